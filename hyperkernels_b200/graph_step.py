"""Forward + backward captured once in a CUDA graph and replayed.

A training step of the attention path is four launches (dQ zeroing, forward, D
pre-pass, backward).  A replay takes the host 3.4 us instead of 17.5 for the two
calls, which it has for other work; the device is no faster for it where the
host keeps ahead (B=8, H=12, T=1024: 142-149 us replayed, 142-146 by calls; B=2,
H=4, T=256: 22.0 and 17.8), since the launches of a call are dependent launches
already and the zeroing is one of its own here.  Zeroing dQ depends on nothing, so it is a
branch beside the forward: its stores (25 MB at B=8, H=12, T=1024) leave the
D pre-pass and fill SMs the forward's last wave leaves idle.  Capture goes through
``hk_attn_forward`` and ``hk_attn_backward`` on a side stream after one eager warm-up step (which sets
the kernels' attributes and resolves the library's device symbols -- neither is
allowed during capture).
"""
from __future__ import annotations

from typing import Optional

from . import attention as att


class GraphedAttentionStep:
    """``O, LSE = fwd(Q, K, V)`` and ``dQ, dK, dV = bwd(dO)`` on fixed device buffers.

    The graph reads ``Q, K, V, dO`` (the tensors given here: refill them in place between replays) and writes
    ``self.O, self.LSE, self.dQ, self.dK, self.dV, self.D``.  With Philox dropout the seed and offset are frozen
    into the graph: every replay draws the same mask; capture again for a new one.
    """

    def __init__(self, Q, K, V, dO, scale: float, causal: bool, *, dropout_p: float = 0.0,
                 philox_seed: Optional[int] = None, philox_offset: int = 0, dropout_scaled: bool = False,
                 bh_pos0: int = 0):
        import torch

        B, H, T, _ = Q.shape
        Tk = K.shape[2]
        dev = Q.device
        self.Q, self.K, self.V, self.dO = Q, K, V, dO
        # one allocation for everything the step writes
        rows_q, rows_k = B * H * T, B * H * Tk
        flat = torch.empty(2 * (rows_q + rows_k) * 64 + 2 * rows_q, dtype=torch.float32, device=dev)
        self.O, self.dQ, self.dK, self.dV, self.LSE, self.D = (
            x.view(shape) for x, shape in zip(flat.split([rows_q * 64] * 2 + [rows_k * 64] * 2 + [rows_q] * 2),
                                              [(B, H, T, 64)] * 2 + [(B, H, Tk, 64)] * 2 + [(B, H, T)] * 2))
        drop = {}
        if dropout_p > 0:
            if philox_seed is None:
                raise ValueError("dropout in a captured step uses the Philox mask: give philox_seed")
            drop = dict(dropout_p=dropout_p, philox_seed=philox_seed, philox_offset=philox_offset,
                        dropout_scaled=dropout_scaled, bh_pos0=bh_pos0)

        zero_stream = torch.cuda.Stream(device=dev)

        def step():
            main = torch.cuda.current_stream(dev)
            zero_stream.wait_stream(main)
            att.attention_forward(Q, K, V, scale, causal, out=self.O, lse=self.LSE, **drop)
            att.zero_dq(self.dQ, zero_stream)
            main.wait_stream(zero_stream)
            att.attention_backward(Q, K, V, self.O, dO, self.LSE, scale, causal, D=self.D,
                                   dQ=self.dQ, dK=self.dK, dV=self.dV, accum_dq=True, **drop)

        n0 = att.launch_count()
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            step()  # eager: first-call set-up happens here, outside the capture
            self.launches_per_replay = att.launch_count() - n0
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=side):
                step()
        torch.cuda.current_stream(dev).wait_stream(side)

    def replay(self) -> None:
        """Enqueue one step on the current stream."""
        self.graph.replay()
