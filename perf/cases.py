"""The work users of this framework have it do: attention calls on B200, smallest to largest.

A case is a dict of plain values.  ``kind`` picks the public entry point:

* ``forward``  ``attention_forward``: inference or the forward half of a step.  ``Tq != Tk`` is a chunk of new queries
  against a key/value cache (chunked prefill; ``Tq`` of a few is decode): the keys are a view of a longer cache buffer
  and the queries are its last positions.
* ``train``    ``attention_forward`` then ``attention_backward``, with the calls' default buffers, as an autograd
  function runs them.  ``Tq != Tk`` without a causal mask is cross-attention.
* ``graph``    ``GraphedAttentionStep.replay``: the step captured once, replayed per batch.
* ``host``     ``HostAttentionStep.step``: tensors in pinned host memory in and out.

``layout`` is how the caller stores its tensors: ``bhtd`` ([B, H, T, 64]) or ``bthd`` ([B, T, H, 64], what a fused QKV
projection leaves).  ``dropout`` is the Philox mask's probability, ``inverted`` the usual 1/(1-p) scaling instead of
drop-then-renormalise, ``det`` the bit-reproducible dQ.
"""
import math

import torch

import hyperkernels_b200 as hk

SCALE = 0.125  # 1 / sqrt(64)


def _case(kind, name, B, H, Tq, Tk, causal, layout="bhtd", dropout=0.0, inverted=False, det=False):
    c = dict(kind=kind, B=B, H=H, Tq=Tq, Tk=Tk, causal=causal, layout=layout, dropout=dropout, inverted=inverted, det=det)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one decoding step of a batch of 16 sequences against their caches: one query row per head, every launch counts
        _case("forward", "decode_b16_kv2047", 16, 12, 1, 2047, True),
        # the smallest forward with a published figure: one short prompt
        _case("forward", "prompt_b1_t512", 1, 12, 512, 512, True),
        # the correctness configuration: a training step too small to fill the chip
        _case("train", "train_small_t256", 2, 4, 256, 256, True),
        # cross-attention with ragged lengths, no mask
        _case("train", "train_cross_777x333", 4, 6, 777, 333, False),
        # chunked prefill: 512 new tokens of one sequence behind 7 680 cached ones, cache stored [B, T, H, 64]
        _case("forward", "prefill_chunk_512_kv8192", 1, 32, 512, 8192, True, layout="bthd"),
        # GPT-2-small batch, inference
        _case("forward", "forward_b8_t1024", 8, 12, 1024, 1024, True),
        # the same batch, the whole step replayed from a graph: the headline configuration
        _case("graph", "graph_b8_t1024", 8, 12, 1024, 1024, True),
        # the same batch, tensors on the host
        _case("host", "host_b8_t1024", 8, 12, 1024, 1024, True),
        # odd length, [B, T, H, 64] storage, reproducible gradients
        _case("train", "train_det_t2000_bthd", 2, 16, 2000, 2000, True, layout="bthd", det=True),
        # GPT-2-XL batch with dropout
        _case("train", "train_b32_t1024_dropout", 32, 25, 1024, 1024, True, dropout=0.1),
        # encoder batch (no mask) with inverted dropout
        _case("train", "train_b16_t2048_full_dropout", 16, 16, 2048, 2048, False, dropout=0.1, inverted=True),
        # one long sequence
        _case("train", "train_b1_t32768", 1, 32, 32768, 32768, True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# rows of the longest tensor, forward + backward operations of a drawn case: below those of the largest listed one
_MAX_ROWS = 1 << 20
_MAX_FLOPS = 4e12


def draw(rng):
    while True:
        kind = rng.choice(["forward", "forward", "train", "train", "train", "graph", "host"])
        B, H = _log_int(rng, 1, 32), rng.choice([1, 4, 6, 8, 12, 16, 20, 25, 32])
        causal = rng.random() < 0.7
        layout = "bthd" if rng.random() < 0.3 and kind != "host" else "bhtd"
        T = _log_int(rng, 64, 16384)
        Tq = Tk = T
        if kind == "forward" and rng.random() < 0.5:  # new queries against a cache
            Tq, causal = min(T, _log_int(rng, 1, 1024)), True
        elif kind == "train" and rng.random() < 0.25:  # cross-attention
            Tk, causal = _log_int(rng, 64, 4096), False
        dropout = 0.1 if kind in ("train", "graph") and rng.random() < 0.3 else 0.0
        det = kind == "train" and max(Tq, Tk) <= 2048 and rng.random() < 0.2
        c = _case(kind, None, B, H, Tq, Tk, causal, layout, dropout, dropout > 0 and rng.random() < 0.5, det)
        rows = B * H * max(Tq, Tk)
        if rows > (_MAX_ROWS if kind != "host" else 1 << 17) or work(c)["flops"] > _MAX_FLOPS:
            continue
        if det and rows * math.ceil(Tk / 128) > (1 << 24):  # one partial dQ per 128 keys: at most 4 GiB
            continue
        return c


def _tensor(case, T, gen, capacity=0):
    """[B, H, T, 64] standard normal values in the case's storage order; capacity: a view of a longer buffer."""
    B, H, n = case["B"], case["H"], max(T, capacity)
    shape = (B, n, H, 64) if case["layout"] == "bthd" else (B, H, n, 64)
    x = torch.randn(shape, generator=gen, device="cuda")
    return (x.transpose(1, 2) if case["layout"] == "bthd" else x)[:, :, :T]


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    # a cache buffer is longer than what it holds so far
    capacity = (c["Tk"] + 1023) // 1024 * 1024 if c["kind"] == "forward" and c["Tq"] != c["Tk"] else 0
    s = {"case": c, "Q": _tensor(c, c["Tq"], gen), "K": _tensor(c, c["Tk"], gen, capacity), "V": _tensor(c, c["Tk"], gen, capacity)}
    if c["kind"] == "forward":
        s["kw"] = {"q_pos0": c["Tk"] - c["Tq"]} if c["causal"] else {}
        return s
    s["dO"] = _tensor(c, c["Tq"], gen)
    s["drop"] = {}
    if c["dropout"] > 0:
        s["drop"] = dict(dropout_p=c["dropout"], philox_seed=seed, dropout_scaled=c["inverted"])
    if c["kind"] == "graph":
        s["step"] = hk.GraphedAttentionStep(s["Q"], s["K"], s["V"], s["dO"], SCALE, c["causal"], **s["drop"])
    elif c["kind"] == "host":
        dims = (c["B"], c["H"], c["Tq"], 64)
        host = lambda *shape: torch.empty(shape, dtype=torch.float32, pin_memory=True)  # noqa: E731
        ins = [host(*dims).copy_(s.pop(k)) for k in ("Q", "K", "V", "dO")]
        outs = [host(*dims), host(*dims[:3]), host(*dims), host(*dims), host(*dims)]
        s["step"], s["args"] = hk.HostAttentionStep(*dims[:3], SCALE, c["causal"]), ins + outs
    return s


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "forward":
        O, LSE = hk.attention_forward(s["Q"], s["K"], s["V"], SCALE, c["causal"], **s["kw"])
        return {"O": O, "LSE": LSE}
    if c["kind"] == "graph":
        g = s["step"]
        g.replay()
        return {"O": g.O, "LSE": g.LSE, "dQ": g.dQ, "dK": g.dK, "dV": g.dV, "D": g.D}
    if c["kind"] == "host":
        s["step"].step(*s["args"])
        return dict(zip(("O", "LSE", "dQ", "dK", "dV"), s["args"][4:]))
    O, LSE = hk.attention_forward(s["Q"], s["K"], s["V"], SCALE, c["causal"], **s["drop"])
    dQ, dK, dV, D = hk.attention_backward(s["Q"], s["K"], s["V"], O, s["dO"], LSE, SCALE, c["causal"],
                                          deterministic_dq=c["det"], **s["drop"])
    return {"O": O, "LSE": LSE, "dQ": dQ, "dK": dK, "dV": dV, "D": D}


def work(case):
    """fp32 tensors read and written once; 2 flops per multiply-add of the products over the (query, key) pairs the mask
    leaves visible: two products forward, five backward."""
    c = case
    bh, Tq, Tk = c["B"] * c["H"], c["Tq"], c["Tk"]
    pairs = Tq * Tk
    if c["causal"]:  # query i of the last Tq positions sees keys 0 .. Tk - Tq + i
        pairs = Tq * (Tk - Tq) + Tq * (Tq + 1) // 2
    fwd_bytes = bh * (2 * Tq * 64 + 2 * Tk * 64 + Tq) * 4          # Q, O; K, V; LSE
    fwd_flops = 4 * 64 * bh * pairs
    if c["kind"] == "forward":
        return {"bytes": fwd_bytes, "flops": fwd_flops}
    # Q, dO in, O, dQ out; K, V in, dK, dV out; LSE and (not on the host) D out
    small = 1 if c["kind"] == "host" else 2
    return {"bytes": bh * (4 * Tq * 64 + 4 * Tk * 64 + small * Tq) * 4, "flops": fwd_flops + 10 * 64 * bh * pairs}


def tolerance(case):
    """fp32 in and out, TF32 (10-bit mantissa) product operands: another correct implementation rounds the
    probabilities and their gradients at other points, 2^-11 each."""
    return {"rel": 1e-3, "max": 2e-2}
