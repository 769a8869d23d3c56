"""Calls whose work items come in several runs of slices (csrc/attn_kernels.cuh, take_in_groups): which calls do, and that each
slice equals the same slice in calls of one run, which other tests compare with the oracle.  Run sizes are asked for, not restated."""
import ctypes as C

import pytest
import torch

import hyperkernels_b200 as hk
from test_work_split import B200, ONE_ITEM, TAKE_OVER, TOGETHER, backward_plan, forward_job

SCALE, P, SEED = 0.125, 0.25, 99

# (BH, Tq, Tk, causal, the forward's job): KV tiles that no query sees, so that the backward's grid has 3 of 4; blocks of more than
# twelve steps; two KV tiles and a second block of few rows
SHAPES = [(700, 300, 500, True, TAKE_OVER), (111, 1000, 1600, False, ONE_ITEM), (1000, 280, 256, True, TAKE_OVER)]


def run_of(backward, BH, Tq, Tk, causal, kind="none", q_pos0=0):
    """slices in a run, BH where there is one"""
    p = hk.MemEfficientBwdParams() if backward else hk.MemEfficientFwdParams()
    p.B, p.nh, p.T, p.kv_len, p.is_causal, p.q_pos0 = 1, BH, Tq, Tk, causal, q_pos0
    if kind != "none":
        p.dropout_p = P
    if kind.startswith("philox"):
        p.flags = hk.FLAG_PHILOX_DROPOUT
    elif kind.startswith("dense"):
        p.dropout_mask = 16  # not read
    n = C.c_int()
    assert (hk.lib().hk_attn_backward_run if backward else hk.lib().hk_attn_forward_run)(C.byref(p), B200, C.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("backward,Tq,Tk,causal,kind,least,run", [
    # least: the fewest slices that come in several runs; up to four blocks of different lengths, and more
    (0, 1024, 1024, True, "none", 256, 64), (0, 1024, 1024, True, "philox", 256, 64), (0, 1024, 1024, True, "dense", 128, 64),
    (0, 1025, 1025, True, "none", 192, 64), (0, 1024, 1024, False, "none", 128, 64), (0, 257, 257, False, "philox", 510, 255),
    # KV tiles: fewer than eight, eight, sixteen, more than 32; runs of two slices
    (1, 512, 512, True, "none", 146, 73), (1, 897, 896, True, "philox", 84, 42), (1, 1024, 1024, True, "none", 93, 37),
    (1, 1024, 1024, False, "dense", 93, 37), (1, 2048, 2048, True, "philox", 45, 18), (1, 2048, 2048, True, "dense", 72, 18),
    (1, 2048, 1920, False, "dense", 48, 19), (1, 4096, 4096, True, "philox", 23, 9), (1, 5067, 5067, True, "philox", 28, 7),
    (1, 5067, 5067, True, "none", 18, 7), (1, 16384, 16384, False, "none", 8, 2)])
def test_calls_of_several_runs(backward, Tq, Tk, causal, kind, least, run):
    assert run_of(backward, least - 1, Tq, Tk, causal, kind) == least - 1
    assert run_of(backward, least, Tq, Tk, causal, kind) == run


@pytest.mark.parametrize("q_pos0,least", [(0, 408), (1, 204), (256, 204)])
def test_runs_of_chunks_behind_keys(q_pos0, least):
    """Keys in front of the queries even out the blocks: two runs of 102 slices, four where there are none."""
    assert run_of(0, least - 1, 512, 768, True, q_pos0=q_pos0) == least - 1
    assert run_of(0, least, 512, 768, True, q_pos0=q_pos0) == 102


@pytest.mark.parametrize("backward,BH,Tq,Tk,causal", [
    (0, 3000, 256, 256, True), (0, 3000, 100, 128, False), (1, 3000, 128, 128, True), (1, 3000, 100, 300, True),  # alone in their slice
    (0, 8, 512, 65536, False), (1, 4, 60000, 300, False)])  # shared by a cluster
def test_calls_of_one_run(backward, BH, Tq, Tk, causal):
    assert run_of(backward, BH, Tq, Tk, causal) == BH
    if BH < 10:
        assert (backward_plan(BH, Tq, Tk, causal, slots=B200)[1] if backward else forward_job(BH, Tq, Tk, causal, slots=B200)) == TOGETHER


@pytest.mark.parametrize("kind", ["none", "philox", "dense"])
@pytest.mark.parametrize("BH,Tq,Tk,causal,job", SHAPES)
def test_shapes_take_several_runs(BH, Tq, Tk, causal, job, kind):
    """Two runs or more in both directions, the last one longer, on the route that the shape stands for."""
    for backward in (0, 1):
        n = run_of(backward, BH, Tq, Tk, causal, kind)
        assert 2 * n <= BH and BH % n
    assert forward_job(BH, Tq, Tk, causal, slots=B200) == job
    assert backward_plan(BH, Tq, Tk, causal, slots=B200) == (1, TAKE_OVER)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "philox", "philox inverted", "dense", "dense inverted"])
@pytest.mark.parametrize("BH,Tq,Tk,causal,job", SHAPES)
def test_every_kind_of_call_in_runs_keeps_its_bits(BH, Tq, Tk, causal, job, kind):
    """O, LSE, dK, dV and the reproducible dQ, stored [B, T, H, 64], and a forward that goes on from a state; gradients added to
    what the buffers hold."""
    part = min(run_of(backward, BH, Tq, Tk, causal, kind) for backward in (0, 1))
    assert all(run_of(backward, part, Tq, Tk, causal, kind) == part for backward in (0, 1))
    gen = torch.Generator(device="cuda").manual_seed(83)
    normal = lambda T: torch.randn((1, T, BH, 64), generator=gen, device="cuda").transpose(1, 2)  # noqa: E731
    Q, dO, K, V = normal(Tq), normal(Tq), normal(Tk), normal(Tk)
    mask = (torch.rand((BH, Tq, Tk), generator=gen, device="cuda") >= P).float() if kind.startswith("dense") else None

    def calls(s):
        """every output of the slices `s`"""
        kw = {} if kind == "none" else dict(dropout_p=P, dropout_scaled=kind.endswith("inverted"))
        if kind.startswith("philox"):
            kw.update(philox_seed=SEED, bh_pos0=s.start)
        second, half = dict(kw), Tk // 16 * 8  # keys in two calls
        if mask is not None:
            kw["dropout_mask"] = mask[s]
        q, k, v, g = Q[:, s], K[:, s], V[:, s], dO[:, s]
        O, L = hk.attention_forward(q, k, v, SCALE, causal, **kw)
        back = lambda **more: hk.attention_backward(q, k, v, O, g, L, SCALE, causal, deterministic_dq=True, **kw, **more)[:3]  # noqa: E731
        grads = back()
        sums = [torch.full_like(x, 0.5) for x in grads]
        back(accum_dq=True, accum_dkdv=True, dQ=sums[0], dK=sums[1], dV=sums[2])
        out = [O, L, *grads, *sums]
        if not kind.endswith("inverted"):
            first = dict(second, dropout_mask=mask[s][:, :, :half].contiguous()) if mask is not None else second
            O2, L2 = hk.attention_forward(q, k[:, :, :half], v[:, :, :half], SCALE, causal, **first)
            if mask is not None:
                second["dropout_mask"] = mask[s][:, :, half:].contiguous()
            hk.attention_forward(q, k[:, :, half:], v[:, :, half:], SCALE, causal, k_pos0=half, continue_state=True, out=O2, lse=L2, **second)
            out += [O2, L2]
        torch.cuda.synchronize()
        assert hk.last_device_status() == 0
        return out

    whole = calls(slice(0, BH))
    for i in range(0, BH, part):
        s = slice(i, min(BH, i + part))
        for got, want in zip(whole, calls(s)):
            assert torch.equal(got[:, s], want)


@pytest.mark.gpu
def test_default_dq_in_runs_differs_by_the_order_of_its_sum():
    """The default dQ adds one term per KV tile in the order of arrival: n terms in two orders, (n - 1) roundings of at most 2^-24 of
    the sum of the magnitudes each."""
    BH, Tq, Tk, causal, _ = SHAPES[0]
    gen = torch.Generator(device="cuda").manual_seed(89)
    normal = lambda T: torch.randn((1, BH, T, 64), generator=gen, device="cuda")  # noqa: E731
    Q, dO, K, V = normal(Tq), normal(Tq), normal(Tk), normal(Tk)
    O, L = hk.attention_forward(Q, K, V, SCALE, causal)
    want, _, _, D = hk.attention_backward(Q, K, V, O, dO, L, SCALE, causal, deterministic_dq=True)
    got = hk.attention_backward(Q, K, V, O, dO, L, SCALE, causal)[0]
    size, tiles = torch.zeros_like(want), -(-Tk // 128)
    for i in range(tiles):  # a KV tile alone
        k, v = (x[:, :, 128 * i:128 * (i + 1)].contiguous() for x in (K, V))
        size += hk.attention_backward(Q, k, v, O, dO, L, SCALE, causal, k_pos0=128 * i, D=D, d_precomputed=True)[0].abs()
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0
    # the sum of magnitudes is itself rounded (n - 1) times, and the zero that dQ starts with is a term without a rounding
    assert bool(((got - want).abs() <= 2 * (tiles - 1) * 2.0 ** -24 * (1 + tiles * 2.0 ** -23) * size).all())
