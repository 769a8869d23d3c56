"""How a call's work is cut over CTAs (mode, key splits, query splits) and what that may change: the choice from sizes
(CPU), and on the GPU every mode and number of splits with every kind of dropout, against the oracle."""
import ctypes as C
import random

import numpy as np
import pytest
import torch

import hyperkernels_b200 as hk
import oracle_lib as ol

SCALE = 0.125
ROWS, ROW, KEYS, DECODE = 0, 1, 2, -1
ONE_ITEM, TAKE_OVER, TOGETHER = 0, 1, 2  # a CTA's items: one, then others that have not started, one that a cluster or two streams share
B200 = (C.c_int * 4)(148, 74, 33, 15)  # resident clusters of 1, 2, 4, 8 CTAs, one CTA per SM


def forward_plan(BH, Tq, Tk, causal=False, q_pos0=0, k_pos0=0, flags=0, dropout_p=0.0, slots=None):
    """(mode, CTAs per block of rows or decoded slice); slots=None: those of the current device"""
    return _forward_plan(BH, Tq, Tk, causal, q_pos0, k_pos0, flags, dropout_p, slots)[:2]


def forward_job(BH, Tq, Tk, causal=False, q_pos0=0, k_pos0=0, slots=None):
    return _forward_plan(BH, Tq, Tk, causal, q_pos0, k_pos0, 0, 0.0, slots)[2]


def _forward_plan(BH, Tq, Tk, causal, q_pos0, k_pos0, flags, dropout_p, slots):
    p = hk.MemEfficientFwdParams()
    p.B, p.nh, p.T, p.kv_len, p.is_causal = 1, BH, Tq, Tk, bool(causal)
    p.q_pos0, p.k_pos0, p.flags, p.dropout_p = q_pos0, k_pos0, flags, dropout_p
    out = (C.c_int * 3)()
    assert hk.lib().hk_attn_forward_plan(C.byref(p), slots, out) == 0
    return tuple(out)


def backward_plan(BH, Tq, Tk, causal=False, q_pos0=0, k_pos0=0, slots=None):
    """(CTAs per KV tile, job)"""
    p = hk.MemEfficientBwdParams()
    p.B, p.nh, p.T, p.kv_len, p.is_causal, p.q_pos0, p.k_pos0 = 1, BH, Tq, Tk, bool(causal), q_pos0, k_pos0
    out = (C.c_int * 2)()
    assert hk.lib().hk_attn_backward_plan(C.byref(p), slots, out) == 0
    return tuple(out)


def backward_splits(BH, Tq, Tk, slots=None):
    return backward_plan(BH, Tq, Tk, slots=slots)[0]


# ---- the choice -----------------------------------------------------------------------------------------------------
def test_training_lengths_are_never_split():
    """kv_len <= 4 096 and < 2 T forward, T < 2 kv_len backward: every slice is summed in one order, whatever the batch."""
    rnd = random.Random(1)
    modes = set()
    for _ in range(3000):
        Tk = int(2 ** rnd.uniform(0, 12))
        Tq = max(Tk // 2 + 1, int(2 ** rnd.uniform(0, 13)))
        BH, causal = int(2 ** rnd.uniform(0, 11)), rnd.random() < 0.5
        mode, splits = forward_plan(BH, Tq, Tk, causal, rnd.choice([0, 0, 300]), rnd.choice([0, 0, 128]), slots=B200)
        assert mode in (ROWS, ROW) and splits == 1, (BH, Tq, Tk, causal)
        modes.add(mode)
        Tq = max(1, int(rnd.uniform(0.01, 2.0) * Tk) - 1)
        assert backward_splits(BH, Tq, Tk, slots=B200) == 1, (BH, Tq, Tk)
    assert modes == {ROWS, ROW}
    assert forward_plan(1, 4096, 4096, True, slots=B200)[1] == 1 and forward_plan(1, 2048, 4095, slots=B200)[1] == 1
    assert backward_splits(1, 1023, 512, slots=B200) == 1


def test_the_batch_decides_outside_training_lengths():
    """The other side of the same lines: a slice alone and the same slice among others are cut differently."""
    assert forward_plan(1, 8192, 8192, True, slots=B200) != forward_plan(32, 8192, 8192, True, slots=B200)
    assert forward_plan(1, 512, 1024, slots=B200)[1] > 1 and forward_plan(64, 512, 1024, slots=B200)[1] == 1
    assert backward_splits(1, 1024, 512, slots=B200) > 1 and backward_splits(64, 1024, 512, slots=B200) == 1
    assert forward_plan(1, 1, 300, True, slots=B200) != forward_plan(192, 1, 3000, True, slots=B200)


def test_decode_kernel_for_one_or_two_rows():
    plan = lambda Tq, Tk, **kw: forward_plan(4, Tq, Tk, slots=B200, **kw)[0]  # noqa: E731
    assert plan(1, 128) == plan(2, 128) == plan(1, 5000, causal=True) == DECODE
    assert DECODE not in (plan(3, 128), plan(1, 127), plan(1, 500, flags=hk.FLAG_CONTINUE_SOFTMAX_STATE),
                          plan(1, 500, flags=hk.FLAG_PHILOX_DROPOUT, dropout_p=0.1))


@pytest.mark.parametrize("job,BH,Tq,Tk,causal,pos", [
    (ONE_ITEM, 148, 128, 128, 0, {}), (TAKE_OVER, 149, 128, 128, 0, {}),  # one CTA more than the device holds
    (TAKE_OVER, 96, 1024, 1536, 0, {}), (ONE_ITEM, 96, 1024, 1537, 0, {}),  # twelve and thirteen steps
    (TAKE_OVER, 96, 2816, 2816, 1, {}), (ONE_ITEM, 96, 2817, 2817, 1, {}),  # 12 and 12.9 on average under the mask
    (TAKE_OVER, 60, 1100, 1100, 1, dict(q_pos0=512, k_pos0=512)), (ONE_ITEM, 60, 1100, 1100, 1, dict(q_pos0=511, k_pos0=512)),
    (TAKE_OVER, 60, 1100, 1100, 0, dict(k_pos0=512)), (TOGETHER, 16, 257, 1000, 0, {}), (TOGETHER, 24, 257, 1000, 1, dict(q_pos0=743))])
def test_row_blocks_that_are_taken_over(job, BH, Tq, Tk, causal, pos):
    """Short ones of a grid larger than the device, each with a key: either side of each line."""
    assert forward_job(BH, Tq, Tk, causal, slots=B200, **pos) == job


@pytest.mark.parametrize("plan,BH,Tq,Tk,causal,pos", [
    ((1, ONE_ITEM), 148, 128, 128, 0, {}), ((1, TAKE_OVER), 149, 128, 128, 0, {}), ((2, TOGETHER), 24, 777, 333, 0, {}),
    ((1, ONE_ITEM), 74, 256, 1000, 1, {}), ((1, TAKE_OVER), 75, 256, 1000, 1, {}), ((1, ONE_ITEM), 75, 256, 1000, 1, dict(k_pos0=128))])
def test_key_tiles_that_are_taken_over(plan, BH, Tq, Tk, causal, pos):
    """A grid larger than the device; KV tiles that no query sees are not in it."""
    assert backward_plan(BH, Tq, Tk, causal, slots=B200, **pos) == plan


# ---- every cut, with every mask -------------------------------------------------------------------------------------
def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _normal(shape, seed):
    return np.random.default_rng(seed).standard_normal(shape).astype(np.float32)


P, SEED, OFFSET = 0.25, 99, 7
MASKS = ["none", "philox", "dense", "philox inverted", "dense inverted"]


def _mask(kind, BH, Tq, Tk, q_pos0=0, k_pos0=0):
    """(keyword arguments of the calls, the oracle's mask); p = 1/4 is exact in 16 bits, so both kinds drop with it"""
    if kind == "none":
        return {}, None
    mask = ol.dropout_mask(BH, Tq, Tk, P, SEED, OFFSET, q_pos0=q_pos0, k_pos0=k_pos0)
    kw = dict(dropout_mask=_dev(mask)) if kind.startswith("dense") else dict(philox_seed=SEED, philox_offset=OFFSET)
    return dict(kw, dropout_p=P, dropout_scaled=kind.endswith("inverted")), mask


def _oracle_forward(kind, mask, q, k, v, causal, **pos):
    if kind.endswith("inverted"):
        return ol.attn_forward_scaled(q, k, v, SCALE, causal, mask, P, **pos)
    return ol.attn_forward_mt(q, k, v, SCALE, causal, mask, **pos)


def _oracle_backward(kind, mask, q, k, v, O, g, L, causal, **pos):
    if kind.endswith("inverted"):
        return ol.attn_backward_scaled(q, k, v, O, g, L, SCALE, causal, mask, P, **pos)
    return ol.attn_backward_mt(q, k, v, O, g, L, SCALE, causal, mask, **pos)


def decode_plan(BH, Tq, Tk, slots=B200):
    """(warps of a CTA, CTAs of a slice)"""
    p = hk.MemEfficientFwdParams()
    p.B, p.nh, p.T, p.kv_len = 1, BH, Tq, Tk
    out = (C.c_int * 3)()
    assert hk.lib().hk_attn_forward_plan(C.byref(p), slots, out) == 0 and out[0] == DECODE
    return out[2], out[1]


def test_decode_puts_one_wave_of_warps_on_the_chip():
    """As many warps as the plan's own estimate of what is resident together (clusters of one CTA per SM, times the CTAs of an
    SM; 0.87 of the places for eight of them), unless one CTA per slice is more already; each with a batch of rows."""
    rnd = random.Random(2)
    for _ in range(3000):
        BH, Tq, Tk = int(2 ** rnd.uniform(0, 12)), rnd.choice([1, 2]), int(2 ** rnd.uniform(7, 15))
        warps, splits = decode_plan(BH, Tq, Tk)
        assert warps in (4, 8, 16) and splits in (1, 2, 4, 8) and warps * splits * 8 <= Tk
        per_sm = 24 if Tq == 1 else 16
        k = per_sm // warps
        fit = dict(zip((1, 2, 4, 8), (k * s for s in B200)))  # clusters that the device is taken to hold
        if k > 1:
            fit[8] = max(fit[8], int(0.87 * 148 * k / 8))
        assert BH <= fit[splits] or splits == 1
        # twice the splits would not fit any more, or leave warps without rows
        if splits < 8 and BH <= fit[2 * splits]:
            assert warps * splits * 2 * 8 > Tk
    assert decode_plan(192, 1, 2047) == (8, 2) and decode_plan(1024, 1, 511) == (8, 1) and decode_plan(12, 1, 2047) == (16, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("BH,Tq,Tk,causal,warps,splits", [
    (4, 1, 129, 1, 16, 1), (4, 2, 257, 0, 8, 4), (2, 1, 2049, 1, 16, 8), (30, 1, 515, 1, 16, 4), (60, 2, 131, 1, 16, 1), (40, 1, 1025, 0, 8, 8),
    (74, 1, 300, 1, 16, 2), (90, 1, 259, 1, 8, 4), (160, 1, 140, 1, 8, 2), (300, 1, 200, 0, 8, 1), (500, 1, 130, 1, 4, 1), (1000, 1, 130, 1, 8, 1), (700, 2, 129, 0, 4, 1), (90, 2, 300, 1, 16, 1)])
def test_every_decode_cut(BH, Tq, Tk, causal, warps, splits):
    from test_attention_gpu import gate, host, lse_check, ok_status

    q, k, v = _normal((1, BH, Tq, 64), 950), _normal((1, BH, Tk, 64), 951), _normal((1, BH, Tk, 64), 952)
    pos = Tk - Tq if causal else 0
    assert decode_plan(BH, Tq, Tk) == (warps, splits)
    O_ref, L_ref = ol.attn_forward_mt(q, k, v, SCALE, causal, q_pos0=pos)
    O, LSE = hk.attention_forward(_dev(q), _dev(k), _dev(v), SCALE, bool(causal), q_pos0=pos)
    ok_status()
    gate("O", host(O), O_ref)
    lse_check(host(LSE), L_ref)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", MASKS)
@pytest.mark.parametrize("mode,splits,BH,Tq,Tk,causal", [
    (ROWS, 1, 64, 129, 400, 0), (ROWS, 2, 16, 257, 1000, 0), (ROWS, 4, 12, 129, 640, 1), (ROWS, 8, 6, 129, 650, 0),
    (ROW, 1, 24, 3, 600, 1), (ROW, 2, 24, 3, 700, 1), (ROW, 4, 12, 3, 640, 1), (ROW, 8, 1, 3, 641, 0),
    (KEYS, 1, 24, 257, 1000, 1), (KEYS, 2, 48, 3, 4200, 0), (KEYS, 4, 24, 3, 8193, 1), (KEYS, 8, 3, 385, 8193, 1)])
def test_every_forward_cut_with_every_mask(mode, splits, BH, Tq, Tk, causal, kind):
    from test_attention_gpu import gate, host, lse_check, ok_status

    q, k, v = _normal((1, BH, Tq, 64), 960), _normal((1, BH, Tk, 64), 961), _normal((1, BH, Tk, 64), 962)
    pos = Tk - Tq if causal else 0
    kw, mask = _mask(kind, BH, Tq, Tk, q_pos0=pos)
    assert forward_plan(BH, Tq, Tk, causal, pos) == (mode, splits)
    O_ref, L_ref = _oracle_forward(kind, mask, q, k, v, causal, q_pos0=pos)
    O, LSE = hk.attention_forward(_dev(q), _dev(k), _dev(v), SCALE, bool(causal), q_pos0=pos, **kw)
    ok_status()
    gate("O", host(O), O_ref)
    lse_check(host(LSE), L_ref)


@pytest.mark.parametrize("tiles,n_q,splits", [
    (148, 20, 1), (149, 20, 2), (74, 4, 2), (75, 4, 1), (80, 58, 4), (33, 40, 4), (34, 40, 2), (15, 80, 8), (16, 80, 4), (150, 1, 1), (1, 2, 1), (1, 4, 4)])
def test_query_splits_by_whole_waves(tiles, n_q, splits):
    """One CTA more than a wave holds is another wave: either side of each line, for 148, 74, 33 and 15 clusters at once."""
    assert backward_splits(tiles, 128 * n_q, 64, slots=B200) == splits


# where the fine estimate of the forward's plan decides: (BH, Tq, Tk, causal, dropout) -> its cut, the coarse one's cut
FINER = [(24, 525, 525, 0, 1, (ROW, 1), (ROWS, 1)), (64, 282, 2017, 1, 0, (ROWS, 1), (KEYS, 1)), (4, 804, 1906, 1, 0, (KEYS, 4), (ROWS, 4)),
         (16, 22, 8399, 1, 0, (KEYS, 4), (ROW, 8)), (8, 390, 8868, 1, 1, (KEYS, 4), (ROWS, 8))]


@pytest.mark.parametrize("BH,Tq,Tk,causal,drop,fine,coarse", FINER)
def test_the_finer_estimate_decides_by_sizes_alone(BH, Tq, Tk, causal, drop, fine, coarse):
    kw = dict(flags=hk.FLAG_PHILOX_DROPOUT, dropout_p=0.1) if drop else {}
    assert forward_plan(BH, Tq, Tk, causal, Tk - Tq if causal else 0, slots=B200, **kw) == fine != coarse


@pytest.mark.gpu
@pytest.mark.parametrize("BH,Tq,Tk,causal,drop,fine,coarse", FINER)
def test_forward_cut_by_the_finer_estimate(BH, Tq, Tk, causal, drop, fine, coarse):
    from test_attention_gpu import gate, host, lse_check, ok_status

    q, k, v = _normal((1, BH, Tq, 64), 970), _normal((1, BH, Tk, 64), 971), _normal((1, BH, Tk, 64), 972)
    kind, pos = "philox" if drop else "none", Tk - Tq if causal else 0
    kw, mask = _mask(kind, 1, Tq, Tk, q_pos0=pos)  # the first slice's
    assert forward_plan(BH, Tq, Tk, causal, pos, **(dict(flags=hk.FLAG_PHILOX_DROPOUT, dropout_p=0.1) if drop else {})) == fine
    O, LSE = hk.attention_forward(_dev(q), _dev(k), _dev(v), SCALE, bool(causal), q_pos0=pos, **kw)
    ok_status()
    s = slice(0, 1)
    O_ref, L_ref = _oracle_forward(kind, mask, q[:, s], k[:, s], v[:, s], causal, q_pos0=pos)
    gate("O", host(O)[:, s], O_ref)
    lse_check(host(LSE)[:, s], L_ref)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", MASKS)
@pytest.mark.parametrize("splits,BH,Tq,Tk,causal", [
    (1, 48, 257, 40, 0), (2, 24, 777, 333, 0), (4, 8, 1024, 129, 0), (4, 1, 257, 128, 0), (8, 1, 4000, 40, 0), (8, 2, 1281, 300, 1)])
def test_every_backward_cut_with_every_mask(splits, BH, Tq, Tk, causal, kind):
    """Beside the default call: dQ through slabs (the same bits on every run, dK and dV those of the default call) and
    results added to what the buffers hold."""
    from test_attention_gpu import gate, host, ok_status

    q, g = _normal((1, BH, Tq, 64), 970), _normal((1, BH, Tq, 64), 971)
    k, v = _normal((1, BH, Tk, 64), 972), _normal((1, BH, Tk, 64), 973)
    pos = dict(k_pos0=(Tq - 200) // 8 * 8 if causal else 0)
    kw, mask = _mask(kind, BH, Tq, Tk, **pos)
    assert backward_splits(BH, Tq, Tk) == splits
    O_ref, L_ref = _oracle_forward(kind, mask, q, k, v, causal, **pos)
    _, *refs = _oracle_backward(kind, mask, q, k, v, O_ref, g, L_ref, causal, **pos)
    args = (_dev(q), _dev(k), _dev(v), _dev(O_ref), _dev(g), _dev(L_ref), SCALE, bool(causal))
    call = lambda **more: hk.attention_backward(*args, **pos, **kw, **more)  # noqa: E731
    plain = call()[:3]
    ok_status()
    for name, got, ref in zip(("dQ", "dK", "dV"), plain, refs):
        gate(name, host(got), ref)
    slabs, again = call(deterministic_dq=True)[:3], call(deterministic_dq=True)[:3]
    ok_status()
    gate("dQ", host(slabs[0]), refs[0])
    assert all(torch.equal(a, b) for a, b in zip(slabs, again))
    assert torch.equal(slabs[1], plain[1]) and torch.equal(slabs[2], plain[2])
    base = [_dev(_normal(r.shape, 974 + i)) for i, r in enumerate(refs)]
    sums = [b.clone() for b in base]
    call(deterministic_dq=True, accum_dq=True, accum_dkdv=True, dQ=sums[0], dK=sums[1], dV=sums[2])
    ok_status()
    for s, b, x in zip(sums, base, slabs):
        # fp32 sums of at most ceil(Tk / 128) + 1 terms in another order
        assert float((s - (b + x)).abs().max()) <= 4 * 2.0 ** -23 * float(x.abs().max() + b.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "philox", "dense inverted"])
@pytest.mark.parametrize("BH,Tq,Tk,causal,pos", [
    (299, 128, 128, 0, {}), (160, 200, 200, 1, {}), (75, 600, 640, 1, {}), (40, 1000, 1100, 0, {}), (200, 100, 150, 0, {}), (40, 1300, 1500, 0, {}),
    (40, 1300, 1800, 0, {}), (60, 1100, 1100, 1, dict(k_pos0=512)), (200, 70, 100, 1, dict(k_pos0=128)),
    # two key tiles, an odd number of row tiles: blocks of one stream before blocks of two
    (96, 379, 200, 0, {}), (96, 640, 256, 1, {}), (48, 1152, 256, 0, {}), (200, 379, 200, 0, {})])
def test_forward_ctas_take_over_row_blocks(BH, Tq, Tk, causal, pos, kind):
    """More blocks of query rows than CTAs start with, of one to twelve steps in one or two streams: first, middle and last slice
    against the oracle, every one against the same call on few enough slices that no CTA takes anything over (the same bits),
    and as a continued state.  Beside them the calls that take none over for another reason: long items (1 800 keys), and blocks
    that see no key (k_pos0 behind their rows; all of them at 70 queries)."""
    from test_attention_gpu import gate, host, lse_check, ok_status

    q, k, v = _normal((1, BH, Tq, 64), 990), _normal((1, BH, Tk, 64), 991), _normal((1, BH, Tk, 64), 992)
    Q, K, V = map(_dev, (q, k, v))
    mode, splits = forward_plan(BH, Tq, Tk, causal, 0, pos.get("k_pos0", 0))
    assert splits == 1 and BH * -(-Tq // (256 if mode == ROWS else 128)) > 148
    assert forward_job(BH, Tq, Tk, causal, **pos) == (ONE_ITEM if Tk == 1800 or pos else TAKE_OVER)
    mask = None if kind == "none" else ol.dropout_mask(BH, Tq, Tk, P, SEED, OFFSET, **pos)
    kw = {} if kind == "none" else dict(_mask(kind, 1, 8, 8)[0])
    if "dropout_mask" in kw:
        kw["dropout_mask"] = _dev(mask)
    O, L = hk.attention_forward(Q, K, V, SCALE, bool(causal), **pos, **kw)
    ok_status()
    for i in (0, BH // 2, BH - 1):
        s = slice(i, i + 1)
        O_ref, L_ref = _oracle_forward(kind, None if mask is None else mask[s], q[:, s], k[:, s], v[:, s], causal, **pos)
        gate("O", host(O[:, s]), O_ref)
        lse_check(host(L[:, s]), L_ref)
    n = 128 // -(-Tq // 128)  # slices whose blocks all start at once
    assert forward_job(n, Tq, Tk, causal, **pos) == ONE_ITEM
    for s0 in range(0, BH, n):
        s = slice(s0, min(BH, s0 + n))
        part = dict(kw, dropout_mask=kw["dropout_mask"][s]) if "dropout_mask" in kw else dict(kw, bh_pos0=s0) if kw else {}
        one = hk.attention_forward(Q[:, s], K[:, s], V[:, s], SCALE, bool(causal), **pos, **part)
        assert torch.equal(one[0], O[:, s]) and torch.equal(one[1], L[:, s])
    if kind == "none":
        # a block that sees no key of the second call keeps what the first one left
        O2, L2 = hk.attention_forward(Q, K, V, SCALE, False, q_pos0=0)
        keep = O2.clone(), L2.clone()
        hk.attention_forward(Q, K, V, SCALE, bool(causal), **pos, continue_state=True, out=O2, lse=L2)
        ok_status()
        blind = min(Tq, pos.get("k_pos0", 0)) if causal else 0
        assert torch.equal(O2[:, :, :blind], keep[0][:, :, :blind]) and torch.equal(L2[:, :, :blind], keep[1][:, :, :blind])
        # twice the same keys: the same O, a normaliser twice as large, where every row sees them all
        if not causal:
            assert float((O2 - keep[0]).norm() / keep[0].norm()) < 1e-3 and float((L2 - keep[1] - np.log(2.0)).abs().max()) < 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "philox", "philox inverted"])
@pytest.mark.parametrize("BH,Tq,Tk,causal", [(299, 128, 128, 0), (60, 640, 640, 1), (75, 100, 300, 0), (90, 257, 384, 1), (60, 130, 1000, 1), (5, 70, 200, 1)])
def test_backward_ctas_take_over_key_tiles(BH, Tq, Tk, causal, kind):
    """More KV tiles than CTAs start with, one to five query tiles each: the CTAs that are through take over the others (not
    where the keys that a query sees make 120 tiles, or none).  First,
    middle and last slice against the oracle, all of them against the same call on 20 slices at a time (every CTA starts with
    its own tile: the same bits), and results added to what the buffers hold.  KV tiles that no query sees (Tk > Tq under the
    mask; all of them where the keys lie behind the queries) leave zeros."""
    from test_attention_gpu import gate, host, ok_status

    q, g = _normal((1, BH, Tq, 64), 980), _normal((1, BH, Tq, 64), 981)
    k, v = _normal((1, BH, Tk, 64), 982), _normal((1, BH, Tk, 64), 983)
    kw, _ = _mask(kind, 1, 8, 8)
    Q, K, V, G = map(_dev, (q, k, v, g))
    for pos in (dict(), dict(k_pos0=1000)) if causal else (dict(),):
        assert backward_plan(BH, Tq, Tk, causal, **pos)[1] == (ONE_ITEM if pos or Tk in (200, 1000) else TAKE_OVER)
        assert backward_plan(20, Tq, Tk, causal, **pos)[1] == ONE_ITEM
        O, L = hk.attention_forward(Q, K, V, SCALE, bool(causal), **pos, **kw)
        call = lambda s, **more: hk.attention_backward(Q[:, s], K[:, s], V[:, s], O[:, s], G[:, s], L[:, s], SCALE, bool(causal), **pos,  # noqa: E731
                                                       **(dict(kw, bh_pos0=s.start) if kw else {}), **more)[:3]
        whole = call(slice(0, BH), deterministic_dq=True)
        ok_status()
        for i in (0, BH // 2, BH - 1):
            s = slice(i, i + 1)
            mask = None if kind == "none" else ol.dropout_mask(BH, Tq, Tk, P, SEED, OFFSET, **pos)[s]
            _, *refs = _oracle_backward(kind, mask, q[:, s], k[:, s], v[:, s], host(O[:, s]), g[:, s], host(L[:, s]), causal, **pos)
            for name, got, ref in zip(("dQ", "dK", "dV"), whole, refs):
                gate(name, host(got[:, s]), ref)
        base = [_dev(_normal(tuple(x.shape), 984 + i)) for i, x in enumerate(whole)]
        sums = [b.clone() for b in base]
        call(slice(0, BH), deterministic_dq=True, accum_dq=True, accum_dkdv=True, dQ=sums[0], dK=sums[1], dV=sums[2])
        for s0 in range(0, BH, 20):
            s = slice(s0, min(BH, s0 + 20))
            for got, ref in zip(call(s, deterministic_dq=True), whole):
                assert torch.equal(got, ref[:, s])
        ok_status()
        for s, b, x in zip(sums, base, whole):
            # fp32 sums of at most ceil(Tk / 128) + 1 terms in another order
            assert float((s - (b + x)).abs().max()) <= 8 * 2.0 ** -23 * float(x.abs().max() + b.abs().max())


# ---- what the cut may change ----------------------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("Tq,Tk,causal,q_pos0", [(4096, 4096, 1, 0), (2048, 4095, 0, 0), (65, 129, 1, 64), (1023, 512, 0, 0), (1500, 1500, 1, 0)])
def test_a_slice_keeps_its_bits_in_any_batch_at_training_lengths(Tq, Tk, causal, q_pos0):
    """Up to the lines themselves: O, LSE, dK and dV of a slice alone and of the same slice among 40, of which the forward
    runs one in row, the other in rows mode."""
    BH = 40
    assert forward_plan(1, Tq, Tk, causal, q_pos0)[0] == ROW and forward_plan(BH, Tq, Tk, causal, q_pos0)[0] == (ROW if Tq <= 128 else ROWS)
    gen = torch.Generator(device="cuda").manual_seed(77)
    Q, dO = (torch.randn((1, BH, Tq, 64), generator=gen, device="cuda") for _ in range(2))
    K, V = (torch.randn((1, BH, Tk, 64), generator=gen, device="cuda") for _ in range(2))
    for kw in ({}, dict(dropout_p=0.1, philox_seed=3)):
        O, LSE = hk.attention_forward(Q, K, V, SCALE, causal, q_pos0=q_pos0, **kw)
        _, dK, dV, _ = hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, causal, q_pos0=q_pos0, **kw)
        for i in (0, 23):
            s = slice(i, i + 1)
            one = dict(kw, bh_pos0=i) if kw else {}
            o, l = hk.attention_forward(Q[:, s], K[:, s], V[:, s], SCALE, causal, q_pos0=q_pos0, **one)
            _, dk, dv, _ = hk.attention_backward(Q[:, s], K[:, s], V[:, s], o, dO[:, s], l, SCALE, causal, q_pos0=q_pos0, **one)
            assert torch.equal(o, O[:, s]) and torch.equal(l, LSE[:, s])
            assert torch.equal(dk, dK[:, s]) and torch.equal(dv, dV[:, s])
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0


@pytest.mark.parametrize("all_", [1, 2, 7, 96, 126, 127, 128, 333, 800])
@pytest.mark.parametrize("n", [1, 2, 9, 64])
def test_every_item_is_handed_out_once(all_, n):
    """Runs of 1, 2, 5, 64 and of more slices than there are: every part of every slice once, a run's slices before those of
    the next, longest parts first inside a run, and only the last run longer (up to, not including, two)."""
    for group in (1, 2, 5, 64, 1000):
        pairs = np.zeros((all_ * n, 2), np.int32)
        hk.lib().hk_attn_item_order(all_, n, C.c_double(2 ** 26 / group), pairs.ctypes.data_as(C.c_void_p))
        assert len({tuple(p) for p in pairs.tolist()}) == all_ * n
        assert pairs.min() == 0 and pairs[:, 0].max() == all_ - 1 and pairs[:, 1].max() == n - 1
        run = np.minimum(pairs[:, 0] // group, max(all_ // group, 1) - 1)
        key = run * n + pairs[:, 1]
        assert (np.diff(key) >= 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("BH,Tq,Tk,causal", [(530, 300, 300, True), (530, 300, 400, False), (171, 1000, 700, False), (2100, 64, 100, True)])
def test_slices_handed_out_in_runs_keep_their_bits(BH, Tq, Tk, causal):
    """More slices than one run of the grid holds (64 MB), the last run longer than the others: every slice equals the same
    slice in calls of one run."""
    def run(seq):  # slices of a run
        return max(1, int(min(BH, 2 ** 26 / (256 * seq) + 0.5)))
    fwd, bwd = run(2 * Tq + 2 * Tk), run(3 * Tq + 4 * Tk)
    part = min(fwd, bwd)
    assert BH >= 2 * bwd and BH % bwd  # several, with a remainder
    gen = torch.Generator(device="cuda").manual_seed(79)
    Q, dO = (torch.randn((1, BH, Tq, 64), generator=gen, device="cuda") for _ in range(2))
    K, V = (torch.randn((1, BH, Tk, 64), generator=gen, device="cuda") for _ in range(2))
    O, LSE = hk.attention_forward(Q, K, V, SCALE, causal)
    got = (O, LSE) + hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, causal, deterministic_dq=True)[:3]
    for i in range(0, BH, part):
        s = slice(i, min(BH, i + part))
        o, l = hk.attention_forward(Q[:, s], K[:, s], V[:, s], SCALE, causal)
        want = (o, l) + hk.attention_backward(Q[:, s], K[:, s], V[:, s], o, dO[:, s], l, SCALE, causal, deterministic_dq=True)[:3]
        for g, w in zip(got, want):
            assert torch.equal(g[:, s], w)
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0


@pytest.mark.gpu
def test_a_chunked_host_step_beyond_them_agrees_within_rounding():
    """One long sequence, its heads one by one or in one call: the forward is cut differently, so a probability is rounded
    to TF32 (2^-11 of itself) relative to another maximum on either side."""
    B, H, T = 1, 4, 6000
    assert forward_plan(1, T, T, True) != forward_plan(H, T, T, True)
    gen = torch.Generator(device="cuda").manual_seed(78)
    Q, K, V, dO = (torch.randn((B, H, T, 64), generator=gen, device="cuda") for _ in range(4))
    O, LSE = hk.attention_forward(Q, K, V, SCALE, True)
    want = (O, LSE) + hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, True)[:3]
    hin = [x.cpu().pin_memory() for x in (Q, K, V, dO)]
    hout = [torch.full(x.shape, float("nan")).pin_memory() for x in want]
    hk.HostAttentionStep(B, H, T, SCALE, True, chunks=H).step(*hin, *hout)
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0
    for got, ref in zip(hout, want):
        ref = ref.cpu().double()
        assert float((got.double() - ref).norm() / ref.norm()) <= 2.0 ** -10
