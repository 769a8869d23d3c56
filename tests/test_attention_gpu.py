"""GPU parity tests: the sm_100a kernels, called through the C ABI, against the
CPU oracle on identical seeded inputs.

Gate (fp32 I/O, TF32 multiplies): max abs error <= 5e-3 and relative L2 error
<= 1e-3 on O, dQ, dK, dV versus the oracle; LSE within 2e-3 absolute; the
reference test's own, looser, peak-relative tolerances (kernels_test.cu:535-537,
589-593) are asserted as well on the reference test's shape.  The dropout
keep-mask is compared bit for bit.
"""
import numpy as np
import pytest
import torch

import hyperkernels_b200 as hk
import oracle_lib as ol

pytestmark = pytest.mark.gpu

MAX_ABS, REL_L2, LSE_ABS = 5e-3, 1e-3, 2e-3
SCALE = 0.125


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def host(t):
    return t.detach().cpu().numpy()


def gate(name, got, ref, max_abs=MAX_ABS, rel=REL_L2):
    """max-abs gate always; relative-L2 gate whenever the oracle tensor is not itself numerical noise
    (with a single visible key dS = p (dP - D) is exactly 0 in real arithmetic, so dQ and dK of such a
    case are pure rounding residue on both sides: RMS below 1e-3 is judged by max-abs only)."""
    assert not np.isnan(got).any(), name
    ma, rl = ol.max_abs(got, ref), ol.rel_l2(got, ref)
    # 5e-3 is stated for outputs of the BASELINE configs' magnitude (|x| below about 5); where a case with
    # very few keys produces gradients of magnitude 10-15 the bound scales with it (1e-3 of the peak)
    bound = max(max_abs, 1e-3 * float(np.abs(ref).max())) if ref.size else max_abs
    assert ma <= bound, f"{name}: max abs {ma:.3e} > {bound}"
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2))) if ref.size else 0.0
    if rms >= 1e-3:
        assert rl <= rel, f"{name}: rel L2 {rl:.3e} > {rel}"


def lse_check(got, ref, tol=LSE_ABS):
    """-inf (fully masked / fully dropped rows) must match exactly, the rest within tol."""
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fin)
    assert np.array_equal(got[~fin], ref[~fin])
    assert ol.max_abs(got[fin], ref[fin]) <= tol


def ok_status():
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0


def normal(shape, seed, sigma=1.0):
    return (np.random.default_rng(seed).standard_normal(shape) * sigma).astype(np.float32)


def run_fwd_bwd_check(Q, K, V, dO, causal, mask=None, fwd_kw=None, bwd_kw=None, q_pos0=0, k_pos0=0, chained=False):
    """Forward vs oracle; backward fed the ORACLE's O/LSE (the reference tests the backward in isolation,
    kernels_test.cu:559-561) unless chained."""
    fwd_kw, bwd_kw = dict(fwd_kw or {}), dict(bwd_kw or {})
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, causal, mask, q_pos0, k_pos0)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(Q, K, V, O_ref, dO, L_ref, SCALE, causal, mask, q_pos0, k_pos0)
    tQ, tK, tV, tdO = dev(Q), dev(K), dev(V), dev(dO)
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, causal, q_pos0=q_pos0, k_pos0=k_pos0, **fwd_kw)
    ok_status()
    gate("O", host(O), O_ref)
    lse_check(host(LSE), L_ref)
    Oin, Lin = (O, LSE) if chained else (dev(O_ref), dev(L_ref))
    dQ, dK, dV, D = hk.attention_backward(tQ, tK, tV, Oin, tdO, Lin, SCALE, causal, q_pos0=q_pos0, k_pos0=k_pos0, **bwd_kw)
    ok_status()
    gate("D", host(D), D_ref, max_abs=2e-2 if chained else 1e-4, rel=1e-3 if chained else 1e-5)
    gate("dQ", host(dQ), dQ_ref)
    gate("dK", host(dK), dK_ref)
    gate("dV", host(dV), dV_ref)
    return dict(O=host(O), LSE=host(LSE), dQ=host(dQ), dK=host(dK), dV=host(dV), refs=(O_ref, L_ref, dQ_ref, dK_ref, dV_ref))


# ---------------------------------------------------------------------------
# the reference's own test: B=2,H=6,T=256, uniform[-1,1] from mt19937_64 seeds 101..104
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("causal", [0, 1])
def test_reference_test_shape(causal):
    B, H, T = 2, 6, 256
    n = B * H * T * 64
    Q, K, V, dO = (ol.rand_vec(n, s).reshape(B, H, T, 64) for s in (101, 102, 103, 104))
    r = run_fwd_bwd_check(Q, K, V, dO, causal)
    O_ref, L_ref, dQ_ref, dK_ref, dV_ref = r["refs"]
    # the reference's peak-relative tolerances (kernels_test.cu:535-537, 589-593)
    assert ol.max_abs(r["O"], O_ref) <= max(2e-3, 0.04 * np.abs(O_ref).max())
    assert ol.max_abs(r["LSE"], L_ref) <= max(2e-3, 0.02 * np.abs(L_ref).max())
    for k, ref in (("dQ", dQ_ref), ("dK", dK_ref), ("dV", dV_ref)):
        assert ol.max_abs(r[k], ref) <= max(2e-3, 0.08 * np.abs(ref).max())


@pytest.mark.parametrize("name", ["attn_ref_T256", "attn_ref_T77"])
@pytest.mark.parametrize("causal", [0, 1])
def test_against_golden_vectors(name, causal):
    import os

    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", name + ".npz"))
    B, H, T, Hd, *seeds = [int(x) for x in g["meta"]]
    n = B * H * T * 64
    Q, K, V, dO = (dev(ol.rand_vec(n, s).reshape(B, H, T, 64)) for s in seeds)
    O, LSE = hk.attention_forward(Q, K, V, SCALE, causal)
    gate("O", host(O), g[f"O_causal{causal}"])
    assert ol.max_abs(host(LSE), g[f"LSE_causal{causal}"]) <= LSE_ABS
    dQ, dK, dV, D = hk.attention_backward(Q, K, V, dev(g[f"O_causal{causal}"]), dO, dev(g[f"LSE_causal{causal}"]), SCALE, causal)
    ok_status()
    gate("D", host(D), g[f"D_causal{causal}"], 1e-4, 1e-5)
    for k, t in (("dQ", dQ), ("dK", dK), ("dV", dV)):
        gate(k, host(t), g[f"{k}_causal{causal}"])


# ---------------------------------------------------------------------------
# BASELINE configs
# ---------------------------------------------------------------------------
def test_config1_B2_H4_N256_causal():
    Q, K, V, dO = (normal((2, 4, 256, 64), s) for s in (0, 1, 2, 3))
    run_fwd_bwd_check(Q, K, V, dO, 1)
    run_fwd_bwd_check(Q, K, V, dO, 1, chained=True)


def test_config2_gpt2_small_full():
    """B=8,H=12,N=1024 causal, every head against the oracle (threads)."""
    Q, K, V, dO = (normal((8, 12, 1024, 64), s) for s in (10, 11, 12, 13))
    run_fwd_bwd_check(Q, K, V, dO, 1)


def _subset_check(B, H, N, causal, p, sigma, heads, seed):
    """Full-size run on the GPU; the listed (b,h) heads are checked against the oracle."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    Q, K, V = (torch.randn((B, H, N, 64), generator=g, device="cuda") * sigma for _ in range(3))
    dO = torch.randn((B, H, N, 64), generator=g, device="cuda")
    kw = dict(dropout_p=p, philox_seed=0x1234ABCD5678, philox_offset=42) if p > 0 else {}
    O, LSE = hk.attention_forward(Q, K, V, SCALE, causal, **kw)
    dQ, dK, dV, D = hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, causal, **kw)
    ok_status()
    for (b, h) in heads:
        q, k, v, g_ = (host(t[b:b + 1, h:h + 1]) for t in (Q, K, V, dO))
        mask = _philox_mask_numpy(b * H + h, N, N, p, 0x1234ABCD5678, 42) if p > 0 else None
        O_ref, L_ref = ol.attn_forward(q, k, v, SCALE, causal, mask)
        D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward(q, k, v, host(O[b:b + 1, h:h + 1]), g_, host(LSE[b:b + 1, h:h + 1]),
                                                         SCALE, causal, mask)
        gate("O", host(O[b:b + 1, h:h + 1]), O_ref)
        lse_check(host(LSE[b:b + 1, h:h + 1]), L_ref)
        gate("dQ", host(dQ[b:b + 1, h:h + 1]), dQ_ref)
        gate("dK", host(dK[b:b + 1, h:h + 1]), dK_ref)
        gate("dV", host(dV[b:b + 1, h:h + 1]), dV_ref)
    return O, LSE, dQ, dK, dV, dO


def _philox_mask_numpy(bh, Tq, Tk, p, seed, offset, q_pos0=0, k_pos0=0):
    """Vectorised numpy Philox4x32-10 keep-mask, identical to csrc/philox.h (checked against it in
    test_dropout_mask_bit_exact): counter {k >> 3, q, bh, lo32(offset)}, 16-bit half number k & 7."""
    M0, M1, W0, W1 = 0xD2511F53, 0xCD9E8D57, 0x9E3779B9, 0xBB67AE85
    assert k_pos0 % 8 == 0
    qi = (np.arange(Tq, dtype=np.uint64) + q_pos0)[:, None]
    k8 = (np.arange((Tk + 7) // 8, dtype=np.uint64) + (k_pos0 >> 3))[None, :]
    c0 = np.broadcast_to(k8, (Tq, k8.shape[1])).astype(np.uint64)
    c1 = np.broadcast_to(qi, c0.shape).astype(np.uint64)
    c2 = np.full(c0.shape, bh, np.uint64)
    c3 = np.full(c0.shape, offset & 0xFFFFFFFF, np.uint64)
    k0 = seed & 0xFFFFFFFF
    k1 = ((seed >> 32) ^ (offset >> 32)) & 0xFFFFFFFF
    for _ in range(10):
        p0 = c0 * np.uint64(M0)
        p1 = c2 * np.uint64(M1)
        hi0, lo0 = p0 >> np.uint64(32), p0 & np.uint64(0xFFFFFFFF)
        hi1, lo1 = p1 >> np.uint64(32), p1 & np.uint64(0xFFFFFFFF)
        n0 = hi1 ^ c1 ^ np.uint64(k0)
        n2 = hi0 ^ c3 ^ np.uint64(k1)
        c0, c1, c2, c3 = n0, lo1, n2, lo0
        k0 = (k0 + W0) & 0xFFFFFFFF
        k1 = (k1 + W1) & 0xFFFFFFFF
    words = np.stack([c0, c1, c2, c3], axis=-1)  # [Tq, groups, 4]
    halves = np.stack([words & np.uint64(0xFFFF), words >> np.uint64(16)], axis=-1).reshape(Tq, -1)[:, :Tk]
    thr = min(int(np.float32(p).astype(np.float64) * 65536.0), 65535)
    return (halves >= np.uint64(thr)).astype(np.float32)[None]


def test_config3_noncausal_dropout_subset():
    """B=16,H=16,N=2048, p=0.1, sigma 0.5; 8 heads against the oracle, incl. first and last."""
    _subset_check(16, 16, 2048, 0, 0.1, 0.5, [(0, 0), (7, 3), (15, 15), (3, 9), (0, 15), (15, 0), (8, 8), (11, 5)], seed=3)


def test_config4_gpt2_xl_causal_dropout_subset():
    """B=32,H=25,N=1024 causal p=0.1; 8 heads against the oracle, incl. first and last."""
    _subset_check(32, 25, 1024, 1, 0.1, 1.0, [(0, 0), (31, 24), (5, 7), (16, 12), (1, 1), (20, 3), (0, 24), (31, 0)], seed=4)


# ---------------------------------------------------------------------------
# edge cases: ragged lengths, tiny T, Tq != Tk, strided layouts, pre-rounded operands
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("T", [1, 5, 64, 127, 128, 129, 200, 333])
@pytest.mark.parametrize("causal", [0, 1])
def test_ragged_lengths(T, causal):
    Q, K, V, dO = (normal((1, 3, T, 64), 100 + s + T) for s in range(4))
    run_fwd_bwd_check(Q, K, V, dO, causal)


@pytest.mark.parametrize("Tq,Tk", [(100, 300), (300, 100), (128, 3), (257, 513)])
def test_different_query_and_key_lengths(Tq, Tk):
    Q, dO = normal((2, 2, Tq, 64), 1), normal((2, 2, Tq, 64), 2)
    K, V = normal((2, 2, Tk, 64), 3), normal((2, 2, Tk, 64), 4)
    run_fwd_bwd_check(Q, K, V, dO, 0)


def test_single_key():
    """One key: P = 1, O = v, dV = sum of dO rows; dS = p (dP - D) cancels exactly in real arithmetic, so dQ and dK
    are the residue of dP (a TF32 product) against D (an fp32 product) -- bounded by the TF32 unit roundoff
    2^-11 * |dP| * scale per element, summed over the 128 query rows for dK."""
    Tq = 128
    Q, dO = normal((1, 2, Tq, 64), 1), normal((1, 2, Tq, 64), 2)
    K, V = normal((1, 2, 1, 64), 3), normal((1, 2, 1, 64), 4)
    O_ref, L_ref = ol.attn_forward(Q, K, V, SCALE, 0)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward(Q, K, V, O_ref, dO, L_ref, SCALE, 0)
    O, LSE = hk.attention_forward(dev(Q), dev(K), dev(V), SCALE, False)
    dQ, dK, dV, D = hk.attention_backward(dev(Q), dev(K), dev(V), O, dev(dO), LSE, SCALE, False)
    ok_status()
    gate("O", host(O), O_ref); lse_check(host(LSE), L_ref); gate("dV", host(dV), dV_ref)
    assert ol.max_abs(host(dQ), dQ_ref) <= 5e-3
    assert ol.max_abs(host(dK), dK_ref) <= 5e-2


@pytest.mark.parametrize("q_pos0,k_pos0,Tq,Tk", [(256, 0, 128, 384), (128, 128, 200, 200), (0, 128, 256, 128), (384, 256, 100, 260)])
def test_causal_blocks_with_positions(q_pos0, k_pos0, Tq, Tk):
    """A block of queries against a block of keys at global positions (ring-attention step);
    rows that see no key in the block give O = 0, LSE = -inf."""
    Q, dO = normal((1, 2, Tq, 64), 5), normal((1, 2, Tq, 64), 6)
    K, V = normal((1, 2, Tk, 64), 7), normal((1, 2, Tk, 64), 8)
    run_fwd_bwd_check(Q, K, V, dO, 1, q_pos0=q_pos0, k_pos0=k_pos0)


def test_strided_bthd_layout_prerounded():
    """[B,T,H,64] storage viewed as [B,H,T,64] (strideM > strideH), operands already TF32-representable:
    the kernels read the caller's tensors directly through TMA, no workspace."""
    B, H, T = 2, 3, 200
    def tf32(x):
        return ((x.view(np.uint32) + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32)
    Qs, Ks, Vs, dOs = (tf32(normal((B, T, H, 64), 30 + s)) for s in range(4))
    Q, K, V, dO = (x.transpose(0, 2, 1, 3) for x in (Qs, Ks, Vs, dOs))  # numpy views [B,H,T,64]
    O_ref, L_ref = ol.attn_forward_mt(np.ascontiguousarray(Q), np.ascontiguousarray(K), np.ascontiguousarray(V), SCALE, 1)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(*(np.ascontiguousarray(x) for x in (Q, K, V)), O_ref,
                                                         np.ascontiguousarray(dO), L_ref, SCALE, 1)
    tQ, tK, tV, tdO = (dev(x).permute(0, 2, 1, 3) for x in (Qs, Ks, Vs, dOs))
    out = torch.empty((B, T, H, 64), device="cuda").permute(0, 2, 1, 3)
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, 1, prerounded=True, out=out)
    gate("O", host(O), O_ref)
    dQ = torch.empty((B, T, H, 64), device="cuda").permute(0, 2, 1, 3)
    dK = torch.empty((B, T, H, 64), device="cuda").permute(0, 2, 1, 3)
    dV = torch.empty((B, T, H, 64), device="cuda").permute(0, 2, 1, 3)
    tO = dev(O_ref)
    hk.attention_backward(tQ, tK, tV, tO, tdO, dev(L_ref), SCALE, 1, prerounded=True, dQ=dQ, dK=dK, dV=dV)
    ok_status()
    gate("dQ", host(dQ), dQ_ref); gate("dK", host(dK), dK_ref); gate("dV", host(dV), dV_ref)


def test_packed_qkv_layout():
    """Packed [B, T, 3, H, 64] storage (the output of a fused QKV projection): Q, K, V are views into one buffer,
    addressed through the reference block's stride triplets (fused_attn_forward_kernel_tc_sm89.cu:24-28); the
    gradients go into a buffer of the same packing.  Arbitrary fp32 inputs, rounded as the loads read the strided views."""
    B, H, T = 2, 4, 333
    qkv = normal((B, T, 3, H, 64), 35)
    dO = normal((B, H, T, 64), 36)
    Q, K, V = (np.ascontiguousarray(qkv[:, :, i].transpose(0, 2, 1, 3)) for i in range(3))
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, 1)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(Q, K, V, O_ref, dO, L_ref, SCALE, 1)
    t_qkv = dev(qkv)
    tQ, tK, tV = (t_qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    assert tQ.stride() == (T * 3 * H * 64, 64, 3 * H * 64, 1)
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, 1)
    ok_status()
    gate("O", host(O), O_ref)
    lse_check(host(LSE), L_ref)
    t_grad = torch.full((B, T, 3, H, 64), float("nan"), device="cuda")
    gQ, gK, gV = (t_grad[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    hk.attention_backward(tQ, tK, tV, O, dev(dO), LSE, SCALE, 1, dQ=gQ, dK=gK, dV=gV)
    ok_status()
    gate("dQ", host(gQ), dQ_ref); gate("dK", host(gK), dK_ref); gate("dV", host(gV), dV_ref)


def test_negative_scale_and_large_scores():
    """Every 64th key row scaled x8 (the long-sequence config's stress of the running max), and a negative scale."""
    Q, K, V, dO = (normal((1, 2, 512, 64), 40 + s) for s in range(4))
    K[:, :, ::64] *= 8.0
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, 1)
    O, LSE = hk.attention_forward(dev(Q), dev(K), dev(V), SCALE, 1)
    # scores reach |s| ~ 60 here: TF32 product error grows with the operand magnitude, gate relative to it
    assert ol.rel_l2(host(O), O_ref) <= 3e-3 and ol.max_abs(host(LSE), L_ref) <= 2e-2
    O_ref2, L_ref2 = ol.attn_forward_mt(Q, normal((1, 2, 512, 64), 41), V, -SCALE, 0)
    O2, L2 = hk.attention_forward(dev(Q), dev(normal((1, 2, 512, 64), 41)), dev(V), -SCALE, 0)
    ok_status()
    gate("O", host(O2), O_ref2)
    assert ol.max_abs(host(L2), L_ref2) <= LSE_ABS


# ---------------------------------------------------------------------------
# dropout
# ---------------------------------------------------------------------------
def test_dropout_mask_bit_exact():
    """Read the kernel's keep-mask out through the forward itself: Q = 0 makes every score equal, V = identity
    makes O[i, j] = keep(i, k_pos0 + j) / (number kept), so O > 0 is the mask.  Compared bit for bit with the host
    twin (hk_attn_dropout_mask) and with the numpy Philox used by the large-config tests."""
    BH_B, BH_H, Tq = 2, 3, 200
    seed, offset, p = 0xDEADBEEFCAFEF00D, 0x1_0000_0007, 0.1
    Q = torch.zeros((BH_B, BH_H, Tq, 64), device="cuda")
    eye = torch.eye(64, device="cuda").expand(BH_B, BH_H, 64, 64).contiguous()
    K = torch.zeros((BH_B, BH_H, 64, 64), device="cuda")
    host_mask = hk.dropout_keep_mask(BH_B * BH_H, Tq, 256, p, seed, offset, q_pos0=16, k_pos0=0)
    assert np.array_equal(host_mask, ol.dropout_mask(BH_B * BH_H, Tq, 256, p, seed, offset, 16, 0))
    for c in range(4):
        O, _ = hk.attention_forward(Q, K, eye, SCALE, False, dropout_p=p, philox_seed=seed, philox_offset=offset,
                                    q_pos0=16, k_pos0=64 * c)
        got = (host(O) > 0).astype(np.float32).reshape(BH_B * BH_H, Tq, 64)
        assert np.array_equal(got, host_mask[:, :, 64 * c:64 * c + 64]), c
    ok_status()
    for bh in (0, 5):
        assert np.array_equal(_philox_mask_numpy(bh, Tq, 256, p, seed, offset, 16, 0)[0], host_mask[bh])
    assert abs(host_mask.mean() - 0.9) < 0.01


@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("mode", ["philox", "dense"])
def test_dropout_forward_backward(causal, mode):
    B, H, T, p, seed, off = 2, 2, 300, 0.25, 777, 12
    Q, K, V, dO = (normal((B, H, T, 64), 50 + s) for s in range(4))
    mask = ol.dropout_mask(B * H, T, T, p, seed, off)
    if mode == "philox":
        kw = dict(dropout_p=p, philox_seed=seed, philox_offset=off)
    else:
        kw = dict(dropout_p=p, dropout_mask=dev(mask))
    r = run_fwd_bwd_check(Q, K, V, dO, causal, mask=mask, fwd_kw=kw, bwd_kw=kw)
    if mode == "dense":
        run_fwd_bwd_check(Q, K, V, dO, causal, mask=mask, fwd_kw=kw, bwd_kw=kw, chained=True)
    assert r is not None


@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("mode", ["philox", "dense"])
def test_inverted_dropout_forward_backward(causal, mode):
    """HK_FLAG_DROPOUT_SCALED: normaliser over all visible keys, kept terms times 1/(1-p); no reference counterpart,
    the oracle for it is pinned by finite differences (tests/test_oracle.py)."""
    B, H, T, p, seed, off = 2, 2, 300, 0.1, 4242, 8
    Q, K, V, dO = (normal((B, H, T, 64), 150 + s) for s in range(4))
    mask = ol.dropout_mask(B * H, T, T, p, seed, off)
    if mode == "philox":
        kw = dict(dropout_p=p, philox_seed=seed, philox_offset=off, dropout_scaled=True)
        p_eff = np.floor(p * 65536.0) / 65536.0  # the 16-bit threshold the mask was drawn with
    else:
        kw = dict(dropout_p=p, dropout_mask=dev(mask), dropout_scaled=True)
        p_eff = p
    O_ref, L_ref = ol.attn_forward_scaled(Q, K, V, SCALE, causal, mask, p_eff)
    _, L_plain = ol.attn_forward(Q, K, V, SCALE, causal)
    assert np.array_equal(L_ref, L_plain)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward_scaled(Q, K, V, O_ref, dO, L_ref, SCALE, causal, mask, p_eff)
    tQ, tK, tV, tdO = dev(Q), dev(K), dev(V), dev(dO)
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, causal, **kw)
    ok_status()
    gate("O", host(O), O_ref)
    lse_check(host(LSE), L_ref)
    for chained in (False, True):
        Oin, Lin = (O, LSE) if chained else (dev(O_ref), dev(L_ref))
        dQ, dK, dV, D = hk.attention_backward(tQ, tK, tV, Oin, tdO, Lin, SCALE, causal, **kw)
        ok_status()
        gate("D", host(D), D_ref, max_abs=2e-2 if chained else 1e-4, rel=1e-3 if chained else 1e-5)
        gate("dQ", host(dQ), dQ_ref)
        gate("dK", host(dK), dK_ref)
        gate("dV", host(dV), dV_ref)
    # the flag is inert without active dropout
    O0, L0 = hk.attention_forward(tQ, tK, tV, SCALE, causal)
    O1, L1 = hk.attention_forward(tQ, tK, tV, SCALE, causal, dropout_scaled=True)
    assert torch.equal(O0, O1) and torch.equal(L0, L1)


def test_fully_dropped_row():
    """Causal row 0 sees only key 0; when that key is dropped the reference gives O = 0, LSE = -inf
    (fused_attn_forward_kernel_tc_sm89.cu:412,424) and the backward must treat the row as p = 0."""
    B, H, T, p, seed = 1, 8, 64, 0.6, 5
    mask = ol.dropout_mask(B * H, T, T, p, seed, 0)
    dropped = [bh for bh in range(B * H) if mask[bh, 0, 0] == 0]
    assert dropped, "pick another seed"
    Q, K, V, dO = (normal((B, H, T, 64), 60 + s) for s in range(4))
    kw = dict(dropout_p=p, philox_seed=seed, philox_offset=0)
    r = run_fwd_bwd_check(Q, K, V, dO, 1, mask=mask, fwd_kw=kw, bwd_kw=kw, chained=True)
    for bh in dropped:
        assert np.all(r["O"][0, bh, 0] == 0) and r["LSE"][0, bh, 0] == -np.inf
        assert np.all(r["dQ"][0, bh, 0] == 0)


# ---------------------------------------------------------------------------
# the other entry points
# ---------------------------------------------------------------------------
def test_precompute_D_reference_shape():
    """kernels_test.cu:459-481: B=16, nh=12, T=1024, seeds 17/18, tolerance 2e-2 there."""
    B, H, T = 16, 12, 1024
    n = B * H * T * 64
    dO, O = ol.rand_vec(n, 17).reshape(B, H, T, 64), ol.rand_vec(n, 18).reshape(B, H, T, 64)
    p = hk.MemEfficientBwdParams()
    tdO, tO = dev(dO), dev(O)
    D = torch.empty((B, H, T), device="cuda")
    p.dO, p.O, p.D = tdO.data_ptr(), tO.data_ptr(), D.data_ptr()
    p.B, p.nh, p.T, p.scale = B, H, T, 1.0
    p.do_strideB, p.do_strideH, p.do_strideM = H * T * 64, T * 64, 64
    p.o_strideB, p.o_strideH, p.o_strideM = H * T * 64, T * 64, 64
    p.d_strideB, p.d_strideH = H * T, T
    hk.mem_efficient_bwd_precompute_D(p)
    ok_status()
    assert ol.max_abs(host(D), ol.precompute_D(dO, O)) <= 1e-4


@pytest.mark.parametrize("hd", [16, 32, 48, 64, 80, 96, 128, 160, 192, 256])
def test_precompute_D_other_head_dims(hd):
    """mem_efficient_bwd_precompute_D_sm89.cu:93-102 instantiates the pre-pass for these head dimensions; rows of a
    [B, T, H, hd] layout (strided heads) and a ragged row count."""
    B, H, T = 2, 3, 517
    rng = np.random.default_rng(hd)
    dO = rng.standard_normal((B, T, H, hd)).astype(np.float32)
    O = rng.standard_normal((B, T, H, hd)).astype(np.float32)
    tdO, tO = dev(dO), dev(O)
    D = torch.empty((B, H, T), device="cuda")
    p = hk.MemEfficientBwdParams()
    p.dO, p.O, p.D = tdO.data_ptr(), tO.data_ptr(), D.data_ptr()
    p.B, p.nh, p.T, p.scale = B, H, T, 1.0
    p.do_strideB, p.do_strideM, p.do_strideH = T * H * hd, H * hd, hd
    p.o_strideB, p.o_strideM, p.o_strideH = T * H * hd, H * hd, hd
    p.d_strideB, p.d_strideH = H * T, T
    hk.mem_efficient_bwd_precompute_D(p, head_dim=hd)
    ok_status()
    ref = (dO.astype(np.float64) * O).sum(-1).transpose(0, 2, 1)
    assert np.abs(host(D) - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    with pytest.raises(hk.HKError):
        hk.mem_efficient_bwd_precompute_D(p, head_dim=72)  # not one of the reference's ten instantiations


def test_backward_with_precomputed_D_and_accumulation():
    B, H, T = 1, 2, 256
    Q, K, V, dO = (normal((B, H, T, 64), 70 + s) for s in range(4))
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, 1)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(Q, K, V, O_ref, dO, L_ref, SCALE, 1)
    t = [dev(x) for x in (Q, K, V, O_ref, dO, L_ref)]
    D = dev(D_ref)
    base = torch.ones((B, H, T, 64), device="cuda")
    dQ, dK, dV = base.clone(), base.clone() * 2, base.clone() * 3
    hk.attention_backward(t[0], t[1], t[2], None, t[4], t[5], SCALE, 1, D=D, d_precomputed=True, accum_dq=True,
                          accum_dkdv=True, dQ=dQ, dK=dK, dV=dV)
    ok_status()
    gate("dQ", host(dQ) - 1, dQ_ref); gate("dK", host(dK) - 2, dK_ref); gate("dV", host(dV) - 3, dV_ref)


def test_backward_reuses_forward_rounded_operands():
    """Same workspace for forward and backward, with the flag that says so: accepted, and the results are those without."""
    B, H, T = 2, 3, 300
    Q, K, V, dO = (normal((B, H, T, 64), 90 + s) for s in range(4))
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, 1)
    D_ref, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(Q, K, V, O_ref, dO, L_ref, SCALE, 1)
    tQ, tK, tV, tdO = dev(Q), dev(K), dev(V), dev(dO)
    ws = torch.empty(4 * B * H * T * 256 + 512, dtype=torch.uint8, device="cuda")
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, True, workspace=ws)
    dQ, dK, dV, D = hk.attention_backward(tQ, tK, tV, O, tdO, LSE, SCALE, True, workspace=ws, reuse_fwd_rounded=True)
    ok_status()
    gate("O", host(O), O_ref); gate("dQ", host(dQ), dQ_ref); gate("dK", host(dK), dK_ref); gate("dV", host(dV), dV_ref)
    dQ2, dK2, dV2, _ = hk.attention_backward(tQ, tK, tV, O, tdO, LSE, SCALE, True)
    assert torch.equal(dK, dK2) and torch.equal(dV, dV2)


@pytest.mark.parametrize("chunks", [1, 2, 4])
def test_host_step_pipeline_matches_direct_calls(chunks):
    """HostAttentionStep (pinned host tensors, batch chunks, copies overlapped with kernels) gives what the direct
    device-tensor calls give: O, LSE, dK, dV bit for bit (each (b,h) slice is computed the same way), dQ up to the
    order of its fp32 reductions."""
    B, H, T = 4, 3, 384
    Q, K, V, dO = (normal((B, H, T, 64), 80 + s) for s in range(4))
    tQ, tK, tV, tdO = dev(Q), dev(K), dev(V), dev(dO)
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, 1)
    dQ, dK, dV, _ = hk.attention_backward(tQ, tK, tV, O, tdO, LSE, SCALE, 1)
    hin = [torch.from_numpy(x).pin_memory() for x in (Q, K, V, dO)]
    hO, hdQ, hdK, hdV = (torch.full((B, H, T, 64), float("nan")).pin_memory() for _ in range(4))
    hLSE = torch.full((B, H, T), float("nan")).pin_memory()
    hs = hk.HostAttentionStep(B, H, T, SCALE, True, chunks=chunks)
    for it in range(3):  # first step issued call by call, second captured in a CUDA graph and replayed, third replayed
        for t in (hO, hdQ, hdK, hdV, hLSE):
            t.fill_(float("nan"))
        hs.step(*hin, hO, hLSE, hdQ, hdK, hdV)
        torch.cuda.synchronize()
        assert torch.equal(hO, O.cpu()) and torch.equal(hdK, dK.cpu()), it
    ok_status()
    assert torch.equal(hO, O.cpu()) and torch.equal(hLSE, LSE.cpu())
    assert torch.equal(hdK, dK.cpu()) and torch.equal(hdV, dV.cpu())
    assert float((hdQ - dQ.cpu()).abs().max()) <= 1e-4
    assert hs.h2d_bytes == 4 * Q.nbytes and hs.d2h_bytes == 4 * Q.nbytes + LSE.numel() * 4


@pytest.mark.parametrize("chunks", [2, 4])
def test_host_step_with_dropout_draws_the_mask_of_the_single_call(chunks):
    """Philox dropout through HostAttentionStep: every chunk passes the index of its first (batch, head) slice
    (bh_pos0) with the same seed and offset, so the chunked step reproduces the direct call over the whole batch
    bit for bit on O, LSE, dK, dV (dQ up to the order of its fp32 reductions)."""
    B, H, T, p, seed, off = 4, 3, 384, 0.1, 0xABCDEF0123, 5
    Q, K, V, dO = (normal((B, H, T, 64), 180 + s) for s in range(4))
    tQ, tK, tV, tdO = dev(Q), dev(K), dev(V), dev(dO)
    kw = dict(dropout_p=p, philox_seed=seed, philox_offset=off)
    O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, 1, **kw)
    dQ, dK, dV, _ = hk.attention_backward(tQ, tK, tV, O, tdO, LSE, SCALE, 1, **kw)
    hin = [torch.from_numpy(x).pin_memory() for x in (Q, K, V, dO)]
    hO, hdQ, hdK, hdV = (torch.full((B, H, T, 64), float("nan")).pin_memory() for _ in range(4))
    hLSE = torch.full((B, H, T), float("nan")).pin_memory()
    hs = hk.HostAttentionStep(B, H, T, SCALE, True, chunks=chunks, **kw)
    hs.step(*hin, hO, hLSE, hdQ, hdK, hdV)
    torch.cuda.synchronize()
    ok_status()
    assert torch.equal(hO, O.cpu()) and torch.equal(hLSE, LSE.cpu())
    assert torch.equal(hdK, dK.cpu()) and torch.equal(hdV, dV.cpu())
    assert float((hdQ - dQ.cpu()).abs().max()) <= 1e-4
    # and the mask really is in play: without dropout the output differs
    O0, _ = hk.attention_forward(tQ, tK, tV, SCALE, 1)
    assert not torch.equal(O0, O)


def test_batch_head_slices_reproduce_the_whole_call_under_dropout():
    """A problem cut into runs of (batch, head) slices (what a batch x head partition over several GPUs does):
    each run, called with bh_pos0 = its first slice, equals those slices of the single call, bit for bit."""
    B, H, T, p, seed, off = 4, 5, 200, 0.2, 99, 3
    Q, K, V, dO = (dev(normal((B, H, T, 64), 190 + s)) for s in range(4))
    kw = dict(dropout_p=p, philox_seed=seed, philox_offset=off)
    O, LSE = hk.attention_forward(Q, K, V, SCALE, 0, **kw)
    dQ, dK, dV, _ = hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, 0, **kw)
    for b0, nb in ((0, 1), (1, 3)):
        sl = slice(b0, b0 + nb)
        q, k, v, g = (t[sl].contiguous() for t in (Q, K, V, dO))
        o, l = hk.attention_forward(q, k, v, SCALE, 0, bh_pos0=b0 * H, **kw)
        dq, dk, dv, _ = hk.attention_backward(q, k, v, o, g, l, SCALE, 0, bh_pos0=b0 * H, **kw)
        assert torch.equal(o, O[sl]) and torch.equal(l, LSE[sl])
        assert torch.equal(dk, dK[sl]) and torch.equal(dv, dV[sl])
        assert float((dq - dQ[sl]).abs().max()) <= 1e-4
    ok_status()


@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("B,H,T", [(2, 3, 640), (1, 2, 556), (1, 1, 1024)])
def test_rounding_in_shared_memory_equals_the_hbm_prepass(B, H, T, causal):
    """HK_FLAG_ROUND_IN_HBM, a workspace and HK_FLAG_REUSE_FWD_ROUNDED come from versions that rounded the operands in a
    pass over HBM or in shared memory; the loads round them now, and these change nothing: O, LSE, dK, dV identical bit
    for bit, dQ up to the order of its additions."""
    Q, K, V, dO = (dev(normal((B, H, T, 64), 900 + s)) for s in range(4))
    O_h, L_h = hk.attention_forward(Q, K, V, SCALE, causal, round_in_hbm=True)
    O_s, L_s = hk.attention_forward(Q, K, V, SCALE, causal)
    ok_status()
    assert torch.equal(O_h, O_s) and torch.equal(L_h, L_s)
    g_h = hk.attention_backward(Q, K, V, O_h, dO, L_h, SCALE, causal, round_in_hbm=True)
    g_s = hk.attention_backward(Q, K, V, O_h, dO, L_h, SCALE, causal)
    ok_status()
    assert torch.equal(g_h[1], g_s[1]) and torch.equal(g_h[2], g_s[2]) and torch.equal(g_h[3], g_s[3])
    assert float((g_h[0] - g_s[0]).abs().max()) <= 1e-4
    # forward and backward sharing one workspace
    p = hk.MemEfficientBwdParams()
    p.B, p.nh, p.T = B, H, T
    ws = torch.empty(hk.bwd_workspace_bytes(p) + 256, dtype=torch.uint8, device="cuda")
    ws.fill_(0x7F)  # nothing may be taken from the workspace
    O_w, L_w = hk.attention_forward(Q, K, V, SCALE, causal, workspace=ws)
    g_w = hk.attention_backward(Q, K, V, O_w, dO, L_w, SCALE, causal, workspace=ws, reuse_fwd_rounded=True)
    ok_status()
    assert torch.equal(O_w, O_h) and torch.equal(L_w, L_h)
    assert torch.equal(g_w[1], g_h[1]) and torch.equal(g_w[2], g_h[2]) and torch.equal(g_w[3], g_h[3])
    assert float((g_w[0] - g_h[0]).abs().max()) <= 1e-4


@pytest.mark.parametrize("Tq,Tk,q_pos0", [(640, 896, 256), (512, 1024, 0), (700, 300, 0)])
def test_workspace_handed_from_forward_to_backward_with_unequal_lengths(Tq, Tk, q_pos0):
    """A workspace full of NaN patterns, handed from the forward to the backward, is not read: causal mask with a query
    offset, more keys than any query sees, fewer keys than queries."""
    B, H = 1, 2
    Q, dO = dev(normal((B, H, Tq, 64), 910)), dev(normal((B, H, Tq, 64), 911))
    K, V = dev(normal((B, H, Tk, 64), 912)), dev(normal((B, H, Tk, 64), 913))
    O_h, L_h = hk.attention_forward(Q, K, V, SCALE, True, q_pos0=q_pos0, round_in_hbm=True)
    g_h = hk.attention_backward(Q, K, V, O_h, dO, L_h, SCALE, True, q_pos0=q_pos0, round_in_hbm=True)
    p = hk.MemEfficientBwdParams()
    p.B, p.nh, p.T, p.kv_len = B, H, Tq, Tk
    ws = torch.empty(hk.bwd_workspace_bytes(p) + 256, dtype=torch.uint8, device="cuda")
    ws.fill_(0x7F)
    O_w, L_w = hk.attention_forward(Q, K, V, SCALE, True, q_pos0=q_pos0, workspace=ws)
    g_w = hk.attention_backward(Q, K, V, O_w, dO, L_w, SCALE, True, q_pos0=q_pos0, workspace=ws, reuse_fwd_rounded=True)
    ok_status()
    assert torch.equal(O_w, O_h) and torch.equal(L_w, L_h)
    assert torch.equal(g_w[1], g_h[1]) and torch.equal(g_w[2], g_h[2])
    assert float((g_w[0] - g_h[0]).abs().max()) <= 1e-4


def random_shapes():
    """24 seeded problems: ragged lengths, unequal query/key lengths, position offsets, Philox dropout."""
    import random

    rnd = random.Random(2024)
    for _ in range(24):
        B, H = rnd.choice([(1, 1), (1, 3), (2, 2), (3, 5)])
        causal = rnd.random() < 0.6
        Tq = rnd.choice([512, 513, 600, 700, 1000, 1024, 1100, 1536, 2047, 2048, 300])
        Tk = rnd.choice([128, 257, 777, 1024, 1500]) if rnd.random() < 0.3 else Tq
        kw = dict(q_pos0=rnd.choice([0, 0, 128, 616]) if causal else 0, k_pos0=rnd.choice([0, 0, 64, 128]) if causal else 0)
        if rnd.random() < 0.3:
            kw.update(dropout_p=0.2, philox_seed=rnd.randrange(1 << 30), philox_offset=8 * rnd.randrange(100))
        yield B, H, Tq, Tk, causal, kw


@pytest.mark.parametrize("case", range(24))
def test_random_shapes_against_the_oracle(case):
    B, H, Tq, Tk, causal, kw = list(random_shapes())[case]
    Q, dO = normal((B, H, Tq, 64), 1000 + case), normal((B, H, Tq, 64), 1100 + case)
    K, V = normal((B, H, Tk, 64), 1200 + case), normal((B, H, Tk, 64), 1300 + case)
    pos = {k: kw.pop(k) for k in ("q_pos0", "k_pos0")}
    mask = None
    if kw:
        mask = ol.dropout_mask(B * H, Tq, Tk, kw["dropout_p"], kw["philox_seed"], kw["philox_offset"], **pos)
    run_fwd_bwd_check(Q, K, V, dO, causal, mask=mask, fwd_kw=kw, bwd_kw=kw, **pos)


def test_random_shapes_the_two_rounding_paths_and_the_workspace_hand_over_agree():
    """The random shapes (their values are held against the oracle above) with HK_FLAG_ROUND_IN_HBM, with a workspace and
    with HK_FLAG_REUSE_FWD_ROUNDED, which change nothing: identical O, LSE, dK, dV (dQ up to the order of its additions)."""
    g = torch.Generator(device="cuda").manual_seed(11)
    same = lambda a, b: torch.equal(torch.nan_to_num(a, nan=0.0, neginf=-1e30), torch.nan_to_num(b, nan=0.0, neginf=-1e30))
    for case, (B, H, Tq, Tk, causal, kw) in enumerate(random_shapes()):
        Q, dO = (torch.randn((B, H, Tq, 64), generator=g, device="cuda") for _ in range(2))
        K, V = (torch.randn((B, H, Tk, 64), generator=g, device="cuda") for _ in range(2))
        O1, L1 = hk.attention_forward(Q, K, V, SCALE, causal, round_in_hbm=True, **kw)
        O2, L2 = hk.attention_forward(Q, K, V, SCALE, causal, **kw)
        p = hk.MemEfficientBwdParams()
        p.B, p.nh, p.T, p.kv_len = B, H, Tq, (Tk if Tk != Tq else 0)
        ws = torch.empty(hk.bwd_workspace_bytes(p) + 256, dtype=torch.uint8, device="cuda")
        ws.fill_(0x7F)
        O3, L3 = hk.attention_forward(Q, K, V, SCALE, causal, workspace=ws, **kw)
        g1 = hk.attention_backward(Q, K, V, O1, dO, L1, SCALE, causal, round_in_hbm=True, **kw)
        g2 = hk.attention_backward(Q, K, V, O1, dO, L1, SCALE, causal, **kw)
        g3 = hk.attention_backward(Q, K, V, O3, dO, L3, SCALE, causal, workspace=ws, reuse_fwd_rounded=True, **kw)
        ok_status()
        what = (case, B, H, Tq, Tk, causal, kw)
        assert same(O1, O2) and same(L1, L2) and same(O1, O3) and same(L1, L3), what
        assert same(g1[1], g2[1]) and same(g1[2], g2[2]) and same(g1[1], g3[1]) and same(g1[2], g3[2]), what
        assert float((g1[0] - g2[0]).abs().max()) <= 1e-3 and float((g1[0] - g3[0]).abs().max()) <= 1e-3, what
        assert bool(torch.isfinite(O2).all()), what


@pytest.mark.parametrize("Tq,Tk,causal,q_pos0", [(333, 333, 1, 0), (640, 640, 0, 0), (200, 384, 1, 184), (1024, 1024, 1, 0)])
def test_deterministic_dq_is_bit_reproducible_and_equal_to_the_default(Tq, Tk, causal, q_pos0):
    """HK_FLAG_DETERMINISTIC_DQ: every KV-tile CTA stores its dQ tiles into a slab of the workspace and a second kernel
    adds the slabs in KV-tile order.  Same inputs, same bits, run after run (the default path adds with bulk reductions
    in whatever order the CTAs finish); the values agree with the default path and pass the oracle gate; accumulation
    into a given dQ works as on the default path."""
    B, H = 2, 3
    Q, dO = normal((B, H, Tq, 64), 920), normal((B, H, Tq, 64), 921)
    K, V = normal((B, H, Tk, 64), 922), normal((B, H, Tk, 64), 923)
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, causal, None, q_pos0, 0)
    _, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(Q, K, V, O_ref, dO, L_ref, SCALE, causal, None, q_pos0, 0)
    tQ, tK, tV, tdO, tO, tL = dev(Q), dev(K), dev(V), dev(dO), dev(O_ref), dev(L_ref)
    runs = [hk.attention_backward(tQ, tK, tV, tO, tdO, tL, SCALE, causal, q_pos0=q_pos0, deterministic_dq=True)
            for _ in range(4)]
    ok_status()
    for r in runs[1:]:
        assert torch.equal(r[0], runs[0][0]) and torch.equal(r[1], runs[0][1]) and torch.equal(r[2], runs[0][2])
    gate("dQ", host(runs[0][0]), dQ_ref)
    gate("dK", host(runs[0][1]), dK_ref)
    gate("dV", host(runs[0][2]), dV_ref)
    dflt = hk.attention_backward(tQ, tK, tV, tO, tdO, tL, SCALE, causal, q_pos0=q_pos0)
    assert float((dflt[0] - runs[0][0]).abs().max()) <= 1e-4
    assert torch.equal(dflt[1], runs[0][1]) and torch.equal(dflt[2], runs[0][2])
    # accumulation into a given dQ
    base = dev(normal((B, H, Tq, 64), 924))
    acc = base.clone()
    hk.attention_backward(tQ, tK, tV, tO, tdO, tL, SCALE, causal, q_pos0=q_pos0, deterministic_dq=True, accum_dq=True, dQ=acc)
    ok_status()
    assert float((acc - (base + runs[0][0])).abs().max()) <= 1e-5  # (base + slab0) + slab1 ... against base + (sum of slabs)


@pytest.mark.parametrize("T,causal", [(333, 1), (129, 0), (640, 1), (1000, 0)])
def test_outputs_stay_inside_their_buffers(T, causal):
    """Canary bands round every output (the memory checker is closed on this pool): O, LSE, dQ, dK, dV and D are views
    into one sentinel-filled allocation with 64 KiB of guard on both sides of each; after a forward and a backward on
    a ragged shape -- whose last tiles the TMA stores must clip -- every guard byte still holds the sentinel, and so
    does the workspace beyond the bytes the library asked for."""
    B, H = 2, 3
    Q, K, V, dO = (dev(normal((B, H, T, 64), 930 + s)) for s in range(4))
    guard = 16384  # floats
    n_big, n_small = B * H * T * 64, B * H * T
    sizes = [n_big, n_small, n_big, n_big, n_big, n_small]  # O, LSE, dQ, dK, dV, D
    pad = lambda x: (x + 63) // 64 * 64  # keeps every view 256-byte aligned; the padding belongs to the guard
    total = guard + sum(pad(x) + guard for x in sizes)
    SENT = 12345.678
    arena = torch.full((total,), SENT, dtype=torch.float32, device="cuda")
    views, off = [], guard
    for x in sizes:
        views.append(arena[off:off + x])
        off += pad(x) + guard
    O, LSE, dQ, dK, dV, D = views
    O, dQ, dK, dV = (t.view(B, H, T, 64) for t in (O, dQ, dK, dV))
    LSE, D = LSE.view(B, H, T), D.view(B, H, T)
    p = hk.MemEfficientBwdParams()
    p.B, p.nh, p.T = B, H, T
    need = hk.bwd_workspace_bytes(p)
    ws = torch.full((need + 256 + 65536,), 0x5A, dtype=torch.uint8, device="cuda")
    hk.attention_forward(Q, K, V, SCALE, causal, out=O, lse=LSE, workspace=ws[:need + 256])
    hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, causal, D=D, dQ=dQ, dK=dK, dV=dV, workspace=ws[:need + 256],
                          reuse_fwd_rounded=True)
    ok_status()
    mask = torch.ones(total, dtype=torch.bool, device="cuda")
    off = guard
    for x in sizes:
        mask[off:off + x] = False
        off += pad(x) + guard
    assert bool((arena[mask] == SENT).all()), "a guard band was written"
    assert bool((ws[need + 256:] == 0x5A).all()), "the workspace was written past the size the library asked for"
    for t in (O, dQ, dK, dV, LSE, D):
        assert bool(torch.isfinite(t).all()) and not bool((t == SENT).all())


def test_graphed_step_replays_the_direct_calls():
    """GraphedAttentionStep (forward + backward captured in a CUDA graph): a replay gives what the direct calls give,
    also after the inputs were refilled in place."""
    B, H, T = 2, 3, 320
    tQ, tK, tV, tdO = (dev(normal((B, H, T, 64), 90 + s)) for s in range(4))
    gs = hk.GraphedAttentionStep(tQ, tK, tV, tdO, SCALE, True)
    assert gs.launches_per_replay == 4  # forward, dQ zeroing beside it, D pre-pass, backward
    for seed in (0, 1):
        if seed:
            for t_, s in zip((tQ, tK, tV, tdO), range(4)):
                t_.copy_(dev(normal((B, H, T, 64), 95 + s)))
        gs.replay()
        torch.cuda.synchronize()
        ok_status()
        O, LSE = hk.attention_forward(tQ, tK, tV, SCALE, 1)
        dQ, dK, dV, _ = hk.attention_backward(tQ, tK, tV, O, tdO, LSE, SCALE, 1)
        assert torch.equal(gs.O, O) and torch.equal(gs.LSE, LSE)
        assert torch.equal(gs.dK, dK) and torch.equal(gs.dV, dV)
        assert float((gs.dQ - dQ).abs().max()) <= 1e-4


def test_merge_partial_equals_full():
    """Keys split into two blocks, each attended separately, merged: equals attention over all keys."""
    B, H, Tq, Tk = 2, 2, 200, 384
    Q, K, V = normal((B, H, Tq, 64), 80), normal((B, H, Tk, 64), 81), normal((B, H, Tk, 64), 82)
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, 1, q_pos0=184)
    tQ, tK, tV = dev(Q), dev(K), dev(V)
    O, LSE = hk.attention_forward(tQ, tK[:, :, :256].contiguous(), tV[:, :, :256].contiguous(), SCALE, True, q_pos0=184, k_pos0=0)
    O2, LSE2 = hk.attention_forward(tQ, tK[:, :, 256:].contiguous(), tV[:, :, 256:].contiguous(), SCALE, True, q_pos0=184, k_pos0=256)
    hk.merge_partial(O, LSE, O2, LSE2)
    ok_status()
    gate("O", host(O), O_ref)
    lse_check(host(LSE), L_ref)


@pytest.mark.parametrize("causal", [0, 1])
def test_chained_forward_over_key_blocks_equals_full(causal):
    """HK_FLAG_CONTINUE_SOFTMAX_STATE: keys split into three blocks, attended one after the other into the same O and
    LSE (the previous result is the starting state): equals attention over all keys; the order of the blocks does not
    matter, and a block no query can see (causal, q_pos0 < k_pos0) leaves the result untouched."""
    B, H, Tq, Tk = 2, 3, 300, 640
    q_pos0 = 200 if causal else 0
    Q, K, V = normal((B, H, Tq, 64), 83), normal((B, H, Tk, 64), 84), normal((B, H, Tk, 64), 85)
    O_ref, L_ref = ol.attn_forward_mt(Q, K, V, SCALE, causal, q_pos0=q_pos0)
    tQ, tK, tV = dev(Q), dev(K), dev(V)
    cuts = [(0, 256), (256, 512), (512, 640)]
    for order in ([0, 1, 2], [2, 0, 1]):
        O = torch.full((B, H, Tq, 64), float("nan"), device="cuda")
        LSE = torch.full((B, H, Tq), float("-inf"), device="cuda")
        for bi in order:
            k0, k1 = cuts[bi]
            hk.attention_forward(tQ, tK[:, :, k0:k1].contiguous(), tV[:, :, k0:k1].contiguous(), SCALE, bool(causal),
                                 q_pos0=q_pos0, k_pos0=k0, out=O, lse=LSE, continue_state=True)
        ok_status()
        gate("O", host(O), O_ref)
        lse_check(host(LSE), L_ref)


# ---------------------------------------------------------------------------
# size-independent properties at full BASELINE sizes
# ---------------------------------------------------------------------------
def test_properties_gpt2_small_shape():
    B, H, N = 8, 12, 1024
    g = torch.Generator(device="cuda").manual_seed(9)
    Q, K, dO = (torch.randn((B, H, N, 64), generator=g, device="cuda") for _ in range(3))
    ones = torch.ones((B, H, N, 64), device="cuda")
    # rows of P sum to 1: V = 1 gives O = 1
    O, LSE = hk.attention_forward(Q, K, ones, SCALE, True)
    assert float((O - 1).abs().max()) < 2e-3
    # column sums of dV equal column sums of dO (sum_j dV_j = sum_i (sum_j p_ij) dO_i)
    V = torch.randn((B, H, N, 64), generator=g, device="cuda")
    O, LSE = hk.attention_forward(Q, K, V, SCALE, True)
    dQ, dK, dV, D = hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, True)
    ok_status()
    s_dv, s_do = dV.double().sum(2), dO.double().sum(2)
    assert float((s_dv - s_do).abs().max()) < 5e-2 and float((s_dv - s_do).norm() / s_do.norm()) < 1e-3
    # softmax shift invariance: sum_j dS_ij = 0, so dQ is unchanged by adding a constant vector to every key
    c = torch.randn((1, 1, 1, 64), generator=g, device="cuda")
    O2, LSE2 = hk.attention_forward(Q, K + c, V, SCALE, True)
    dQ2, _, _, _ = hk.attention_backward(Q, K + c, V, O2, dO, LSE2, SCALE, True)
    assert float((dQ2 - dQ).norm() / dQ.norm()) < 3e-3
    # determinism of everything but the atomically accumulated dQ
    dQ3, dK3, dV3, _ = hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, True)
    assert torch.equal(dK3, dK) and torch.equal(dV3, dV)
    assert float((dQ3 - dQ).abs().max()) < 1e-4


def test_long_sequence_rows_against_oracle():
    """Long-sequence shape (N = 32768, every 64th key x8), 2 heads: the last 128 query rows, and the gradients of a
    key block, against the oracle evaluated on just those rows / that block (position-addressed oracle)."""
    H, N = 2, 32768
    g = torch.Generator(device="cuda").manual_seed(11)
    Q, K, V, dO = (torch.randn((1, H, N, 64), generator=g, device="cuda") for _ in range(4))
    K[:, :, ::64] *= 8.0
    O, LSE = hk.attention_forward(Q, K, V, SCALE, True)
    dQ, dK, dV, D = hk.attention_backward(Q, K, V, O, dO, LSE, SCALE, True)
    ok_status()
    r0 = N - 128
    O_ref, L_ref = ol.attn_forward_mt(host(Q[:, :, r0:]), host(K), host(V), SCALE, 1, q_pos0=r0)
    # |scores| reach ~60 with the x8 keys: the TF32 product error scales with it (the reference kernel's does too)
    assert ol.rel_l2(host(O[:, :, r0:]), O_ref) <= 3e-3
    assert ol.max_abs(host(LSE[:, :, r0:]), L_ref) <= 2e-2
    # dQ of those rows: needs every key
    _, dQ_ref, _, _ = ol.attn_backward_mt(host(Q[:, :, r0:]), host(K), host(V), host(O[:, :, r0:]), host(dO[:, :, r0:]),
                                          host(LSE[:, :, r0:]), SCALE, 1, q_pos0=r0)
    assert ol.rel_l2(host(dQ[:, :, r0:]), dQ_ref) <= 5e-3
    # dK, dV of key block [k0, k0+128): needs every query at or after k0
    k0 = N - 2048
    _, _, dK_ref, dV_ref = ol.attn_backward_mt(host(Q[:, :, k0:]), host(K[:, :, k0:k0 + 128]), host(V[:, :, k0:k0 + 128]),
                                               host(O[:, :, k0:]), host(dO[:, :, k0:]), host(LSE[:, :, k0:]), SCALE, 1,
                                               q_pos0=k0, k_pos0=k0)
    assert ol.rel_l2(host(dK[:, :, k0:k0 + 128]), dK_ref) <= 5e-3
    assert ol.rel_l2(host(dV[:, :, k0:k0 + 128]), dV_ref) <= 5e-3


# ---------------------------------------------------------------------------
# failure detection: a wait that cannot complete ends by itself and is reported
# ---------------------------------------------------------------------------
def test_bounded_wait_reports_timeout_and_context_survives():
    """Self-test case 3 waits on an mbarrier nothing arrives at.  No fault, no trap: the wait gives up after its
    limit (2 s), the kernel frees its tensor memory and returns, the status word says so once, and the next
    kernels run normally."""
    import time

    L = hk.lib()
    z = torch.zeros(128 * 128, device="cuda")
    t0 = time.time()
    assert L.hk_attn_selftest(3, z.data_ptr(), z.data_ptr(), z.data_ptr(), None) == 0
    assert hk.last_device_status() == -8  # HK_ERR_DEVICE_TIMEOUT (synchronises)
    assert 1.5 < time.time() - t0 < 10.0
    assert hk.last_device_status() == 0  # reported once, then cleared
    Q, K, V = (dev(normal((1, 2, 256, 64), 300 + s)) for s in range(3))
    O, LSE = hk.attention_forward(Q, K, V, SCALE, True)
    ok_status()
    O_ref, _ = ol.attn_forward_mt(host(Q), host(K), host(V), SCALE, 1)
    gate("O", host(O), O_ref)


@pytest.mark.parametrize("Tq,Tk,causal", [(1, 128, 1), (2, 129, 1), (1, 1000, 0), (2, 2047, 1), (3, 300, 1), (1, 4100, 1)])
def test_few_queries_against_a_cache(Tq, Tk, causal):
    """One or two query rows run in the decode kernel, three in the tensor-core one: run boundaries of the key splits,
    keys that only the last row sees, rows that see no key (k_pos0 beyond them)."""
    B, H = 2, 3
    q = normal((B, H, Tq, 64), 930)
    k, v = normal((B, H, Tk, 64), 931), normal((B, H, Tk, 64), 932)
    for q_pos0, k_pos0 in ((Tk - Tq, 0), (Tk // 2, 0), (5, 6)) if causal else ((0, 0),):
        O_ref, L_ref = ol.attn_forward_mt(q, k, v, SCALE, causal, q_pos0=q_pos0, k_pos0=k_pos0)
        O, LSE = hk.attention_forward(dev(q), dev(k), dev(v), SCALE, causal, q_pos0=q_pos0, k_pos0=k_pos0)
        ok_status()
        gate("O", host(O), O_ref)
        L, seen = host(LSE), np.isfinite(L_ref)
        assert np.array_equal(np.isfinite(L), seen) and (not seen.any() or np.abs(L[seen] - L_ref[seen]).max() <= 2e-3)


@pytest.mark.parametrize("BH,Tq,Tk,causal", [
    (1, 3, 641, 0), (12, 3, 640, 1), (6, 129, 650, 0), (12, 129, 640, 1), (16, 257, 1000, 0), (24, 3, 700, 1),
    (24, 257, 1000, 1), (48, 3, 4200, 0), (24, 3, 8193, 1)])
def test_key_splits_of_short_query_blocks(BH, Tq, Tk, causal):
    """Few queries against many keys: 2, 4, 8 key splits of one and of two blocks of 128 rows, and the even / odd key tiles
    of one block, each plain, with the Philox mask and continued from the state of the first keys."""
    q, k, v = normal((1, BH, Tq, 64), 940), normal((1, BH, Tk, 64), 941), normal((1, BH, Tk, 64), 942)
    pos, cut = (Tk - Tq if causal else 0), 136  # the second part starts inside a key tile
    tq, tk, tv = dev(q), dev(k), dev(v)
    mask = ol.dropout_mask(BH, Tq, Tk, 0.25, 99, 7, q_pos0=pos)
    for kw, m in (({}, None), (dict(dropout_p=0.25, philox_seed=99, philox_offset=7), mask)):
        O_ref, L_ref = ol.attn_forward_mt(q, k, v, SCALE, causal, m, q_pos0=pos)
        O, LSE = hk.attention_forward(tq, tk, tv, SCALE, bool(causal), q_pos0=pos, **kw)
        ok_status()
        gate("O", host(O), O_ref)
        lse_check(host(LSE), L_ref)
        O, LSE = hk.attention_forward(tq, tk[:, :, :cut], tv[:, :, :cut], SCALE, bool(causal), q_pos0=pos, **kw)
        hk.attention_forward(tq, tk[:, :, cut:], tv[:, :, cut:], SCALE, bool(causal), q_pos0=pos, k_pos0=cut, out=O, lse=LSE,
                             continue_state=True, **kw)
        ok_status()
        gate("O", host(O), O_ref)
        lse_check(host(LSE), L_ref)


@pytest.mark.parametrize("BH,Tq,Tk,causal", [(1, 257, 128, 0), (8, 1024, 129, 0), (1, 4000, 40, 0), (24, 777, 333, 0), (2, 1281, 300, 1)])
def test_query_splits_of_few_key_tiles(BH, Tq, Tk, causal):
    """Many queries against few keys: 2, 4, 8 CTAs share the query tiles of a KV tile, splits without a tile of their own,
    key tiles (causal, k_pos0) that few or no queries see; plain, with the Philox mask, into accumulated dK and dV."""
    q, k, v, g = normal((1, BH, Tq, 64), 950), normal((1, BH, Tk, 64), 951), normal((1, BH, Tk, 64), 952), normal((1, BH, Tq, 64), 953)
    k_pos0 = Tq - 200 if causal else 0
    mask = ol.dropout_mask(BH, Tq, Tk, 0.25, 99, 7, k_pos0=k_pos0 // 8 * 8)
    for kw, m in (({}, None), (dict(dropout_p=0.25, philox_seed=99, philox_offset=7), mask)):
        kp = k_pos0 // 8 * 8
        O_ref, L_ref = ol.attn_forward_mt(q, k, v, SCALE, causal, m, k_pos0=kp)
        _, dQ_ref, dK_ref, dV_ref = ol.attn_backward_mt(q, k, v, O_ref, g, L_ref, SCALE, causal, m, k_pos0=kp)
        args = (dev(q), dev(k), dev(v), dev(O_ref), dev(g), dev(L_ref), SCALE, bool(causal))
        dQ, dK, dV, _ = hk.attention_backward(*args, k_pos0=kp, **kw)
        ok_status()
        for name, got, ref in (("dQ", dQ, dQ_ref), ("dK", dK, dK_ref), ("dV", dV, dV_ref)):
            gate(name, host(got), ref)
        dK2, dV2 = dK.clone(), dV.clone()
        hk.attention_backward(*args, k_pos0=kp, dK=dK2, dV=dV2, accum_dkdv=True, **kw)
        ok_status()
        assert torch.equal(dK2, dK + dK) and torch.equal(dV2, dV + dV)
