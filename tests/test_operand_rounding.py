"""How the tensor-map loads round the operands: to TF32, to nearest, ties to even, for every map of the two kernels.

Each map is read out through the kernels bit for bit.  With one key and a score of zero the probability is exactly 1, so
O = V and dV = dO; with P = 1, D = 0 and one-hot operands dS, and through it dQ and dK, is a single product of a rounded
value and a power of two.  The scores of the forward are read out through LSE = score * scale, whose own error (a few
2^-24) is far below the 2^-11 between neighbouring TF32 values."""
import numpy as np
import pytest
import torch

import hyperkernels_b200 as hk

pytestmark = pytest.mark.gpu
SCALE = 0.125
BH, D = 64, 64


def _rne(x):
    """fp32 -> TF32 (10 mantissa bits), to nearest, ties to even"""
    b = np.ascontiguousarray(x, np.float32).view(np.uint32)
    return ((b + np.uint32(0xFFF) + ((b >> np.uint32(13)) & np.uint32(1))) & np.uint32(0xFFFFE000)).view(np.float32)


def _values(shape, seed, lo=-20, hi=20):
    """random signs, exponents and mantissas; every fourth a tie, others one ulp beside one, all ones, or exact"""
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    sign = rng.integers(0, 2, n, dtype=np.uint32) << np.uint32(31)
    exponent = rng.integers(127 + lo, 127 + hi, n).astype(np.uint32) << np.uint32(23)
    mantissa = rng.integers(0, 1 << 23, n, dtype=np.uint32)
    top, kind = mantissa & np.uint32(0x7FE000), rng.integers(0, 12, n)
    for k, low in ((0, 0x1000), (1, 0x1000), (2, 0x1000), (3, 0x0FFF), (4, 0x1001), (5, 0)):
        mantissa = np.where(kind == k, top | np.uint32(low), mantissa)
    mantissa = np.where(kind == 6, np.uint32(0x7FFFFF), mantissa)
    return (sign | exponent | mantissa).astype(np.uint32).view(np.float32).reshape(shape)


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _host(t):
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0
    return t.cpu().numpy()


def _hot(rows):
    """[1, BH, rows, 64], in slice j a one in column j of every row"""
    x = np.zeros((1, BH, rows, D), np.float32)
    x[0, np.arange(BH), :, np.arange(BH)] = 1.0
    return x


def _eye():
    """[1, BH, 64, 64], row i a one in column i"""
    return np.broadcast_to(np.eye(D, dtype=np.float32), (1, BH, D, D))


def _backward(Q, K, V, dO):
    """dQ, dK, dV with LSE = 0 (P = 1 where the scores are 0) and D = 0"""
    rows = torch.zeros((1, BH, Q.shape[2]), device="cuda")
    dQ, dK, dV, _ = hk.attention_backward(_dev(Q), _dev(K), _dev(V), None, _dev(dO), rows, SCALE, False, D=rows.clone(),
                                          d_precomputed=True)
    return _host(dQ), _host(dK), _host(dV)


def _same(got, x):
    assert np.array_equal(got.view(np.uint32), _rne(x).view(np.uint32))
    assert not np.array_equal(got, x)


ROWS = 200  # a whole tile and a part of one
ZERO = lambda rows: np.zeros((1, BH, rows, D), np.float32)  # noqa: E731


def test_forward_v():
    V = _values((1, BH, 1, D), 1)
    O, _ = hk.attention_forward(_dev(_values((1, BH, ROWS, D), 2)), _dev(ZERO(1)), _dev(V), SCALE, False)
    for row in (0, 127, 128, ROWS - 1):
        _same(_host(O)[:, :, row], V[:, :, 0])


def test_forward_v_denormals():
    V = np.random.default_rng(12).integers(0, 1 << 23, (1, BH, 1, D), dtype=np.uint32)
    V[0, 0, 0, :6] = [0x1000, 0x3000, 0x0FFF, 0x1001, 0x7FFFFF, 0x2000]
    V = V.view(np.float32)
    O, _ = hk.attention_forward(_dev(ZERO(ROWS)), _dev(ZERO(1)), _dev(V), SCALE, False)
    for row in (0, ROWS - 1):
        _same(_host(O)[:, :, row], V[:, :, 0])


def _from_lse(LSE):
    """the TF32 value nearest to score = LSE / scale"""
    return _rne((_host(LSE).astype(np.float64) / SCALE).astype(np.float32))


def test_forward_q():
    Q = _values((1, BH, ROWS, D), 3)
    _, LSE = hk.attention_forward(_dev(Q), _dev(_hot(1)), _dev(ZERO(1)), SCALE, False)
    _same(_from_lse(LSE), Q[0, np.arange(BH), :, np.arange(BH)][None])


def test_forward_k():
    K = _values((1, BH, 1, D), 4)
    _, LSE = hk.attention_forward(_dev(_eye()), _dev(K), _dev(ZERO(1)), SCALE, False)
    _same(_from_lse(LSE), K[:, :, 0])


def test_backward_do_over_the_queries():
    """dV = P^T dO, one query"""
    dO = _values((1, BH, 1, D), 5)
    _, _, dV = _backward(ZERO(1), ZERO(1), ZERO(1), dO)
    _same(dV, dO)


def test_backward_q_over_the_queries():
    """dK = dS^T Q, one query, dS = scale * (V . dO) = 1"""
    Q, eight = _values((1, BH, 1, D), 6), 8.0 * _hot(1)
    _, dK, _ = _backward(Q, ZERO(1), eight, _hot(1))
    _same(dK, Q)


def test_backward_k_over_the_keys():
    """dQ = dS K, one key, dS = 1"""
    K = _values((1, BH, 1, D), 7)
    dQ, _, _ = _backward(ZERO(ROWS), K, 8.0 * _hot(1), _hot(ROWS))
    for row in (0, 127, 128, ROWS - 1):
        _same(dQ[:, :, row], K[:, :, 0])


def test_backward_v_over_the_columns():
    """dP = V dO^T = V[i] in row i; dQ = scale * dP * 8 in column 0"""
    V, K = _values((1, BH, 1, D), 8), ZERO(1)
    K[..., 0] = 8.0
    dQ, _, _ = _backward(ZERO(D), K, V, _eye())
    _same(np.ascontiguousarray(dQ[..., 0]), V[:, :, 0])


def test_backward_do_over_the_columns():
    dO, K = _values((1, BH, ROWS, D), 9), ZERO(1)
    K[..., 0] = 8.0
    dQ, _, _ = _backward(ZERO(ROWS), K, _hot(1), dO)
    _same(np.ascontiguousarray(dQ[..., 0]), dO[0, np.arange(BH), :, np.arange(BH)][None])


@pytest.mark.parametrize("which", ["Q", "K"])
def test_backward_q_and_k_over_the_columns(which):
    """S = K Q^T: P = 2^(S c - LSE log2e), c = scale * log2e.  Scores between 1 and 2, a scale of 256 and LSE = 256 * the
    rounded score: P is 1 but for the roundings of c and of LSE * log2e (together 2^-23 of an exponent below 740) and its
    own rounding to TF32; a score one unit off (2^-10) would make it 2^+-0.36, half a unit 2^+-0.18."""
    x, hot = _values((1, BH, 1, D), 10, 0, 1), _hot(1)
    picked = x[0, np.arange(BH), 0, np.arange(BH)]
    lse = (256.0 * _rne(picked))[None, :, None]
    Q, K = (x, hot) if which == "Q" else (hot, x)
    _, _, dV, _ = hk.attention_backward(_dev(Q), _dev(K), _dev(ZERO(1)), None, _dev(hot), _dev(lse), 256.0, False,
                                        D=torch.zeros((1, BH, 1), device="cuda"), d_precomputed=True)
    p = _host(dV)[0, np.arange(BH), 0, np.arange(BH)]
    assert np.abs(p - 1.0).max() <= 2.0 ** -11 + 740 * 2.0 ** -23
