"""CPU tests of the calls on torch tensors (csrc/hk_torch.cpp): what they refuse, and that nothing they meet ends the
process.  No call here gets as far as a launch."""
import os
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (what throws, the call): each in a process of its own, which an exception that escapes the native code would end
THROWS = {
    "forward: the current stream of a machine without a device": "hk.attention_forward(x, x, x, 0.125, True)",
    "backward: the same": "hk.attention_backward(x, x, x, x, x, l, 0.125, True)",
    "zero_dq: the same": "att.zero_dq(x)",
    "forward: a tensor without data": "vmap(lambda y: hk.attention_forward(x, y, x, 0.125, True, stream=0))(x[None])",
    "backward: the same ": "vmap(lambda y: hk.attention_backward(x, x, x, x, y, l, 0.125, True, stream=0))(x[None])",
    "zero_dq: the same ": "vmap(lambda y: att.zero_dq(y, 0))(x[None])",
    "forward: no memory for the result": "hk.attention_forward(x.expand(1 << 24, 1 << 24, 64, 64), x, x, 0.125, True, stream=0)",
    "backward: the same  ": "hk.attention_backward(x.expand(1 << 24, 1 << 24, 64, 64), x, x, x, x, l, 0.125, True, stream=0)",
    "forward: a result without the dimensions": "hk.attention_forward(x, x, x, 0.125, True, lse=l[0, 0], stream=0)",
}


@pytest.mark.skipif(torch.cuda.is_available(), reason="host tensors: a kernel must not get them")
@pytest.mark.parametrize("what", THROWS)
def test_exceptions_of_the_native_calls_reach_the_caller(what):
    code = f"""
import torch, hyperkernels_b200 as hk, hyperkernels_b200.attention as att
from torch.func import vmap
x, l = torch.zeros(1, 1, 64, 64), torch.zeros(1, 1, 64)
try:
    {THROWS[what]}
except (RuntimeError, IndexError) as e:
    print("caught", not isinstance(e, hk.HKError))
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "caught True", (r.returncode, r.stdout, r.stderr[-400:])


FORWARD_TENSORS = ["Q", "K", "V", "dropout_mask", "workspace", "out", "lse"]
BACKWARD_TENSORS = ["Q", "K", "V", "O", "dO", "LSE", "dropout_mask", "workspace", "D", "dQ", "dK", "dV"]


@pytest.mark.parametrize("call,name", [("forward", n) for n in FORWARD_TENSORS] + [("backward", n) for n in BACKWARD_TENSORS])
@pytest.mark.parametrize("kind", ["numpy array", "list", "address", "False"])
def test_what_is_no_tensor_is_refused(call, name, kind):
    """A mask that is no tensor must not run without dropout, a buffer that is none must not be left unwritten."""
    import numpy as np

    import hyperkernels_b200 as hk

    x, l = torch.zeros(1, 1, 64, 64), torch.zeros(1, 1, 64)
    wrong = {"numpy array": np.ones((1, 64, 64), np.float32), "list": [1.0], "address": 4096, "False": False}[kind]
    args = dict(Q=x, K=x, V=x) if call == "forward" else dict(Q=x, K=x, V=x, O=x, dO=x, LSE=l)
    args.update(scale=0.125, causal=True, dropout_p=0.1)
    args[name] = wrong
    with pytest.raises(TypeError, match=f"^{name}: expected a tensor"):
        (hk.attention_forward if call == "forward" else hk.attention_backward)(**args)


@pytest.mark.parametrize("name", ["Q", "K", "V", "dO", "LSE"])
def test_none_is_refused_where_a_tensor_is_needed(name):
    import hyperkernels_b200 as hk
    import hyperkernels_b200.attention as att

    x, l = torch.zeros(1, 1, 64, 64), torch.zeros(1, 1, 64)
    args = dict(Q=x, K=x, V=x, O=x, dO=x, LSE=l, scale=0.125, causal=True)
    args[name] = None
    with pytest.raises(TypeError, match=f"^{name}: expected a tensor"):
        hk.attention_backward(**args)
    with pytest.raises(TypeError, match="^dQ: expected a tensor"):
        att.zero_dq(None)


def test_an_offset_without_a_seed_is_not_read():
    """philox_offset=None beside philox_seed=None, as a caller that forwards its own defaults passes them."""
    import hyperkernels_b200 as hk

    x, l = torch.zeros(1, 1, 64, 64), torch.zeros(1, 1, 64)
    # dropout_p = 1 is refused by the library, behind all reading of arguments and in front of any launch
    for call in (lambda **kw: hk.attention_forward(x, x, x, 0.125, True, dropout_p=1.0, stream=0, **kw),
                 lambda **kw: hk.attention_backward(x, x, x, x, x, l, 0.125, True, dropout_p=1.0, stream=0, **kw)):
        with pytest.raises(hk.HKError, match="dropout"):
            call(philox_offset=None)
        with pytest.raises(TypeError):
            call(philox_seed=1, philox_offset=None)


@pytest.mark.parametrize("status,address,dims,strides", [
    (-1, 0, (1, 1, 64), (4096, 4096, 64)), (-2, 4096, (1, 1, 0), (4096, 4096, 64)), (-2, 4096, (0, 1, 64), (4096, 4096, 64)),
    (-2, 4096, (1, 0, 64), (4096, 4096, 64)), (-3, 4100, (1, 1, 64), (4096, 4096, 64)), (-3, 4096, (1, 1, 64), (4096, 4096, 66)),
    (-3, 4096, (2, 1, 64), (4097, 4096, 64)), (-3, 4096, (1, 2, 64), (4096, 4098, 64))])
def test_zero_dq_refuses_what_its_kernel_cannot_write(status, address, dims, strides):
    """No rows (a division by zero on the host), no memory, or rows that are not on 16 bytes (a fault on the device).
    In a process of its own: the unchecked call ended it."""
    code = f"""
import ctypes as C, hyperkernels_b200 as hk
p = hk.MemEfficientBwdParams()
p.dQ = {address} or None
p.B, p.nh, p.T = {dims}
p.dq_strideB, p.dq_strideH, p.dq_strideM = {strides}
print(hk.lib().hk_attn_zero_dq(C.byref(p), None))
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == str(status), (r.returncode, r.stdout, r.stderr[-400:])


@pytest.mark.gpu
def test_no_memory_for_the_result_is_torchs_own_error():
    """torch.OutOfMemoryError, which programs catch to free memory and try again, not a bare RuntimeError."""
    import hyperkernels_b200 as hk

    x = torch.zeros(1, 1, 64, 64, device="cuda")
    with pytest.raises(torch.OutOfMemoryError):
        hk.attention_forward(x.expand(1 << 20, 1 << 10, 64, 64), x, x, 0.125, True)


@pytest.mark.gpu
def test_slabs_of_a_backward_on_another_stream_are_not_handed_on():
    """The slabs of the deterministic dQ are given back when the call returns.  Called with a stream that is not the
    current one and still busy, the kernels write them later: a tensor made meanwhile must not get that memory."""
    import hyperkernels_b200 as hk

    B, H, T = 1, 8, 1000
    g = torch.Generator(device="cuda").manual_seed(5)
    Q, K, V, dO = (torch.randn((B, H, T, 64), generator=g, device="cuda") for _ in range(4))
    O, LSE = hk.attention_forward(Q, K, V, 0.125, True)
    want = hk.attention_backward(Q, K, V, O, dO, LSE, 0.125, True, deterministic_dq=True)
    dQ, dK, dV = (torch.empty_like(Q) for _ in range(3))
    D = torch.empty_like(LSE)
    slab_floats = (T + 127) // 128 * B * H * T * 64 + 64
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)  # about 0.1 s
    hk.attention_backward(Q, K, V, O, dO, LSE, 0.125, True, deterministic_dq=True, dQ=dQ, dK=dK, dV=dV, D=D, stream=side)
    others = [torch.full((slab_floats,), 7.0, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0
    assert all(bool((t == 7.0).all()) for t in others)
    assert torch.equal(dQ, want[0]) and torch.equal(dK, want[1]) and torch.equal(dV, want[2])


@pytest.mark.gpu
@pytest.mark.parametrize("handle", [0, 1, 2])
def test_slabs_under_the_streams_that_have_no_object(handle):
    """0, cudaStreamLegacy and cudaStreamPerThread, as numbers."""
    import hyperkernels_b200 as hk

    g = torch.Generator(device="cuda").manual_seed(6)
    Q, K, V, dO = (torch.randn((1, 2, 300, 64), generator=g, device="cuda") for _ in range(4))
    O, LSE = hk.attention_forward(Q, K, V, 0.125, True)
    want = hk.attention_backward(Q, K, V, O, dO, LSE, 0.125, True, deterministic_dq=True)
    torch.cuda.synchronize()
    got = hk.attention_backward(Q, K, V, O, dO, LSE, 0.125, True, deterministic_dq=True, stream=handle)
    torch.cuda.synchronize()
    assert hk.last_device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(got, want))
