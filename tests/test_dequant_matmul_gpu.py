"""`x @ dequantize(W).T` of the i-matrix formats in one kernel: tile edges in rows and tokens, one to many weight columns, the
window of a tensor's last row, and the calls that must keep the two-step path."""
import pytest
import torch

from kaillm_b200 import capi, linear
from tests.gpu_util import act, dev, wire

pytestmark = pytest.mark.gpu
# fp32 accumulation and one rounding of the output: unit roundoff of the type (2^-11, 2^-8) plus k * 2^-24 < 4e-4
BOUND = {"f16": 2.0 ** -11 + 4e-4, "bf16": 2.0 ** -8 + 4e-4}


def want(wt, qt, xt):
    n, k = wt.shape[0], xt.shape[1]
    return xt.double() @ capi.dequantize(wt, qt, n * k, xt.dtype).view(n, k).double().T


def fused(wt, xt, qt):
    (m, k), n = xt.shape, wt.shape[0]
    y = torch.empty((m, n), dtype=xt.dtype, device=xt.device)
    assert capi.lib.kq_dequant_mul_mat(wt.data_ptr(), qt, n, k, xt.data_ptr(), capi._DT[xt.dtype], m, xt.stride(0), y.data_ptr(), n,
                                       torch.cuda.current_stream().cuda_stream) == 0
    return y


def rel(y, ref):
    return float((y.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("qt", [20, 21, 23])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("n,k,m", [(1, 256, 9), (127, 512, 16), (128, 768, 63), (129, 256, 64), (300, 5632, 65), (64, 1024, 128),
                                   (257, 512, 129), (40, 2048, 256), (72, 256, 300)])
def test_matches_dequantize_and_matmul(qt, dt, n, k, m):
    _, wt = wire(qt, n, k, seed=qt + n)
    _, xt = act(m, k, seed=m, dt=dt)
    y = fused(wt, xt, qt)
    assert rel(y, want(wt, qt, xt)) < BOUND[dt]
    status = capi.ctypes.c_int(0)
    assert capi.lib.kq_dequant_mul_mat_status(capi.ctypes.byref(status), 0) == 0 and status.value == 0


def test_exact_on_small_integers():
    """One-hot activations pick single weights: the operand rounding is kq_dequantize's, bit for bit."""
    for qt in (20, 21, 23):
        n, k = 130, 512
        _, wt = wire(qt, n, k, seed=qt)
        for dt in (torch.float16, torch.bfloat16):
            x = torch.eye(k, dtype=dt, device=dev())[3::7][:70].contiguous()
            y = fused(wt, x, qt)
            assert torch.equal(y, capi.dequantize(wt, qt, n * k, dt).view(n, k).T[3::7][:70])


def test_other_forms_keep_the_two_steps():
    qt, n, k, m = 21, 12300, 512, 12
    assert capi.lib.kq_dequant_mul_mat_preferred(n, m) == 1 and capi.lib.kq_dequant_mul_mat_preferred(4096, m) == 0
    _, wt = wire(qt, n, k, seed=3)
    _, big = act(m, 2 * k + 8, seed=4, dt="bf16")
    for x in (big[:, :k], big[:, 1:k + 1], big[:, ::2][:, :k], big.t().contiguous().t()[:, :k], big[:, :k].float().contiguous()):
        y = linear.fused_mul_mat_gguf(x, wt, qt)
        assert y.dtype == x.dtype and rel(y, want(wt, qt, x)) < BOUND["bf16"]
    x = big[:, :k].contiguous()
    assert torch.equal(linear.fused_mul_mat_gguf(x, wt, qt), fused(wt, x, qt))
    x = x.requires_grad_()
    linear.fused_mul_mat_gguf(x, wt, qt).float().sum().backward()
    assert x.grad is not None and bool(x.grad.abs().sum() > 0)
    _, w32 = wire(20, 70, 288, seed=5)                  # K no multiple of 256
    _, x32 = act(33, 288, seed=6, dt="f16")
    assert rel(linear.fused_mul_mat_gguf(x32, w32, 20), want(w32, 20, x32)) < BOUND["f16"]
