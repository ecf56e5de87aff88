"""Merged projections of mixed types with one quantization against the calls they stand for."""
import pytest
import torch

from kaillm_b200 import linear
from tests.gpu_util import act, dev, wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types,rows", [((12, 12, 14), (300, 64, 65)), ((13, 8), (40, 24)), ((10, 2, 12), (6000, 33, 1)), ((12, 21), (96, 32))])
@pytest.mark.parametrize("m", [1, 2, 5, 8, 17, 49, 80])
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_merged_equals_the_shards(types, rows, m, dt):
    k = 1024
    ws = [wire(t, n, k, seed=i)[1] for i, (t, n) in enumerate(zip(types, rows))]
    _, x = act(m, k, seed=m, dt=dt)
    x = x * 0.01
    layer = linear.GGUFLinear(list(zip(ws, types)))
    bias = torch.randn(sum(rows), device=dev()).to(x.dtype)
    want = torch.cat([linear.fused_mul_mat_gguf(x, w, t) for w, t in zip(ws, types)], dim=1) + bias
    got = layer.apply(x, bias)
    # the same integer dots; the kernels may add a row's fp32 terms in another order (1-2 tokens) and then round once more
    tol = {"f32": 2e-5, "f16": 2.0 ** -11 + 2e-5, "bf16": 2.0 ** -8 + 2e-5}[dt]
    assert got.dtype == want.dtype and float((got.double() - want.double()).norm() / want.double().norm()) <= tol
    strided = torch.cat([x, x], dim=1)[:, :k]
    assert torch.equal(layer.apply(strided, bias), got)
