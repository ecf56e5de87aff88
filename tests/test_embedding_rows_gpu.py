"""The embedding op at row lengths around its 256-thread chunks, against the C ABI and the whole dequantized table."""
import pytest
import torch

from kaillm_b200 import capi, linear
from tests.gpu_util import dev, wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qt", [2, 12, 13, 14, 21])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("k,shape", [(256, (1,)), (2304, (3, 5)), (4096, (700,)), (512, (0,))])
def test_embedding_rows(qt, dt, k, shape):
    n = 50
    _, w = wire(qt, n, k, seed=qt)
    ids = torch.randint(0, n, shape, device=dev())
    if ids.numel() > 2:
        ids.view(-1)[1] = n                       # outside the table: zeros
    got = linear.apply_gguf_embedding(ids, w, qt, k, dt)
    assert got.shape == (*shape, k) and torch.equal(got, capi.dequantize_rows(w, qt, k, ids, dt, qt in (12, 13, 14)))
    if qt in (2, 21) and ids.numel():
        full = capi.dequantize(w, qt, n * k, dt).view(n, k)
        flat = ids.view(-1)
        want = torch.where((flat < n)[:, None], full[flat.clamp(max=n - 1)], torch.zeros((), dtype=dt, device=dev()))
        assert torch.equal(got.view(-1, k), want)
    assert torch.equal(linear.apply_gguf_embedding(ids.to(torch.int32), w, qt, k, dt), got)
