"""Under autocast the calls that have an op of their own keep the chain of torch ops, whose result types autocast decides."""
import pytest
import torch

from kaillm_b200 import linear
from tests.gpu_util import act, dev, wire
from tests.test_moe_gpu import experts_wire, routing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [5, 70])
def test_moe(tokens):
    e, hidden, inter, top_k = 4, 256, 256, 2
    _, w1 = experts_wire(12, e, 2 * inter, hidden, seed=1)
    _, w2 = experts_wire(8, e, 64, inter, seed=2)
    _, x = act(tokens, hidden, seed=3, dt="bf16")
    x = x * 0.004
    ids = torch.from_numpy(routing(tokens, top_k, e, seed=4)).to(dev())
    tw = torch.rand((tokens, top_k), device=dev())
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got = linear.fused_moe_gguf(x, w1, w2, tw, ids, 12, 8)
        chain = linear.fused_moe_gguf(x.clone().requires_grad_(), w1, w2, tw, ids, 12, 8)
    assert got.dtype == chain.dtype == torch.float32 and torch.equal(got, chain.detach())


def test_i_matrix_linear():
    qt, n, k, m = 21, 12300, 512, 12                 # sizes at which one kernel does the two steps
    _, w = wire(qt, n, k, seed=3)
    _, x = act(m, k, seed=4, dt="f16")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got = linear.fused_mul_mat_gguf(x * 0.01, w, qt)
    assert got.dtype == torch.bfloat16
    assert linear.fused_mul_mat_gguf(x * 0.01, w, qt).dtype == torch.float16
