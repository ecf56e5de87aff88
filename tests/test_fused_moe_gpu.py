"""The whole feed-forward as one call against the chain of ops it stands for (a differentiated input keeps that chain)."""
import numpy as np
import pytest
import torch

from kaillm_b200 import capi, linear, ops
from tests.gpu_util import TDT, act, dev
from tests.test_moe_gpu import experts_wire, routing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total,e,seed", [(1, 1, 0), (31, 3, 1), (1024, 32, 2), (1000, 60, 3), (8192, 1024, 4), (96, 256, 5)])
def test_align_kernel_equals_the_torch_ops(total, e, seed):
    rng = np.random.default_rng(seed)
    ids = torch.from_numpy(rng.integers(0, max(1, e - 1), size=(total, 1)).astype(np.int32)).to(dev())
    s, ex, tot = linear.moe_align_block_size(ids, 8, e)
    gs, gex, post = torch.empty_like(s), torch.empty_like(ex), torch.empty(2, dtype=torch.int32, device=dev())
    rc = capi.lib.kq_moe_align
    P, L = capi.ctypes.c_void_p, capi.ctypes.c_int64
    assert rc(P(ids.data_ptr()), L(total), L(e), P(gs.data_ptr()), L(gs.numel()), P(gex.data_ptr()), L(gex.numel()), P(post.data_ptr()),
              P(torch.cuda.current_stream().cuda_stream)) == 0
    assert torch.equal(gs, s) and torch.equal(gex, ex) and post.tolist() == [int(tot), 0]


@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("t1,t2,tokens,top_k,e", [(12, 8, 1, 1, 3), (8, 14, 7, 3, 5), (12, 8, 64, 2, 8), (10, 6, 65, 2, 8), (12, 12, 100, 6, 9),
                                                  (21, 20, 80, 2, 4)])
def test_one_call_equals_the_chain(dt, t1, t2, tokens, top_k, e):
    hidden, inter = 512, 256
    _, w1 = experts_wire(t1, e, 2 * inter, hidden, seed=t1)
    _, w2 = experts_wire(t2, e, 200, inter, seed=t2)
    _, x = act(tokens, hidden, seed=tokens, dt=dt)
    x = x * 0.004                                    # the output grows as x^2: keeps the fp16 chain itself finite (2^16 at 0.02)
    ids = torch.from_numpy(routing(tokens, top_k, e, seed=e)).to(dev())
    tw = torch.rand((tokens, top_k), device=dev())
    with torch.no_grad():
        got = linear.fused_moe_gguf(x, w1, w2, tw, ids.to(torch.int64), t1, t2)
    chain = linear.fused_moe_gguf(x.clone().requires_grad_(), w1, w2, tw, ids, t1, t2).detach()
    assert got.dtype == TDT[dt] and bool(torch.isfinite(chain).all())
    # same kernels and roundings up to the fp32 sum over top_k <= 6 products: one rounding of the output type apart
    tol = {"f32": 6 * 2.0 ** -24, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dt]
    assert float((got.double() - chain.double()).norm() / chain.double().norm()) <= tol


def test_invalid_expert_ids():
    e, hidden, inter, top_k = 3, 256, 256, 2
    _, w1 = experts_wire(12, e, 2 * inter, hidden, seed=1)
    _, w2 = experts_wire(8, e, 64, inter, seed=2)
    for tokens in (5, 70):
        _, x = act(tokens, hidden, seed=3, dt="bf16")
        ids = torch.from_numpy(routing(tokens, top_k, e, seed=4)).to(dev())
        ids[2, 1] = -1
        tw = torch.rand((tokens, top_k), device=dev())
        if tokens > 64:                              # the expert-sorted branch refuses them
            with pytest.raises(RuntimeError):
                linear.fused_moe_gguf(x, w1, w2, tw, ids, 12, 8)
        else:                                        # the per-pair branch counts them as nothing
            got = linear.fused_moe_gguf(x, w1, w2, tw, ids, 12, 8)
            only = linear.fused_moe_gguf(x[2:3], w1, w2, tw[2:3, :1].contiguous(), ids[2:3, :1].contiguous(), 12, 8)
            assert torch.equal(got[2:3], only)
    assert ops.ggml_moe_get_block_size(12) == 8


@pytest.mark.parametrize("total,e,kind", [(8192, 2, "one"), (33, 7, "bad"), (5000, 1000, "bad"), (1025, 33, "skewed")])
def test_align_kernel_order_and_invalid_ids(total, e, kind):
    """Against the definition: slots of an expert in slot order, runs padded to 8, invalid ids in no run and flagged."""
    rng = np.random.default_rng(total)
    ids = np.full(total, 1) if kind == "one" else rng.integers(0, e, size=total)
    if kind == "skewed":
        ids = np.minimum(ids, rng.integers(0, e, size=total))
    if kind == "bad":
        ids[::5] = rng.choice([-1, e, 2 ** 31 - 1, -2 ** 31], size=ids[::5].size)
    nb = (total + e * 7 + 7) // 8
    want_s, want_e = [], []
    for ex in range(e):
        z = np.nonzero(ids == ex)[0]
        pad = -z.size % 8
        want_s += list(z) + [total] * pad
        want_e += [ex] * ((z.size + pad) // 8)
    post_want = len(want_s)
    want_s += [total] * (8 * nb - len(want_s))
    want_e += [-1] * (nb - len(want_e))
    it = torch.from_numpy(ids.astype(np.int32)).to(dev())
    s, ex, post = (torch.empty(n, dtype=torch.int32, device=dev()) for n in (8 * nb, nb, 2))
    P, L = capi.ctypes.c_void_p, capi.ctypes.c_int64
    assert capi.lib.kq_moe_align(P(it.data_ptr()), L(total), L(e), P(s.data_ptr()), L(8 * nb), P(ex.data_ptr()), L(nb), P(post.data_ptr()),
                                 P(torch.cuda.current_stream().cuda_stream)) == 0
    assert s.tolist() == want_s and ex.tolist() == want_e and post.tolist() == [post_want, int(kind == "bad")]
