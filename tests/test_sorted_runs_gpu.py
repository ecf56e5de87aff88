"""The expert-sorted op beyond one scan step, one item per CTA and one alignment of the weights: long runs that cross the scan's 32-block
steps, more items than CTA groups, a K that ends inside a column, weights off the 16-byte grid, a side stream."""
import numpy as np
import pytest
import torch

from kaillm_b200 import capi, linear
from oracle import gguf_oracle as O
from tests.gpu_util import act, dev, rel_l2, to_np, wire
from tests.test_moe_gpu import align, experts_wire

pytestmark = pytest.mark.gpu
TIGHT = 2.1e-5      # as tests/test_int_gemm_gpu.py: at most K / 16 = 352 fp32 terms in another order


def by_expert(w, qt, x, ids):
    """Oracle rows of every (token, expert) pair, an expert at a time."""
    flat = ids.reshape(-1)
    out = np.zeros((flat.size, w.shape[1]), np.float32)
    for ex in range(w.shape[0]):
        z = np.nonzero(flat == ex)[0]
        if z.size:
            out[z] = O.mul_mat(w[ex], qt, x[z // ids.shape[1]], "mmq")
    return out


def sorted_op(wt, xt, ids, qt, moe_smem=1):
    s, ex, tot = (torch.from_numpy(a).to(dev()) for a in align(ids, 8, wt.shape[0]))
    capi.set_option("moe_smem", moe_smem)
    try:
        return capi.moe_a8(wt, xt, s, ex, tot, ids.shape[1], qt, out_dtype=torch.float32)
    finally:
        capi.set_option("moe_smem", 1)


@pytest.mark.parametrize("qt,k,n", [(8, 1408, 33), (6, 96, 65), (12, 256, 40), (14, 512, 7)])
@pytest.mark.parametrize("moe_smem", [0, 1])
def test_runs_cross_the_scan_steps(qt, k, n, moe_smem):
    e, tokens = 5, 700                               # about 90 blocks: runs of 10, 50, 0, 25 and 3
    w, wt = experts_wire(qt, e, n, k, seed=qt)
    x, xt = act(tokens, k, seed=k, dt="bf16")
    ids = np.repeat(np.array([0, 1, 3, 4], np.int32), [80, 396, 200, 24]).reshape(-1, 1)
    np.random.default_rng(0).shuffle(ids)
    assert rel_l2(to_np(sorted_op(wt, xt, ids, qt, moe_smem)), by_expert(w, qt, x, ids)) < TIGHT


def test_more_items_than_groups():
    qt, e, n, k, tokens = 8, 3, 16400, 64, 900       # 129 row tiles leave ten groups of CTAs for about fifteen items
    _, wt = experts_wire(qt, e, n, k, seed=1)
    _, xt = act(tokens, k, seed=2, dt="bf16")
    ids = np.random.default_rng(3).integers(0, e, size=(tokens, 1)).astype(np.int32)
    assert rel_l2(to_np(sorted_op(wt, xt, ids, qt)), to_np(sorted_op(wt, xt, ids, qt, 0))) < TIGHT


@pytest.mark.parametrize("qt,off", [(8, 2), (8, 14), (14, 6), (12, 4), (10, 12)])
def test_weights_off_the_16_byte_grid(qt, off):
    e, n, k, tokens = 3, 70, 512, 100
    w, wt = experts_wire(qt, e, n, k, seed=qt)
    x, xt = act(tokens, k, seed=off, dt="bf16")
    buf = torch.zeros(wt.numel() + 32, dtype=torch.uint8, device=dev())
    buf[off:off + wt.numel()] = wt.view(-1)
    ids = np.random.default_rng(off).integers(0, e, size=(tokens, 1)).astype(np.int32)
    got = sorted_op(buf[off:off + wt.numel()].view(wt.shape), xt, ids, qt)
    assert rel_l2(to_np(got), by_expert(w, qt, x, ids)) < TIGHT


def test_merged_layer_reaches_the_integer_gemm_with_a_wide_row_stride():
    k, m = 512, 70
    shards = [(wire(13, 8200, k, seed=1)[1], 13), (wire(14, 65, k, seed=2)[1], 14)]
    x = act(m, k, seed=3, dt="f16")[1] * 0.01
    layer = linear.GGUFLinear(shards)
    want = torch.cat([linear.fused_mul_mat_gguf(x, w, t) for w, t in shards], dim=1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = layer.apply(x)
    torch.cuda.current_stream().wait_stream(side)
    # one rounding to f16 and the order of fp32 terms apart, as tests/test_merged_gpu.py
    assert float((got.double() - want.double()).norm() / want.double().norm()) <= 2.0 ** -11 + 2e-5
