"""The integer GEMM (many tokens, formats without a tcgen05 GEMM; expert-sorted blocks) at the edges of its tiles: 64 and
128-row tiles, 64-token tiles, half columns of 128 weights, a K that ends inside a column, rows whose copy windows end with
the tensor, runs of one expert longer than an item."""
import numpy as np
import pytest
import torch

from kaillm_b200 import capi, synth
from oracle import gguf_oracle as O
from tests.gpu_util import act, dev, rel_l2, to_np, wire
from tests.test_moe_gpu import align, expected, experts_wire

pytestmark = pytest.mark.gpu
# Same exact integers and scales as the oracle; fp32 sums of at most K / 16 = 352 terms in another order: 352 * 2^-24 = 2.1e-5
TIGHT = 2.1e-5
MORE_32 = [t for t in O.MORE_QTYPES if synth.BLOCK[t][0] == 32]


@pytest.mark.parametrize("qt", O.MORE_QTYPES)
@pytest.mark.parametrize("mmq", [False, True])
@pytest.mark.parametrize("n,k,m", [(1, 256, 9), (63, 256, 64), (65, 768, 65), (129, 512, 17), (257, 5632, 130)])
def test_matches_oracle(qt, mmq, n, k, m):
    if mmq and qt in O.NO_MMQ:
        pytest.skip("no MMQ flavour")
    w, wt = wire(qt, n, k, seed=qt + n)
    x, xt = act(m, k, seed=m, dt="bf16")
    capi.set_option("mmq_min_m", 9)
    try:
        y = capi.mul_mat(wt, xt, qt, mmq=mmq, out_dtype=torch.float32)
    finally:
        capi.set_option("mmq_min_m", 0)
    assert rel_l2(to_np(y), O.mul_mat(w, qt, x, "mmq" if mmq else "mmvq")) < TIGHT


@pytest.mark.parametrize("qt", MORE_32)
@pytest.mark.parametrize("k", [32, 96, 160, 288])
def test_k_ends_inside_a_column(qt, k):
    n, m = 70, 33
    w, wt = wire(qt, n, k, seed=qt + k)
    x, xt = act(m, k, seed=k, dt="f16")
    capi.set_option("mmq_min_m", 9)
    try:
        y = capi.mul_mat(wt, xt, qt, out_dtype=torch.float32)
    finally:
        capi.set_option("mmq_min_m", 0)
    assert rel_l2(to_np(y), O.mul_mat(w, qt, x, "mmvq")) < TIGHT


def test_large_grid_takes_128_row_tiles():
    qt, n, k, m = 13, 15000, 256, 190          # 118 row tiles x 3 token tiles
    w, wt = wire(qt, n, k, seed=1)
    x, xt = act(m, k, seed=2, dt="bf16")
    y = capi.mul_mat(wt, xt, qt, mmq=True, out_dtype=torch.float32)
    assert rel_l2(to_np(y), O.mul_mat(w, qt, x, "mmq")) < TIGHT


@pytest.mark.parametrize("qt", [q for q in O.ALL_QTYPES if q not in O.NO_MMQ])
@pytest.mark.parametrize("e,n,tokens,top_k,one", [(5, 130, 40, 2, False), (3, 64, 150, 1, True)])
def test_expert_runs(qt, e, n, tokens, top_k, one):
    """Runs of 1 to 19 blocks; `one`: every token goes to the same expert, the others have no block."""
    k = 512
    w, wt = experts_wire(qt, e, n, k, seed=qt)
    x, xt = act(tokens, k, seed=tokens, dt="bf16")
    rng = np.random.default_rng(qt)
    ids = np.full((tokens, 1), 1, np.int32) if one else np.stack([rng.choice(e, size=top_k, replace=False, p=[.5, .2, .1, .1, .1])
                                                                  for _ in range(tokens)]).astype(np.int32)
    s, ex, tot = (torch.from_numpy(a).to(dev()) for a in align(ids, 8, e))
    y = capi.moe_a8(wt, xt, s, ex, tot, top_k, qt, out_dtype=torch.float32)
    assert rel_l2(to_np(y), expected(w, qt, x, ids, "mmq")) < TIGHT


def one_run(tokens):
    """Sorted blocks of one expert's run: tokens 0 .. tokens - 1."""
    s = np.full((tokens + 7) // 8 * 8, tokens, np.int32)
    s[:tokens] = np.arange(tokens)
    return [torch.from_numpy(a).to(dev()) for a in (s, np.zeros(s.size // 8, np.int32), np.array([s.size], np.int32))]


@pytest.mark.parametrize("qt", O.ALL_QTYPES)
@pytest.mark.parametrize("k", [256, 512, 5632])
def test_fp32_error_is_not_above_the_kernels_it_stands_for(qt, k):
    """Against the exact value, in fp32: the GEMV passes (formats without a tcgen05 GEMM) and the one-warp-per-row block op add a
    row in 32 lanes and a tree.  3840 outputs: the two errors are known to about 1.1 %, so 5 % is three deviations of their ratio."""
    n, m = 96, 40
    w, wt = wire(qt, n, k, seed=qt + k)
    x, xt = act(m, k, seed=k, dt="bf16")

    def linear(new):
        capi.set_option("mmq_min_m", 9 if new else 1 << 30)
        try:
            return capi.mul_mat(wt, xt, qt, mmq=qt not in O.NO_MMQ, out_dtype=torch.float32)
        finally:
            capi.set_option("mmq_min_m", 0)

    def sorted_op(new):
        capi.set_option("moe_smem", int(new))
        try:
            return capi.moe_a8(wt.view(1, n, -1), xt, *one_run(m), 1, qt, out_dtype=torch.float32)
        finally:
            capi.set_option("moe_smem", 1)

    ref = O.mul_mat(w, qt, x, "mmvq" if qt in O.NO_MMQ else "mmq")
    for call in ([linear] if qt in O.MORE_QTYPES else []) + ([sorted_op] if qt not in O.NO_MMQ else []):
        old, new = rel_l2(to_np(call(False)), ref), rel_l2(to_np(call(True)), ref)
        assert new <= 1.05 * old, (call.__name__, old, new)


@pytest.mark.parametrize("n,k,m,launches", [(2048, 5120, 89, 12), (2048, 1024, 89, 1), (2048, 5120, 112, 1), (8192, 5120, 33, 5), (8192, 5120, 40, 1)])
def test_dispatch_looks_at_k(n, k, m, launches):
    """Long rows of few-row matrices keep the GEMV passes (8 tokens each, then 4, 2, 1) longer: launches beside the quantizer's."""
    qt = 13
    _, wt = wire(qt, n, k, seed=1)
    _, xt = act(m, k, seed=2, dt="bf16")
    capi.mul_mat(wt, xt, qt, mmq=True)
    before = capi.get_option("launch_count")
    capi.mul_mat(wt, xt, qt, mmq=True)
    assert capi.get_option("launch_count") - before == launches + 1
