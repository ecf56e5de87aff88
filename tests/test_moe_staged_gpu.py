"""The per-pair MoE op with staged weight rows: bit-identical to the one-warp-per-row kernel (option moe_smem = 0) at the edges of
its 128-row tiles and row pairs, for rows that start 2, 4 .. 14 bytes past a 16-byte boundary, at the tensor's end, and with rows
too long to stage."""
import numpy as np
import pytest
import torch

from kaillm_b200 import capi
from oracle import gguf_oracle as O
from tests.gpu_util import act, dev
from tests.test_moe_gpu import experts_wire, routing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qt", O.ALL_QTYPES)
@pytest.mark.parametrize("n,k", [(1, 256), (2, 512), (127, 256), (129, 1024), (131, 2304), (9, 8192)])
def test_same_bits_as_the_unstaged_kernel(qt, n, k):
    e, tokens, top_k = 3, 5, 2
    _, w = experts_wire(qt, e, n, k, seed=qt + n)
    _, x = act(tokens, k, seed=k, dt="bf16")
    ids = routing(tokens, top_k, e, seed=n)
    ids[1, 1] = e                                    # no such expert: the row keeps its zeros
    idt = torch.from_numpy(ids.astype(np.int32)).to(dev())
    got = capi.moe_a8_vec(w, x, idt, qt, out_dtype=torch.float32)
    capi.set_option("moe_smem", 0)
    try:
        want = capi.moe_a8_vec(w, x, idt, qt, out_dtype=torch.float32)
    finally:
        capi.set_option("moe_smem", 1)
    assert torch.equal(got, want) and not bool(got[3].any())


@pytest.mark.parametrize("qt", O.ALL_QTYPES)
@pytest.mark.parametrize("n,k,tokens", [(1, 256, 2), (63, 512, 3), (65, 1024, 3), (129, 2304, 5), (200, 256, 310)])
def test_forced_staging_has_the_same_bits(qt, n, k, tokens):
    """Edges of the 64-row tiles (128-row ones from 592 tiles on: the last shape), whatever the dispatch would choose."""
    e, top_k = 3, 1
    _, w = experts_wire(qt, e, n, k, seed=qt + n)
    _, x = act(tokens, k, seed=k, dt="bf16")
    idt = torch.from_numpy(routing(tokens, top_k, e, seed=n).astype(np.int32)).to(dev())
    out = []
    for mode in (0, 1, 2):
        capi.set_option("moe_smem", mode)
        try:
            out.append(capi.moe_a8_vec(w, x, idt, qt, out_dtype=torch.float32))
        finally:
            capi.set_option("moe_smem", 1)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
