"""The status readers synchronise with the whole device: work on a non-blocking side stream has ended when they return."""
import pytest
import torch

from kaillm_b200 import capi
from tests.gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["dequant_mul_mat", "arrival", "scratch", "static"])
def test_reader_waits_for_side_streams(which):
    scratch = torch.zeros(capi.workspace_bytes(12, 1, 64, 256), dtype=torch.uint8, device=dev())
    status = capi.ctypes.c_int(7)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                # about ten milliseconds
        done = torch.cuda.Event()
        done.record()
    if which == "dequant_mul_mat":
        assert capi.lib.kq_dequant_mul_mat_status(capi.ctypes.byref(status), 0) == 0 and status.value == 0
    elif which == "arrival":
        assert capi.arrival_status() == 0
    elif which == "scratch":
        assert capi.read_status(12, 1, 64, 256, scratch) == 0
    else:
        assert capi.read_status_static() == 0
    assert done.query()
