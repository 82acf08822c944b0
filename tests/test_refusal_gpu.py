"""A checked apply with a bad argument is refused at once, not after the work
that its stream holds, and the next call is right."""

import pytest

from conftest import golden
from qhmat_gb300 import HMatrix, PrecisionHMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cls", [HMatrix, PrecisionHMatrix])
def test_bad_arguments_do_not_wait(cuda_device, cls):
    import torch

    h = cls.from_bytes(golden("cfg1")[0])
    call = h._lib.qh_matmul_device_checked if cls is HMatrix else h._lib.qh_pmatmul_device_checked
    x = torch.ones(h.order, 3, dtype=torch.float64, device="cuda")
    expect = h.matmul(x)
    y = torch.empty_like(x)
    ws = torch.empty(h.workspace_bytes(3) + 256, dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(1_000_000_000)  # half a second
        busy = torch.cuda.Event()
        busy.record()
    a = (h._h, x.data_ptr(), y.data_ptr(), 3, ws.data_ptr(), ws.numel(), s.cuda_stream)
    for at, bad in ((1, None), (2, None), (3, 0), (3, 1 << 62), (4, ws.data_ptr() + 8), (5, 256)):
        args = list(a)
        args[at] = bad
        assert call(*args) in (1, 3), at  # QH_EINVAL, QH_EOVERFLOW
    assert not busy.query()
    assert call(*a) == 0
    assert torch.equal(y, expect)
