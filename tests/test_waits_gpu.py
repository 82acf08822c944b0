"""A block of the tensor-memory kernels gives up as a whole: one warp's wait runs
out of its tests, and another warp's, which has tests left, ends because the block
has been told; every lane of both agrees.  Nothing is in flight, and the context
stays usable."""

import pytest

from conftest import golden
from qhmat_gb300 import HMatrix, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [1, 255, 256, 3000])
def test_block_gives_up_as_a_whole(cuda_device, polls):
    lib = _lib.load_library()
    assert lib.qh_debug_wait_timeout(cuda_device, polls) == _lib.QH_ERUNTIME
    assert lib.qh_last_error().decode() == "device copy wait timed out"
    data, g = golden("cfg1")
    assert abs(HMatrix.from_bytes(data).matmul(g["x"]) - g["y"]).max() <= 1e-12 * abs(g["y"]).max()
