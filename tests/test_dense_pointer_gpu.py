"""to_dense into a pointer that is not pageable host memory although the caller
says host: the copy judges it (an error code or the matrix), the host does not
touch it.  A pinned buffer receives the matrix."""

import numpy as np
import pytest

from qhmat_gb300 import HMatrix

pytestmark = pytest.mark.gpu


@pytest.fixture()
def handle(cuda_device):
    n = 800  # 5.1 MB: large enough for its pages to be populated
    rng = np.random.default_rng(1)
    h = HMatrix.from_arrays(n, rng.permutation(n), [(0, n, 0, n, 0, 0, 0, 1)], rng.standard_normal(n * n),
                            np.zeros(1, np.uint32), np.zeros(1, np.uint32), [], [], [], [], [])
    return h, h.to_dense()


def test_device_pointer_called_host(handle):
    import torch

    h, expect = handle
    out = torch.full(expect.shape, float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = h._lib.qh_matrix_reconstruct(h._h, out.data_ptr(), out.numel(), 0)
    if rc == 0:
        np.testing.assert_array_equal(out.cpu().numpy(), expect)
    np.testing.assert_array_equal(h.to_dense(), expect)


def test_pinned_buffer(handle):
    import torch

    h, expect = handle
    out = torch.full(expect.shape, float("nan"), dtype=torch.float64).pin_memory()
    assert h._lib.qh_matrix_reconstruct(h._h, out.data_ptr(), out.numel(), 0) == 0
    np.testing.assert_array_equal(out.numpy(), expect)
