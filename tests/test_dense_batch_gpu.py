"""Dense reconstruction of a block-diagonal handle: entries outside every
stored block are exact zeros, whatever the output buffer held before."""

import ctypes as C

import numpy as np
import pytest

from conftest import golden
from qhmat_gb300 import HMatrix, load_library
from qhmat_gb300._lib import raise_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("names", [["cuda10", "ragged300"], ["tiny2", "cfg1", "tiny2"]])
def test_off_diagonal_blocks_are_zero(cuda_device, names):
    import torch

    lib = load_library()
    images = [golden(name)[0] for name in names]
    bufs = [C.create_string_buffer(b, len(b)) for b in images]
    ptrs = (C.c_void_p * len(images))(*[C.addressof(b) for b in bufs])
    lens = (C.c_size_t * len(images))(*[len(b) for b in images])
    offs = (C.c_uint64 * len(images))()
    h = C.c_void_p()
    raise_for(lib.qh_matrix_from_batch(ptrs, lens, len(images), cuda_device, C.byref(h), offs))
    try:
        parts = [HMatrix.from_bytes(b).to_dense() for b in images]
        n = sum(len(p) for p in parts)
        expect = np.zeros((n, n))
        for o, p in zip(offs, parts):
            expect[o:o + len(p), o:o + len(p)] = p
        out = np.full((n, n), np.nan)
        raise_for(lib.qh_matrix_reconstruct(h, out.ctypes.data, out.size, 0))
        np.testing.assert_array_equal(out, expect)
        dev = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        raise_for(lib.qh_matrix_reconstruct(h, dev.data_ptr(), dev.numel(), 1))
        np.testing.assert_array_equal(dev.cpu().numpy(), expect)
    finally:
        lib.qh_matrix_destroy(h)
