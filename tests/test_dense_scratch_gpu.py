"""The scratch of a dense reconstruction: four bytes a factor entry (and a few
megabytes), so that an output that nearly fills the device still fits beside it.
Seen from outside: the device's free memory, polled during a call that computes
for some tens of milliseconds."""

import threading

import numpy as np
import pytest

from qhmat_gb300 import HMatrix

pytestmark = pytest.mark.gpu


def test_four_bytes_a_factor_entry(cuda_device):
    import torch

    n, half, rank, w = 4096, 2048, 2000, 8
    rng = np.random.default_rng(5)
    blocks, nd = [], 0
    for k, (r, c) in enumerate([(0, 0), (0, half), (half, 0), (half, half)]):
        dense = r == c
        blocks.append((r, r + half, c, c + half, 0 if dense else rank, 0 if dense else (k - 1) * rank, nd, int(dense)))
        nd += half * half if dense else 0
    nw = half * w // 32
    offs = [nw * j for j in range(2 * rank)]
    words = [rng.integers(0, 1 << 32, 2 * rank * nw, dtype=np.uint32) for _ in range(2)]
    h = HMatrix.from_arrays(n, np.arange(n), blocks, np.zeros(nd), *words, offs, offs, [1.0] * (2 * rank),
                            [1.0] * (2 * rank), [w] * (2 * rank))
    out = torch.empty(n * n, dtype=torch.float64, device="cuda")
    assert h._lib.qh_matrix_reconstruct(h._h, out.data_ptr(), out.numel(), 1) == 0  # (kernels loaded)
    torch.cuda.synchronize()
    before, least, done = torch.cuda.mem_get_info()[0], [], threading.Event()

    def poll():
        torch.cuda.set_device(0)
        while not done.is_set():
            least.append(torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=poll)
    t.start()
    rc = h._lib.qh_matrix_reconstruct(h._h, out.data_ptr(), out.numel(), 1)
    done.set()
    t.join()
    assert rc == 0
    entries = 2 * rank * 2 * half
    used = before - min(least)
    assert 0 < used <= 4 * entries + (16 << 20), used
