"""Applies of several columns whose structure takes them off the usual path:
a long 1-D matrix with small leaves, which stays on the column-by-column kernels
at some column counts and leaves them at others; a row tile whose items have
more than 32 steps (two runs of step descriptors); matrices of different sizes
applied at the same time on streams of their own.  Every column equals its own
one-column apply bit for bit."""

import numpy as np
import pytest

from qhmat_gb300 import HMatrix
from qhmat_gb300.construct import spatial_partition

pytestmark = pytest.mark.gpu


def _matrix(n, perm, blocks, rng):
    """A matrix with the given blocks (row0, row1, col0, col1, rank; 0: dense),
    random codes of 2 .. 32 bits."""
    descs, widths, offs, scales, nd, at = [], [], ([], []), ([], []), 0, [0, 0]
    for r0, r1, c0, c1, rank in blocks:
        if rank == 0:
            descs.append((r0, r1, c0, c1, 0, 0, nd, 1))
            nd += (r1 - r0) * (c1 - c0)
            continue
        descs.append((r0, r1, c0, c1, rank, len(widths), 0, 0))
        for j in range(rank):
            w = (32, 24, 16, 12, 8, 4, 2)[7 * j // rank]
            widths.append(w)
            for side, m in enumerate((r1 - r0, c1 - c0)):
                offs[side].append(at[side])
                scales[side].append(2.0 ** (1 - w))
                at[side] += (m * w + 31) // 32
    words = [rng.integers(0, 1 << 32, k, dtype=np.uint32) for k in at]
    return HMatrix.from_arrays(n, perm, descs, rng.standard_normal(nd), *words, *offs, *scales, widths)


def _points(n, dim, leaf, rank, seed):
    rng = np.random.default_rng(seed)
    perm, rects = spatial_partition(rng.random((n, dim)), leaf)
    blocks = [(*r[:4], 0 if r[:2] == r[2:4] else min(rank, r[1] - r[0], r[3] - r[2])) for r in map(tuple, rects)]
    return _matrix(n, perm, blocks, rng)


def _single(h, x):
    return np.stack([h.matmul(np.ascontiguousarray(x[:, k])) for k in range(x.shape[1])], axis=1)


def _check(h, columns, seed):
    x = np.random.default_rng(seed).standard_normal((h.order, max(columns)))
    one = _single(h, x)
    for p in columns:
        assert np.array_equal(h.matmul(np.ascontiguousarray(x[:, :p])), one[:, :p]), p


def test_long_1d_matrix(cuda_device):
    _check(_points(12001, 1, 16, 6, 1), (2, 3, 4, 5, 8, 9, 17), 2)


def test_row_items_of_more_than_32_steps(cuda_device):
    # 68 blocks of rank 64 beside one tile's rows: 69 k-pairs a split, 35 steps
    n, c = 64 * 69, range(0, 64 * 69, 64)
    rng = np.random.default_rng(3)
    blocks = [(r, r + 64, k, k + 64, 0 if r == k else 64 if r == 0 else 1) for r in c for k in c]
    _check(_matrix(n, rng.permutation(n), blocks, rng), (3, 4, 5, 9, 17), 4)


def test_matrices_at_the_same_time(cuda_device):
    import torch

    jobs = []
    for k, (n, dim, leaf, rank, p) in enumerate([(300, 2, 64, 12, 3), (1000, 2, 64, 14, 8), (2049, 1, 32, 6, 4),
                                                 (3001, 2, 32, 14, 16), (700, 3, 64, 20, 5), (64, 1, 64, 1, 9)]):
        h = _points(n, dim, leaf, rank, 10 + k)
        x = torch.from_numpy(np.random.default_rng(20 + k).standard_normal((n, p))).cuda()
        ws = torch.empty(h.workspace_bytes(p), dtype=torch.uint8, device="cuda")
        jobs.append((h, x, h.matmul(x), ws, torch.cuda.Stream()))
    torch.cuda.synchronize()
    got = [[] for _ in jobs]
    for _ in range(20):
        for k, (h, x, _, ws, s) in enumerate(jobs):
            with torch.cuda.stream(s):
                got[k].append(h.matmul(x, workspace=ws, check=False))
    torch.cuda.synchronize()
    for ys, (_, _, y, _, _) in zip(got, jobs):
        assert all(torch.equal(y, v) for v in ys)
