"""Applies of several columns whose structure takes them off the usual path:

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
