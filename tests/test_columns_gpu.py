"""The several-column kernels (three right-hand sides and more) at the sizes
where they can go wrong: tasks of 1 .. 32 components and items of one to four
of them, odd chunk counts, row tiles of 1 .. 4 16-row M-tiles in both row
shapes, every code width (nibble and byte top planes), tasks split along their
columns, and accumulator segments full of the largest digits times the largest
limbs (their FP32 sums have to stay exact).

Every column equals the one-column kernels' result bit for bit, whatever the
number of columns: both sum integers.  (The one-column kernels are compared
with the oracle in test_matvec_gpu.py.)
"""

import numpy as np
import pytest

from qhmat_gb300 import HMatrix
from test_oracle import _pack_codes

pytestmark = pytest.mark.gpu

# (rows of the first cluster, rows of the second, rank, widths)
SHAPES = [
    (33, 31, 1, [2]),
    (17, 18, 16, [3, 32]),
    (64, 64, 33, list(range(2, 33))),
    (48, 257, 40, [8, 9, 12, 13]),
    (100, 97, 97, [4, 5, 16, 17, 20, 24, 25, 28, 29, 32]),
    (130, 705, 130, [7, 14, 21, 32, 2, 31]),
]


def _matrix(a, b, rank, widths, kind, rng):
    """Dense diagonal clusters of a and b rows, off-diagonal blocks of `rank`."""
    n = a + b
    perm = rng.permutation(n)
    rects = [(0, a, 0, a), (0, a, a, n), (a, n, 0, a), (a, n, a, n)]
    blocks, dense, words, offs, scales, ws, nd = [], [], ([], []), ([], []), ([], []), [], 0
    for k, (r0, r1, c0, c1) in enumerate(rects):
        if k in (0, 3):
            d = rng.standard_normal((r1 - r0, c1 - c0)) / n
            blocks.append((r0, r1, c0, c1, 0, 0, nd, 1))
            dense.append(d.ravel())
            nd += d.size
            continue
        blocks.append((r0, r1, c0, c1, rank, len(ws), 0, 0))
        for j in range(rank):
            w = widths[(j + k) % len(widths)]
            ws.append(w)
            for side, m in enumerate((r1 - r0, c1 - c0)):
                if kind == "random":
                    codes = rng.integers(-(1 << (w - 1)) + 1, 1 << (w - 1), m)
                else:  # digits 255 .. 255 and the largest top digit
                    codes = np.full(m, (1 << (w - 1)) - 1)
                # (one component in eight adds nothing)
                s = 0.0 if kind == "random" and j % 8 == 7 and side else float(2.0 ** (1 - w) * (1 + 0.5 * rng.random()))
                p = _pack_codes(codes, w)
                offs[side].append(sum(map(len, words[side])))
                words[side].append(p)
                scales[side].append(s)
    return HMatrix.from_arrays(n, perm, blocks, np.concatenate(dense), np.concatenate(words[0]),
                               np.concatenate(words[1]), offs[0], offs[1], scales[0], scales[1], ws)


def _columns(n, p, kind, rng):
    if kind == "random":
        x = rng.standard_normal((n, p)) * np.exp2(rng.integers(-20, 20, (n, 1)))
        x[:, p // 2] = 0.0
        return x
    # X = x 2^8: limbs 63, 127, 127, .. and -63, -128, -128, ..
    x = np.full((n, p), float(0x3F7F7F7F7F7F7E))
    x[:, 1::2] = -float(0x3F808080808080)
    return x


@pytest.mark.parametrize("kind", ["random", "extreme"])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_columns_equal_single_columns(cuda_device, monkeypatch, shape, kind):
    a, b, rank, widths = SHAPES[shape]
    rng = np.random.default_rng(1000 + shape)
    h = _matrix(a, b, rank, widths, kind, rng)
    x = _columns(h.order, 17, kind, rng)
    one = np.stack([h.matmul(np.ascontiguousarray(x[:, k])) for k in range(17)], axis=1)
    monkeypatch.setenv("QHMAT_GB300_PART_CHUNKS", "1")
    split = _matrix(a, b, rank, widths, kind, np.random.default_rng(1000 + shape))
    for p in (2, 3, 4, 5, 8, 9, 17):
        xp = np.ascontiguousarray(x[:, :p])
        assert np.array_equal(h.matmul(xp), one[:, :p]), p
        assert np.array_equal(split.matmul(xp), one[:, :p]), p
