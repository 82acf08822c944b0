"""to_dense at the edges of its kernels' tiles (32 x 32 entries, 16 components)
and of the page handling (buffers of several megabytes): equal bit for bit to
the reference's loop (factors scaled, then one multiply and one add per
component, in order)."""

import numpy as np
import pytest

from qhmat_gb300 import HMatrix
from test_oracle import _pack_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b,rank", [(1, 1, 1), (31, 33, 15), (32, 64, 16), (33, 65, 17), (100, 90, 33), (700, 801, 49)])
def test_to_dense_tiles(cuda_device, a, b, rank):
    n = a + b
    rng = np.random.default_rng(n)
    perm = rng.permutation(n)
    full = np.zeros((n, n))
    blocks, dense, ws, nd = [], [], [], 0
    words, offs, scales = ([], []), ([], []), ([], [])
    for k, (r0, r1, c0, c1) in enumerate([(0, a, 0, a), (0, a, a, n), (a, n, 0, a), (a, n, a, n)]):
        if k in (0, 3):
            d = rng.standard_normal((r1 - r0, c1 - c0))
            blocks.append((r0, r1, c0, c1, 0, 0, nd, 1))
            dense.append(d.ravel())
            nd += d.size
            full[r0:r1, c0:c1] = d
            continue
        blocks.append((r0, r1, c0, c1, rank, len(ws), 0, 0))
        for j in range(rank):
            w = int(rng.integers(2, 33))
            ws.append(w)
            f = []
            for side, m in enumerate((r1 - r0, c1 - c0)):
                codes = rng.integers(-(1 << (w - 1)) + 1, 1 << (w - 1), m)
                s = float(rng.random())
                offs[side].append(sum(map(len, words[side])))
                words[side].append(_pack_codes(codes, w))
                scales[side].append(s)
                f.append(codes.astype(np.float64) * s)
            full[r0:r1, c0:c1] += np.outer(f[0], f[1])
    h = HMatrix.from_arrays(n, perm, blocks, np.concatenate(dense), np.concatenate(words[0]), np.concatenate(words[1]),
                            offs[0], offs[1], scales[0], scales[1], ws)
    out = np.zeros((n, n))
    out[np.ix_(perm, perm)] = full
    for _ in range(2):
        np.testing.assert_array_equal(h.to_dense(), out)
    for side in (0, 1):
        got = h.debug_decode(side)
        expect = []
        for r0, r1, c0, c1, r, first, _, is_dense in blocks:
            if not is_dense:
                for j in range(first, first + r):
                    m = (r1 - r0, c1 - c0)[side]
                    raw = np.unpackbits(words[side][j].view(np.uint8), bitorder="little")[: m * ws[j]].reshape(m, ws[j])
                    v = raw.astype(np.int64) @ (1 << np.arange(ws[j], dtype=np.int64))
                    expect.append(v - (v >> (ws[j] - 1) << ws[j]))
        assert np.array_equal(got, np.concatenate(expect).astype(np.int32))
