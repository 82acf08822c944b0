"""The right-hand side's exponent and limbs at the orders where the cluster
kernel's grid has remainders or ends (8192 padded entries; above: the
cooperative launch), with padding past the order.

y is compared with the same factors multiplied in extended precision, within
the 1e-13 (in norm) that the library states, and columns with their own
one-column applies bit for bit.
"""

import numpy as np
import pytest

from conftest import rel_err
from qhmat_gb300 import HMatrix
from test_oracle import _pack_codes

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.mark.parametrize("n", [2, 31, 33, 8159, 8160, 8161, 16385])
def test_orders_at_the_cluster_edges(cuda_device, n):
    import torch

    w = 16
    rng = np.random.default_rng(n)
    perm = rng.permutation(n)
    blocks, dense, words, offs, scales, ws, factors = [], [], ([], []), ([], []), ([], []), [], []

    def cut(r0, r1):  # dense diagonal blocks of up to 64, rank 1 off the diagonal
        if r1 - r0 <= 64:
            d = rng.standard_normal((r1 - r0, r1 - r0))
            blocks.append((r0, r1, r0, r1, 0, 0, sum(map(len, dense)), 1))
            dense.append(d.ravel())
            factors.append((r0, r1, r0, r1, d, None))
            return
        m = (r0 + r1) // 2
        for a0, a1, b0, b1 in ((r0, m, m, r1), (m, r1, r0, m)):
            blocks.append((a0, a1, b0, b1, 1, len(ws), 0, 0))
            ws.append(w)
            f = []
            for side, k in enumerate((a1 - a0, b1 - b0)):
                codes = rng.integers(-(1 << (w - 1)) + 1, 1 << (w - 1), k)
                offs[side].append(sum(map(len, words[side])))
                words[side].append(_pack_codes(codes, w))
                scales[side].append(2.0**-15)
                f.append(codes.astype(np.longdouble) * np.longdouble(2.0**-15))
            factors.append((a0, a1, b0, b1, *f))
        cut(r0, m)
        cut(m, r1)

    cut(0, n)
    words = [w if w else [np.zeros(1, np.uint32)] for w in words]
    h = HMatrix.from_arrays(n, perm, blocks, np.concatenate(dense), np.concatenate(words[0]), np.concatenate(words[1]),
                            offs[0], offs[1], scales[0], scales[1], ws)
    x = rng.standard_normal((n, 3)) * np.array([1.0, 2.0**300, 0.0])
    x[n - 1, 2] = 1.0  # the last entry alone
    xc = x[perm].astype(np.longdouble)
    yc = np.zeros((n, 3), np.longdouble)
    for r0, r1, c0, c1, p, q in factors:
        yc[r0:r1] += p @ xc[c0:c1] if q is None else np.outer(p, q @ xc[c0:c1])
    y = h.matmul(x)
    for k in range(3):
        assert rel_err(y[perm, k] / 2.0**(300 * (k == 1)), yc[:, k] / np.longdouble(2.0**(300 * (k == 1)))) <= TOL
        assert np.array_equal(h.matmul(np.ascontiguousarray(x[:, k])), y[:, k])
    bad = torch.from_numpy(x).cuda()
    bad[n - 1, 1] = float("inf")
    with pytest.raises(ValueError, match="nonfinite right-hand side"):
        h.matmul(bad)
    assert np.array_equal(h.matmul(torch.from_numpy(x).cuda()).cpu().numpy(), y)
