"""Slots past a row tile's k axis add nothing, whatever the workspace held:
matrices whose factor arrays start after a gap (component 0 belongs to no
block) and whose rank is not a multiple of 32, with a workspace full of 0x80
bytes.  The right-hand side meets only zero codes of the right factors, so y
is a column of the dense diagonal blocks, exactly."""

import numpy as np
import pytest

from qhmat_gb300 import HMatrix
from test_oracle import _pack_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b,rank", [(33, 31, 5), (64, 64, 33), (100, 300, 70)])
def test_slots_past_the_k_axis(cuda_device, a, b, rank):
    import torch

    n, gap = a + b, 3
    rng = np.random.default_rng(n)
    col = {0: a // 2, a: b // 3}  # the column of each cluster that x meets
    blocks, dense, words, offs, scales = [], [], ([np.zeros(1, np.uint32)], [np.zeros(1, np.uint32)]), ([], []), ([], [])
    ws = [2] * gap
    for side in (0, 1):
        offs[side].extend([0] * gap)
        scales[side].extend([0.0] * gap)
    full = np.zeros((n, n))
    for k, (r0, r1, c0, c1) in enumerate([(0, a, 0, a), (0, a, a, n), (a, n, 0, a), (a, n, a, n)]):
        if k in (0, 3):
            d = rng.standard_normal((r1 - r0, c1 - c0))
            blocks.append((r0, r1, c0, c1, 0, 0, sum(map(len, dense)), 1))
            dense.append(d.ravel())
            full[r0:r1, c0:c1] = d
            continue
        r = min(rank, a - 1, b - 1)
        blocks.append((r0, r1, c0, c1, r, len(ws), 0, 0))
        for j in range(r):
            w = 3 + (j * 7 + k) % 30
            ws.append(w)
            for side, m in enumerate((r1 - r0, c1 - c0)):
                codes = rng.integers(-(1 << (w - 1)) + 1, 1 << (w - 1), m)
                if side:
                    codes[col[c0]] = 0
                offs[side].append(sum(map(len, words[side])))
                words[side].append(_pack_codes(codes, w))
                scales[side].append(float(2.0 ** (1 - w)))
    h = HMatrix.from_arrays(n, np.arange(n), blocks, np.concatenate(dense), np.concatenate(words[0]),
                            np.concatenate(words[1]), offs[0], offs[1], scales[0], scales[1], ws)
    for p in (1, 2, 3, 4, 5, 9):
        x = np.zeros((n, p))
        for j in range(p):
            x[[0, a][j % 2] + col[[0, a][j % 2]], j] = 1.0 + j
        need = h.workspace_bytes(p)
        ws_buf = torch.full((need,), 0x80, dtype=torch.uint8, device="cuda")
        y = h.matmul(torch.from_numpy(x).cuda(), workspace=ws_buf).cpu().numpy()
        np.testing.assert_array_equal(y, full @ x, err_msg=str(p))
