"""The apply on device tensors with the status check: each call reports its own
right-hand side's nonfinite entries, also when threads apply the same handle
on streams of their own, and a failed call leaves the next ones right."""

import threading

import numpy as np
import pytest

from conftest import golden
from qhmat_gb300 import HMatrix, PrecisionHMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cls", [HMatrix, PrecisionHMatrix])
@pytest.mark.parametrize("p", [1, 2, 3, 9])
def test_status_is_per_call(cuda_device, cls, p):
    import torch

    data, _ = golden("cfg1")
    h = cls.from_bytes(data)
    x = torch.from_numpy(np.random.default_rng(p).standard_normal((h.order, p))).cuda()
    bad = x.clone()
    bad[h.order // 3, p - 1] = float("nan")
    expect = h.matmul(x)
    assert torch.equal(h.matmul(x, check=False), expect)
    torch.cuda.synchronize()
    wrong = []

    def run(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(20):
                try:
                    y = h.matmul(bad if (i + k) % 3 == 0 else x)
                    if (i + k) % 3 == 0 or not torch.equal(y, expect):
                        wrong.append((k, i, "value"))
                except ValueError as e:
                    if (i + k) % 3 or "nonfinite right-hand side" not in str(e):
                        wrong.append((k, i, str(e)))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
    assert torch.equal(h.matmul(x), expect)
