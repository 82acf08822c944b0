"""The precision form's exponent and limb kernels at the column counts and
orders where their blocks (16 rows, 2^k >= p columns) have remainders, on
columns that stress the limbs: magnitudes spread over 2^-40 .. 2^40, a zero
column, a subnormal column, a single spike.

x carries about 33 bits below its column's largest entry and sums are FP32, so
a column's y is within 1e-5 in norm of the plain form's (the form's stated
tolerance); powers of two in x only move exponents, so they scale y to 1e-12.
"""

import numpy as np
import pytest

from conftest import golden, rel_err
from qhmat_gb300 import HMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3, 5, 8, 9, 17, 33, 63, 64, 65])
@pytest.mark.parametrize("name", ["cuda10", "ragged300", "cfg1"])
def test_limbs_at_block_edges(cuda_device, name, p):
    data, _ = golden(name)
    h = HMatrix.from_bytes(data, precision=True)
    rng = np.random.default_rng(p)
    x = rng.standard_normal((h.order, p))
    x[:, 1::5] *= np.exp2(rng.integers(-40, 40, (h.order, 1)))
    x[:, 2::5] = 0.0
    x[h.order // 2, 2::10] = -3.0
    x[:, 3::5] *= 2.0**-1060  # subnormal: no exponent, taken as zero
    y = h.matmul(x, form="precision")
    plain = h.matmul(x)
    for k in range(p):
        if k % 5 == 3:
            assert not y[:, k].any()
        else:
            assert rel_err(y[:, k], plain[:, k]) <= 1e-5, k
    y2 = h.matmul(x * 2.0**60, form="precision")
    ok = [k for k in range(p) if k % 5 != 3]
    assert rel_err(y2[:, ok], y[:, ok] * 2.0**60) <= 1e-12
