"""The plain form's update of rows down to FP64's smallest numbers: slice products
(zone_update_oz.cu) against the CUDA-core products (simt_gram=True).

Tolerance: that of test_gpu_update_oz.py relative to a row's largest element, plus a unit of the
last place of subnormals (2^-1074) for each of the N + 1 roundings that either side makes there.
"""
import numpy as np
import pytest

import oak_gb300 as oak
from test_gpu_isqrt import _lambda_max, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(20, 32, 9), (70, 33, 64)])
def test_rows_down_to_subnormals(sizes):
    N = 64
    p = _problem(N, 3, 11, lambda m, rng: rng.uniform(0.1, 1.0, m))
    rng = np.random.default_rng(12)
    n = sum(sizes)
    Sf = rng.standard_normal((n, N))
    scale = 2.0 ** np.linspace(-900.0, -1022.0, n)
    Sf *= scale[:, None]
    Sf[3::7] = np.ldexp(rng.integers(-9, 10, (len(Sf[3::7]), N)).astype(float), -1074)  # subnormal
    Sf[4::7] *= np.where(np.arange(N) == 5, 1.0, 2.0 ** -60)  # one element far above the others
    p = dict(p, zone_size=np.array(sizes, np.int32), xf=np.zeros(n), Sf=np.asfortranarray(Sf))
    a = oak.loc_analysis(**p)
    b = oak.loc_analysis(**p, simt_gram=True)
    tol = N * 2.0 ** -53 * (2.0 + _lambda_max(p)) * np.sqrt(N)
    row = np.abs(Sf).max(axis=1)
    assert row.min() < 1e-320 and row.max() > 1e-275
    bound = np.ldexp(np.ldexp(row, 600) * tol, -600) + (N + 1) * 5e-324
    assert (np.abs(a[1] - b[1]).max(axis=1) <= bound).all()
    assert (np.abs(a[1]).max(axis=1) > 0).all()
