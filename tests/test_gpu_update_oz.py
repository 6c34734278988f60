"""The plain form's update on the tensor cores (zone_update_oz.cu) against the CUDA-core products
(simt_gram=True): row counts at the edges of its tiles (32 | 33, 64 | 65, several tiles, tiles
split over CTAs), both storage types, in place of nothing.

Tolerance: N u relative to the rows' norms for the update (u = 2^-53), plus what the two forms'
transforms may differ by, N u (1 + lambda_max) (test_gpu_isqrt.py); FP32 storage rounds both to
2^-24.
"""
import numpy as np
import pytest

import oak_gb300 as oak
from test_gpu_isqrt import _lambda_max, _problem

pytestmark = pytest.mark.gpu


def _resized(p, sizes, seed):
    rng = np.random.default_rng(seed)
    n, N = int(sizes.sum()), p["Sf"].shape[1]
    Sf = rng.standard_normal((n, N)) * 10.0 ** rng.uniform(-6, 6, (n, 1))
    return dict(p, zone_size=sizes.astype(np.int32), xf=rng.standard_normal(n), Sf=np.asfortranarray(Sf))


@pytest.mark.parametrize("N", [47, 63, 64])
@pytest.mark.parametrize("sizes", [(1, 31, 32, 7), (33, 1, 64, 20), (65, 129, 3, 500), (20_001, 40, 1, 64)])
def test_update_matches_the_cuda_cores(N, sizes):
    p = _resized(_problem(N, 4, N, lambda m, rng: rng.uniform(0.1, 1.0, m)), np.array(sizes), 3)
    a = oak.loc_analysis(**p)
    b = oak.loc_analysis(**p, simt_gram=True)
    tol = N * 2.0 ** -53 * (2.0 + _lambda_max(p))
    row = np.linalg.norm(p["Sf"], axis=1)
    assert (np.linalg.norm(a[1] - b[1], axis=1) <= tol * row).all()
    # the mean's increment is Sf ampl: |ampl| <= |A^-1 g|, both forms'
    inc = np.abs(b[0] - p["xf"]) + np.abs(p["xf"]) + row
    assert (np.abs(a[0] - b[0]) <= 64 * tol * inc).all()


def test_float_storage_and_zones_without_observations():
    p = _resized(_problem(64, 5, 2, lambda m, rng: rng.uniform(0.1, 1.0, m)), np.array([40, 5, 70, 33, 64]), 4)
    p["max_len"] = np.where(np.arange(5) == 2, 1e-9, p["max_len"])  # zone 2 sees no observation
    f = {k: (v.astype(np.float32) if k in ("xf", "Hxf", "yo", "Sf", "HSf", "r_diag") else v)
         for k, v in p.items()}
    wide = {k: (v.astype(np.float64) if k in ("xf", "Hxf", "yo", "Sf", "HSf", "r_diag") else v)
            for k, v in f.items()}
    a, b = oak.loc_analysis(**f), oak.loc_analysis(**wide)
    assert a[3][2] == 0 and b[3][2] == 0
    # the same analysis, rounded once at the boundary
    assert np.array_equal(a[0], b[0].astype(np.float32))
    assert np.array_equal(a[1], b[1].astype(np.float32))
    rows = slice(45, 115)
    assert np.array_equal(b[1][rows], wide["Sf"][rows]) and np.array_equal(b[0][rows], wide["xf"][rows])


def test_infinite_and_nan_rows():
    """A row with an infinity or a NaN gets what the sum of its products is, and no other row does."""
    p = _resized(_problem(64, 3, 6, lambda m, rng: rng.uniform(0.1, 1.0, m)), np.array([20, 70, 33]), 5)
    Sf = p["Sf"]
    Sf[3, 0], Sf[25, 63], Sf[30, [5, 40]], Sf[95, 17] = np.inf, -np.inf, (np.inf, -np.inf), np.nan
    a = oak.loc_analysis(**p)
    b = oak.loc_analysis(**p, simt_gram=True)
    odd = [3, 25, 30, 95]
    for x, y in ((a[0][odd], b[0][odd]), (a[1][odd], b[1][odd])):
        assert not np.isfinite(x).any()
        assert np.array_equal(x, y, equal_nan=True)
    rest = np.setdiff1d(np.arange(Sf.shape[0]), odd)
    assert np.isfinite(a[1][rest]).all() and np.isfinite(a[0][rest]).all()
