"""The amplitudes A^-1 g of the plain form's Newton transform (zone_isqrt_oz.cu, 17 <= N <= 64), which
are refined by g - A a: the increments X a that they give at the observations are no further from
the exact ones than the CUDA-core form's (an FP64 eigensolve), in the geometric mean over the zones.

G and g are exact on both sides (observations at the zone, r = 1, anomalies and innovations with few
bits, as in test_gpu_isqrt_residual.py); the reference is refined with exact residuals.
"""
import numpy as np
import pytest

import oak_gb300 as oak
from test_gpu_isqrt_residual import _anomalies, _product

pytestmark = pytest.mark.gpu


def _exact(x, d):
    """A^-1 X^T d as hi + lo."""
    import torch
    G, g = x.mT @ x, x.mT @ d  # exact
    A = G + torch.eye(x.shape[-1], device="cuda", dtype=torch.float64)
    L = torch.linalg.cholesky(A)
    column = lambda v: torch.nn.functional.pad(v, (0, v.shape[1] - 1))
    hi, lo = torch.cholesky_solve(g, L), torch.zeros_like(g)
    for _ in range(4):
        ph, pl = _product(A, column(hi))
        r = (g - ph[..., :1]) - pl[..., :1] - A @ lo
        lo = lo + torch.cholesky_solve(r, L)
        new = hi + lo
        hi, lo = new, lo - (new - hi)
    return hi, lo


@pytest.mark.parametrize("shape,N,lo,hi", [("lin", 20, 3, 4), ("lin", 48, 3, 4), ("lin", 64, 2, 3),
                                           ("two", 64, 1.5, 2.5), ("geom", 40, 2, 3),
                                           ("one", 33, 2, 3), ("flat", 17, 1, 2)])
def test_increments_are_as_exact_as_the_eigensolve(shape, N, lo, hi):
    torch = pytest.importorskip("torch")
    Z = 300
    rng = np.random.default_rng(N)
    X = _anomalies(shape, N, 10.0 ** rng.uniform(lo, hi, Z), rng)
    p = X.shape[1]
    d = rng.integers(-64, 65, (Z, p)).astype(float)
    zp = np.zeros((Z, 4))
    zp[:, 0] = 10.0 * np.arange(Z)
    m = Z * p
    args = (np.ones(Z, np.int32), np.zeros(Z), np.zeros(m), d.reshape(m),
            np.asfortranarray(rng.standard_normal((Z, N))), np.asfortranarray(X.reshape(m, N)),
            np.ones(m), zp, (np.repeat(zp[:, 0], p), np.zeros(m), None, None), np.full(Z, 3.0),
            np.full(Z, 4.0))
    x, dv = torch.as_tensor(X, device="cuda"), torch.as_tensor(d, device="cuda")[:, :, None]
    ah, al = _exact(x, dv)
    size = torch.linalg.vector_norm(x @ ah, dim=(1, 2))
    err = []
    for simt in (False, True):
        _, _, ampl, nobs = oak.loc_analysis(*args, ampl_always=True, simt_gram=simt)
        assert (nobs == p).all()
        a = torch.as_tensor(np.ascontiguousarray(ampl.T), device="cuda")[..., None]
        rel = torch.linalg.vector_norm(x @ ((a - ah) - al), dim=(1, 2)) / size
        err.append(float(torch.log(rel + 2.0 ** -60).mean().exp()))
    assert err[0] <= err[1], err
