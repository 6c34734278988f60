"""The plain form's update over uneven zones, narrower ensembles and in place (zone_update_oz.cu):
Sf T and xf + Sf ampl from the transforms and amplitudes of a second call, whose state rows are the
identity, with the tolerance of test_gpu_update_oz.py.
"""
import numpy as np
import pytest

import oak_gb300 as oak
from test_gpu_isqrt import _lambda_max, _problem
from test_gpu_update_oz import _resized

pytestmark = pytest.mark.gpu


def _check(p):
    xa, Sa, _, nobs = oak.loc_analysis(**p)
    Z, N = p["zone_size"].size, p["Sf"].shape[1]
    q = dict(p, zone_size=np.full(Z, N, np.int32), xf=np.zeros(Z * N),
             Sf=np.asfortranarray(np.tile(np.eye(N), (Z, 1))))
    _, T, ampl, n2 = oak.loc_analysis(**q, ampl_always=True)
    assert np.array_equal(nobs, n2)
    T = np.ascontiguousarray(T).reshape(Z, N, N)
    first = np.cumsum(p["zone_size"]) - p["zone_size"]
    tol = N * 2.0 ** -53 * (2.0 + _lambda_max(p))
    row = np.linalg.norm(p["Sf"], axis=1)
    for z in range(Z):
        r = slice(first[z], first[z] + p["zone_size"][z])
        S = np.ascontiguousarray(p["Sf"][r])
        assert (np.linalg.norm(Sa[r] - S @ T[z], axis=1) <= tol * row[r]).all(), z
        ref = p["xf"][r] + S @ ampl[:, z]
        inc = np.abs(ref - p["xf"][r]) + np.abs(p["xf"][r]) + row[r]
        assert (np.abs(xa[r] - ref) <= 64 * tol * inc).all(), z


def _uneven(Z, seed, long_rows):
    rng = np.random.default_rng(seed)
    sizes = rng.integers(0, 41, Z)
    sizes[rng.integers(0, Z)] = long_rows
    return sizes


# fewer zones than SMs, as many, several rounds; the longest zone within a tile, many tiles
@pytest.mark.parametrize("N", [26, 33, 46, 64])
@pytest.mark.parametrize("Z,long_rows", [(3, 40_000), (200, 30_000), (200, 65), (2000, 31), (5000, 9_000)])
def test_uneven_zones(N, Z, long_rows):
    sizes = np.minimum(_uneven(Z, Z + N, long_rows), max(long_rows, 31))
    p = _resized(_problem(N, Z, N, lambda m, rng: rng.uniform(0.1, 1.0, m)), sizes, 7)
    _check(p)


@pytest.mark.parametrize("N,sizes", [(64, (20, 32, 9)), (40, (500, 70, 0)), (64, (33, 64, 4000))])
def test_in_place(N, sizes):
    """Sa over Sf and xa over xf, one zone without observations."""
    torch = pytest.importorskip("torch")
    p = _resized(_problem(N, 3, N, lambda m, rng: rng.uniform(0.1, 1.0, m)), np.array(sizes), 8)
    p["max_len"] = np.where(np.arange(3) == 1, 1e-9, p["max_len"])

    def dev(x):
        if isinstance(x, tuple):
            return tuple(dev(t) if t is not None else None for t in x)
        if x.ndim == 2 and x.flags.f_contiguous:
            return torch.as_tensor(np.ascontiguousarray(x.T), device="cuda").t()
        return torch.as_tensor(x, device="cuda")

    d = {k: dev(v) for k, v in p.items()}
    xa, Sa, _, nobs = oak.loc_analysis(**d)
    assert nobs[1] == 0 and nobs[0] > 0
    oak.loc_analysis(**d, out=(d["xf"], d["Sf"]))
    assert torch.equal(d["xf"], xa) and torch.equal(d["Sf"], Sa)
