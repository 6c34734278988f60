"""The plain form's square-root transform from the tridiagonal form (zone_sqrt64.cu, 65 <= N <=
128) against the analysis in observation space, in extended precision: with X the weighted
observed anomalies of a zone, K = I + X X^T, A = I + X^T X,
    xa = xf + Sf X^T K^-1 d,  Sa Sa^T = Sf A^-1 Sf^T = Sf Sf^T - (Sf X^T) K^-1 (Sf X^T)^T,
and, rotated, Sa 1 = 0. Odd and even row strides, one and two blocks an SM, every count of
poles, zones beyond its range.

Tolerance: the transform perturbs A by at most ~N u ||A|| (u = 2^-53), which moves A^(-1/2),
A^-1 and A^-1 g by at most N u (1 + lambda_max) relative to their norms (||A^-1|| <= 1, the
derivative of A^(-1/2) at A >= I is bounded by 1/2).
"""
import numpy as np
import pytest

import oak_gb300 as oak
from test_gpu_isqrt import _lambda_max, _problem

pytestmark = pytest.mark.gpu


def _exact(p):
    xa, P = p["xf"].copy(), []
    for z in range(p["zone_size"].size):
        e = slice(3 * z, 3 * z + 3)
        d = np.abs(p["obs_pos"][0] - p["zone_pos"][z, 0])
        s = d <= 4.0
        w = np.exp(-(d[s] / 3.0) ** 2) / np.sqrt(p["r_diag"][s])
        X = (p["HSf"][s] * w[:, None]).astype(np.longdouble)
        Sf = p["Sf"][e].astype(np.longdouble)
        rhs = np.column_stack([((p["yo"] - p["Hxf"])[s] * w).astype(np.longdouble), X @ Sf.T])
        K = np.eye(int(s.sum())) + X @ X.T
        y = np.zeros_like(rhs)
        for _ in range(6):  # refined from FP64 solves
            y = y + np.linalg.solve(K.astype(float), (rhs - K @ y).astype(float))
        xa[e] += (Sf @ (X.T @ y[:, 0])).astype(float)
        P.append((Sf @ Sf.T - (X @ Sf.T).T @ y[:, 1:]).astype(float))
    return xa, np.array(P)


def _compare(p, tol, rotate=True):
    xa, Sa, _, _ = oak.loc_analysis(**p, rotate=rotate)
    xe, P = _exact(p)
    norm = np.linalg.norm
    assert norm(xa - xe) <= tol * max(norm(xe - p["xf"]), norm(p["xf"]))
    S3 = np.ascontiguousarray(Sa).reshape(-1, 3, Sa.shape[1])
    assert norm(S3 @ S3.transpose(0, 2, 1) - P) <= tol * norm(p["Sf"]) ** 2
    if rotate:
        assert norm(Sa.sum(axis=1)) <= tol * norm(p["Sf"]) * np.sqrt(Sa.shape[1])
    else:
        b = oak.loc_analysis(**p, rotate=False, simt_gram=True)
        assert norm(Sa - b[1]) <= tol * norm(b[1])


@pytest.mark.parametrize("N", [65, 66, 96, 97, 102, 103, 127, 128])
@pytest.mark.parametrize("Z,rotate", [(2, True), (7, False), (307, True)])
def test_transform_matches_eigensolve(N, Z, rotate):
    p = _problem(N, Z, 100 * N + Z, lambda m, rng: rng.uniform(0.05, 0.5, m))
    _compare(p, N * 2.0 ** -53 * (1.0 + _lambda_max(p)), rotate=rotate)


# lambda_max ~ 100 / r: the Gershgorin bound passes 4^1, 4^4, 4^7, 4^10 and ends below 4^13
@pytest.mark.parametrize("r", [300.0, 30.0, 1.0, 3e-2, 1e-3, 2e-5])
def test_every_pole_count(r):
    p = _problem(100, 5, 17, lambda m, rng: np.full(m, r))
    _compare(p, 100 * 2.0 ** -53 * (1.0 + _lambda_max(p)))


def test_zero_gram_gives_the_prior():
    p = _problem(70, 9, 5, lambda m, rng: np.ones(m))
    p["HSf"] = np.zeros_like(p["HSf"])
    xa, Sa, _, _ = oak.loc_analysis(**p)
    assert np.allclose(xa, p["xf"], rtol=0, atol=1e-14)
    assert np.linalg.norm(Sa - p["Sf"]) <= 70 * 2.0 ** -50 * np.linalg.norm(p["Sf"])


def test_zones_beyond_the_range_take_the_eigensolve():
    """Every third zone has r = 1e-8 (lambda ~ 1e10): those go to the eigenvalue stages, the
    others keep their results to the bit, in a direct call and in a captured plan."""
    torch = pytest.importorskip("torch")
    Z, N = 50, 100
    p = _problem(N, Z, 3, lambda m, rng: np.full(m, 0.5))
    q = dict(p, r_diag=np.where((np.arange(40 * Z) // 40) % 3 == 0, 1e-8, 0.5))
    a = oak.loc_analysis(**p)
    b = oak.loc_analysis(**q)
    c = oak.loc_analysis(**q, simt_gram=True)
    rows = np.repeat(np.arange(Z) % 3 != 0, 3)
    assert np.array_equal(a[0][rows], b[0][rows]) and np.array_equal(a[1][rows], b[1][rows])
    # the same stages on the same Gram
    assert np.array_equal(b[1][~rows], c[1][~rows])

    def dev(x):
        if isinstance(x, tuple):
            return tuple(None if t is None else dev(t) for t in x)
        if x.ndim == 2 and x.flags.f_contiguous:
            return torch.as_tensor(np.ascontiguousarray(x.T), device="cuda").t()
        return torch.as_tensor(x, device="cuda")

    plan = oak.Plan(*[dev(q[k]) for k in ("zone_size", "xf", "Hxf", "yo", "Sf", "HSf", "r_diag",
                                          "zone_pos", "obs_pos", "corr_len", "max_len")])
    xa, Sa, _ = plan.execute()
    assert np.array_equal(xa.cpu().numpy(), b[0]) and np.array_equal(Sa.cpu().numpy(), b[1])
