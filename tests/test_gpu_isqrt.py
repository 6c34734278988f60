"""The plain form's square-root transform by Newton steps from FP32 eigenpairs
(zone_isqrt_oz.cu, 17 <= N <= 64) against the FP64 eigensolve on the CUDA cores
(simt_gram=True) and, for a few zones, the oracle.

Tolerance: both sides perturb A = I + G by at most ~N u ||A|| (u = 2^-53), which moves
A^(-1/2) and A^-1 g by at most N u (1 + lambda_max) relative to their norms (||A^(-1/2)|| <= 1,
the derivative of A^(-1/2) at A >= I is bounded by 1/2, and each side counts once).
"""
import numpy as np
import pytest

import oak_gb300 as oak

pytestmark = pytest.mark.gpu


def _problem(N, Z, seed, r):
    """Z zones of 3 elements on a line, 40 observations near each; r per observation."""
    rng = np.random.default_rng(seed)
    m, n = 40 * Z, 3 * Z
    ox = np.repeat(np.arange(Z) * 10.0, 40) + rng.uniform(-3.0, 3.0, m)
    HS = rng.standard_normal((m, N))
    HS -= HS.mean(axis=1, keepdims=True)
    Sf = rng.standard_normal((n, N))
    Sf -= Sf.mean(axis=1, keepdims=True)
    zp = np.zeros((Z, 4))
    zp[:, 0] = np.arange(Z) * 10.0
    return dict(zone_size=np.full(Z, 3, np.int32), xf=rng.standard_normal(n),
                Hxf=rng.standard_normal(m), yo=rng.standard_normal(m),
                Sf=np.asfortranarray(Sf), HSf=np.asfortranarray(HS), r_diag=r(m, rng),
                zone_pos=zp, obs_pos=(ox, np.zeros(m), None, None),
                corr_len=np.full(Z, 3.0), max_len=np.full(Z, 4.0))


def _lambda_max(p):
    lam = 0.0
    for z in range(p["zone_size"].size):
        d = np.abs(p["obs_pos"][0] - p["zone_pos"][z, 0])
        s = d <= 4.0
        X = p["HSf"][s] * (np.exp(-(d[s] / 3.0) ** 2) / np.sqrt(p["r_diag"][s]))[:, None]
        lam = max(lam, np.linalg.norm(X, 2) ** 2)
    return lam


def _compare(p, tol, **opts):
    a = oak.loc_analysis(**p, **opts)
    b = oak.loc_analysis(**p, simt_gram=True, **opts)
    assert np.array_equal(a[3], b[3])
    inc = np.linalg.norm(b[0] - p["xf"])
    assert np.linalg.norm(a[0] - b[0]) <= tol * max(inc, np.linalg.norm(p["xf"]))
    assert np.linalg.norm(a[1] - b[1]) <= tol * np.linalg.norm(b[1])
    return a


@pytest.mark.parametrize("N", [17, 32, 33, 63, 64])
@pytest.mark.parametrize("Z,rotate", [(2, True), (7, False), (311, True)])
def test_newton_transform_matches_eigensolve(N, Z, rotate):
    p = _problem(N, Z, 100 * N + Z, lambda m, rng: rng.uniform(0.05, 0.5, m))
    tol = N * 2.0 ** -53 * (1.0 + _lambda_max(p))
    _compare(p, tol, rotate=rotate)


def test_zero_gram_gives_the_prior():
    p = _problem(40, 9, 5, lambda m, rng: np.ones(m))
    p["HSf"] = np.zeros_like(p["HSf"])
    xa, Sa, _, _ = oak.loc_analysis(**p)
    # T = A^(-1/2) Omega with A = I: Omega is the identity up to rounding
    assert np.allclose(xa, p["xf"], rtol=0, atol=1e-14)
    assert np.linalg.norm(Sa - p["Sf"]) <= 40 * 2.0 ** -50 * np.linalg.norm(p["Sf"])


def test_zones_beyond_fp32_take_the_eigensolve():
    """Every third zone has r = 1e-8 (lambda ~ 1e10): those are handed to the FP64 eigensolve and
    the others keep their results, in a direct call and in a captured plan."""
    torch = pytest.importorskip("torch")
    Z, N = 160, 64
    p = _problem(N, Z, 9, lambda m, rng: np.full(m, 0.1))
    q = dict(p, r_diag=np.where((np.arange(40 * Z) // 40) % 3 == 0, 1e-8, 0.1))
    a = oak.loc_analysis(**p)
    b = oak.loc_analysis(**q)
    c = oak.loc_analysis(**q, simt_gram=True)
    rows = np.repeat(np.arange(Z) % 3 != 0, 3)
    # the Gram's fixed point follows the call's largest |HS| / sqrt(r) (below 2^17 here), so an
    # element of the other zones (below 20) is rounded to 2^-38: G moves by at most 2 * 40 * 20 *
    # 2^-38 = 6e-9 an element, T by half its norm (<= 64 elements a row)
    assert np.abs(a[1][rows] - b[1][rows]).max() <= 32 * 6e-9 * np.abs(p["Sf"]).max() * N
    tol = N * 2.0 ** -53 * (1.0 + _lambda_max(q))
    assert np.linalg.norm(b[1][~rows] - c[1][~rows]) <= tol * np.linalg.norm(p["Sf"][~rows])

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
