"""Zones out of the reach of the plain form's Newton transform (17 <= N <= 64) among zones within it and
zones without observations: those whose Gram matrix is large are left by the first stage, those
with a wide spectrum by the second, those whose iteration does not settle by the transform itself,
and all take the FP64 stages with the tensor-core products. Against the CUDA-core form
(simt_gram=True).

Tolerance, a zone: A = I + G is perturbed by N u (1 + lambda_max) as in test_gpu_isqrt.py and by what
the Gram's fixed point leaves out (2^-54 of the call's largest element an observation, times the
zone's largest): e. T moves by at most 2 e (e / 2 and as much by the rotation's v, twice), A^-1 g by
e |A^-1 g|.
"""
import numpy as np
import pytest

import oak_gb300 as oak
from test_gpu_isqrt import _problem

pytestmark = pytest.mark.gpu

# r a zone, by turns: within reach; near its end; a wide spectrum; a large Gram matrix; no observation
_R = (1.0, 3e-5, 2e-6, 1e-9, None)


@pytest.mark.parametrize("N", [17, 32, 50, 64])
@pytest.mark.parametrize("Z,rotate", [(10, True), (400, False), (400, True)])
def test_zones_out_of_reach(N, Z, rotate):
    p = _problem(N, Z, N + Z, lambda m, rng: np.ones(m))
    p["r_diag"] = np.repeat([_R[z % 5] or 1.0 for z in range(Z)], 40)
    p["max_len"] = np.where(np.arange(Z) % 5 == 4, 1e-9, p["max_len"])
    a = oak.loc_analysis(**p, rotate=rotate)
    b = oak.loc_analysis(**p, rotate=rotate, simt_gram=True, ampl_always=True)
    assert np.array_equal(a[3], b[3]) and (a[3][4::5] == 0).all()
    top = np.log2(np.abs(p["HSf"] / np.sqrt(p["r_diag"])[:, None]).max()) + 1.0
    u = 2.0 ** -53
    for z in range(Z):
        d = np.abs(p["obs_pos"][0] - p["zone_pos"][z, 0])
        s = d <= p["max_len"][z]
        e = slice(3 * z, 3 * z + 3)
        if not s.any():
            assert np.array_equal(a[1][e], p["Sf"][e])
            continue
        X = p["HSf"][s] * (np.exp(-(d[s] / 3.0) ** 2) / np.sqrt(p["r_diag"][s]))[:, None]
        lam = np.linalg.norm(X, 2) ** 2
        fixed = s.sum() * 2.0 ** (top - 53) * np.abs(X).max()  # an element of G
        err = N * u * (1.0 + lam) + N * fixed
        S = np.linalg.norm(p["Sf"][e])
        assert np.linalg.norm(a[1][e] - b[1][e]) <= 2 * err * S, (z, lam)
        assert (np.linalg.norm(a[0][e] - b[0][e])
                <= err * np.linalg.norm(b[2][:, z]) * S + 4 * u * np.linalg.norm(a[0][e])), (z, lam)


def test_every_zone_out_of_reach_in_a_plan():
    torch = pytest.importorskip("torch")
    N, Z = 40, 30
    p = _problem(N, Z, 1, lambda m, rng: np.full(m, 1e-10))
    b = oak.loc_analysis(**p)

    def dev(x):
        if isinstance(x, tuple):
            return tuple(None if t is None else dev(t) for t in x)
        if x.ndim == 2 and x.flags.f_contiguous:
            return torch.as_tensor(np.ascontiguousarray(x.T), device="cuda").t()
        return torch.as_tensor(x, device="cuda")

    plan = oak.Plan(*[dev(p[k]) for k in ("zone_size", "xf", "Hxf", "yo", "Sf", "HSf", "r_diag",
                                          "zone_pos", "obs_pos", "corr_len", "max_len")])
    for _ in range(2):
        xa, Sa, _ = plan.execute()
        assert np.array_equal(xa.cpu().numpy(), b[0]) and np.array_equal(Sa.cpu().numpy(), b[1])
