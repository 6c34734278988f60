"""Adjoint of the local analysis mean for 17 to 64 members (the tensor-core Gram on the list of
seeded zones) against the FP64 reference gradient, also beside one far more exact observation that no
seeded zone sees: the Gram's fixed point follows the call's largest element, and zones that it would
be too coarse for take the FP64 products.

Tolerance: that of test_gpu_adjoint.py against the same reference.
"""
import numpy as np
import pytest

from oracle import oakref_torch
from test_gpu_adjoint import _J_and_seed, _forward, _problem

pytestmark = pytest.mark.gpu


def _exact_observation(P, r, at):
    """P with one more observation of error variance r at `at`."""
    rng = np.random.default_rng(9)
    N = P["HSf"].shape[1]
    h = rng.standard_normal(N) / np.sqrt(N - 1)
    far = dict(P, HSf=np.asfortranarray(np.vstack([P["HSf"], h - h.mean()])), Hxf=np.r_[P["Hxf"], 0.3],
               yo=np.r_[P["yo"], 0.4], r=np.r_[P["r"], r])
    far["obs_pos"] = tuple(np.r_[c, v] for c, v in zip(P["obs_pos"], (*at, 0.0, 0.0)))
    return far


def _check(oakg, P):
    import torch
    s, kind = 1.05, P["kind"]
    xa = _forward(oakg, P, P["yo"], P["r"], 1.0, s)
    _, seed = _J_and_seed(xa, P)
    dyo, dr, dlen, dinfl = oakg.loc_analysis_adjoint(
        P["zs"], P["Hxf"], P["yo"], P["Sf"], P["HSf"], P["r"], P["zone_pos"], P["obs_pos"],
        P["corr"], P["maxl"], seed, inflation=s, weight=kind)
    sels = oakref_torch.selections(P["zone_pos"], P["obs_pos"], P["corr"], P["maxl"], kind=kind)
    yo = torch.tensor(P["yo"], requires_grad=True)
    r = torch.tensor(P["r"], requires_grad=True)
    kap = torch.tensor(1.0, dtype=torch.float64, requires_grad=True)
    st = torch.tensor(s, dtype=torch.float64, requires_grad=True)
    xt = oakref_torch.loc_analysis_mean(P["zs"], P["xf"], P["Hxf"], P["Sf"], P["HSf"], P["corr"],
                                        sels, yo, r, kap, st, kind)
    # the cost's gradient at the reference's own analysis: the seed is a given of the adjoint call
    (xt * torch.tensor(seed)).sum().backward()
    rel = lambda a, b: np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)
    assert rel(dyo, yo.grad.numpy()) < 1e-9
    assert rel(dr, r.grad.numpy()) < 1e-9
    assert abs(dlen - float(kap.grad)) <= 1e-9 * max(1.0, abs(float(kap.grad)))
    assert abs(dinfl - float(st.grad)) <= 1e-9 * max(1.0, abs(float(st.grad)))


@pytest.mark.parametrize("kind,N", [(0, 17), (1, 33), (0, 48), (1, 64)])
def test_wider_ensembles(oakg, kind, N):
    _check(oakg, _problem(kind=kind, N=N))


@pytest.mark.parametrize("kind,N", [(0, 5), (1, 20), (0, 64)])
def test_beside_one_exact_observation(oakg, kind, N):
    P = _exact_observation(_problem(kind=kind, N=N), 1e-24, (500.0, 400.0))
    _check(oakg, P)
