"""Adjoint of the local analysis mean over more seeded zones than one chunk of zone matrices holds
(16 GiB: 516,000 zones of 64 members): the gradients are linear in the seed, so that a call is the
sum of two calls with half of the zones seeded each, which take one chunk. A tenth of the zones see
an observation of error variance 1e-12, so that both chunks have zones that the fixed point is too
coarse for and zones that it is not.

Tolerance: a zone's terms are the same in both; their sums (at most 3.6 million terms, u = 2^-53
each) are in another order. Zones of a group have terms of one sign and 500 groups differ, which
leaves a sum above 1/50 of the sum of magnitudes: 3.6e6 u 50 = 2e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_call_of_two_chunks_is_the_sum_of_its_halves(oakg):
    import torch
    N, Z, groups, p = 64, 600_000, 500, 6
    rng = np.random.default_rng(11)
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    F = lambda a: torch.as_tensor(np.ascontiguousarray(a.T), device="cuda").t()
    g = np.arange(Z) % groups
    zp = np.zeros((Z, 4))
    zp[:, 0] = 100.0 * g
    anomalies = lambda k: (lambda x: (x - x.mean(1, keepdims=True)) / np.sqrt(N - 1))(
        rng.standard_normal((k, N)))
    m = groups * p
    r = rng.uniform(0.05, 0.5, m)
    exact = np.arange(0, m, 10 * p)
    r[exact] = 1e-12
    args = (T(np.ones(Z, np.int32)), T(np.zeros(m)), T(rng.standard_normal(m)),
            F(anomalies(groups)[g]), F(anomalies(m)), T(r), T(zp),
            (T(np.repeat(100.0 * np.arange(groups), p) + rng.uniform(-3.0, 3.0, m)), T(np.zeros(m)),
             None, None), T(np.full(Z, 3.0)), T(np.full(Z, 4.0)))
    seed = rng.uniform(0.5, 1.5, Z)

    def grads(s):
        dyo, dr, dlen, dinfl = oakg.loc_analysis_adjoint(*args, T(s), weight=1)
        dyo, dr = dyo.cpu().numpy(), dr.cpu().numpy()
        rest = np.ones(m, bool)
        rest[exact] = False
        return [dyo[rest], dyo[exact], dr[rest], dr[exact], np.array([dlen]), np.array([dinfl])]

    low = np.arange(Z) < Z // 2
    for a, b, c in zip(grads(seed), grads(seed * low), grads(seed * ~low)):
        norm = np.linalg.norm
        assert np.isfinite(a).all() and norm(a) > 0
        assert norm(a - (b + c)) <= 2e-8 * max(norm(b), norm(c))
