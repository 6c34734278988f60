"""The tensor-core Gram over a call in which every CTA goes for several seconds without an observation
to stage: waits for the workers' progress do not expire (only those for the tensor core are bounded,
2^22 polls of about 1.5 us each)."""
import numpy as np
import pytest

import oak_gb300 as oak

pytestmark = pytest.mark.gpu


def test_a_long_run_of_zones_that_select_nothing():
    """Every observation is within the cut-off of every zone, so all are tested, but beyond twice
    the length scale, where the weight vanishes; the last zones lie among the observations."""
    torch = pytest.importorskip("torch")
    f64 = dict(device="cuda", dtype=torch.float64)
    N, m, Z, last = 2, 4_000_000, 62_000, 152
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    zone_pos = torch.zeros((Z, 4), **f64)
    zone_pos[:-last, 0] = 1000.0
    oak.release()
    HSf = torch.randn((N, m), generator=g, **f64).t()
    args = (torch.ones(Z, device="cuda", dtype=torch.int32), torch.zeros(Z, **f64),
            torch.zeros(m, **f64), torch.randn(m, generator=g, **f64),
            torch.randn((N, Z), generator=g, **f64).t(), HSf, torch.full((m,), 1e3, **f64), zone_pos,
            (torch.rand(m, generator=g, **f64), torch.rand(m, generator=g, **f64), None, None),
            torch.full((Z,), 10.0, **f64), torch.full((Z,), 5000.0, **f64))
    xa, Sa, _, nobs = oak.loc_analysis(*args, weight=oak.GASPARI_COHN, want_ampl=False, cell_size=0.002)
    ms = oak.last_timings()["gram"]
    oak.release()
    print(f"Gram stage {ms:.0f} ms")
    assert int(nobs[:-last].sum()) == 0 and (nobs[-last:] == m).all()
    assert torch.equal(Sa[:-last], args[4][:-last]) and torch.isfinite(Sa).all()
    assert (Sa[-last:] != args[4][-last:]).any()
    assert ms > 6500.0  # long enough to mean something
