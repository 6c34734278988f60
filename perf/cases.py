"""Performance cases of the local ensemble square-root analysis: the calls a data-assimilation
system makes, with the sizes of its configurations.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the inputs (and the plan) a program holds before the call, on the GPU
    run(state)           one pass through the public entry points, and its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    what run() returns, from plain torch in 64 bits

Inputs follow the repository's workloads: Gaussian random fields (horizontal length 8 cells,
vertical 3 levels) as ensemble members, a zone per water column, observations of single state
elements, most of them clustered on satellite-like tracks, the rest uniform.

Keys of a case. entry: the entry point; precision: fp64, mixed or refined (the mixed form with
FP64-accurate eigenpairs); f32: FP32 storage of the state and observation arrays; nx, ny, nz,
nvar: grid, levels and 3-D variables; surface: one more 2-D variable; N: members; m:
observations; tracks, track_len: number of tracks and the part of the grid's width each covers;
weight: gc (Gaspari-Cohn) or gauss; metric: cartesian (cell units) or spherical (degrees);
radius: localisation cut-off in cells; ragged: columns end at a bathymetry, land has none;
rough_r: error sd drawn from 0.05-0.5 instead of 0.1 of the variable's sd.
"""
import math

import numpy as np
import torch

import oak_gb300 as oak

DEV = "cuda"
_SD = (1.0, 0.2, 0.1, 0.1)
_SD_SURFACE = 0.05
_PREC = {"fp64": oak.PREC_FP64, "mixed": oak.PREC_MIXED, "refined": oak.PREC_MIXED_FP64EIG}
_EARTH = 6378137.0  # metres, the radius of the spherical metric
_DEG = 0.125        # grid step of the spherical cases, degrees
_LAT0 = 36.0        # southern edge of the spherical cases


def _case(name, entry, **kw):
    c = {"name": name, "entry": entry, "precision": "fp64", "f32": False, "nx": 100, "ny": 80,
         "nz": 1, "nvar": 1, "surface": False, "N": 30, "m": 500, "tracks": 8, "track_len": 1.0,
         "weight": "gc", "metric": "cartesian", "radius": 12.0, "ragged": False,
         "rough_r": False}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a global analysis of one 2-D field, every observation used once
        _case("global-small", "analysis"),
        # a global analysis of a 3-D state with many observations: one zone on the whole chip
        _case("global-wide", "analysis", nx=360, ny=180, nz=5, N=64, m=20_000, tracks=40),
        # a regional model's daily cycle: lon/lat grid with land, prepared once, run each day
        _case("regional-plan", "plan", nx=72, ny=54, nz=15, N=40, m=3_000, weight="gauss",
              metric="spherical", ragged=True, radius=9.0, tracks=6),
        # a small ensemble taken whole: H Ef, anomalies, local analysis, inflation, new members
        _case("cycle-ensemble", "ens", nx=120, ny=60, nz=20, N=30, m=5_500, tracks=13),
        # the plain form at the configuration the library is quoted on
        _case("local-fp64", "loc", nx=360, ny=180, nz=20, N=64, m=50_000, tracks=40),
        # the plain form with a wide ensemble and a column of five variables
        _case("columns-fp64-n100", "loc", nx=180, ny=90, nz=30, nvar=4, surface=True, N=100,
              m=12_500, tracks=2, track_len=0.25),
        # the mixed form at the quoted configuration, FP32 arrays
        _case("local-mixed", "loc", precision="mixed", f32=True, nx=360, ny=180, nz=20, N=64,
              m=50_000, tracks=40),
        # the batched five-variable configuration at half its grid
        _case("columns-mixed-n100", "loc", precision="mixed", f32=True, nx=360, ny=180, nz=30,
              nvar=4, surface=True, N=100, m=50_000, tracks=4, track_len=0.25),
        # the large two-variable configuration at a quarter of its grid
        _case("columns-mixed-n128", "loc", precision="mixed", f32=True, nx=360, ny=180, nz=50,
              nvar=2, N=128, m=62_500, tracks=4, track_len=0.25, radius=10.0, rough_r=True),
        # FP32 arrays with eigenpairs refined to FP64 accuracy
        _case("local-refined", "loc", precision="refined", f32=True, nx=180, ny=90, nz=20, N=64,
              m=12_500, tracks=20),
        # observation impact: the gradient of a cost over a 60 x 40 sub-region
        _case("adjoint", "adjoint", nx=360, ny=180, nz=20, N=64, m=50_000, tracks=40),
        # members to mean and anomalies and back, without an analysis: memory traffic only
        _case("convert", "convert", nx=360, ny=180, nz=20, N=64, m=50_000, tracks=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("analysis", "plan", "ens", "loc-fp64", "loc-fp64", "loc-fp64-wide",
                       "loc-mixed", "loc-mixed-wide", "loc-refined", "adjoint", "convert"))
    c = _case("", kind.split("-")[0])
    del c["name"]
    nx = _log_int(rng, 24, 330)
    c.update(nx=nx, ny=max(12, int(nx * rng.uniform(0.4, 0.55))), nz=_log_int(rng, 2, 22),
             N=rng.randint(12, 64))
    if kind == "analysis":
        c.update(nz=rng.randint(1, 5), N=rng.randint(12, 100))
    elif kind in ("loc-fp64-wide", "loc-mixed-wide"):
        if kind == "loc-fp64-wide":
            c.update(nx=min(nx, 150), ny=min(c["ny"], 75))
        surface = rng.random() < 0.5
        c.update(N=rng.randint(65, 128 if kind == "loc-mixed-wide" else 100),
                 nvar=4 if surface else 2, surface=surface, nz=rng.randint(8, 28),
                 track_len=0.25, rough_r=rng.random() < 0.5)
    elif kind == "loc-refined":
        c.update(nx=min(nx, 170), ny=min(c["ny"], 85))
    if kind.startswith("loc-mixed") or kind == "loc-refined":
        c.update(precision="mixed" if "mixed" in kind else "refined", f32=True)
    c["radius"] = round(rng.uniform(4.0, 12.0), 2)
    cells = c["nx"] * c["ny"]
    c["m"] = max(20, int(cells * math.exp(rng.uniform(math.log(0.08), math.log(0.75)))))
    if kind == "analysis":
        c["m"] = min(c["m"], 20_000)
    c["tracks"] = max(1, c["nx"] // (80 if c["track_len"] < 1.0 else 9))
    if kind in ("plan", "loc-fp64") and rng.random() < 0.5:
        c.update(weight="gauss", metric="spherical", ragged=True,
                 nx=min(c["nx"], 150), ny=min(c["ny"], 75))
        c["m"] = min(c["m"], c["nx"] * c["ny"])
    return c


# --------------------------------------------------------------------------------- inputs

def _fields(shape, lengths, count, gen, dtype):
    """`count` white-noise fields convolved with exp(-(r/l)^2) per axis, sd 1."""
    filt = None
    for ax, (size, length) in enumerate(zip(shape, lengths)):
        f = torch.fft.rfftfreq if ax == len(shape) - 1 else torch.fft.fftfreq
        k = f(size, device=DEV, dtype=dtype)
        t = torch.exp(-(math.pi * length * k) ** 2)
        t = t.reshape([-1 if i == ax else 1 for i in range(len(shape))])
        filt = t if filt is None else filt * t
    dims = tuple(range(1, len(shape) + 1))
    noise = torch.randn((count, *shape), generator=gen, device=DEV, dtype=dtype)
    out = torch.fft.irfftn(torch.fft.rfftn(noise, dim=dims) * filt, s=shape, dim=dims)
    return out / out.std(dim=dims, keepdim=True)


def _members(c, gen, dtype, mask, count):
    """(count, n) states: column by column, in a column variable by variable, level by level."""
    ny, nx, nz = c["ny"], c["nx"], c["nz"]
    n_col = c["nvar"] * nz + int(c["surface"])
    rows = []
    step = max(1, (1 << 28) // (ny * nx * max(n_col, nz) * 8))
    for k0 in range(0, count, step):
        k = min(step, count - k0)
        x = torch.empty((k, ny, nx, n_col), device=DEV, dtype=dtype)
        for v in range(c["nvar"]):
            x[..., v * nz:(v + 1) * nz] = _SD[v] * _fields((ny, nx, nz), (8.0, 8.0, 3.0), k, gen,
                                                           dtype)
        if c["surface"]:
            x[..., -1] = _SD_SURFACE * _fields((ny, nx), (8.0, 8.0), k, gen, dtype)
        x = x.reshape(k, -1)
        rows.append(x if mask is None else x[:, mask])
    return torch.cat(rows)


def _track_cells(c, m, rng):
    """Grid cells (i, j) under `tracks` great-circle-like tracks."""
    nx, ny, tracks = c["nx"], c["ny"], c["tracks"]
    t = rng.integers(0, tracks, m)
    slope = np.tan(np.deg2rad(rng.uniform(10.0, 80.0, tracks)))[t]
    start = rng.uniform(0.0, nx, tracks)[t]
    at = rng.uniform(0.0, (1.0 - c["track_len"]) * (nx - 1), tracks)[t]
    i = at + rng.uniform(0.0, c["track_len"] * (nx - 1), m)
    j = ny / 2 * (1.0 + np.arctan(slope * np.sin(2 * np.pi * (i - start) / nx)) / (np.pi / 2))
    return (np.clip(np.rint(i), 0, nx - 1).astype(np.int64),
            np.clip(np.rint(j), 0, ny - 1).astype(np.int64))


def _inputs(c, seed):
    """Everything the entry points take, in 64 bits or in FP32 storage, on the GPU."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    dtype = torch.float32 if c["f32"] else torch.float64
    ny, nx, nz, N, m = c["ny"], c["nx"], c["nz"], c["N"], c["m"]
    n_col = c["nvar"] * nz + int(c["surface"])
    depth = np.full(ny * nx, n_col, dtype=np.int64)
    mask = None
    if c["ragged"]:
        # the bathymetry belongs to the model: every seed's inputs have the same
        basin = torch.Generator(device=DEV)
        basin.manual_seed(7)
        sea = _fields((ny, nx), (8.0, 8.0), 1, basin, torch.float64)[0].reshape(-1)
        levels = torch.clamp(torch.round(n_col * (0.75 + 0.6 * sea)), 0, n_col).long()
        levels[torch.argmax(sea)] = n_col
        mask = (torch.arange(n_col, device=DEV)[None, :] < levels[:, None]).reshape(-1)
        depth = levels.cpu().numpy()
    first = np.cumsum(depth) - depth  # each column's first state element
    wet = np.flatnonzero(depth)

    E = _members(c, gen, dtype, mask, N + 1)
    truth, E = E[N], E[:N]

    on_track = int(round(0.7 * m))
    ti, tj = _track_cells(c, on_track, rng)
    col = np.concatenate([tj * nx + ti, wet[rng.integers(0, wet.size, m - on_track)]])
    dry = depth[col] == 0
    col[dry] = wet[rng.integers(0, wet.size, int(dry.sum()))]
    off = (rng.uniform(0.0, 1.0, m) * depth[col]).astype(np.int64)
    index = torch.as_tensor(first[col] + off, device=DEV)
    if c["surface"]:
        sd = np.array([*np.repeat(_SD[:c["nvar"]], nz), _SD_SURFACE])[off]
    else:
        sd = np.repeat(_SD[:c["nvar"]], nz)[off]
    err = rng.uniform(0.05, 0.5, m) if c["rough_r"] else 0.1 * sd
    yo = truth[index] + torch.as_tensor(rng.standard_normal(m) * err, device=DEV, dtype=dtype)

    x, y = col % nx, col // nx
    zx, zy = wet % nx, wet // nx
    if c["metric"] == "spherical":
        pos = [p * _DEG + o for p, o in ((x, 0.0), (y, _LAT0), (zx, 0.0), (zy, _LAT0))]
        reach = c["radius"] * _DEG * math.pi / 180.0 * _EARTH
    else:
        pos = [p.astype(np.float64) for p in (x, y, zx, zy)]
        reach = c["radius"]
    zone_pos = np.zeros((wet.size, 4))
    zone_pos[:, 0], zone_pos[:, 1] = pos[2], pos[3]
    f64 = dict(device=DEV, dtype=torch.float64)
    s = {
        "case": c, "truth": truth, "index": index, "yo": yo,
        "r": torch.as_tensor(err * err, device=DEV, dtype=dtype),
        "zone_size": torch.as_tensor(depth[wet].astype(np.int32), device=DEV),
        "zone_cell": torch.as_tensor(wet, device=DEV),
        "zone_pos": torch.as_tensor(zone_pos, **f64),
        "obs_pos": (torch.as_tensor(pos[0], **f64), torch.as_tensor(pos[1], **f64), None, None),
        "corr_len": torch.full((wet.size,), reach / 2.0, **f64),
        "max_len": torch.full((wet.size,), reach, **f64),
    }
    if c["entry"] in ("ens", "convert"):
        s["Ef"] = E.t()
        s["H_index"] = index.reshape(m, 1).contiguous()
        s["H_weight"] = torch.ones((m, 1), **f64)
        if c["entry"] == "convert":
            s["max_correction"] = torch.full((E.shape[1],), 0.5, **f64)
        return s
    mean = E.mean(0)
    E = (E - mean).div_(math.sqrt(N - 1.0))
    s.update(xf=mean, Sf=E.t(), Hxf=mean[index].contiguous(),
             HSf=E[:, index].contiguous().t())
    if c["entry"] == "adjoint":
        # J = mean squared (analysis mean - truth) over a sub-region a sixth (a ninth) as wide
        # (high): dJ/dxa at the forecast mean
        cell = s["zone_cell"]
        i0, j0, w, h = nx // 3, ny // 3, max(1, nx // 6), max(1, 2 * ny // 9)
        inside = ((cell % nx >= i0) & (cell % nx < i0 + w)
                  & (cell // nx >= j0) & (cell // nx < j0 + h))
        rows = torch.repeat_interleave(inside, s["zone_size"].long())
        s["seed"] = torch.where(rows, 2.0 * (mean - truth) / rows.sum(), torch.zeros_like(mean))
    return s


def _options(c):
    return dict(weight=oak.GASPARI_COHN if c["weight"] == "gc" else oak.GAUSS_CUTOFF,
                metric=oak.SPHERICAL if c["metric"] == "spherical" else oak.CARTESIAN)


def _geometry(s):
    return s["zone_pos"], s["obs_pos"], s["corr_len"], s["max_len"]


_INFLATION = 1.05


def prepare(case, seed):
    s = _inputs(case, seed)
    if case["entry"] == "plan":
        s["plan"] = oak.Plan(s["zone_size"], s["xf"], s["Hxf"], s["yo"], s["Sf"], s["HSf"],
                             s["r"], *_geometry(s), precision=_PREC[case["precision"]],
                             **_options(case))
    return s


def run(s):
    c = s["case"]
    entry = c["entry"]
    if entry == "analysis":
        return oak.analysis(s["xf"], s["Hxf"], s["yo"], s["Sf"], s["HSf"], s["r"])
    if entry == "plan":
        return s["plan"].execute()
    if entry == "ens":
        return oak.ens_loc_analysis(s["zone_size"], s["Ef"], s["H_index"], s["H_weight"],
                                    s["yo"], s["r"], *_geometry(s), inflation=_INFLATION,
                                    **_options(c))
    if entry == "adjoint":
        return oak.loc_analysis_adjoint(s["zone_size"], s["Hxf"], s["yo"], s["Sf"], s["HSf"],
                                        s["r"], *_geometry(s), s["seed"], inflation=_INFLATION,
                                        **_options(c))
    if entry == "convert":
        xf, Sf, Hxf, HSf = oak.ensemble_prologue(s["Ef"], s["H_index"], s["H_weight"])
        Ea = oak.ensemble_epilogue(s["truth"], xf, Sf, inflation=_INFLATION,
                                   max_correction=s["max_correction"])
        return xf, Sf, Hxf, HSf, Ea
    xa, Sa, _, nobs = oak.loc_analysis(s["zone_size"], s["xf"], s["Hxf"], s["yo"], s["Sf"],
                                       s["HSf"], s["r"], *_geometry(s), want_ampl=False,
                                       precision=_PREC[c["precision"]], **_options(c))
    return xa, Sa, nobs


# ----------------------------------------------------------------------- what a pass needs

def work(case):
    c = case
    N, m, b = c["N"], c["m"], 4 if c["f32"] else 8
    cells = c["nx"] * c["ny"]
    n = cells * (c["nvar"] * c["nz"] + int(c["surface"])) * (0.7 if c["ragged"] else 1.0)
    zones = cells * (0.85 if c["ragged"] else 1.0)
    obs = m * (N + 3) * b
    if c["entry"] == "analysis":
        return {"bytes": 2 * n * (N + 1) * b + obs,
                "flops": m * N * (N + 3.0) + 9.0 * N ** 3 + 2.0 * n * N * (N + 1)}
    if c["entry"] == "convert":
        return {"bytes": (3 * n * N + 4 * n + m * (N + 5)) * b, "flops": 5.0 * n * N}
    p = min(m, math.pi * c["radius"] ** 2 * m / cells)
    gram = p * N * (N + 3.0)
    if c["entry"] == "adjoint":
        part = 1.0 / 27.0
        return {"bytes": n * b + part * n * N * b + obs + 2 * m * b,
                "flops": part * zones * (gram + N ** 3 / 3.0 + 8.0 * p * N) + 4 * part * n * N}
    # a zone's square-root transform counts as a symmetric eigensolve with vectors
    return {"bytes": 2 * n * (N + 1) * b + obs + zones * 60,
            "flops": zones * (gram + 9.0 * N ** 3) + 2.0 * n * N * (N + 1)}


# ------------------------------------------------------------------------ the same, in 64 bits

def _locfun(r):
    near = (((-r / 4.0 + 0.5) * r + 0.625) * r - 5.0 / 3.0) * r * r + 1.0
    s = torch.clamp(r, min=1.0)
    far = ((((s / 12.0 - 0.5) * s + 0.625) * s + 5.0 / 3.0) * s - 5.0) * s + 4.0 - 2.0 / (3.0 * s)
    return torch.where(r <= 1.0, near, torch.where(r <= 2.0, far, torch.zeros_like(r)))


def _locfun_slope(r):
    near = (((-1.25 * r + 2.0) * r + 1.875) * r - 10.0 / 3.0) * r
    s = torch.clamp(r, min=1.0)
    far = ((((5.0 / 12.0 * s - 2.0) * s + 1.875) * s + 10.0 / 3.0) * s - 5.0) + 2.0 / (3.0 * s * s)
    return torch.where(r <= 1.0, near, torch.where(r <= 2.0, far, torch.zeros_like(r)))


def _distances(s, zones):
    ox, oy = s["obs_pos"][0][None, :], s["obs_pos"][1][None, :]
    zx, zy = s["zone_pos"][zones, 0][:, None], s["zone_pos"][zones, 1][:, None]
    if s["case"]["metric"] == "cartesian":
        dx, dy = zx - ox, zy - oy
        return torch.sqrt(dx * dx + dy * dy)
    rad = math.pi / 180.0
    a, b, d = oy * rad, zy * rad, (zx - ox) * rad
    t = torch.sin(b) * torch.sin(a) + torch.cos(b) * torch.cos(a) * torch.cos(d)
    return _EARTH * torch.arccos(torch.clamp(t, -1.0, 1.0))


def _weights(s, zones):
    """(weight, selected) of every observation for the zones given."""
    d = _distances(s, zones)
    t = d / s["corr_len"][zones][:, None]
    inside = d <= s["max_len"][zones][:, None]
    if s["case"]["weight"] == "gauss":
        return torch.exp(-t * t), inside, t
    w = _locfun(t)
    return w, inside & (w != 0.0), t


def _groups(s, zones, width):
    """Zones in groups of alike observation counts: (zones, observation indices, weights as
    zero-padded rows, scaled distances)."""
    m = s["yo"].shape[0]
    step = max(1, (1 << 27) // m)
    counts = torch.cat([_weights(s, zones[k:k + step])[1].sum(1)
                        for k in range(0, zones.numel(), step)])
    order = torch.argsort(counts)
    zones, counts = zones[order], counts[order].cpu().numpy()
    k = int(np.searchsorted(counts, 1))
    while k < counts.size:
        fit = 1
        while (k + fit < counts.size and fit < step
               and (fit + 1) * int(counts[k + fit]) * width < (1 << 27)):
            fit += 1
        z, p = zones[k:k + fit], int(counts[k + fit - 1])
        w, sel, t = _weights(s, z)
        at, q = torch.nonzero(sel, as_tuple=True)
        count = sel.sum(1)
        slot = torch.arange(at.numel(), device=DEV) - (torch.cumsum(count, 0) - count)[at]
        idx = torch.zeros((fit, p), device=DEV, dtype=torch.long)
        idx[at, slot] = q
        filled = torch.arange(p, device=DEV)[None, :] < count[:, None]
        w = torch.where(filled, torch.gather(w, 1, idx), 0.0)
        yield z, idx, w, torch.gather(t, 1, idx)
        k += fit


def _inverse(A):
    """Inverses of symmetric positive definite matrices."""
    L = torch.linalg.cholesky(A)
    L = torch.linalg.solve_triangular(L, torch.eye(A.shape[-1], device=DEV, dtype=A.dtype)
                                      .expand_as(A), upper=False)
    return L.mT @ L


def _roots(A):
    """A^(1/2) and A^(-1/2) of symmetric positive definite matrices: the eigenvectors for a
    few, the Denman-Beavers iteration with scaling (a batched eigensolver takes milliseconds a
    matrix) for many."""
    if A.shape[0] <= 128:
        lam, U = torch.linalg.eigh(A)
        root = torch.sqrt(torch.clamp(lam, min=1.0))[:, None, :]
        return (U * root) @ U.mT, (U / root) @ U.mT
    N = A.shape[-1]
    Y, Z = A, torch.eye(N, device=DEV, dtype=A.dtype).expand_as(A)
    for _ in range(20):
        iY, iZ = _inverse(Y), _inverse(Z)
        # the Frobenius scaling of each step; 1 near convergence
        mu = torch.sqrt((iY.flatten(1).norm(dim=1) * iZ.flatten(1).norm(dim=1))
                        / (Y.flatten(1).norm(dim=1) * Z.flatten(1).norm(dim=1))).sqrt()
        mu = torch.where((mu - 1.0).abs() < 1e-2, 1.0, mu)[:, None, None]
        Yn, Zn = 0.5 * (mu * Y + iZ / mu), 0.5 * (mu * Z + iY / mu)
        step = float(((Zn - Z).flatten(1).norm(dim=1) / Zn.flatten(1).norm(dim=1)).max())
        Y, Z = 0.5 * (Yn + Yn.mT), 0.5 * (Zn + Zn.mT)
        if step < 1e-13:
            break
    return Y, Z


def _transform(G, g):
    """Amplitudes (I + G)^-1 g and the mean-preserving transform (I + G)^(-1/2) Omega."""
    N = G.shape[-1]
    root, T = _roots(G + torch.eye(N, device=DEV, dtype=G.dtype))
    ampl = (T @ (T @ g[..., None]))[..., 0]
    v = root.sum(-1)
    v = v / v.norm(dim=-1, keepdim=True)
    # Omega = P_v P_w + (1 - s_v) v w^T: P_x = I - u u^T / (1 + |x_N|), u = x + sign(x_N) e_N
    w = torch.full_like(v, N ** -0.5)

    def reflect(A, x):
        sign = torch.where(x[..., -1] >= 0, 1.0, -1.0)
        u = x.clone()
        u[..., -1] += sign
        return A - (A @ u[..., None]) * u[..., None, :] / (1.0 + x[..., -1].abs())[..., None, None]

    sign = torch.where(v[..., -1] >= 0, 1.0, -1.0)
    extra = (1.0 - sign)[..., None] * (T @ v[..., None])[..., 0]
    return ampl, reflect(reflect(T, v), w) + extra[..., None] * w[..., None, :]


def _local_exact(s, xf, Sf, Hxf, HSf):
    zones = torch.arange(s["zone_size"].numel(), device=DEV)
    size = s["zone_size"].long()
    first = torch.cumsum(size, 0) - size
    xa, Sa = xf.double().clone(), Sf.double().t().contiguous()  # Sa as (N, n)
    HS, d, r = HSf.double(), s["yo"].double() - Hxf.double(), s["r"].double()
    N = HS.shape[1]
    for z, idx, w, _ in _groups(s, zones, N):
        X = HS[idx] * (w / torch.sqrt(r[idx]))[..., None]
        g = (HS[idx] * (w * w / r[idx] * d[idx])[..., None]).sum(1)
        ampl, T = _transform(X.mT @ X, g)
        del X
        rows = first[z][:, None] + torch.arange(int(size[z].max()), device=DEV)[None, :]
        keep = torch.arange(rows.shape[1], device=DEV)[None, :] < size[z][:, None]
        at = torch.where(keep, rows, first[z][:, None])
        old = Sa[:, at.reshape(-1)].t().reshape(z.numel(), -1, N)
        xa[rows[keep]] += (old @ ampl[..., None])[..., 0][keep]
        Sa[:, rows[keep]] = (old @ T)[keep].t()
    return xa, Sa.t()


def _adjoint_exact(s):
    infl = _INFLATION
    size = s["zone_size"].long()
    first = torch.cumsum(size, 0) - size
    owner = torch.repeat_interleave(torch.arange(size.numel(), device=DEV), size)
    zones = torch.unique(owner[s["seed"] != 0.0])
    HS, d, r = s["HSf"], s["yo"] - s["Hxf"], s["r"]
    N = HS.shape[1]
    dyo, dr = torch.zeros_like(d), torch.zeros_like(r)
    dlen = dinfl = 0.0
    eye = torch.eye(N, device=DEV, dtype=torch.float64)
    for z, idx, w, t in _groups(s, zones, N):
        h, dq, rq = HS[idx], d[idx], r[idx]
        c = w * w / rq
        A = eye + infl * infl * (h.mT @ (h * c[..., None]))
        g = (h * (c * dq)[..., None]).sum(1)
        rows = first[z][:, None] + torch.arange(int(size[z].max()), device=DEV)[None, :]
        keep = torch.arange(rows.shape[1], device=DEV)[None, :] < size[z][:, None]
        at = torch.where(keep, rows, first[z][:, None])
        seed = torch.where(keep, s["seed"][at], 0.0)
        b = infl * (s["Sf"][at].mT @ seed[..., None])[..., 0]
        sol = torch.linalg.solve(A, torch.stack([b, infl * g], -1))
        t1 = infl * (h @ sol[..., :1])[..., 0]
        t2 = infl * (h @ sol[..., 1:])[..., 0]
        dc = t1 * (dq - t2)
        dyo.index_add_(0, idx.reshape(-1), (c * t1).reshape(-1))
        dr.index_add_(0, idx.reshape(-1), (-dc * c / rq).reshape(-1))
        slope = 2.0 * t * t * w if s["case"]["weight"] == "gauss" else -t * _locfun_slope(t)
        dlen += float((dc * 2.0 * w / rq * slope).sum())
        dinfl += float(((b * sol[..., 1]).sum() + (c * t1 * (dq - 2.0 * t2)).sum()) / infl)
    return dyo, dr, dlen, dinfl


def exact(case, seed):
    s = _inputs(case, seed)
    entry, N = case["entry"], case["N"]
    if entry == "adjoint":
        return _adjoint_exact(s)
    if entry in ("ens", "convert"):
        Ef = s["Ef"]
        xf = Ef.mean(1)
        Sf = (Ef - xf[:, None]) / math.sqrt(N - 1.0)
        Hxf, HSf = xf[s["index"]], Sf[s["index"]]
        if entry == "convert":
            old = s["truth"]
            xa = torch.minimum(torch.maximum(xf, old - s["max_correction"]),
                               old + s["max_correction"])
            return xf, Sf, Hxf, HSf, xa[:, None] + _INFLATION * math.sqrt(N - 1.0) * Sf
        xa, Sa = _local_exact(s, xf, Sf, Hxf, HSf)
        return xa[:, None] + _INFLATION * math.sqrt(N - 1.0) * Sa
    if entry == "analysis":
        X = s["HSf"] / torch.sqrt(s["r"])[:, None]
        g = s["HSf"].t() @ ((s["yo"] - s["Hxf"]) / s["r"])
        ampl, T = _transform((X.t() @ X)[None], g[None])
        return s["xf"] + s["Sf"] @ ampl[0], s["Sf"] @ T[0], ampl[0]
    xa, Sa = _local_exact(s, s["xf"], s["Sf"], s["Hxf"], s["HSf"])
    return xa, Sa, None
