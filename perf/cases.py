"""Workloads of the framework's public entry points, for timing and for comparing builds.

Kinds of case:

``analysis`` / ``synthesis``
    The Gauss-Legendre transform of ``make_sht("cuda", ...)``: one NumPy grid or spectrum (``io =
    "host"``, what an unmodified reference solver does per transform), one CUDA tensor in the dense
    layout (``"dense"``, what the segmented guess and the rate read-out do) or a list of CUDA tensors
    in the packed layout (``"packed"``, what an ensemble does).
``solve``
    One time step of one solve (``SeaLevelSolver`` / ``OptSeaLevelSolver``), NumPy ice in, topography
    and radial displacement out: what the forward and outer drivers do each step.
``batch``
    One time step of a ``SolverBatch``, ice in device memory, every member's sea-level change out:
    what the ensemble runner and the serving loop do each step.
``guess``
    The segmented initial-topography guess before an outer run, ice states on the device.

Solves step through a short cycle of ice states (growing, then shrinking), so that a pass can be
repeated for as long as it takes.
"""

import functools
import math

import numpy as np
import torch

SQRT2_LEGACY = 1.41421356   # the transform's own literal, part of its convention
PI = math.pi
NSTATES = 6                 # ice states of a solve's cycle: 0, 1, .. 5, 4, .. 1, 0, 1, ..
MODES = 8
SHEETS = ((60.0, 265.0, 20.0, 3500.0), (63.0, 15.0, 12.0, 2500.0), (-90.0, 0.0, 22.0, 3000.0))


def listed():
    return [
        # the smallest grid in use (the reference's small test case), one transform of a NumPy grid as
        # an unmodified reference solver asks for it: latency of the call
        {"name": "analysis_64_host", "kind": "analysis", "precision": "fp64", "nlat": 64, "nlon": 128, "lmax": 63,
         "fields": 1, "io": "host"},
        # one full-size field on the device, each direction: a driver's own transforms around the step
        {"name": "analysis_512", "kind": "analysis", "precision": "fp64", "nlat": 512, "nlon": 1024, "lmax": 511,
         "fields": 1, "io": "dense"},
        {"name": "synthesis_512", "kind": "synthesis", "precision": "fp64", "nlat": 512, "nlon": 1024, "lmax": 511,
         "fields": 1, "io": "dense"},
        # an odd number of fields on a ragged grid (latitudes no multiple of 32, truncation below the
        # grid's): post-processing of a few output fields
        {"name": "analysis_180x512_x7", "kind": "analysis", "precision": "fp64", "nlat": 180, "nlon": 512, "lmax": 170,
         "fields": 7, "io": "packed"},
        # a full launch of the mixed-precision transforms, each direction: the ensemble's transforms
        {"name": "mixed_analysis_512_x32", "kind": "analysis", "precision": "mixed", "nlat": 512, "nlon": 1024,
         "lmax": 511, "fields": 32, "io": "packed"},
        {"name": "mixed_synthesis_512_x32", "kind": "synthesis", "precision": "mixed", "nlat": 512, "nlon": 1024,
         "lmax": 511, "fields": 32, "io": "packed"},
        # a partly filled launch on a truncated grid
        {"name": "mixed_synthesis_192_x5", "kind": "synthesis", "precision": "mixed", "nlat": 192, "nlon": 512,
         "lmax": 170, "fields": 5, "io": "packed"},
        # the smallest solve, the reference's plain form: latency of a step
        {"name": "solve_64", "kind": "solve", "precision": "fp64", "nlat": 64, "nlon": 128, "lmax": 63, "dt": 1.0,
         "form": "plain"},
        # a glacial-cycle solve at the production degree in the default precision
        {"name": "solve_512", "kind": "solve", "precision": "fp64", "nlat": 512, "nlon": 1024, "lmax": 511,
         "dt": 200.0, "form": "opt"},
        # the benchmark's ensemble step
        {"name": "batch_512_x32", "kind": "batch", "precision": "mixed", "nlat": 512, "nlon": 1024, "lmax": 511,
         "dt": 200.0, "members": 32},
        # a half-full batch of the serving mix's smallest degree
        {"name": "batch_128_x12", "kind": "batch", "precision": "mixed", "nlat": 128, "nlon": 256, "lmax": 127,
         "dt": 200.0, "members": 12},
        # the outer driver's start: thirteen ice states of two glacial cycles
        {"name": "guess_256", "kind": "guess", "nlat": 256, "nlon": 512, "lmax": 255, "states": 13},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, precision):
    """A grid and a truncation: latitudes even (mixed precision: a multiple of 64), longitudes a power
    of two, the degree at most what both carry."""
    if precision == "mixed":
        nlat = 64 * _log_int(rng, 1, 8)
    else:
        nlat = 2 * _log_int(rng, 24, 256)
    nlon = 8
    while nlon < 1.5 * nlat:
        nlon *= 2
    full = min(nlat - 1, nlon // 2 - 1)
    lmax = full if rng.random() < 0.5 else rng.randint(2 * full // 3, full)
    return {"nlat": nlat, "nlon": nlon, "lmax": lmax}


def draw(rng):
    kind = rng.choice(("analysis", "synthesis", "analysis", "synthesis", "solve", "batch", "batch", "guess"))
    precision = rng.choice(("fp64", "mixed"))
    if kind in ("analysis", "synthesis"):
        c = {"kind": kind, "precision": precision, **_grid(rng, precision), "fields": 1,
             "io": rng.choice(("host", "dense", "packed", "packed"))}
        if c["io"] == "packed":
            c["fields"] = _log_int(rng, 1, 32)
        return c
    if kind == "solve":
        return {"kind": kind, "precision": precision, **_grid(rng, precision), "dt": rng.choice((1.0, 10.0, 200.0)),
                "form": rng.choice(("plain", "opt"))}
    if kind == "batch":
        precision = "mixed" if rng.random() < 0.75 else "fp64"
        most = 32 if precision == "mixed" else 8
        return {"kind": kind, "precision": precision, **_grid(rng, precision), "dt": rng.choice((1.0, 200.0)),
                "members": _log_int(rng, 2, most)}
    return {"kind": kind, **_grid(rng, "fp64"), "states": rng.randint(7, 17)}


# ------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=16)
def _nodes(nlat):
    """Gauss nodes (north to south) and weights."""
    x, w = np.polynomial.legendre.leggauss(nlat)
    return x[::-1].copy(), w[::-1].copy()


def _sphere(nlat, nlon):
    """Unit vectors of the grid points, (3, nlat, nlon), and the row weights."""
    x, w = _nodes(nlat)
    z = torch.from_numpy(x).cuda()[:, None]
    s = torch.sqrt(1.0 - z * z)
    lon = torch.arange(nlon, dtype=torch.float64, device="cuda")[None, :] * (2.0 * PI / nlon)
    return torch.stack([s * torch.cos(lon), s * torch.sin(lon), z.expand(nlat, nlon)]), torch.from_numpy(w).cuda()


def _smooth(pos, rng, kmax, waves=40):
    """A smooth random field on the sphere: plane waves of falling amplitude."""
    k = np.exp(rng.uniform(0.0, math.log(max(kmax, 2.0)), waves))
    d = rng.standard_normal((waves, 3))
    d *= (k / np.linalg.norm(d, axis=1))[:, None]
    ph, amp = rng.uniform(0.0, 2.0 * PI, waves), k ** -1.0
    f = torch.zeros(pos.shape[1:], dtype=torch.float64, device="cuda")
    for i in range(waves):
        f += amp[i] * torch.cos(d[i, 0] * pos[0] + d[i, 1] * pos[1] + d[i, 2] * pos[2] + ph[i])
    return f


def _mm(f):
    return torch.round(f * 1000.0) / 1000.0


def _topography(pos, w, rng, lmax):
    """70 % ocean by area, mean ocean depth 4000 m, highest land 3000 m, whole millimetres; a marine
    bed of -500 to -1500 m under the south polar cap."""
    g = _smooth(pos, rng, min(lmax, 48))
    area = w[:, None].expand_as(g).reshape(-1)
    v, order = torch.sort(g.reshape(-1), stable=True)
    cum = torch.cumsum(area[order], 0) / area.sum()
    g = g - v[int((cum < 0.70).sum())]
    sea = g < 0
    depth = (w[:, None] * g * sea).sum() / (w[:, None] * sea).sum()
    topo = torch.where(sea, g * (-4000.0 / depth), g * (3000.0 / g.max()))
    colat = torch.arccos((-pos[2]).clamp(-1.0, 1.0)) * (180.0 / PI)
    return _mm(torch.where(colat < 22.0, -500.0 - 1000.0 * (1.0 - colat / 22.0), topo))


def _sheets(pos):
    """Ice thickness of the three sheets at full extent."""
    ice = torch.zeros(pos.shape[1:], dtype=torch.float64, device="cuda")
    for lat, lon, radius, height in SHEETS:
        a, o = math.radians(lat), math.radians(lon)
        c = pos[0] * (math.cos(a) * math.cos(o)) + pos[1] * (math.cos(a) * math.sin(o)) + pos[2] * math.sin(a)
        d = torch.arccos(c.clamp(-1.0, 1.0)) * (180.0 / PI) / radius
        ice = torch.maximum(ice, height * (1.0 - d.clamp(max=1.0) ** (4.0 / 3.0)).clamp(min=0.0) ** 0.375)
    return ice


def _amplitude(k, dt):
    """Extent of the ice at state k of a cycle: 200-year steps of a 90-kyr growth, shorter steps faster."""
    return 0.85 + (0.0022 if dt >= 100.0 else 0.0008) * k


def _state_of(i):
    """Ice state of pass i = 1, 2, ...: 1 2 3 4 5 4 3 2 1 0 1 ..."""
    p = i % (2 * (NSTATES - 1))
    return p if p < NSTATES else 2 * (NSTATES - 1) - p


def _spectrum(rng, lmax):
    """Dense coefficients [l, m] of a field of some hundred metres, m = 0 real."""
    l = np.arange(lmax + 1)
    amp = 300.0 * np.maximum(l, 1.0) ** -1.5
    c = (rng.standard_normal((lmax + 1, lmax + 1)) + 1j * rng.standard_normal((lmax + 1, lmax + 1))) * amp[:, None]
    c[:, 0] = c[:, 0].real
    return np.tril(c)


def _packed_index(lmax):
    """Rows l and columns m of the packed order (order-major: m = 0 with l = 0 .. L, then m = 1, ...)."""
    m, l = np.triu_indices(lmax + 1)
    return l, m


def _transform_input(case, seed):
    """The grids (fields, nlat, nlon) on the device, or the dense spectra on the host."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "synthesis":
        return np.stack([_spectrum(rng, case["lmax"]) for _ in range(case["fields"])])
    pos, _ = _sphere(case["nlat"], case["nlon"])
    grids = []
    for _ in range(case["fields"]):
        # a sea-level field that ends at the coast, as the step analyses it
        f, coast = _smooth(pos, rng, min(case["lmax"], 60), 24), _smooth(pos, rng, 12, 12)
        grids.append(100.0 * f * (coast < 0.5))
    return torch.stack(grids)


def _prepare_transform(case, seed):
    from slevolve_b200 import make_sht

    sht = make_sht("cuda", case["nlat"], case["nlon"], case["lmax"], precision=case["precision"])
    x = _transform_input(case, seed)
    ana = case["kind"] == "analysis"
    if case["io"] == "host":
        return {"case": case, "sht": sht, "x": x[0].cpu().numpy() if ana else x[0]}
    if case["io"] == "dense":
        x = x[0].contiguous() if ana else torch.from_numpy(x[0]).cuda()
        shape = (case["lmax"] + 1,) * 2 if ana else (case["nlat"], case["nlon"])
        out = torch.empty(shape, dtype=torch.complex128 if ana else torch.float64, device="cuda")
        return {"case": case, "sht": sht, "x": x, "out": out}
    n = case["fields"]
    if ana:
        out = torch.empty((n, sht.ncoef), dtype=torch.complex128, device="cuda")
    else:
        l, m = _packed_index(case["lmax"])
        x = torch.from_numpy(np.ascontiguousarray(x[:, l, m])).cuda()
        out = torch.empty((n, case["nlat"], case["nlon"]), dtype=torch.float64, device="cuda")
    return {"case": case, "sht": sht, "x": [x[f] for f in range(n)], "out": out, "outs": [out[f] for f in range(n)]}


def _run_transform(s):
    from slevolve_b200 import _lib

    sht, ana, io = s["sht"], s["case"]["kind"] == "analysis", s["case"]["io"]
    if io == "host":
        return sht.analysis(s["x"]) if ana else sht.synthesis(s["x"])
    if io == "dense":
        return sht.analysis(s["x"], out=s["out"]) if ana else sht.synthesis(s["x"], out=s["out"])
    if ana:
        sht.analysis_device(s["x"], s["outs"], layout=_lib.LAYOUT_PACKED)
    else:
        sht.synthesis_device(s["x"], s["outs"], layout=_lib.LAYOUT_PACKED)
    return s["out"]


def _prepare_solve(case, seed):
    from slevolve_b200 import OptSeaLevelSolver, SeaLevelSolver, SyntheticEarth, make_sht

    rng = np.random.default_rng(seed)
    nlat, nlon, lmax, dt = case["nlat"], case["nlon"], case["lmax"], case["dt"]
    pos, w = _sphere(nlat, nlon)
    topo, sheets = _topography(pos, w, rng, lmax), _sheets(pos)
    ice = [_mm(_amplitude(k, dt) * sheets).cpu().numpy() for k in range(NSTATES)]
    sht = make_sht("cuda", nlat, nlon, lmax, precision=case["precision"])
    love = SyntheticEarth(lmax, MODES, int(rng.integers(1 << 30)))
    kw = {"norder": lmax, "dt": dt, "precision": case["precision"]}
    if case["form"] == "plain":
        slv = SeaLevelSolver(sht, love, topo.cpu().numpy(), ice[0], **kw)
    else:
        slv = OptSeaLevelSolver(sht, love, topo.cpu().numpy(), ice[0], opt={"dsl", "diag"}, inner="extrap", **kw)
    return {"case": case, "solver": slv, "ice": ice, "pass": 0}


def _run_solve(s):
    s["pass"] += 1
    rec = s["solver"].step(s["ice"][_state_of(s["pass"])])
    return {"tgrid": rec["tgrid"], "R": rec["R"], "numiter": rec["numiter"], "ocean_area": rec["ocean_area"],
            "gmslc_ocn": rec["gmslc_ocn"], "ice_volume": rec["ice_volume"], "il": rec["il"], "mm": rec["mm"]}


def _prepare_batch(case, seed):
    from slevolve_b200 import SyntheticEarth
    from slevolve_b200.batch import SolverBatch

    rng = np.random.default_rng(seed)
    nlat, nlon, lmax, dt, n = case["nlat"], case["nlon"], case["lmax"], case["dt"], case["members"]
    pos, w = _sphere(nlat, nlon)
    topo, sheets = _topography(pos, w, rng, lmax), _sheets(pos)
    earths = [SyntheticEarth(lmax, MODES, int(rng.integers(1 << 30)), relax_scale=float(np.exp(rng.uniform(-1.1, 1.1))))
              for _ in range(min(n, 4))]
    amps = [1.0] + [float(a) for a in rng.uniform(0.5, 1.5, n - 1)]
    bt = SolverBatch(nlat, nlon, lmax, n, max_modes=MODES, precision=case["precision"], opt=("dsl", "diag"), inner="extrap")
    ice = [{b: _mm(amps[b] * _amplitude(k, dt) * sheets) for b in range(n)} for k in range(NSTATES)]
    for b in range(n):
        bt.load(b, earths[b % len(earths)], topo, ice[0][b], dt)
    out = torch.empty((n, nlat, nlon), dtype=torch.float64, device="cuda")
    return {"case": case, "batch": bt, "ice": ice, "out": out, "outs": [out[b] for b in range(n)], "pass": 0}


def _run_batch(s):
    s["pass"] += 1
    bt = s["batch"]
    infos = bt.step(s["ice"][_state_of(s["pass"])])
    for b, o in enumerate(s["outs"]):
        bt.get(b, "deltasl", out=o)
    info = [infos[b] for b in range(len(s["outs"]))]
    return {"deltasl": s["out"], "numiter": np.array([i["numiter"] for i in info]),
            "ocean_area": np.array([i["ocean_area"] for i in info]),
            "gmslc_ocn": np.array([i["gmslc_ocn"] for i in info]),
            "ice_volume": np.array([i["ice_volume"] for i in info])}


def _prepare_guess(case, seed):
    from slevolve_b200 import SyntheticEarth, make_sht

    rng = np.random.default_rng(seed)
    nlat, nlon, lmax, n = case["nlat"], case["nlon"], case["lmax"], case["states"]
    pos, w = _sphere(nlat, nlon)
    topo, sheets = _topography(pos, w, rng, lmax), _sheets(pos)
    t = np.linspace(0.0, 1.0, n)
    amp = 0.35 + 0.65 * np.abs(np.sin(2.2 * PI * t)) * (1.0 - 0.4 * t)
    ice = [_mm(float(a) * sheets) for a in amp]
    return {"case": case, "topo": topo, "ice": ice, "love": SyntheticEarth(lmax, MODES, int(rng.integers(1 << 30))),
            "sht": make_sht("cuda", nlat, nlon, lmax)}


def _run_guess(s):
    from slevolve_b200.init_topo import segmented_guess

    t0, info = segmented_guess(s["topo"], s["ice"], s["love"], s["case"]["lmax"], 10.0, sht=s["sht"])
    return {"T0": t0, "c": info["c"], "iters": info["iters"]}


_KINDS = {"analysis": (_prepare_transform, _run_transform), "synthesis": (_prepare_transform, _run_transform),
          "solve": (_prepare_solve, _run_solve), "batch": (_prepare_batch, _run_batch),
          "guess": (_prepare_guess, _run_guess)}


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return _KINDS[state["case"]["kind"]][1](state)


def work(case):
    """One read of each input and one write of each output; the Legendre sums as 4 flops per
    (coefficient, latitude of one hemisphere)."""
    ng, nc = case["nlat"] * case["nlon"], (case["lmax"] + 1) * (case["lmax"] + 2) // 2
    leg = 4.0 * (case["nlat"] // 2) * nc
    if case["kind"] in ("analysis", "synthesis"):
        coefs = nc if case["io"] == "packed" else (case["lmax"] + 1) ** 2
        return {"bytes": case["fields"] * (8.0 * ng + 16.0 * coefs), "flops": case["fields"] * leg}
    if case["kind"] == "guess":
        # some eight iterations of three operators, each an analysis and a synthesis
        return {"bytes": 8.0 * ng * (case["states"] + 2), "flops": 48 * leg}
    # the ice in, topography and two displacement grids out, the modal state through; about five
    # iterations of a synthesis and two analyses, and three transforms around them
    n = case.get("members", 1)
    return {"bytes": n * (32.0 * ng + 2 * MODES * 16.0 * nc), "flops": n * 18 * leg}


# ------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """The transforms in plain torch FP64 (the recursion over degrees for all orders at once); None
    for whole solves."""
    if case["kind"] not in ("analysis", "synthesis"):
        return None
    nlat, nlon, lmax, ana = case["nlat"], case["nlon"], case["lmax"], case["kind"] == "analysis"
    nh, nm, x = nlat // 2, lmax + 1, _transform_input(case, seed)
    nodes, weights = _nodes(nlat)
    mu = torch.from_numpy(nodes[:nh].copy()).cuda()
    m = torch.arange(nm, device="cuda")
    odd_m = (m % 2 == 1)[:, None]
    if ana:
        f = torch.fft.rfft(x, dim=2)[:, :, :nm] * (torch.from_numpy(weights).cuda()[None, :, None] / nlon)
        north, south = f[:, :nh].transpose(1, 2), f[:, nh:].flip(1).transpose(1, 2)
        plus, minus = north + south, north - south
        by_parity = [torch.where(odd_m, minus, plus), torch.where(odd_m, plus, minus)]
        dense = torch.zeros((case["fields"], nm, nm), dtype=torch.complex128, device="cuda")
    else:
        c = torch.from_numpy(x).cuda() * SQRT2_LEGACY
        sums = [torch.zeros((case["fields"], nm, nh), dtype=torch.complex128, device="cuda") for _ in range(2)]
    mf = m.to(torch.float64)
    a, b = torch.zeros((nm, nh), dtype=torch.float64, device="cuda"), torch.zeros((nm, nh), dtype=torch.float64, device="cuda")
    prod = torch.full((nh,), 0.5, dtype=torch.float64, device="cuda")
    for l in range(nm):
        if l:
            eps = torch.sqrt((l * l - mf * mf).clamp(min=0.0) / (4.0 * l * l - 1.0))[:l, None]
            eps1 = torch.sqrt(((l - 1.0) ** 2 - mf * mf).clamp(min=0.0) / (4.0 * (l - 1.0) ** 2 - 1.0))[:l, None]
            new = torch.zeros_like(b)
            new[:l] = (mu * b[:l] - eps1 * a[:l]) / eps
            a, b = b, new
            prod = prod * (1.0 - mu * mu) * (2.0 * l + 1.0) / (2.0 * l)
        b[l] = torch.sqrt(prod)
        if ana:
            dense[:, l, : l + 1] = (b[: l + 1] * by_parity[l % 2][:, : l + 1]).sum(2) / SQRT2_LEGACY
        else:
            sums[l % 2][:, : l + 1] += c[:, l, : l + 1, None] * b[: l + 1]
    if ana:
        if case["io"] == "packed":
            li, mi = _packed_index(lmax)
            return dense[:, torch.from_numpy(li).cuda(), torch.from_numpy(mi).cuda()]
        out = dense[0]
        return out.cpu().numpy() if case["io"] == "host" else out
    even = torch.where(odd_m, sums[1], sums[0])   # sums of even and of odd l - m
    odd = torch.where(odd_m, sums[0], sums[1])
    rows = torch.cat([(even + odd).transpose(1, 2), (even - odd).transpose(1, 2).flip(1)], dim=1)
    full = torch.zeros((case["fields"], nlat, nlon // 2 + 1), dtype=torch.complex128, device="cuda")
    full[:, :, :nm] = rows
    full[:, :, 0] = full[:, :, 0].real.to(torch.complex128)
    g = torch.fft.irfft(full, n=nlon, dim=2) * nlon
    if case["io"] == "packed":
        return g
    return g[0].cpu().numpy() if case["io"] == "host" else g[0]
