"""Workloads the engine is timed on, through its public entry points.

A case is a dict of plain values: `kind` names the entry point, the rest its sizes and options.
`listed()` holds one case per kind of work a user has the engine do, at the sizes of this
repository's configurations, tests and benchmark; `draw(rng)` makes more of the same ranges.

The specimens are crystal slabs with a small static strain drawn from the seed, the frozen-phonon
seed follows the input seed, and the calls run on one simulator handle, as a program that simulates
many specimens keeps it.  Forward and gradient calls on caller potentials keep the potential on the
GPU (the ABI's on-device arguments); the simulator calls take host atoms and return host arrays.

`exact` restates the simulation in 64 bits with numpy and torch: phonon displacements, slicing,
radial splines, probe, transmission, Fresnel propagation, lens, detectors and the loss gradient
(autograd).  Decisions made on float32 values (slice membership, aperture and detector masks) use
the same float32 arithmetic as the definition of the simulation.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import cudaem_b200 as cb
from cudaem_b200 import _abi as abi

A_STO, A_SI = 3.905, 5.431
BASIS = {
    "sto": (A_STO, [38, 22, 8, 8, 8], [(0, 0, 0), (.5, .5, .5), (.5, .5, 0), (.5, 0, .5), (0, .5, .5)]),
    "si": (A_SI, [14] * 8, [(0, 0, 0), (.5, .5, 0), (.5, 0, .5), (0, .5, .5), (.25, .25, .25), (.75, .75, .25),
                            (.75, .25, .75), (.25, .75, .75)]),
}
R_MIN, R_MAX, N_R = 0.01, 3.0, 128


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a quick look at a 128^2 pattern (the smoke configuration)
        dict(name="cbed_128", kind="cbed", crystal="si", cells_x=2, cells_y=2, cells_z=4, nx=128, ny=128, dz=1.358,
             E0=300.0, aper=0.020, nconf=2),
        # one HRTEM image on a plane wave: a single 512^2 wave, bound by each slice's latency
        dict(name="hrtem_512", kind="tem", crystal="sto", cells_x=10, cells_y=10, cells_z=20, nx=512, ny=512,
             dz=A_STO / 2, E0=200.0, aper=0.020, c10=-100.0, c30=1.0e7, nconf=1),
        # a through-focus series of complex waves with a few phonon configurations, small grid
        dict(name="series_256_wave", kind="series", crystal="sto", cells_x=5, cells_y=5, cells_z=9, nx=256, ny=256,
             dz=A_STO / 2, E0=200.0, aper=0.020, c10=-60.0, c30=1.0e7, nconf=3, n_defocus=7, wave=True),
        # thickness series: the filtered intensity after every slice, 256^2
        dict(name="thickness_256", kind="thickness", crystal="sto", cells_x=6, cells_y=6, cells_z=12, nx=256, ny=256,
             dz=A_STO / 2, E0=200.0, aper=0.020, nconf=2, det=0.040),
        # the headline workload: frozen-phonon CBED, 1024^2, 240 slices, 8 configurations
        dict(name="cbed_1024_8conf", kind="cbed", crystal="si", cells_x=16, cells_y=16, cells_z=60, nx=1024, ny=1024,
             dz=1.358, E0=300.0, aper=0.020, nconf=8),
        # the largest grid: 2048^2, periodic potentials, an odd number of configurations
        dict(name="cbed_2048_wrap", kind="cbed", crystal="si", cells_x=30, cells_y=30, cells_z=8, nx=2048, ny=2048,
             dz=1.358, E0=200.0, aper=0.015, nconf=3, wrap=True),
        # ADF STEM: one configuration of a 16 x 16 scan at 1024^2, 50 slices
        dict(name="stem_1024_16x16", kind="stem", crystal="sto", cells_x=16, cells_y=16, cells_z=25, nx=1024, ny=1024,
             dz=A_STO / 2, E0=200.0, aper=0.022, nconf=1, scan_x=16, scan_y=16, n_det=1),
        # a ragged scan on a rectangular grid with three detectors and phonons
        dict(name="stem_512x256_13x7", kind="stem", crystal="sto", cells_x=10, cells_y=5, cells_z=9, nx=512, ny=256,
             dz=1.71, E0=120.0, aper=0.025, nconf=3, scan_x=13, scan_y=7, n_det=3),
        # differentiable STEM on potentials held on the GPU: the forward model and its gradient
        dict(name="forward_512_16", kind="forward", crystal="sto", cells_x=10, cells_y=10, cells_z=40, nx=512, ny=512,
             dz=A_STO / 2, E0=200.0, aper=0.022, c10=-20.0, c30=1.0e4, n_probe=16, n_det=1),
        dict(name="backward_512_16", kind="backward", crystal="sto", cells_x=10, cells_y=10, cells_z=40, nx=512, ny=512,
             dz=A_STO / 2, E0=200.0, aper=0.022, c10=-20.0, c30=1.0e4, n_probe=16, n_det=1, ckpt=8),
        # projected potentials of one phonon configuration, left on the GPU
        dict(name="potential_512", kind="potential", crystal="sto", cells_x=10, cells_y=10, cells_z=40, nx=512, ny=512,
             dz=A_STO / 2, E0=200.0, aper=0.022, nconf=1),
        # an uneven batch: 20 simulations of mixed grids (256^2..2048^2) and slice counts in one call
        dict(name="uneven_20", kind="many", n_sim=20, mix=42, max_slices=200),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


MOST_PIXELS = 3.0e9   # wave pixels x slices of a drawn case (the largest listed one has 1.3e10)


def draw(rng):
    kind = rng.choice(["cbed", "cbed", "tem", "series", "thickness", "stem", "stem", "forward", "backward",
                       "potential", "many"])
    if kind == "many":
        return dict(kind="many", n_sim=rng.randint(2, 14), mix=rng.randint(0, 1 << 30),
                    max_slices=_logint(rng, 12, 120))
    crystal = rng.choice(["sto", "si"])
    a = BASIS[crystal][0]
    sizes = [128, 256, 512, 1024, 2048]
    nx = rng.choice(sizes)
    ny = nx if rng.random() < 0.6 else rng.choice(sizes)
    cx = max(2, min(40, int(round(nx * rng.uniform(0.06, 0.1) / a))))
    cy = max(2, min(40, int(round(ny * rng.uniform(0.06, 0.1) / a))))
    c = dict(kind=kind, crystal=crystal, cells_x=cx, cells_y=cy, nx=nx, ny=ny, dz=round(rng.uniform(1.1, 3.0), 3),
             E0=round(rng.uniform(80.0, 300.0), 1), aper=round(rng.uniform(0.010, 0.030), 4))
    waves = 1
    if kind in ("cbed", "tem", "series", "thickness"):
        c["nconf"] = _logint(rng, 1, 12)
        waves = c["nconf"]
    if kind in ("tem", "series", "forward", "backward"):
        c["c10"], c["c30"] = round(rng.uniform(-200.0, 0.0), 2), 10.0 ** rng.uniform(4, 7)
    if kind in ("cbed", "tem", "series"):
        c["wave"] = rng.random() < 0.3
    if kind in ("cbed", "tem", "stem", "potential"):
        c["wrap"] = rng.random() < 0.4
    if kind == "series":
        c["n_defocus"] = rng.randint(1, 11)
    if kind == "thickness":
        c["det"] = round(rng.uniform(0.010, 0.040), 4)
    if kind == "stem":
        c["nconf"], c["n_det"] = rng.randint(1, 3), rng.randint(1, 4)
        c["scan_x"], c["scan_y"] = _logint(rng, 1, 24), _logint(rng, 1, 24)
        waves = c["nconf"] * c["scan_x"] * c["scan_y"]
    if kind == "potential":
        c["nconf"] = 1
    if kind in ("forward", "backward"):
        c["n_probe"], c["n_det"] = _logint(rng, 1, 24), rng.randint(1, 3)
        waves = 4 * c["n_probe"]
        if kind == "backward":
            c["ckpt"] = rng.randint(1, 12)
    slices = _logint(rng, 3, 240)
    if kind == "thickness":
        slices = min(slices, max(3, int(1.2e7 / (nx * ny))))
    slices = max(1, min(slices, int(MOST_PIXELS / (nx * ny * waves))))
    c["cells_z"] = max(1, int(round(slices * c["dz"] / a)))
    return c


# ---------------------------------------------------------------------------
# inputs: specimens and parameters as plain values (shared by prepare and exact)
# ---------------------------------------------------------------------------
def _slab(crystal, cx, cy, cz, sigma, seed):
    a, Z, frac = BASIS[crystal]
    cells = np.stack(np.meshgrid(np.arange(cx), np.arange(cy), np.arange(cz), indexing="ij"), -1).reshape(-1, 1, 3)
    pos = ((cells + np.asarray(frac)[None]) * a).reshape(-1, 3)
    n = pos.shape[0]
    rng = np.random.default_rng([seed, 11])
    pos[:, :2] += rng.normal(0.0, 0.01, (n, 2))   # static strain in the plane
    f = np.float32
    return dict(Z=np.tile(np.asarray(Z, np.int32), n // len(Z)), x=pos[:, 0].astype(f), y=pos[:, 1].astype(f),
                z=pos[:, 2].astype(f), sigma=np.full(n, sigma, f), occ=np.ones(n, f))


def _problems(case, seed):
    """The simulations of one call: a list of (parameters, atoms) as plain dicts."""
    if case["kind"] == "many":
        mix = np.random.default_rng(case["mix"])
        out = []
        for i in range(case["n_sim"]):
            n = int(mix.choice([256, 512, 1024, 2048]))
            crystal = "sto" if mix.integers(0, 2) else "si"
            a = BASIS[crystal][0]
            per = 2 if crystal == "sto" else 4
            nsl = int(mix.integers(min(10, case["max_slices"]), case["max_slices"] + 1))
            cells = max(2, int(round(n * 0.08 / a)))
            sub = dict(kind="cbed", crystal=crystal, cells_x=cells, cells_y=cells, cells_z=max(1, -(-nsl // per)),
                       nx=n, ny=n, dz=a / per, E0=float(mix.uniform(80, 300)), aper=float(mix.uniform(0.010, 0.030)),
                       nconf=1)
            out += _problems(sub, seed * 1009 + i)
        return out
    crystal = case["crystal"]
    a = BASIS[crystal][0]
    sigma = 0.08 if crystal == "sto" else 0.075
    atoms = _slab(crystal, case["cells_x"], case["cells_y"], case["cells_z"], sigma, seed)
    rng = np.random.default_rng([seed, 7])
    lx, ly = case["cells_x"] * a, case["cells_y"] * a
    p = dict(nx=case["nx"], ny=case["ny"], lx=lx, ly=ly, dz=case["dz"], E0=case["E0"], nconf=case.get("nconf", 0),
             pn_seed=int(rng.integers(1, 1 << 30)), wrap=bool(case.get("wrap")), wave=bool(case.get("wave")),
             aper=case["aper"], c10=case.get("c10", 0.0), c30=case.get("c30", 0.0),
             iw_x=lx / 2 + float(rng.uniform(-0.5, 0.5)) * a, iw_y=ly / 2 + float(rng.uniform(-0.5, 0.5)) * a,
             det=[])
    if case["kind"] == "thickness":
        p["det"] = [(0.0, case["det"])]
    elif "n_det" in case:
        p["det"] = [(0.060, 0.200), (0.0, 0.012), (0.025, 0.060), (0.012, 0.025)][:case["n_det"]]
        # small grids do not reach 200 mrad: keep the annuli inside the band limit
        gmax = min(case["nx"] / 2 / lx, case["ny"] / 2 / ly) * 2 / 3
        lim = math.asin(min(0.9, gmax * _physics(case["E0"])[0]))
        p["det"] = [(min(i, 0.4 * lim), min(o, lim)) for i, o in p["det"]]
    if case["kind"] == "stem":
        step = 0.2
        p.update(scan_x=case["scan_x"], scan_y=case["scan_y"], step=step,
                 scan_x0=p["iw_x"] - case["scan_x"] * step / 2, scan_y0=p["iw_y"] - case["scan_y"] * step / 2)
    if case["kind"] in ("forward", "backward"):
        p["xy"] = np.array([p["iw_x"], p["iw_y"]]) + rng.uniform(-a, a, (case["n_probe"], 2))
        if case["kind"] == "backward":
            # measured intensities: a few per cent of the beam on every detector
            frac = rng.uniform(0.02, 0.2, (case["n_probe"], len(p["det"])))
            p["target"] = (frac * float(_probe_mask(p).sum()) * (p["nx"] * p["ny"]) ** 2).astype(np.float32)
    return [(p, atoms)]


_SIM = {"tem": abi.MS_SIM_HRTEM, "series": abi.MS_SIM_HRTEM, "thickness": abi.MS_SIM_HRTEM, "cbed": abi.MS_SIM_CBED,
        "many": abi.MS_SIM_CBED, "potential": abi.MS_SIM_CBED}
_ONE = None


def _simulator():
    global _ONE
    if _ONE is None:
        _ONE = cb.ThicknessSimulator()
    return _ONE


def _fptr(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_float))


def prepare(case, seed):
    kind = case["kind"]
    jobs = []
    for p, at in _problems(case, seed):
        q = cb.MultisliceParams(
            simulation_type=_SIM.get(kind, abi.MS_SIM_STEM), nx=p["nx"], ny=p["ny"], lx=p["lx"], ly=p["ly"],
            dz=p["dz"], E0=p["E0"], pn_seed=p["pn_seed"], pot_wrap=int(p["wrap"]), iw_x=p["iw_x"], iw_y=p["iw_y"],
            phonon_model=abi.MS_PHONON_FROZEN if p["nconf"] else abi.MS_PHONON_STILL, pn_nconf=max(1, p["nconf"]),
            data_record=abi.MS_RECORD_WAVE if p["wave"] else abi.MS_RECORD_INTENSITY)
        lens = q.obj_lens if kind in ("tem", "series", "thickness") else q.cond_lens
        lens.outer_aper_ang, lens.c10, lens.c30 = p["aper"], p["c10"], p["c30"]
        q.set_detectors(p["det"])
        if kind == "stem":
            q.scan_nx, q.scan_ny, q.scan_dx, q.scan_dy = p["scan_x"], p["scan_y"], p["step"], p["step"]
            q.scan_x0, q.scan_y0 = p["scan_x0"], p["scan_y0"]
        else:
            q.scan_nx = q.scan_ny = 1
        jobs.append((q, cb.Atoms(**at)))
    s = dict(kind=kind, sim=_simulator(), jobs=jobs)
    p, at = _problems(case, seed)[0] if kind != "many" else (None, None)
    if kind == "series":
        s["defocus"] = _defocus(case)
    if kind in ("forward", "backward"):
        V, z0 = _guess(p, at)
        s.update(V=V.float().contiguous(), z0=z0, xy=np.ascontiguousarray(p["xy"]), n_det=len(p["det"]))
        if kind == "backward":
            jobs[0][0].ckpt_interval = case["ckpt"]
            s.update(target=p["target"], gV=torch.empty_like(s["V"]))
        else:
            s["I"] = np.empty((len(p["xy"]), len(p["det"])), np.float32)
    if kind == "potential":
        ns = C.c_int()
        q, atoms = jobs[0][0].c(), jobs[0][1].c()
        ctx = s["sim"].ctx
        ctx.check(cb.lib().ms_projected_potential(ctx.handle, C.byref(q), C.byref(atoms), 1, None, 0, 0, C.byref(ns)))
        s["V"] = torch.empty((ns.value, p["ny"], p["nx"]), dtype=torch.float32, device="cuda")
    return s


def run(s):
    kind, sim = s["kind"], s["sim"]
    params, atoms = s["jobs"][0]
    if kind == "cbed":
        return _image(sim.executionCBED(params, atoms))
    if kind == "tem":
        return _image(sim.executionTEM(params, atoms))
    if kind == "series":
        return _image(sim.executionTEMDefocusSeries(params, atoms, s["defocus"]))
    if kind == "thickness":
        return sim.run(params, atoms).thickness_frames
    if kind == "stem":
        return sim.executionSTEM(params, atoms).stem_intensity
    if kind == "many":
        return [o.image_intensity for o in sim.executionMany(s["jobs"])[0]]
    p, ctx, L = params.c(), sim.ctx, cb.lib()
    if kind == "potential":
        ns, a = C.c_int(), atoms.c()
        ctx.check(L.ms_projected_potential(ctx.handle, C.byref(p), C.byref(a), 1, _fptr(s["V"]), s["V"].numel(), 1,
                                           C.byref(ns)))
        return s["V"]
    V, xy = s["V"], s["xy"]
    xyp = xy.ctypes.data_as(C.POINTER(C.c_double))
    if kind == "forward":
        ctx.check(L.ms_stem_forward_potential(ctx.handle, C.byref(p), _fptr(V), V.shape[0], 1, s["z0"], xyp, len(xy),
                                              s["I"].ctypes.data_as(C.POINTER(C.c_float))))
        return s["I"]
    loss, g10, g30 = C.c_double(), C.c_double(), C.c_double()
    ctx.check(L.ms_stem_backward(ctx.handle, C.byref(p), _fptr(V), V.shape[0], 1, s["z0"], xyp, len(xy),
                                 s["target"].ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss), _fptr(s["gV"]),
                                 C.byref(g10), C.byref(g30)))
    return {"loss": loss.value, "dV": s["gV"], "dC10": g10.value, "dC30": g30.value}


def _image(o):
    return o.image_intensity if o.image_intensity is not None else [o.image_real, o.image_imag]


def _defocus(case):
    return np.linspace(-120.0, 150.0, case["n_defocus"])


# ---------------------------------------------------------------------------
# what one pass cannot do without: the atoms (or the potential) in, the result out, and the
# transforms, products and spline values of the definition
# ---------------------------------------------------------------------------
def work(case):
    if case["kind"] == "many":
        mix = np.random.default_rng(case["mix"])
        total = dict(bytes=0.0, flops=0.0)
        for _ in range(case["n_sim"]):
            n = int(mix.choice([256, 512, 1024, 2048]))
            crystal = "sto" if mix.integers(0, 2) else "si"
            per = 2 if crystal == "sto" else 4
            nsl = int(mix.integers(min(10, case["max_slices"]), case["max_slices"] + 1))
            mix.uniform(80, 300), mix.uniform(0.010, 0.030)
            cells = max(2, int(round(n * 0.08 / BASIS[crystal][0])))
            w = work(dict(kind="cbed", crystal=crystal, cells_x=cells, cells_y=cells, cells_z=max(1, -(-nsl // per)),
                          nx=n, ny=n, dz=BASIS[crystal][0] / per, nconf=1))
            total = {k: total[k] + w[k] for k in total}
        return total
    kind = case["kind"]
    a, Z, _ = BASIS[case["crystal"]]
    nx, ny = case["nx"], case["ny"]
    N = nx * ny
    n_atoms = case["cells_x"] * case["cells_y"] * case["cells_z"] * len(Z)
    S = max(1, int(case["cells_z"] * a / case["dz"]))
    fft = 5.0 * N * math.log2(N)
    conf = max(1, case.get("nconf", 1))
    disc = math.pi * R_MAX ** 2 * (nx / (case["cells_x"] * a)) * (ny / (case["cells_y"] * a))
    splines = conf * n_atoms * disc * 10.0
    step = 2 * fft + 12.0 * N
    out = {"cbed": N, "tem": N, "series": N * case.get("n_defocus", 1), "thickness": N * S, "potential": N * S,
           "stem": case.get("scan_x", 1) * case.get("scan_y", 1) * case.get("n_det", 1),
           "forward": case.get("n_probe", 1), "backward": N * S}[kind]
    if case.get("wave"):
        out *= 2
    nbytes = 4.0 * out + 24.0 * n_atoms
    if kind == "potential":
        return dict(bytes=nbytes, flops=splines)
    if kind in ("forward", "backward"):
        k = case["n_probe"] * S
        if kind == "forward":
            return dict(bytes=4.0 * (out + N * S), flops=k * step)
        return dict(bytes=4.0 * (out + N * S), flops=k * (2 * step + 8.0 * N))
    waves = conf * case.get("scan_x", 1) * case.get("scan_y", 1)
    flops = splines + waves * S * step
    if kind == "series":
        flops += conf * case["n_defocus"] * (fft + 6.0 * N)
    if kind == "thickness":
        flops += waves * S * (fft + 3.0 * N)
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------------------
# the same simulations in 64 bits (numpy and torch only)
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _physics(E0):
    h, me, qe, c = 6.62607015e-34, 9.1093837015e-31, 1.602176634e-19, 299792458.0
    E = E0 * 1e3
    g = 1 + qe * E / (me * c * c)
    lam = h / math.sqrt(2 * me * qe * E * (1 + qe * E / (2 * me * c * c)))
    return lam * 1e10, 2 * math.pi * g * me * qe * lam / h ** 2 * 1e-10


def _freq(n, L):
    k = np.where(np.arange(n) < n // 2, np.arange(n), np.arange(n) - n)
    return k / L, k.astype(np.float32) * (np.float32(1.0) / np.float32(L))


def _g2_float(p):
    fx, fy = _freq(p["nx"], p["lx"])[1], _freq(p["ny"], p["ly"])[1]
    return (fx * fx)[None, :] + (fy * fy)[:, None]


def _threshold(ang, lam):
    g = np.float32(math.sin(ang) / lam)
    return g * g


def _probe_mask(p):
    return _g2_float(p) < _threshold(p["aper"], _physics(p["E0"])[0])


def _annuli(p):
    lam, g2 = _physics(p["E0"])[0], _g2_float(p)
    return [torch.from_numpy((_threshold(i, lam) <= g2) & (g2 <= _threshold(o, lam))).to(_dev()) for i, o in p["det"]]


def _mix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _gauss(seed, conf, n, stream):
    """Two unit Gaussians per atom: SplitMix64 keyed by (seed, configuration, atom, stream), polar method."""
    one = np.array([seed], np.uint64)
    key = _mix64(_mix64(_mix64(one) ^ np.uint64(conf)) ^ ((np.arange(n, dtype=np.uint64) << np.uint64(2)) | np.uint64(stream)))
    g0, g1, left = np.zeros(n), np.zeros(n), np.arange(n)
    for it in range(64):
        k = key[left]
        u = (_mix64(k + np.uint64(2 * it)) >> np.uint64(11)).astype(np.float64)
        v = (_mix64(k + np.uint64(2 * it + 1)) >> np.uint64(11)).astype(np.float64)
        u, v = 2.0 * ((u + 0.5) * 2.0 ** -53) - 1.0, 2.0 * ((v + 0.5) * 2.0 ** -53) - 1.0
        s = u * u + v * v
        ok = (s < 1.0) & (s > 0.0)
        f = np.sqrt(-2.0 * np.log(s[ok]) / s[ok])
        g0[left[ok]], g1[left[ok]] = u[ok] * f, v[ok] * f
        left = left[~ok]
        if not left.size:
            break
    return g0, g1


def _displaced(p, at, conf):
    x, y, z = at["x"], at["y"], at["z"]
    if conf:
        gx, gy = _gauss(p["pn_seed"], conf, len(x), 0)
        gz, _ = _gauss(p["pn_seed"], conf, len(x), 1)
        s = at["sigma"].astype(np.float64)
        x, y, z = x + (s * gx).astype(np.float32), y + (s * gy).astype(np.float32), z + (s * gz).astype(np.float32)
    return x, y, z


def _slices(p, z, top):
    """Slice planes (float32) and every atom's slice; `top`: planes counted from the highest atom down."""
    f = np.float32
    lo, hi, dz, eps = z.min(), z.max(), f(p["dz"]), f(1e-4)
    nv = int(np.floor(((hi - lo) + eps) / dz)) + 2
    i = np.arange(nv).astype(f)
    b = (hi + f(2) * eps) - i[::-1] * dz if top else (lo - f(2) * eps) + i * dz
    s = np.searchsorted(b, z, side="right") - 1
    s = np.where((z >= b[0]) & (z < b[-1]), s, np.where((z == b[-1]) & (z == hi), nv - 2, -1))
    return b, s, nv - 1


def _spline(Z):
    """Radial spline of the projected potential in R^2: nodes and the four coefficients per node."""
    aTF = 0.88534138 * 0.529177210903 * float(Z) ** (-1.0 / 3.0)
    R = torch.tensor([R_MIN * (R_MAX / R_MIN) ** (i / (N_R - 1)) for i in range(N_R)], dtype=torch.float64)
    R[-1] = R_MAX
    V, dV = torch.zeros_like(R), torch.zeros_like(R)
    for al, be in ((0.35, 0.3), (0.55, 1.2), (0.10, 6.0)):
        cl, k = 14.399645478425668 * Z * al, be / aTF
        V = V + 2.0 * cl * torch.special.modified_bessel_k0(k * R)
        dV = dV - cl * k * torch.special.modified_bessel_k1(k * R) / R
    R2 = R * R
    tap0 = (0.85 * R_MAX) ** 2
    w = math.pi / (2.0 * (R_MAX ** 2 - tap0))
    t = R2 > tap0
    c, s = torch.cos(w * (R2 - tap0)), torch.sin(w * (R2 - tap0))
    dV = torch.where(t, dV * c - w * V * s, dV)
    V = torch.where(t, V * c, V)
    h = 1.0 / (R2[1:] - R2[:-1])
    m, n = (V[1:] - V[:-1]) * h, dV[:-1] + dV[1:]
    co = torch.stack([V[:-1], dV[:-1], (3.0 * m - n - dV[:-1]) * h, (n - 2.0 * m) * h * h])
    return R2, co


def _potential(p, at, conf, top):
    """sigma V of every slice in 64 bits [S][ny][nx], the first slice's middle, the slice count."""
    dev = _dev()
    x, y, z = _displaced(p, at, conf)
    b, sl, S = _slices(p, z, top)
    nx, ny = p["nx"], p["ny"]
    dx, dy = p["lx"] / nx, p["ly"] / ny
    V = torch.zeros(S * ny * nx, dtype=torch.float64, device=dev)
    kx, ky = int(R_MAX / dx) + 2, int(R_MAX / dy) + 2
    ox, oy = torch.arange(-kx, kx + 1, device=dev), torch.arange(-ky, ky + 1, device=dev)
    per = max(1, int(2.0e7 / (len(ox) * len(oy))))
    sig = _physics(p["E0"])[1]
    for Z in np.unique(at["Z"]):
        R2, co = (t.to(dev) for t in _spline(int(Z)))
        pick = np.flatnonzero((at["Z"] == Z) & (sl >= 0))
        for i in range(0, len(pick), per):
            q = pick[i:i + per]
            xa = torch.from_numpy(x[q].astype(np.float64)).to(dev)
            ya = torch.from_numpy(y[q].astype(np.float64)).to(dev)
            sa = torch.from_numpy(sl[q].astype(np.int64)).to(dev)
            ix = torch.round(xa / dx).long()[:, None] + ox
            iy = torch.round(ya / dy).long()[:, None] + oy
            r2 = ((iy * dy - ya[:, None]) ** 2)[:, :, None] + ((ix * dx - xa[:, None]) ** 2)[:, None, :]
            use = r2 < R_MAX ** 2
            if p["wrap"]:
                ix, iy = ix % nx, iy % ny
            else:
                use = use & ((ix >= 0) & (ix < nx))[:, None, :] & ((iy >= 0) & (iy < ny))[:, :, None]
            at_px = ((sa[:, None, None] * ny + iy[:, :, None]) * nx + ix[:, None, :])[use]
            r2 = r2[use]
            k = (torch.searchsorted(R2, r2, right=True) - 1).clamp_(0, N_R - 2)
            d = r2 - R2[k]
            V.index_add_(0, at_px, sig * (((co[3][k] * d + co[2][k]) * d + co[1][k]) * d + co[0][k]))
    z0 = float(np.float32(0.5 * float(b[0] + b[1])))
    return V.view(S, ny, nx), z0, S


def _grids(p):
    gx = torch.from_numpy(_freq(p["nx"], p["lx"])[0]).to(_dev())[None, :]
    gy = torch.from_numpy(_freq(p["ny"], p["ly"])[0]).to(_dev())[:, None]
    return gx, gy, gx ** 2 + gy ** 2


def _propagator(p):
    lam = _physics(p["E0"])[0]
    _, _, g2 = _grids(p)
    gl = 2.0 * min((p["nx"] // 2) / p["lx"], (p["ny"] // 2) / p["ly"]) / 3.0
    alpha = math.log(99.0) / ((gl + 0.25) ** 2 - gl ** 2)
    amp = 1.0 / (p["nx"] * p["ny"]) / (1.0 + torch.exp(alpha * (g2 - gl ** 2)))
    return torch.polar(amp, -math.pi * lam * p["dz"] * g2)


def _lens(p, c10, c30, mask):
    lam = _physics(p["E0"])[0]
    _, _, g2 = _grids(p)
    chi = -math.pi * lam * c10 * g2 - math.pi * lam ** 3 / 2.0 * c30 * g2 ** 2
    m = torch.from_numpy(mask).to(_dev()).double()
    return torch.complex(m * torch.cos(chi), m * torch.sin(chi))


def _probe(p, x, y, lens):
    gx, gy, _ = _grids(p)
    ph = -2.0 * math.pi * (x * gx + y * gy)
    return torch.fft.ifft2(lens * torch.complex(torch.cos(ph), torch.sin(ph)), norm="forward")


def _exit(V, P, psi):
    """The exit wave in reciprocal space."""
    for s in range(V.shape[0]):
        psi = torch.fft.fft2(psi * torch.polar(torch.ones_like(V[s]), V[s]))
        if s < V.shape[0] - 1:
            psi = torch.fft.ifft2(P * psi, norm="forward")
    return psi


def _guess(p, at):
    """The current estimate of the potential in a reconstruction: float32 values, kept in 64 bits."""
    V, z0, _ = _potential(p, at, 0, False)
    return (0.8 * V).float().double(), z0


def _exact_one(kind, case, p, at):
    confs = list(range(1, p["nconf"] + 1)) or [0]
    P = _propagator(p) if kind != "potential" else None
    w = 1.0 / len(confs)
    N = p["nx"] * p["ny"]
    ones = torch.ones((p["ny"], p["nx"]), dtype=torch.complex128, device=_dev())
    out = None
    add = lambda acc, v: v if acc is None else acc + v  # noqa: E731
    if kind == "potential":
        return _potential(p, at, 1, False)[0]
    if kind in ("forward", "backward"):
        V, z0 = _guess(p, at)
        ann = _annuli(p)
        c10, c30 = (torch.tensor(p[k], dtype=torch.float64, device=_dev()) for k in ("c10", "c30"))
        if kind == "backward":
            V, c10, c30 = (t.requires_grad_() for t in (V, c10, c30))
        loss, rows = 0.0, []
        for i, (x, y) in enumerate(p["xy"]):
            W = _exit(V, P, _probe(p, x, y, _lens(p, c10 + z0, c30, _probe_mask(p))))
            a2 = W.real ** 2 + W.imag ** 2
            I = torch.stack([(a2 * m).sum() for m in ann])
            if kind == "backward":
                l = ((I - torch.from_numpy(p["target"][i]).double().to(_dev())) ** 2).sum()
                l.backward()
                loss += float(l.detach())
            rows.append(I.detach())
        if kind == "forward":
            return torch.stack(rows)
        return {"loss": torch.tensor(loss, dtype=torch.float64), "dV": V.grad, "dC10": c10.grad, "dC30": c30.grad}
    for conf in confs:
        if kind == "stem":
            V, z0, _ = _potential(p, at, conf, False)
            ann = _annuli(p)
            lens = _lens(p, p["c10"] + z0, p["c30"], _probe_mask(p))
            I = torch.zeros((len(ann), p["scan_y"], p["scan_x"]), dtype=torch.float64, device=_dev())
            for iy in range(p["scan_y"]):
                for ix in range(p["scan_x"]):
                    W = _exit(V, P, _probe(p, p["scan_x0"] + ix * p["step"], p["scan_y0"] + iy * p["step"], lens))
                    a2 = W.real ** 2 + W.imag ** 2
                    for d, m in enumerate(ann):
                        I[d, iy, ix] = (a2 * m).sum()
            out = add(out, w * I)
            continue
        top = kind in ("tem", "series", "thickness")
        V, z0, S = _potential(p, at, conf, top)
        if kind == "cbed":
            W = _exit(V, P, _probe(p, p["iw_x"], p["iw_y"], _lens(p, p["c10"] + z0, p["c30"], _probe_mask(p))))
            r = torch.fft.fftshift(torch.stack([W.real, W.imag]), dim=(1, 2)) if p["wave"] else \
                torch.fft.fftshift(W.real ** 2 + W.imag ** 2)
            out = add(out, w * r)
        elif kind == "thickness":
            frames = _slices(p, at["z"], True)[2]
            if out is None:
                out = torch.zeros((frames, p["ny"], p["nx"]), dtype=torch.float64, device=_dev())
            psi, m = ones, _annuli(p)[0]
            for s in range(frames):
                F = P * torch.fft.fft2(psi * torch.polar(torch.ones_like(V[s]), V[s]) if s < S else psi)
                f = torch.fft.ifft2(F * m, norm="forward")
                out[s] += w * (f.real ** 2 + f.imag ** 2)
                psi = torch.fft.ifft2(F, norm="forward")
        else:
            W = _exit(V, P, ones)
            imgs = []
            for df in (_defocus(case) if kind == "series" else [0.0]):
                im = torch.fft.ifft2(W * _lens(p, p["c10"] + df, p["c30"], _probe_mask(p)), norm="forward")
                imgs.append(torch.stack([im.real, im.imag]) if p["wave"] else im.real ** 2 + im.imag ** 2)
            r = torch.stack(imgs, dim=1 if p["wave"] else 0)
            if kind == "tem":
                r = r[:, 0] if p["wave"] else r[0]
            out = add(out, w * r)
    return [out[0], out[1]] if p["wave"] else out


def exact(case, seed):
    kind = case["kind"]
    res = [_exact_one("cbed" if kind == "many" else kind, case, p, at) for p, at in _problems(case, seed)]
    return res if kind == "many" else res[0]
