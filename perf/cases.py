"""Timed cases of the scattering-amplitude path, one for each way a program uses the library.

Every case goes through the public Python mirror of the C ABI (`sassena_gb300.abi`). A state
holds what such a program keeps between calls: the plan with its staged trajectory, the
q-vectors and class factors, the batch, the network. Trajectories are seeded random walks,
generated on the GPU with the densities, step lengths and q ranges of the benchmark workloads
(`sassena_gb300/synth.py`).

Results of the FP64 form are returned as the library gives them (complex128). The FP32 form's
results have FP32 accuracy (its phases, amplitudes and power spectra are FP32) and are kept as
complex64, as a program that chose that form would store them.
"""
import math

import numpy as np
import torch

from sassena_gb300 import abi, synth

COHERENT = [-3.7390, 6.6460, 9.3600, 5.8030, 2.8470]  # H C N O S, fm
INCOHERENT = [25.274, 0.089, 1.990, 0.080, 0.236]
RATIOS = [50, 30, 8, 10, 2]
MASSES = [1.008, 12.011, 14.007, 15.999, 32.06]
AXIS = (0.0, 0.0, 1.0)


def _phase(name, na, nf, nq, nm, precision, scattering="all", dsp="autocorrelate", qmin=0.05, qmax=3.0,
           density=0.08, scan="linear", factors="neutron"):
    return dict(name=name, kind="phase", na=na, nf=nf, nq=nq, nm=nm, precision=precision, scattering=scattering,
                dsp=dsp, qmin=qmin, qmax=qmax, density=density, scan=scan, factors=factors)


def listed():
    return [
        # A small selection at a few q, host frames in and results out: what a script that walks
        # over many selections or windows calls again and again. Latency and launches count.
        dict(_phase("small_call_fp64", 200, 50, 4, 12, "fp64", qmin=0.2, qmax=2.5), kind="call"),
        # Coherent S(q,t) in the driver's default precision (FP64), a modest solution.
        _phase("coherent_fp64", 3000, 250, 12, 60, "fp64"),
        # The headline: coherent S(q,t) of 10,000 atoms, 1,024 frames, 20 shells x 500 directions.
        _phase("coherent_fp32", 10000, 1024, 20, 500, "fp32"),
        # Static X-ray I(q) of a 100,000-atom system: many finely spaced shells, form factors that
        # fall off with q, square instead of a correlation. The largest job.
        _phase("static_xray_fp32", 100000, 16, 100, 250, "fp32", dsp="square", qmin=0.01, qmax=0.5, density=0.075,
               factors="xray"),
        # Incoherent F(q,t): one series per atom and direction, 128 frames; the fast form and the
        # default one.
        _phase("incoherent_fp32", 1000, 128, 10, 100, "fp32", scattering="self", qmin=0.1, qmax=2.0, density=0.037),
        _phase("incoherent_fp64", 1000, 128, 10, 100, "fp64", scattering="self", qmin=0.1, qmax=2.0, density=0.037),
        # A long trajectory of a small system (padded length 32,768: transforms through HBM).
        _phase("long_series_fp32", 1500, 12000, 8, 40, "fp32"),
        # Independent systems of uneven size with unevenly spaced shells, one graph-captured batch.
        dict(name="batch_uneven_fp32", kind="batch", nsys=8, na_min=500, na_max=6000, nf_min=250, nf_max=900,
             nq_min=5, nq_max=30, nm_min=50, nm_max=200, sizes=4),
        # The learned control variate on a layered system, network in hand.
        dict(name="control_variate_fp32", kind="cv", na=4000, nf=200, nq=24, nm=128, qmin=0.1, qmax=1.5),
        # Multipole averages (FP64 devices) at the default resolution.
        dict(name="multipole_sphere", kind="sphere", na=5000, nf=64, nq=10, resolution=20, qmin=0.05, qmax=3.0),
        dict(name="multipole_cylinder", kind="cylinder", na=5000, nf=64, nq=10, resolution=20, qmin=0.05, qmax=3.0),
        # Staging with alignments: centre, then fit every frame onto the first; host frames in.
        dict(name="prepass_fit", kind="prepass", na=10000, nf=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: sizes log-uniform, capped at the listed cost."""
    kind = rng.choice(["call", "phase32", "phase32", "phase64", "static", "self32", "self64", "long", "batch", "cv",
                       "sphere", "cylinder", "prepass"])
    if kind == "call":
        c = _phase("", _log(rng, 20, 600), _log(rng, 8, 100), _log(rng, 1, 8), _log(rng, 1, 24), "fp64",
                   dsp=rng.choice(["autocorrelate", "square", "plain"]), qmin=0.2, qmax=2.5)
        c["kind"] = "call"
    elif kind in ("phase32", "phase64"):
        f32 = kind == "phase32"
        na, nf = _log(rng, 300, 12000), _log(rng, 40, 1100)
        nq = _log(rng, 2, 40)
        cap = 1.0e11 if f32 else 5e8
        nm = max(1, min(_log(rng, 10, 600), int(cap / (float(na) * nf * nq))))
        c = _phase("", na, nf, nq, nm, "fp32" if f32 else "fp64", dsp=rng.choice(["autocorrelate", "autocorrelate",
                   "square", "plain"]), scan=rng.choice(["linear", "linear", "random"]))
    elif kind == "static":
        na, nf, nq = _log(rng, 20000, 120000), _log(rng, 4, 70), _log(rng, 30, 200)
        nm = max(1, min(_log(rng, 50, 1000), int(4e10 / (float(na) * nf * nq))))
        c = _phase("", na, nf, nq, nm, "fp32", dsp="square", qmin=0.01, qmax=0.5, density=0.075, factors="xray")
    elif kind in ("self32", "self64"):
        f32 = kind == "self32"
        nf = _log(rng, 20, 600)
        nq, nm = _log(rng, 1, 15), _log(rng, 5, 120)
        na = max(1, min(_log(rng, 100, 3000), int((1.28e8 if f32 else 4e7) * 128 / (float(nf) * nf * nq * nm))))
        c = _phase("", na, nf, nq, nm, "fp32" if f32 else "fp64", scattering="self", qmin=0.1, qmax=2.0, density=0.037,
                   dsp=rng.choice(["autocorrelate", "autocorrelate", "square"]))
    elif kind == "long":
        c = _phase("", _log(rng, 300, 2000), _log(rng, 4200, 16000), _log(rng, 3, 9), _log(rng, 8, 40), "fp32")
    elif kind == "batch":
        c = dict(kind="batch", nsys=rng.randint(2, 8), na_min=300, na_max=_log(rng, 1000, 6000), nf_min=100,
                 nf_max=_log(rng, 300, 900), nq_min=3, nq_max=rng.randint(8, 30), nm_min=30, nm_max=rng.randint(60, 200),
                 sizes=rng.randint(1, 1000))
    elif kind == "cv":
        c = dict(kind="cv", na=_log(rng, 500, 4500), nf=_log(rng, 50, 220), nq=_log(rng, 6, 26), nm=_log(rng, 16, 128),
                 qmin=0.1, qmax=1.5)
    elif kind in ("sphere", "cylinder"):
        c = dict(kind=kind, na=_log(rng, 500, 5500), nf=_log(rng, 10, 64), nq=_log(rng, 2, 10),
                 resolution=rng.randint(4, 20), qmin=0.05, qmax=3.0)
    else:
        c = dict(kind="prepass", na=_log(rng, 500, 10500), nf=_log(rng, 20, 250))
    return {k: v for k, v in c.items() if k != "name"}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _walk(na, nf, density, seed, sigma=0.05, rmsd=1.0):
    """float32 [nf, na, 3] on the GPU: uniform positions, harmonically held Gaussian steps."""
    g = _gen(seed)
    box = (na / density) ** (1.0 / 3.0)
    r0 = torch.rand((na, 3), generator=g, device="cuda", dtype=torch.float64) * box
    k = 1.0 - math.sqrt(1.0 - 3.0 * sigma * sigma / (rmsd * rmsd))
    out = torch.empty((nf, na, 3), device="cuda", dtype=torch.float32)
    d = torch.zeros_like(r0)
    for t in range(nf):
        out[t] = r0 + d
        d.mul_(1.0 - k).add_(torch.randn((na, 3), generator=g, device="cuda", dtype=torch.float64), alpha=sigma)
    return out


def _classes(na, seed):
    rng = np.random.default_rng(seed)
    counts = np.floor(np.asarray(RATIOS) / sum(RATIOS) * na).astype(int)
    counts[0] += na - counts.sum()
    c = np.repeat(np.arange(len(RATIOS)), counts)
    rng.shuffle(c)
    return c.astype(np.int32)


def _shells(nq, qmin, qmax, scan, seed):
    if scan == "random":
        return np.sort(np.random.default_rng(seed + 5).uniform(qmin, qmax, nq))
    return np.linspace(qmin, qmax, nq)


def _factors(c, shells, seed):
    if c.get("factors") == "xray":  # four-Gaussian form factors, coil and solvent
        p = synth.xray_form_factor_params(np.random.default_rng(seed + 9), 2)
        return np.stack([synth.sfactor_type2(v, shells) for v in p], axis=1)
    return np.tile(np.asarray(INCOHERENT if c.get("scattering") == "self" else COHERENT), (len(shells), 1))


def _inputs(c, seed):
    """Trajectory (GPU), classes, shells, unit directions, class factors of a phase case."""
    coords = _walk(c["na"], c["nf"], c["density"], seed)
    if c["factors"] == "xray":  # 1 coil bead for 4 solvent atoms
        cls = (np.arange(c["na"]) >= c["na"] // 5).astype(np.int32)
    else:
        cls = _classes(c["na"], seed + 1)
    shells = _shells(c["nq"], c["qmin"], c["qmax"], c["scan"], seed)
    return coords, cls, shells, synth.sphere_directions(c["nm"], seed + 1000), _factors(c, shells, seed)


def _batch_systems(c, seed):
    rng = np.random.default_rng(c["sizes"])  # the sizes belong to the case, the contents to the seed
    out = []
    for i in range(c["nsys"]):
        def pick(k):
            return int(round(math.exp(rng.uniform(math.log(c[k + "_min"]), math.log(c[k + "_max"])))))
        na, nf, nq, nm = pick("na"), pick("nf"), pick("nq"), pick("nm")
        out.append((_walk(na, nf, 0.1, seed * 100 + i, sigma=0.1, rmsd=2.0), _classes(na, seed + i),
                    _shells(nq, 0.1, 2.5, "random", seed + i), synth.sphere_directions(nm, seed * 1000 + i)))
    return out


def _moments(kind, res):
    if kind == "sphere":
        return [(0, 0)] + [(l, m) for l in range(1, res + 1) for m in range(-l, l + 1)]
    return [(0, 0)] + [(l, m) for l in range(1, res + 1) for m in range(4)]


def _mp_inputs(c, seed):
    coords = _walk(c["na"], c["nf"], 0.08, seed)
    shells = np.linspace(c["qmin"], c["qmax"], c["nq"])
    qv = shells[:, None] * synth.sphere_directions(c["nq"], seed + 7)
    return coords, _classes(c["na"], seed + 1), qv, np.tile(np.asarray(COHERENT), (c["nq"], 1))


def _layered(c, seed):
    """Density modulated along z (period 8 A), so the intensity depends on the direction."""
    coords = _walk(c["na"], c["nf"], 0.1, seed)
    z = coords[0, :, 2].double()
    coords[:, :, 2] += (0.35 * torch.sin(2 * math.pi * z / 8.0)).float()
    return coords, _classes(c["na"], seed + 1), np.linspace(c["qmin"], c["qmax"], c["nq"])


def _network(c, coords, cls, shells, seed):
    """A network fitted to log intensities of the first frames (computed here, in 64 bits)."""
    n = 1024
    rng = np.random.default_rng(seed + 3)
    u, q = synth.sphere_directions(n, seed + 17), rng.uniform(shells[0], shells[-1], n)
    b = torch.tensor(COHERENT, device="cuda", dtype=torch.float64)[torch.from_numpy(cls).cuda().long()]
    sv = torch.from_numpy(q[:, None] * u).cuda()
    inten = torch.zeros(n, device="cuda", dtype=torch.float64)
    for t in range(4):
        p = sv @ coords[t * (len(coords) // 4)].double().T
        inten += (torch.cos(p) @ b) ** 2 + (torch.sin(p) @ b) ** 2
    y = torch.log(inten / 4 / c["na"]).cpu().numpy()
    mid, half = 0.5 * (shells[0] + shells[-1]), 0.5 * (shells[-1] - shells[0])
    net = abi.MLP(seed=seed)
    net.set_scaling(mid, half, float(y.mean()) + math.log(c["na"]), float(y.std()))
    net.train(np.concatenate([u, ((q - mid) / half)[:, None]], axis=1), (y - y.mean()) / y.std(), steps=100, batch=1024)
    return net


def prepare(case, seed):
    c = case
    if c["kind"] in ("phase", "call"):
        coords, cls, shells, dirs, cf = _inputs(c, seed)
        sv = (shells[:, None, None] * dirs[None]).reshape(-1, 3)
        offs = np.arange(c["nq"] + 1, dtype=np.uintp) * c["nm"]
        plan = abi.Plan(c["na"], c["nf"], cf.shape[1], c["scattering"], c["dsp"], "fftw", c["precision"])
        plan.set_classes(cls)
        torch.cuda.synchronize()
        if c["kind"] == "call":
            frames = coords.cpu().numpy()
        else:
            frames = None
            plan.stage(coords.data_ptr(), on_device=True)
        return dict(case=c, plan=plan, offs=offs, sv=sv, cf=cf, frames=frames)
    if c["kind"] == "batch":
        ws = []
        for coords, cls, shells, dirs in _batch_systems(c, seed):
            ws.append(synth.Workload("system", coords.cpu().numpy(), cls, ["H", "C", "N", "O", "S"],
                                     np.tile(np.asarray(COHERENT), (len(shells), 1)), shells, dirs))
        return dict(case=c, batch=abi.Batch(ws, precision="fp32"), n=len(ws))
    if c["kind"] == "cv":
        coords, cls, shells = _layered(c, seed)
        plan = abi.Plan(c["na"], c["nf"], 5, "all", "autocorrelate", "fftw", "fp32")
        plan.set_classes(cls)
        net = _network(c, coords, cls, shells, seed)
        torch.cuda.synchronize()
        plan.stage(coords.data_ptr(), on_device=True)
        return dict(case=c, plan=plan, net=net, shells=shells, dirs=synth.sphere_directions(c["nm"], seed + 1000),
                    cf=np.tile(np.asarray(COHERENT), (c["nq"], 1)))
    if c["kind"] in ("sphere", "cylinder"):
        coords, cls, qv, cf = _mp_inputs(c, seed)
        plan = abi.Plan(c["na"], c["nf"], 5, "all", "autocorrelate", "fftw", "fp64")
        plan.set_classes(cls)
        torch.cuda.synchronize()
        plan.stage(coords.data_ptr(), on_device=True)
        return dict(case=c, plan=plan, qv=qv, cf=cf, moments=_moments(c["kind"], c["resolution"]))
    frames, masses, steps = _prepass_inputs(c, seed)
    plan = abi.Plan(c["na"], c["nf"], 5, "all", "autocorrelate", "fftw", "fp32")
    return dict(case=c, plan=plan, frames=frames, masses=masses, steps=steps, target=np.arange(c["na"], dtype=np.uintp))


def _prepass_inputs(c, seed):
    """A system that drifts and turns: every frame a rotated, shifted copy plus thermal motion."""
    coords = _walk(c["na"], c["nf"], 0.08, seed).double()
    mid = coords[0].mean(dim=0)
    t = torch.arange(c["nf"], device="cuda", dtype=torch.float64)
    ca, sa = torch.cos(0.003 * t)[:, None], torch.sin(0.003 * t)[:, None]
    x, y, z = (coords - mid).unbind(-1)
    turned = torch.stack([ca * x - sa * y, sa * x + ca * y, z], dim=-1) + mid + 0.01 * t[:, None, None]
    frames = turned.float().cpu().numpy()
    atoms = np.arange(c["na"], dtype=np.uintp)
    masses = np.asarray(MASSES)[_classes(c["na"], seed + 1)]
    steps = [dict(type="center", selection=atoms, reference_selection=atoms),
             dict(type="fitrottrans", selection=atoms, reference_selection=atoms,
                  reference=frames[0].astype(np.float64), fit_target=atoms, fit_source=atoms)]
    return frames, masses, steps


def _kept(out, precision):
    return tuple(a.astype(np.complex64) for a in out) if precision == "fp32" else tuple(out)


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        b = state["batch"]
        b.run()
        b.sync()
        return [_kept(b.results(i), "fp32") for i in range(state["n"])]
    p = state["plan"]
    if c["kind"] in ("phase", "call"):
        if state["frames"] is not None:
            p.stage(state["frames"])
        return _kept(p.compute(state["offs"], state["sv"], state["cf"]), c["precision"])
    if c["kind"] == "cv":
        return _kept(abi.compute_cv(p, state["net"], state["shells"], state["dirs"], state["cf"])[:4], "fp32")
    if c["kind"] in ("sphere", "cylinder"):
        return p.multipole(c["kind"], state["qv"], state["cf"], state["moments"], AXIS)
    return p.stage_prepass(state["frames"], state["masses"], state["steps"], state["target"])


def _work_phase(na, nf, nq, nm, scattering, esize):
    """Read the frames, write the rows; per term a complex product and sum (4 operations at the
    least), per direction (and shell) the transforms where each atom has its own series."""
    terms = float(na) * nf * nq * nm
    flops = 4.0 * terms + 5.0 * na * nf * nm
    if scattering == "self":
        flops += 5.0 * terms * 2 * math.log2(max(2, 2 * nf))
    return {"bytes": 12.0 * na * nf + 2.0 * esize * nq * (nf + 2) + 24.0 * nq * nm, "flops": flops}


def work(case):
    c = case
    if c["kind"] in ("phase", "call"):
        return _work_phase(c["na"], c["nf"], c["nq"], c["nm"], c["scattering"], 8)
    if c["kind"] == "batch":  # geometric means of the ranges
        g = {k: math.sqrt(float(c[k + "_min"]) * c[k + "_max"]) for k in ("na", "nf", "nq", "nm")}
        w = _work_phase(g["na"], g["nf"], g["nq"], g["nm"], "all", 8)
        return {k: v * c["nsys"] for k, v in w.items()}
    if c["kind"] == "cv":
        return _work_phase(c["na"], c["nf"], c["nq"], c["nm"], "all", 8)
    if c["kind"] in ("sphere", "cylinder"):
        n = float(c["na"]) * c["nf"] * c["nq"] * len(_moments(c["kind"], c["resolution"]))
        return {"bytes": 12.0 * c["na"] * c["nf"] + 16.0 * c["nq"] * (c["nf"] + 2), "flops": 4.0 * n}
    n = float(c["na"]) * c["nf"]
    return {"bytes": 24.0 * n, "flops": 60.0 * n}


# ---- plain 64-bit values ---------------------------------------------------------------


def _amplitudes(coords, cls, shells, dirs, cf, linear):
    """A[q, m, t] in complex128: sums per class of exp(i q u.r), weighted by the factors."""
    nq, nd, (nf, na) = len(shells), len(dirs), coords.shape[:2]
    order = np.argsort(cls, kind="stable")
    idx = torch.from_numpy(order).cuda()
    bounds = np.searchsorted(cls[order], np.arange(cf.shape[1] + 1))
    u = torch.from_numpy(dirs).cuda()
    out = torch.zeros((nq, nd, nf), device="cuda", dtype=torch.complex128)
    w = torch.from_numpy(cf).cuda()
    chunk = max(1, int(6e7 // na))  # (frame, direction) pairs at a time
    for f0 in range(0, nf, max(1, chunk // nd)):
        f1 = min(nf, f0 + max(1, chunk // nd))
        r = coords[f0:f1][:, idx].double()
        for d0 in range(0, nd, chunk):
            d1 = min(nd, d0 + chunk)
            s = torch.einsum("dk,tjk->dtj", u[d0:d1], r)
            if linear and nq > 2:
                z = torch.polar(torch.ones_like(s), s * shells[0])
                step = torch.polar(torch.ones_like(s), s * ((shells[-1] - shells[0]) / (nq - 1)))
            for k in range(nq):
                if not (linear and nq > 2):
                    z = torch.polar(torch.ones_like(s), s * shells[k])
                for a in range(cf.shape[1]):
                    if bounds[a + 1] > bounds[a]:
                        out[k, d0:d1, f0:f1] += w[k, a] * z[..., bounds[a]:bounds[a + 1]].sum(dim=-1)
                if linear and nq > 2 and k + 1 < nq:
                    z.mul_(step)
    return out


def _dsp(a, kind):
    """Correlated (or squared, or plain) series along the last axis."""
    nf = a.shape[-1]
    if kind == "plain":
        return a
    if kind == "square":
        return (a.real ** 2 + a.imag ** 2).to(torch.complex128)
    x = torch.fft.fft(a, n=2 * nf)
    c = torch.fft.ifft((x.real ** 2 + x.imag ** 2).to(torch.complex128))[..., :nf]
    return c / (nf - torch.arange(nf, device=a.device, dtype=torch.float64))


def _average(series, kind, inv):
    """(fqt, fq, fq2) of series [n, nf], summed and scaled by `inv`."""
    c = _dsp(series, kind)
    m = c.mean(dim=-1)
    return c.sum(dim=0) * inv, m.sum() * inv, (m * m.conj()).sum() * inv


def _rows(parts):
    return tuple(torch.stack([p[i] for p in parts]).cpu().numpy() for i in range(3))


def _exact_coherent(coords, cls, shells, dirs, cf, dsp, linear):
    a = _amplitudes(coords, cls, shells, dirs, cf, linear)
    return _rows([_average(a[k], dsp, 1.0 / len(dirs)) for k in range(len(shells))])


def _exact_self(coords, cls, shells, dirs, cf, dsp):
    r = coords.double()
    b = torch.from_numpy(cf).cuda()[:, torch.from_numpy(cls).cuda().long()]
    u = torch.from_numpy(dirs).cuda()
    parts = []
    for k in range(len(shells)):
        acc = None
        for d in range(len(dirs)):
            p = torch.einsum("tjk,k->jt", r, u[d] * shells[k])
            v = _average(torch.polar(b[k][:, None].expand_as(p).contiguous(), p), dsp, 1.0 / len(dirs))
            acc = v if acc is None else tuple(x + y for x, y in zip(acc, v))
        parts.append(acc)
    return _rows(parts)


def _exact_sphere(c, seed):
    coords, cls, qv, cf = _mp_inputs(c, seed)
    L, nq = c["resolution"], len(qv)
    x, y, z = coords.double().unbind(-1)
    r = torch.sqrt(x * x + y * y + z * z)
    theta = torch.acos(z / r).float().double()
    phi = torch.remainder(torch.atan2(y, x), 2 * math.pi).float().double()
    r = r.float().double()
    b = torch.from_numpy(cf).cuda()[:, torch.from_numpy(cls).cuda().long()]
    ql = torch.from_numpy(np.linalg.norm(qv, axis=1)).cuda()
    amps = torch.zeros((nq, (L + 1) ** 2, c["nf"]), device="cuda", dtype=torch.complex128)
    for f0 in range(0, c["nf"], 16):
        f1 = min(c["nf"], f0 + 16)
        xq = ql[:, None, None] * r[f0:f1][None]                       # [q, t, j]
        # ratios j_{l+1} / j_l downwards for small arguments, upwards recurrence beyond L
        rho, t = [None] * L, torch.zeros_like(xq)
        for l in range(L + 40, -1, -1):
            t = xq / (2 * l + 3 - xq * t)
            if l < L:
                rho[l] = t
        up0, up1 = torch.sin(xq) / xq, (torch.sin(xq) / xq - torch.cos(xq)) / xq
        jl, down, big = [up0], up0, xq > L
        for l in range(1, L + 1):
            down = down * rho[l - 1]
            if l > 1:
                up0, up1 = up1, (2 * l - 1) / xq * up1 - up0
            jl.append(torch.where(big, up1, down))
        ct, st = torch.cos(theta[f0:f1]), torch.sin(theta[f0:f1]).abs()
        P = {(0, 0): torch.full_like(ct, math.sqrt(0.25 / math.pi))}
        for m in range(L + 1):
            if m > 0:
                P[m, m] = -math.sqrt((2 * m + 1) / (2.0 * m)) * st * P[m - 1, m - 1]
            if m < L:
                P[m + 1, m] = math.sqrt(2 * m + 3) * ct * P[m, m]
            for l in range(m + 2, L + 1):
                f = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
                g = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1))
                P[l, m] = f * (ct * P[l - 1, m] - g * P[l - 2, m])
        for l in range(L + 1):
            bj = (4 * math.pi * b[:, None, :] * jl[l]).permute(1, 0, 2)  # [t, q, j]
            ym = []
            for m in range(-l, l + 1):
                v = P[l, abs(m)] * (-1.0 if m < 0 and m % 2 else 1.0)
                ym.append(torch.polar(torch.ones_like(v), -m * phi[f0:f1]) * v)
            a = torch.matmul(bj.to(torch.complex128), torch.stack(ym, dim=-1)) * (1j ** l)
            amps[:, l * l:(l + 1) ** 2, f0:f1] = a.permute(1, 2, 0)
    return _rows([_average(amps[k], "autocorrelate", 0.25 / math.pi) for k in range(nq)])


def _exact_cylinder(c, seed):
    coords, cls, qv, cf = _mp_inputs(c, seed)
    L, nq = c["resolution"], len(qv)
    # the frame of the z axis: e_r = y x z = x, e_phi = z x e_r = y
    x, y, z = coords.double().unbind(-1)
    r = torch.sqrt(x * x + y * y).float().double()
    phi = torch.atan(y / x) + torch.where(x < 0, torch.copysign(torch.full_like(y, float(np.float32(math.pi))), y), 0.0)
    phi = torch.where(phi < 0, phi + 2 * math.pi, phi).float().double()  # the half turn is a float, as staged
    b = torch.from_numpy(cf).cuda()[:, torch.from_numpy(cls).cuda().long()]
    amps = torch.zeros((nq, 4 * L + 1, c["nf"]), device="cuda", dtype=torch.complex128)
    N = 2 * L
    for k in range(nq):
        qr, qz = math.hypot(qv[k, 0], qv[k, 1]), qv[k, 2]
        qphi = math.atan(qv[k, 1] / qv[k, 0])
        if qv[k, 0] < 0:
            qphi += math.copysign(float(np.float32(math.pi)), qv[k, 1])
        xq = qr * r
        t = torch.zeros_like(xq)
        rho = [None] * (N + 1)
        for n in range(N + int(float(xq.max())) + 50, 0, -1):  # J_n / J_{n-1}, downwards
            t = xq / (2 * n - xq * t)
            if n <= N:
                rho[n] = t
        e = torch.polar((b[k][None] * math.sqrt(2 * math.pi)).expand_as(z).contiguous(), (z * qz).abs())
        J = torch.special.bessel_j0(xq)
        amps[k, 0] = (J * e).sum(dim=-1)
        for n in range(1, N + 1):
            J = J * rho[n]
            l = (n + 1) // 2
            sign = (-1.0) ** (l if n % 2 == 0 else l - 1)
            w = e * J * (math.sqrt(2.0) * sign)
            if n % 2:
                w = w * 1j
            at = 1 + 4 * (l - 1) + (2 if n % 2 else 0)
            amps[k, at] = (w * torch.cos(n * (phi - qphi))).sum(dim=-1)
            amps[k, at + 1] = (w * torch.sin(n * (phi - qphi))).sum(dim=-1)
    return _rows([_average(amps[k], "autocorrelate", 0.5 / math.pi) for k in range(nq)])


def _exact_prepass(c, seed):
    frames, masses, _ = _prepass_inputs(c, seed)
    r, m = torch.from_numpy(frames).cuda().double(), torch.from_numpy(masses).cuda()
    ref = r[0]
    r = r - (r * m[:, None]).sum(dim=1, keepdim=True) / m.sum()  # centred
    com = (ref * m[:, None]).sum(dim=0) / m.sum()
    u, v = ref - com, r - (r * m[:, None]).sum(dim=1, keepdim=True) / m.sum()
    K = torch.einsum("j,ja,tjb->tab", m, u, v)
    U, _, Vt = torch.linalg.svd(K)
    D = torch.diag_embed(torch.stack([torch.ones(len(r), device="cuda", dtype=torch.float64)] * 2
                                     + [torch.linalg.det(U @ Vt)], dim=-1))
    return (v @ (U @ D @ Vt).transpose(1, 2) + com).cpu().numpy()


def exact(case, seed):
    c = case
    if c["kind"] in ("phase", "call"):
        coords, cls, shells, dirs, cf = _inputs(c, seed)
        if c["scattering"] == "self":
            return _exact_self(coords, cls, shells, dirs, cf, c["dsp"])
        return _exact_coherent(coords, cls, shells, dirs, cf, c["dsp"],
                               c["scan"] == "linear" and c["precision"] == "fp32")
    if c["kind"] == "batch":
        cf = np.asarray(COHERENT)
        return [_exact_coherent(r, cls, s, d, np.tile(cf, (len(s), 1)), "autocorrelate", False)
                for r, cls, s, d in _batch_systems(c, seed)]
    if c["kind"] == "cv":  # the plain average on the same directions (halves of equal weight)
        coords, cls, shells = _layered(c, seed)
        dirs, cf, h = synth.sphere_directions(c["nm"], seed + 1000), np.tile(np.asarray(COHERENT), (c["nq"], 1)), c["nm"] // 2
        a, b = (_exact_coherent(coords, cls, shells, d, cf, "autocorrelate", True) for d in (dirs[:h], dirs[h:]))
        return (None, 0.5 * (a[0] + b[0]), None, 0.5 * (a[1] + b[1]))
    if c["kind"] == "sphere":
        return _exact_sphere(c, seed)
    if c["kind"] == "cylinder":
        return _exact_cylinder(c, seed)
    return _exact_prepass(c, seed)
