"""The work that users of kpolaris_b200 wait for, as measurable cases: images
of the analytic RIAF in Cartesian Kerr-Schild and of GRMHD snapshots in FMKS,
alone and in batches, with fixed and adaptive steps, one to four frequencies,
in FP64 and under the mixed policy, from thumbnails to production frames; the
line-of-sight analysis image; slow light on resident snapshots.

`exact` evaluates the same images with plain torch in 64 bits: the method the
library documents (backward pass A, forward pass B, classical RK4 with step
doubling, thermal synchrotron fits, semi-analytic Stokes transfer), written
for whole arrays of rays, without the library's code.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import kpolaris_b200 as kp
from kpolaris_b200 import _abi, configs, synthetic

FREQUENCIES = [230.0e9, 86.0e9, 345.0e9, 690.0e9]
STOKES = ("image_i", "image_q", "image_u", "image_v")

# kinds: what is called and how
#   riaf   image_riaf          (precision, schedule)
#   batch  batch_riaf          (sizes "256x256,64x64": one job each)
#   grmhd  image_grmhd         on one resident snapshot
#   slow   image_grmhd_slow_light on `snapshots` resident snapshots
#   analysis  image_riaf_analysis


def listed():
    return [
        # the smallest call, all options at their defaults: a thumbnail or a
        # unit test of a user's pipeline
        dict(name="riaf_fp64_fixed_16", kind="riaf", sizes="16x16", precision="fp64", schedule="per_pixel",
             adaptive=False, nfreq=1, spin=0.9375, inclination=17.0),
        # the reference's CPU configuration: 64^2, fixed step 1 M
        dict(name="riaf_fp64_fixed_64", kind="riaf", sizes="64x64", precision="fp64", schedule="per_pixel",
             adaptive=False, nfreq=1, spin=0.9375, inclination=17.0),
        # default options with the recommended transfer controls, an odd-sized
        # multi-frequency image
        dict(name="riaf_fp64_adaptive_97x61_4f", kind="riaf", sizes="97x61", precision="fp64", schedule="per_pixel",
             adaptive=True, nfreq=4, spin=0.5, inclination=60.0),
        # a parameter survey in FP64: several images in one launch
        dict(name="riaf_fp64_batch", kind="batch", sizes="128x128,96x96,33x57", precision="fp64",
             schedule="persistent", adaptive=True, nfreq=2, spin=0.9, inclination=35.0),
        # interactive preview under the mixed policy, replayed as a graph
        dict(name="riaf_mixed_31x24", kind="riaf", sizes="31x24", precision="mixed", schedule="graph",
             adaptive=True, nfreq=1, spin=0.7, inclination=50.0),
        # the headline image: 256^2, four frequencies
        dict(name="riaf_mixed_256_4f", kind="riaf", sizes="256x256", precision="mixed", schedule="persistent",
             adaptive=True, nfreq=4, spin=0.9375, inclination=17.0),
        # an uneven batch of a parameter survey under the mixed policy
        dict(name="riaf_mixed_batch_uneven", kind="batch", sizes="256x256,256x256,192x108,97x97,64x64,32x32",
             precision="mixed", schedule="persistent", adaptive=True, nfreq=4, spin=0.8, inclination=140.0),
        # a GRMHD snapshot imaged in FP64
        dict(name="grmhd_fp64_48", kind="grmhd", sizes="48x48", precision="fp64", schedule="persistent",
             adaptive=True, nfreq=1, spin=0.9375, inclination=163.0, grid="96x64x64", snapshots=1),
        # the production GRMHD frame under the mixed policy
        dict(name="grmhd_mixed_192", kind="grmhd", sizes="192x192", precision="mixed", schedule="graph",
             adaptive=True, nfreq=1, spin=0.9375, inclination=163.0, grid="192x96x96", snapshots=1),
        # slow light over resident snapshots
        dict(name="grmhd_slow_mixed_72x50", kind="slow", sizes="72x50", precision="mixed", schedule="graph",
             adaptive=True, nfreq=1, spin=0.9375, inclination=150.0, grid="96x48x48", snapshots=4),
        # line-of-sight diagnostics of an FP64 image
        dict(name="riaf_analysis_48", kind="analysis", sizes="48x48", precision="fp64", schedule="per_pixel",
             adaptive=True, nfreq=1, spin=0.9375, inclination=17.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["riaf", "riaf", "riaf", "batch", "batch", "grmhd", "grmhd", "slow", "analysis"])
    precision = rng.choice(["fp64", "mixed", "mixed"])
    if kind == "analysis":
        precision = "fp64"
    # fixed steps are the plain kernel's configuration (the reference's own)
    adaptive = kind != "riaf" or precision != "fp64" or rng.random() < 0.5
    spin = round(rng.uniform(0.0, 0.99), 4)
    inclination = round(rng.choice([rng.uniform(10.0, 80.0), rng.uniform(100.0, 170.0)]), 2)
    if kind == "batch":
        sizes = ",".join("%dx%d" % (_log_int(rng, 16, 128), _log_int(rng, 16, 128)) for _ in range(rng.randint(2, 5 if precision == "mixed" else 3)))
    else:
        top = {"riaf": 200 if precision == "mixed" else 96, "analysis": 48, "slow": 72,
               "grmhd": 160 if precision == "mixed" else 48}[kind]
        sizes = "%dx%d" % (_log_int(rng, 12, top), _log_int(rng, 12, top))
    case = dict(kind=kind, sizes=sizes, precision=precision, schedule="persistent", adaptive=adaptive,
                nfreq=rng.randint(1, 4) if kind in ("riaf", "batch") else 1, spin=spin, inclination=inclination)
    if kind == "riaf":
        if precision == "mixed":
            case["schedule"] = rng.choice(["persistent", "graph"])
        elif not adaptive or rng.random() < 0.7:
            case["schedule"] = "per_pixel"
    elif kind == "analysis":
        case["schedule"] = "per_pixel"
    elif kind in ("grmhd", "slow"):
        case["schedule"] = rng.choice(["persistent", "graph"])
        case["grid"] = "%dx%dx%d" % (rng.choice([96, 128]), rng.choice([48, 64]), rng.choice([48, 64]))
        case["snapshots"] = 1 if kind == "grmhd" else rng.randint(2, 4)
        case["spin"] = round(rng.uniform(0.5, 0.95), 4)
    return case


# ---------------------------------------------------------------- inputs

def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]


def _riaf_jobs(case, seed):
    """(params, model, frequencies) per image: the case's geometry with the
    plasma and, over the jobs of a batch, the spin and the viewing angle that
    a parameter survey steps through."""
    rng = random.Random(1000003 * int(seed) + 17)
    jobs = []
    for i, (nx, ny) in enumerate(_sizes(case)):
        if case["adaptive"]:
            p = configs.config2(nx, ny)[0]
        else:
            p = configs.config1(nx, ny)[0]
        spin = min(0.99, max(0.0, case["spin"] - 0.05 * i))
        p.spin = spin
        p.inner_radius = configs.reference_horizon(spin) * 1.05
        inc = case["inclination"] + rng.uniform(-2.0, 2.0) + (3.0 * i if case["inclination"] < 90.0 else -3.0 * i)
        p.camera.inclination = configs.inclination_from_degrees(inc)
        fov = 2.0 * 80.0 / p.camera.radius
        p.camera.fov = fov
        p.camera.fov_y = fov * ny / nx
        m = configs.riaf_model(ne_unit=4.0e6 * rng.uniform(0.8, 1.25), te_unit=1.5e11 * rng.uniform(0.9, 1.1))
        nf = case["nfreq"]
        jobs.append((p, m, FREQUENCIES[:nf] if i % 2 == 0 else FREQUENCIES[:nf][::-1]))
    return jobs


def _grmhd_inputs(case, seed):
    n1, n2, n3 = (int(v) for v in case["grid"].split("x"))
    rng = random.Random(1000003 * int(seed) + 29)
    torus = int(seed) % (1 << 31)
    m_unit = 1.0e27 * rng.uniform(0.8, 1.25)
    # 160 M between the first and the last snapshot: the light travel times
    # over the radiating region
    times = [160.0 * k / max(1, case["snapshots"] - 1) for k in range(case["snapshots"])]
    prims = []
    for t in times:
        f, model = synthetic.fm_torus(n1, n2, n3, spin=case["spin"], seed=torus, M_unit=m_unit, time=t)
        prims.append(f)
    (nx, ny), = _sizes(case)
    p = synthetic.fmks_pass_a_params(model, nx, ny, inclination_deg=case["inclination"] + rng.uniform(-2.0, 2.0),
                                     adaptive=int(case["adaptive"]))
    p.camera.fov_y = p.camera.fov * ny / nx
    # the light of the flow is seen about r + 2 ln(r) later than it leaves it
    return p, model, prims, times, 0.5 * times[-1] + p.camera.radius + 2.0 * math.log(p.camera.radius)


def _options(case):
    return dict(precision=_abi.PRECISION_MIXED if case["precision"] == "mixed" else _abi.PRECISION_FP64,
                schedule={"per_pixel": _abi.SCHEDULE_PER_PIXEL, "persistent": _abi.SCHEDULE_PERSISTENT,
                          "graph": _abi.SCHEDULE_GRAPH}[case["schedule"]])


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "options": _options(case), "mixed": case["precision"] == "mixed"}
    if kind in ("riaf", "batch", "analysis"):
        state["jobs"] = _riaf_jobs(case, seed)
    else:
        p, model, prims, times, t_obs = _grmhd_inputs(case, seed)
        state.update(params=p, frequencies=FREQUENCIES[:case["nfreq"]], times=times, t_obs=t_obs,
                     grids=[kp.Grid(model, f) for f in prims])
    return state


def _outputs(image, short):
    """FP64 images come whole, with their closure diagnostics and step
    counts.  A mixed-policy image is its Stokes maps and how each ray ended:
    its remaining diagnostics measure that policy's rounding itself, and its
    step counts follow from it.  (The analysis image, too, comes as `short`
    as that, beside its line-of-sight arrays.)"""
    if short:
        out = {k: image.arrays[k] for k in STOKES}
        out["reason"] = image.arrays["reason"]
        return out
    return dict(image.arrays)


def run(state):
    kind, opt = state["kind"], state["options"]
    if kind == "batch":
        return [_outputs(r, state["mixed"]) for r in kp.batch_riaf(state["jobs"], **opt)]
    if kind == "riaf":
        p, m, f = state["jobs"][0]
        return [_outputs(kp.image_riaf(p, m, f, **opt), state["mixed"])]
    if kind == "analysis":
        p, m, _ = state["jobs"][0]
        image, lines = kp.image_riaf_analysis(p, m)
        return [_outputs(image, True), dict(lines.arrays)]
    if kind == "grmhd":
        return [_outputs(kp.image_grmhd(state["params"], state["grids"][0], state["frequencies"], **opt),
                         state["mixed"])]
    return [_outputs(kp.image_grmhd_slow_light(state["params"], state["grids"], state["times"], state["t_obs"],
                                               state["frequencies"], **opt), state["mixed"])]


def work(case):
    """Operations of the method on these rays.  One right-hand side of the
    three transports, its shared connection evaluated once, is 320 operations
    in Kerr-Schild and 430 in FMKS; an adaptive step takes 11 of them, a
    fixed one 4, and one radiating step about 420 operations of plasma state
    and 330 per frequency."""
    rays = sum(nx * ny for nx, ny in _sizes(case))
    fixed = not case["adaptive"]
    grmhd = case["kind"] in ("grmhd", "slow")
    if grmhd:
        steps, near, rhs = 2000, 160, 430
    elif fixed:
        steps, near, rhs = 2200, 260, 320
    else:
        steps, near, rhs = 1250, 225, 320
    flops = rays * (steps * ((4 if fixed else 11) * (rhs + 96)) + near * (420 + 330 * case["nfreq"]))
    bytes_ = rays * (4 * 8 * case["nfreq"] + 11 * 8 + 3 * 4)
    if grmhd:
        n1, n2, n3 = (int(v) for v in case["grid"].split("x"))
        bytes_ += n1 * n2 * n3 * 80 * case["snapshots"]
    return {"bytes": float(bytes_), "flops": float(flops)}


# ---------------------------------------------------------------- exact
# The images in plain 64-bit torch.  A ray is Y[4, 4]: position, wavevector
# and the two transported screen vectors.  Every function takes all rays of a
# case at once; c is a dict of per-ray constants.

F64 = torch.float64
EE, ME, CL, HPL, MP = 4.803204712570263e-10, 9.1093837015e-28, 2.99792458e10, 6.62607015e-27, 1.67262192369e-24
KBOL = 1.380649e-16
TINY = 1e-300


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def exact(case, seed):
    kind = case["kind"]
    if kind in ("riaf", "batch", "analysis"):
        jobs = _riaf_jobs(case, seed)
        scene = _Riaf(jobs, 1 if kind == "analysis" else None)
    else:
        p, model, prims, times, t_obs = _grmhd_inputs(case, seed)
        scene = _Grmhd(p, model, prims, times, t_obs, FREQUENCIES[:case["nfreq"]], kind == "slow")
        jobs = [(p, model, FREQUENCIES[:case["nfreq"]])]
    stokes, reason = _image(scene)
    names = STOKES + (() if case["precision"] == "mixed" or kind == "analysis" else _abi.DIAG_FIELDS + _abi.INT_FIELDS)
    out, at = [], 0
    for p, _, freqs in jobs:
        n = p.camera.nx * p.camera.ny
        nf = 1 if kind == "analysis" else len(freqs)
        part = stokes[at:at + n, :nf].permute(2, 1, 0).cpu().numpy()
        img = {k: None for k in names}
        for i, k in enumerate(STOKES):
            img[k] = np.ascontiguousarray(part[i])
        img["reason"] = reason[at:at + n].to(torch.int32).cpu().numpy()
        out.append(img)
        at += n
    if kind == "analysis":
        out.append({k: None for k in _abi.AnalysisHostData.allocate(1, 1).arrays})
    return out


def _advance(step, state, every=8):
    """Repeats step(state) (in place, masked by state["on"]) until no ray is
    on.  The rays still on are packed together now and then; on a GPU one
    repetition is a captured graph."""
    idx = torch.arange(state["on"].shape[0], device=state["on"].device)
    while idx.numel():
        cur = {k: v[idx].clone() for k, v in state.items()}
        if cur["on"].is_cuda:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                step({k: v.clone() for k, v in cur.items()})
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step(cur)
            once = graph.replay
        else:
            def once():
                step(cur)
        left = idx.numel()
        while left and left > 0.7 * idx.numel():
            for _ in range(every):
                once()
            left = int(cur["on"].sum())
        for k, v in state.items():
            v[idx] = cur[k]
        idx = idx[cur["on"]]


def _set(state, mask, **new):
    for k, v in new.items():
        old = state[k]
        m = mask.reshape(mask.shape + (1,) * (old.dim() - 1))
        if isinstance(v, torch.Tensor):
            old.copy_(torch.where(m, v.to(old.dtype), old))
        else:
            old.masked_fill_(m, v)


def _rk4(rhs, c, Y, h, k1=None):
    h = h[:, None, None]
    k1 = rhs(c, Y) if k1 is None else k1
    k2 = rhs(c, Y + k1 * (0.5 * h))
    k3 = rhs(c, Y + k2 * (0.5 * h))
    k4 = rhs(c, Y + k3 * h)
    return Y + (k1 + 2.0 * k2 + 2.0 * k3 + k4) * (h / 6.0)


def _attempt(scene, c, Y, h):
    """One step of each ray: endpoint, radiation sample and error."""
    if not scene.adaptive:
        end = _rk4(scene.rhs, c, Y, h)
        return end, end, torch.zeros_like(h)
    k1 = scene.rhs(c, Y)
    half = _rk4(scene.rhs, c, Y, 0.5 * h, k1)
    two = _rk4(scene.rhs, c, half, 0.5 * h)
    full = _rk4(scene.rhs, c, Y, h, k1)
    scale = torch.clamp(torch.maximum(full.abs(), two.abs()), min=1.0)
    return two, half, ((full - two).abs() / scale).amax((1, 2))


def _grown(c, h, err, lo, hi):
    factor = torch.clamp(0.9 * (c["tol"] / err.clamp(min=TINY)) ** 0.2, 0.2, 2.0)
    factor = torch.where(err > 0.0, factor, torch.full_like(factor, 2.0))
    return torch.minimum(hi, torch.maximum(lo, h.abs() * factor))


def _shrunk(c, h, err):
    return h * torch.clamp(0.9 * (c["tol"] / err.clamp(min=TINY)) ** 0.25, 0.1, 0.8)


def _begin(s, fresh, want, lo, hi):
    h = torch.minimum(torch.maximum(want.abs(), lo), hi)
    _set(s, fresh, h=torch.where(want < 0.0, -h, h), lo=lo, hi=hi, attempt=0, fresh=False)


def _rejected(scene, s, c, bad, err):
    """Shrinks the rejected steps; returns the rays that gave up, with the
    size of their next step."""
    _set(s, bad, attempt=s["attempt"] + 1)
    floor = s["h"].abs() <= s["lo"] * 1.0001
    _set(s, bad & ~floor, h=_shrunk(c, s["h"], err))
    lost = bad & (floor | (s["attempt"] >= 10))
    return lost, torch.maximum(s["lo"], s["h"].abs() * 0.5)


def _pass_a(scene, s, c):
    on = s["on"]
    r = scene.radius(c, s["Y"])
    top = on & s["fresh"]
    _set(s, top & (s["n"] >= c["max_steps"]), on=False)
    top = top & s["on"]
    inner = top & s["entered"] & (r <= c["inner"])
    outer = top & s["entered"] & ~inner & (s["inside"] > 0) & (r >= c["outer"])
    _set(s, inner, reason=2, on=False)
    _set(s, outer, reason=3, on=False)
    _set(s, top & ~s["entered"] & (r <= c["outer"]), entered=True, inside=0)
    top = top & s["on"]
    _set(s, top, old_r=r)
    if scene.adaptive:
        _begin(s, top, s["want"], torch.minimum(c["min_step"], s["want"].abs()), c["max_step"])
    else:
        _set(s, top, h=s["want"])
    new, _, err = _attempt(scene, c, s["Y"], s["h"])
    ok = s["on"] & (err <= c["tol"])
    if scene.adaptive:
        lost, next_h = _rejected(scene, s, c, s["on"] & ~ok, err)
        _set(s, lost, want=-next_h, fresh=True, n=s["n"] + 1)
        _set(s, lost & (next_h <= c["min_step"] * 1.0001), reason=7, on=False)
        _set(s, ok, want=-_grown(c, s["h"], err, s["lo"], s["hi"]))
    _set(s, ok, fresh=True)
    next_r = scene.radius(c, new)
    enters = ok & ~s["entered"] & (next_r <= c["outer"])
    misses = ok & ~s["entered"] & ~enters & (next_r >= s["old_r"])
    _set(s, enters, entered=True, inside=0)
    _set(s, misses, Y=new, reason=3, on=False)
    go = ok & ~misses
    hits = go & s["entered"] & (s["old_r"] > c["inner"]) & (next_r <= c["inner"])
    leaves = go & s["entered"] & ~hits & (s["inside"] > 0) & (s["old_r"] < c["outer"]) & (next_r >= c["outer"])
    _set(s, hits | leaves, cross=True, on=False, full_h=s["h"], end=new,
         surf=torch.where(hits, c["inner"], c["outer"]))
    _set(s, hits, reason=2)
    _set(s, leaves, reason=3)
    go = go & ~hits & ~leaves
    _set(s, go, Y=new, n=s["n"] + 1)
    _set(s, go & s["entered"], inside=s["inside"] + 1)


def _surface(scene, s, c):
    """The last point on the near side of the crossed surface."""
    def path(h):
        if not scene.adaptive:
            return _rk4(scene.rhs, c, s["Y"], h)
        return _rk4(scene.rhs, c, _rk4(scene.rhs, c, s["Y"], 0.5 * h), 0.5 * h)

    def finite(y):
        return torch.isfinite(y).all(2).all(1)

    best = s["Y"].clone()
    lo, hi = torch.zeros_like(s["h"]), torch.ones_like(s["h"])
    flo = scene.radius(c, s["Y"]) - s["surf"]
    end = path(s["full_h"])
    fhi = scene.radius(c, end) - s["surf"]
    on = s["cross"] & (flo != 0.0) & finite(s["end"]) & finite(end) & torch.isfinite(fhi)
    best = torch.where((on & (fhi == 0.0))[:, None, None], end, best)
    on = on & (fhi != 0.0) & ((flo > 0.0) != (fhi > 0.0))
    secant_ok = torch.ones_like(on)
    for _ in range(12):
        width = hi - lo
        trial = 0.5 * (lo + hi)
        denom = flo - fhi
        sec = lo + width * flo / torch.where(denom == 0.0, torch.ones_like(denom), denom)
        use = secant_ok & (denom.abs() > TINY) & (sec > lo + 0.1 * width) & (sec < hi - 0.1 * width)
        trial = torch.where(use, sec, trial)
        y = path(s["full_h"] * trial)
        ft = scene.radius(c, y) - s["surf"]
        bad = on & ~(finite(y) & torch.isfinite(ft))
        hit = on & ~bad & (ft == 0.0)
        near = on & ~bad & ~hit & ((flo > 0.0) == (ft > 0.0))
        far = on & ~bad & ~hit & ~near
        best = torch.where((hit | near)[:, None, None], y, best)
        lo = torch.where(near, trial, lo)
        flo = torch.where(near, ft, flo)
        hi = torch.where(far | bad, trial, hi)
        fhi = torch.where(far, ft, fhi)
        secant_ok = secant_ok & ~bad
        on = on & ~hit
    s["Y"].copy_(torch.where(s["cross"][:, None, None], best, s["Y"]))


def _pow2_at_least(ratio):
    """The smallest power of two that is at least `ratio`, from 1 to 4096."""
    m, e = torch.frexp(ratio.clamp(min=0.5, max=8192.0))
    e = torch.where(m > 0.5, e, e - 1).clamp(0, 12)
    return torch.ldexp(torch.ones_like(ratio), e)


def _substeps(c, k, h, max_rad):
    """Substeps that keep every depth of one step under its limit, over the
    frequencies of the image; k the coefficients [N, F]."""
    dl = h[:, None].abs() * c["dls"].abs()
    one = torch.ones_like(h)
    n = torch.where(max_rad > 0.0, _pow2_at_least(h.abs() / torch.where(max_rad > 0.0, max_rad, one)), one)
    alim = torch.where(c["max_abs"] >= 0.0, c["max_abs"], c["max_depth"])
    flim = torch.where(c["max_far"] >= 0.0, c["max_far"], c["max_depth"])
    for lim, depth in ((alim, k["aI"].abs() + torch.sqrt(k["aQ"] ** 2 + k["aU"] ** 2 + k["aV"] ** 2)),
                       (flim, torch.sqrt(k["rQ"] ** 2 + k["rU"] ** 2 + k["rV"] ** 2))):
        ratio = (depth * dl * c["live"]).amax(1) / torch.where(lim > 0.0, lim, one)
        n = torch.maximum(n, torch.where(lim > 0.0, _pow2_at_least(ratio), one))
    return n


def _pass_b(scene, s, c):
    _set(s, s["on"] & s["fresh"] & (s["steps"] >= c["max_steps"]), reason=4, on=False)
    r = scene.radius(c, s["Y"])
    top = s["on"] & s["fresh"]
    want = torch.where((r <= c["outer"]) & (s["cap"] > 0.0), torch.minimum(s["want"], s["cap"]), s["want"])
    _set(s, top, old_r=r, cam=False)
    if scene.adaptive:
        _begin(s, top, want, c["min_step"], c["max_step"])
    else:
        _set(s, top, h=want, fresh=False)
    new, mid, err = _attempt(scene, c, s["Y"], s["h"])
    ok = s["on"] & (err <= c["tol"])
    h = s["h"].abs()
    if scene.adaptive:
        lost, next_h = _rejected(scene, s, c, s["on"] & ~ok, err)
        _set(s, lost, want=next_h, fresh=True)
        _set(s, lost & ~s["cam"] & (next_h <= c["min_step"] * 1.0001), reason=4 if scene.slow else 7, on=False)
        _set(s, ok & ~s["cam"], want=_grown(c, s["h"], err, s["lo"], s["hi"]))
    # the camera's surface
    s0 = s["old_r"] - c["camera"]
    s1 = scene.radius(c, new) - c["camera"]
    meets = (s0 == 0.0) | (s1 == 0.0) | ((s0 < 0.0) != (s1 < 0.0))
    crosses = s["cam"] | meets
    denom = s0 - s1
    frac = torch.where(denom.abs() <= TINY, torch.ones_like(s0),
                       (s0 / torch.where(denom == 0.0, torch.ones_like(denom), denom)).clamp(0.0, 1.0))
    first = ok & ~s["cam"] & meets
    none = first & ((h * frac).abs() <= 1e-14)
    part = first & ~none & (frac < 0.999999999999)
    h = torch.where(none, torch.zeros_like(h), h)
    new = torch.where(none[:, None, None], s["Y"], new)
    mid = torch.where(none[:, None, None], s["Y"], mid)
    hc = h * frac
    lo = torch.minimum(c["min_step"], hc)
    if scene.adaptive:
        _begin(s, part, hc, lo, torch.maximum(lo, hc))
    else:
        _set(s, part, h=hc, fresh=False)
    _set(s, part, cam=True)
    ok = ok & ~part
    # radiation at the sample point
    mid_r = scene.radius(c, mid)
    new_r = scene.radius(c, new)
    near = (s["old_r"] <= c["outer"]) | (mid_r <= c["outer"]) | (new_r <= c["outer"])
    max_rad = torch.where((c["max_rad"] > 0.0) & near, c["max_rad"], torch.zeros_like(h))
    if scene.slow:
        inside = (mid_r >= c["inner"]) & (mid_r < c["outer"])
        late = ok & inside & ~scene.resident(mid)
        _set(s, late, reason=6, on=False)
        ok = ok & ~late
    else:
        inside = (mid_r > c["inner"]) & (mid_r < c["outer"])
    k = scene.coefficients(c, mid, inside)
    required = _substeps(c, k, h, max_rad)
    pred = _substeps(c, k, s["want"], max_rad)
    short = ok & (required > 1.0) & (h > c["min_step"] * 1.0001)
    less = torch.maximum(c["min_step"], h / required)
    _set(s, short, want=less, cap=less, fresh=True)
    ok = ok & ~short
    limited = (max_rad > 0.0) | (c["max_depth"] > 0.0) | (c["max_abs"] > 0.0) | (c["max_far"] > 0.0)
    cap = torch.where(limited & (pred > 1.0), torch.maximum(c["min_step"], s["want"] / pred), c["max_step"])
    _set(s, ok, cap=cap, S=_transfer(s["S"], k, h[:, None] * c["dls"]), Y=new, steps=s["steps"] + 1, fresh=True)
    _set(s, ok & crosses, reason=1, on=False)


def _transfer(S, k, dl):
    """Faraday half step, absorption and emission, Faraday half step."""
    def rotate(P):
        rho = torch.stack([k["rQ"], k["rU"], k["rV"]], -1)
        norm = torch.sqrt((rho * rho).sum(-1, keepdim=True))
        th = norm * (0.5 * dl)[..., None]
        n = rho / torch.where(norm == 0.0, torch.ones_like(norm), norm)
        cross = torch.linalg.cross(n, P)
        f = (n * P).sum(-1, keepdim=True) * (2.0 * torch.sin(0.5 * th) ** 2)
        return P * torch.cos(th) + n * f + cross * torch.sin(th)

    def fade(a):
        return torch.exp(-(a * dl))

    def source(a):
        x = a * dl
        small = x.abs() < 1e-6
        safe = torch.where(small, torch.ones_like(a), a)
        return torch.where(small, dl * (1.0 - x / 2.0 + x * x / 6.0 - x * x * x / 24.0), -torch.expm1(-x) / safe)

    I, P = S[..., 0], rotate(S[..., 1:])
    a = torch.stack([k["aQ"], k["aU"], k["aV"]], -1)
    j = torch.stack([k["jQ"], k["jU"], k["jV"]], -1)
    an = torch.sqrt((a * a).sum(-1))
    n = a / torch.where(an < TINY, torch.ones_like(an), an)[..., None]
    par, jpar = (n * P).sum(-1), (n * j).sum(-1)
    kp_, km = k["aI"] + an, k["aI"] - an
    sp = fade(kp_) * (I + par) + source(kp_) * (k["jI"] + jpar)
    sm = fade(km) * (I - par) + source(km) * (k["jI"] - jpar)
    e, f = fade(k["aI"])[..., None], source(k["aI"])[..., None]
    P2 = n * (0.5 * (sp - sm))[..., None] + (P - n * par[..., None]) * e + (j - n * jpar[..., None]) * f
    return torch.cat([(0.5 * (sp + sm))[..., None], rotate(P2)], -1)


def _image(scene):
    """Observed Stokes [rays, frequencies, 4] and how each ray ended."""
    Y0, c = scene.rays()
    n, nf, dev = Y0.shape[0], c["dls"].shape[1], Y0.device
    zero = torch.zeros(n, dtype=F64, device=dev)
    yes, no = torch.ones(n, dtype=torch.bool, device=dev), torch.zeros(n, dtype=torch.bool, device=dev)
    whole = torch.zeros(n, dtype=torch.int64, device=dev)
    a = dict(on=yes.clone(), fresh=yes.clone(), entered=no.clone(), cross=no.clone(), Y=Y0.clone(), end=Y0.clone(),
             want=-c["step"].abs(), h=zero.clone(), lo=zero.clone(), hi=zero.clone(), old_r=zero.clone(),
             full_h=zero.clone(), surf=zero.clone(), attempt=whole.clone(), n=whole.clone(), inside=whole.clone(),
             reason=whole + 4)

    def masked(step, keys):
        def go(s):
            step(scene, s, {k: s["c_" + k] for k in keys})
        return go

    consts = {"c_" + k: v for k, v in c.items()}
    full = {**a, **consts}
    _advance(masked(_pass_a, list(c)), full)
    _surface(scene, full, c)
    go = full["entered"] & ((full["reason"] == 2) | (full["reason"] == 3))
    cap = torch.where(c["max_rad"] > 0.0, c["max_rad"], c["max_step"])
    b = dict(on=go.clone(), fresh=yes.clone(), cam=no.clone(), Y=full["Y"], want=c["step"].clone(), cap=cap,
             h=zero.clone(), lo=zero.clone(), hi=zero.clone(), old_r=zero.clone(), attempt=whole.clone(),
             steps=whole.clone(), reason=torch.where(go, whole + 4, full["reason"]),
             S=torch.zeros(n, nf, 4, dtype=F64, device=dev))
    full = {**b, **consts}
    keep = torch.nonzero(go).flatten()
    if keep.numel():
        part = {k: v[keep].clone() for k, v in full.items()}
        _advance(masked(_pass_b, list(c)), part)
        for k, v in full.items():
            v[keep] = part[k]
    # to the observer's screen
    g = scene.metric(c, full["Y"])
    R = torch.einsum("nij,nai,nbj->nab", g, Y0[:, 2:], full["Y"][:, 2:])
    r11, r12, r21, r22 = (R[:, i, j, None] for i in (0, 1) for j in (0, 1))
    I, Q, U, V = full["S"].unbind(-1)
    obs = torch.stack([I, 0.5 * Q * (r11 ** 2 - r12 ** 2 - r21 ** 2 + r22 ** 2) + U * (r11 * r12 - r21 * r22),
                       Q * (r11 * r21 - r12 * r22) + U * (r11 * r22 + r12 * r21), (r11 * r22 - r12 * r21) * V], -1)
    return torch.where(go[:, None, None], obs, torch.zeros_like(obs)), full["reason"]


def _pass_constants(p, n, dev):
    def col(v):
        return torch.full((n,), float(v), dtype=F64, device=dev)

    return dict(inner=col(p.inner_radius), outer=col(p.outer_radius), step=col(p.step), min_step=col(abs(p.min_step)),
                max_step=col(p.max_step), tol=col(max(p.adaptive_tolerance, 8.0 * 2.0 ** -52)),
                max_rad=col(p.max_radiation_step), max_depth=col(p.max_radiation_depth),
                max_abs=col(p.max_absorption_depth), max_far=col(p.max_faraday_depth), max_steps=col(p.max_steps),
                camera=col(p.camera.radius), spin=col(p.spin))


def _frequency_constants(freqs, mbh_solar, width, n, dev):
    length = 6.67430e-8 * mbh_solar * 1.98847e33 / (CL * CL)
    f = list(freqs) + [freqs[0]] * (width - len(freqs))
    row = torch.tensor(f, dtype=F64, device=dev)
    live = torch.tensor([1.0] * len(freqs) + [0.0] * (width - len(freqs)), dtype=F64, device=dev)
    return dict(freq=row.expand(n, -1).clone(), dls=(length / row).expand(n, -1).clone(),
                live=live.expand(n, -1).clone())


def _screen_rays(p, g, x, frame, dev):
    """Pinhole rays of one image from its tetrad (numpy) at x."""
    e0, e1, e2, e3 = (torch.tensor(v, dtype=F64, device=dev) for v in frame)
    g = torch.tensor(g, dtype=F64, device=dev)
    cam = p.camera
    pix = torch.arange(cam.nx * cam.ny, device=dev)
    fov_y = cam.fov_y if cam.fov_y > 0.0 else cam.fov
    sx = (((pix % cam.nx).to(F64) + 0.5) / cam.nx - 0.5) * cam.fov + cam.x_offset
    sy = ((torch.div(pix, cam.nx, rounding_mode="floor").to(F64) + 0.5) / cam.ny - 0.5) * fov_y + cam.y_offset
    norm = torch.sqrt(1.0 + sx * sx + sy * sy)
    t1, t2, t3 = (sx / norm)[:, None], (sy / norm)[:, None], (1.0 / norm)[:, None]
    d = e1 * t1 + e2 * t2 + e3 * t3

    def dot(u, v):
        return ((u @ g) * v).sum(-1, keepdim=True)

    f1 = e1 - d * t1
    f1 = f1 / torch.sqrt(dot(f1, f1))
    f2 = e2 - d * t2
    f2 = f2 - f1 * (dot(f2, f1) / dot(f1, f1))
    f2 = f2 / torch.sqrt(dot(f2, f2))
    pos = torch.tensor(x, dtype=F64, device=dev).expand_as(d)
    return torch.stack([pos, e0 + d, f1, f2], 1)


def _tetrad(g, u, toward, trial2, trial1):
    """The observer's orthonormal frame by Gram-Schmidt (numpy)."""
    def dot(a, b):
        return a @ g @ b

    def unit(v):
        return v / math.sqrt(abs(dot(v, v)))

    def without(v, *others):
        for w in others + others:
            v = v - w * (dot(v, w) / dot(w, w))
        return v

    e0 = unit(u)
    e3 = unit(without(toward, e0))
    e2 = unit(without(trial2, e0, e3))
    e1 = unit(without(trial1, e0, e2, e3))
    if np.linalg.det(np.stack([e0, e1, e2, e3])) < 0.0:
        e1 = -e1
    return e0, e1, e2, e3


# ---- Cartesian Kerr-Schild with the analytic RIAF

def _ks_radius(a, x):
    s = (x[..., 1:] ** 2).sum(-1) - a * a
    return torch.sqrt((0.5 * (s + torch.sqrt(s * s + 4.0 * a * a * x[..., 3] ** 2))).clamp(min=TINY))


def _ks_metric(a, x):
    r = _ks_radius(a, x)
    r2, a2, z = r * r, a * a, x[..., 3]
    l = torch.stack([torch.ones_like(r), (r * x[..., 1] + a * x[..., 2]) / (r2 + a2),
                     (r * x[..., 2] - a * x[..., 1]) / (r2 + a2), z / r], -1)
    amp = 2.0 * r2 * r / (r2 * r2 + a2 * z * z)
    eta = torch.eye(4, dtype=F64, device=x.device)
    eta[0, 0].neg_()
    return eta + amp[..., None, None] * l[..., :, None] * l[..., None, :]


def _ks_rhs(c, Y):
    a = c["spin"]
    x, y, z = Y[:, 0, 1], Y[:, 0, 2], Y[:, 0, 3]
    a2 = a * a
    s = x * x + y * y + z * z - a2
    disc = torch.sqrt(s * s + 4.0 * a2 * z * z)
    r2 = 0.5 * (s + disc)
    r = torch.sqrt(r2)
    den = r2 * r2 + a2 * z * z
    rp = r2 + a2
    f = 2.0 * r2 * r / den
    f_r = -2.0 * r2 * (r2 * r2 - 3.0 * a2 * z * z) / (den * den)
    l1, l2, l3 = (r * x + a * y) / rp, (r * y - a * x) / rp, z / r
    g12 = (1.0 + s / disc) * 0.5 / r
    d1, d2 = x * g12, y * g12
    d3 = z * (1.0 + (s + 2.0 * a2) / disc) * 0.5 / r
    df = torch.stack([f_r * d1, f_r * d2, (6.0 * r2 * d3 - f * (4.0 * r * r2 * d3 + 2.0 * a2 * z)) / den], -1)
    u1, u2, u3 = x - 2.0 * r * l1, y - 2.0 * r * l2, -z / r2
    # dl[nu][i] = d l_nu / d x^i
    dl = torch.stack([(r + u1 * d1) / rp, (a + u1 * d2) / rp, u1 * d3 / rp,
                      (-a + u2 * d1) / rp, (r + u2 * d2) / rp, u2 * d3 / rp,
                      u3 * d1, u3 * d2, (r - z * d3) / r2], -1).reshape(-1, 1, 3, 3)
    l = torch.stack([l1, l2, l3], -1)[:, None]
    df, f = df[:, None], f[:, None]
    q0, q = Y[:, 1:, 0], Y[:, 1:, 1:]
    lq = q0 + (q * l).sum(-1)
    Mq = (dl * q[:, :, None, :]).sum(-1)
    dq = (dl * q[:, :, :, None]).sum(-2)
    Dq = (q * df).sum(-1)
    lk, Dk, Mk, dk, k = lq[:, :1], Dq[:, :1], Mq[:, :1], dq[:, :1], q[:, :1]
    common = lq * Dk + lk * Dq + f * ((k * dq).sum(-1) + (q * dk).sum(-1))
    fe, lqe, lke = f[..., None], lq[..., None], lk[..., None]
    t = l * common[..., None] + fe * (lqe * (Mk - dk) + lke * (Mq - dq)) - df * (lke * lqe)
    lt = f * ((l * t).sum(-1) - common)
    out = torch.empty_like(Y)
    out[:, 0] = Y[:, 1]
    out[:, 1:, 0] = 0.5 * (common - lt)
    out[:, 1:, 1:] = -0.5 * (t - l * lt[..., None])
    return out


class _Riaf:
    slow = False

    def __init__(self, jobs, width=None):
        self.jobs = [(p, m, f if width is None else [m.freq_cgs]) for p, m, f in jobs]
        self.adaptive = bool(jobs[0][0].adaptive)

    rhs = staticmethod(_ks_rhs)

    @staticmethod
    def radius(c, Y):
        return _ks_radius(c["spin"], Y[:, 0])

    @staticmethod
    def metric(c, Y):
        return _ks_metric(c["spin"], Y[:, 0])

    def rays(self):
        dev = _device()
        width = max(len(f) for _, _, f in self.jobs)
        Ys, cs = [], []
        for p, m, freqs in self.jobs:
            a, R, th = p.spin, p.camera.radius, p.camera.inclination
            si, ci = math.sin(th), math.cos(th)
            x = np.array([0.0, R * si, a * si, R * ci])
            g = _ks_metric(torch.tensor(a, dtype=F64), torch.tensor(x, dtype=F64)).numpy()
            gi = np.linalg.inv(g)
            xx, yy, zz = x[1:]
            s = xx * xx + yy * yy + zz * zz - a * a
            disc = math.sqrt(s * s + 4.0 * a * a * zz * zz)
            q = 0.5 / (0.5 * (s + disc))
            toward = gi @ np.array([1.0, xx * (1.0 + s / disc) * q, yy * (1.0 + s / disc) * q,
                                    zz * (1.0 + (s + 2.0 * a * a) / disc) * q])

            def native(v0, v1, v2, v3):
                vr, vt = R * v1, math.pi * v2
                return np.array([v0, vr * si + vt * R * ci - v3 * a * si, vt * a * ci + v3 * R * si,
                                 vr * ci - vt * R * si])

            frame = _tetrad(g, -gi[:, 0], toward, native(0.0, 0.0, 1.0, 0.0), native(1.0, 1.0, 1.0, 1.0))
            Y = _screen_rays(p, g, x, frame, dev)
            n = Y.shape[0]
            hor = 1.0 + math.sqrt(max(1.0 - a * a, 0.0))
            z1 = 1.0 + np.cbrt(1.0 - a * a) * (np.cbrt(1.0 + a) + np.cbrt(1.0 - a))
            z2 = math.sqrt(3.0 * a * a + z1 * z1)
            isco = 3.0 + z2 - math.copysign(1.0, a) * math.sqrt((3.0 - z1) * (3.0 + z1 + 2.0 * z2))
            c = {**_pass_constants(p, n, dev), **_frequency_constants(freqs, m.mbh_solar, width, n, dev)}
            for k, v in dict(hor=hor, isco=isco, h_disk=m.disk_h, pow_n=m.pow_nth, pow_t=m.pow_T, ne0=m.nth0 * m.ne_unit,
                             te0=m.Te0 * m.te_unit * KBOL / (ME * CL * CL), r_lo=max(m.r_min, hor + m.horizon_buffer),
                             r_hi=m.r_max).items():
                c[k] = torch.full((n,), float(v), dtype=F64, device=dev)
            Ys.append(Y)
            cs.append(c)
        self.model = self.jobs[0][1]
        return torch.cat(Ys), {k: torch.cat([c[k] for c in cs]) for k in cs[0]}

    def coefficients(self, c, Y, inside):
        a, x = c["spin"], Y[:, 0]
        r = _ks_radius(a, x)
        ct = (x[:, 3] / r).clamp(-1.0, 1.0)
        st = torch.sqrt(((x[:, 1] ** 2 + x[:, 2] ** 2) / (r * r + a * a)).clamp(min=1e-60))
        cp, sp = r * x[:, 1] + a * x[:, 2], r * x[:, 2] - a * x[:, 1]
        np_ = torch.sqrt((cp * cp + sp * sp).clamp(min=TINY))
        cp, sp = cp / np_, sp / np_
        emits = inside & (r > c["r_lo"]) & (r <= c["r_hi"])
        # plasma
        ne = c["ne0"] * torch.exp(-(ct * ct) / (2.0 * st * st * c["h_disk"] ** 2)) * r ** c["pow_n"]
        emits = emits & (ne > 0.0)
        te = (c["te0"] * r ** c["pow_t"]).clamp(min=self.model.min_thetae)
        b = torch.sqrt(8.0 * math.pi * 0.1 * ne * MP * CL * CL / (6.0 * r)).clamp(min=1e-12)
        # flow: circular Keplerian outside the ISCO, plunging from it inside
        def bl(r):
            s2, sig = st * st, r * r + a * a * ct * ct
            dlt = r * r - 2.0 * r + a * a
            tt, tp = -(1.0 - 2.0 * r / sig), -2.0 * a * r * s2 / sig
            pp = (r * r + a * a + 2.0 * a * a * r * s2 / sig) * s2
            itt = -((r * r + a * a) ** 2 - a * a * dlt * s2) / (sig * dlt)
            itp = -2.0 * a * r / (sig * dlt)
            ipp = (dlt - a * a * s2) / (sig * dlt * s2)
            return tt, tp, pp, sig / dlt, itt, itp, ipp, dlt / sig

        tt, tp, pp, rr, itt, itp, ipp, irr = bl(r)
        om = 1.0 / (r * torch.sqrt(r) + a)
        ri = c["isco"]
        tti, tpi, ppi = bl(ri)[:3]
        omi = 1.0 / (ri * torch.sqrt(ri) + a)
        uti = 1.0 / torch.sqrt((-(tti + 2.0 * omi * tpi + omi * omi * ppi)).clamp(min=TINY))
        E, L = (tti + tpi * omi) * uti, (tpi + ppi * omi) * uti
        kk = itt * E * E + 2.0 * itp * E * L + ipp * L * L
        vr_in = -irr * torch.sqrt((-(1.0 + kk) / irr).clamp(min=0.0))
        om_in = (itp * E + ipp * L) / (itt * E + itp * L)
        plunge = r < ri
        om = torch.where(plunge, om_in, om)
        vr = torch.where(plunge, vr_in, torch.zeros_like(r))
        vt = torch.sqrt((-(1.0 + vr * vr * rr) / (tt + 2.0 * om * tp + om * om * pp)).clamp(min=0.0))
        dlt = r * r - 2.0 * r + a * a

        def to_ks(vt, vr, vp):
            vp = vp + a / dlt * vr
            return torch.stack([vt + 2.0 * r / dlt * vr, vr * cp * st - vp * (r * sp + a * cp) * st,
                                vr * sp * st + vp * (r * cp - a * sp) * st, vr * ct], -1)

        g = _ks_metric(a, x)
        u = to_ks(vt, vr, om * vt)
        B = to_ks(torch.zeros_like(r), torch.zeros_like(r), torch.ones_like(r))
        return _screen_coefficients(c, self.model, g, Y, u, B, True, ne, te, b, emits, self.model.min_sin_theta)


def _dot(g, u, v):
    return (u * (g @ v[..., None])[..., 0]).sum(-1)


def _screen_coefficients(c, model, g, Y, u, B, project, ne, te, b, emits, min_sin):
    """Coefficients [N, F] in the transported screen basis of a plasma with
    four-velocity u and field direction B (unnormalised; projected normal to
    u when `project`)."""
    if project:
        u = u / torch.sqrt((-_dot(g, u, u)).clamp(min=TINY))[:, None]
        B = B + u * _dot(g, u, B)[:, None]
    B = B / torch.sqrt(_dot(g, B, B).abs().clamp(min=TINY))[:, None]
    k, e1, e2 = Y[:, 1], Y[:, 2], Y[:, 3]
    uk = _dot(g, u, k)
    nu = uk.abs().clamp(min=1e-8)
    ct = (_dot(g, k, B) / nu).clamp(-1.0, 1.0)
    st = torch.sqrt((1.0 - ct * ct).clamp(min=0.0)).clamp(min=min_sin)
    eK = -k / uk[:, None] - u
    uB, kB = _dot(g, u, B), _dot(g, eK, B)
    b1 = _dot(g, e1, B) + _dot(g, u, e1) * uB - _dot(g, eK, e1) * kB
    b2 = _dot(g, e2, B) + _dot(g, u, e2) * uB - _dot(g, eK, e2) * kB
    bb = (b1 * b1 + b2 * b2).clamp(min=1e-30)
    c2, s2 = ((b2 * b2 - b1 * b1) / bb)[:, None], (-2.0 * b1 * b2 / bb)[:, None]
    one = torch.ones_like(ne)

    def safe(v):
        return torch.where(emits, v, one)[:, None]

    t = _thermal(model, safe(nu) * c["freq"], safe(ne), safe(te), safe(b), safe(st), safe(ct))
    z = torch.zeros_like(c["freq"])
    m = emits[:, None] & (c["live"] > 0.0)
    out = {"jI": t["jI"], "jV": t["jV"], "aI": t["aI"], "aV": t["aV"], "rV": t["rV"]}
    for n in ("j", "a", "r"):
        out[n + "Q"], out[n + "U"] = t[n + "Q"] * c2, t[n + "Q"] * s2
    return {n: torch.where(m & torch.isfinite(v), v, z) for n, v in out.items()}


def _poly(y, *cs):
    p = torch.full_like(y, cs[-1])
    for v in cs[-2::-1]:
        p = v + y * p
    return p


def _bessel_ratios(x):
    """K0/K2 and K1/K2 with the polynomial fits that the method prescribes."""
    xs, xl = x.clamp(max=2.0), x.clamp(min=2.0)
    y, t = xs * xs / 4.0, (xs / 3.75) ** 2
    i0 = _poly(t, 1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813)
    i1 = xs * _poly(t, 0.5, 0.87890594, 0.51498869, 0.15084934, 0.02658733, 0.00301532, 0.00032411)
    lg = torch.log(xs / 2.0)
    k0 = -lg * i0 + _poly(y, -0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698, 0.00010750, 0.00000740)
    k1 = lg * i1 + _poly(y, 1.0, 0.15443144, -0.67278579, -0.18156897, -0.01919402, -0.00110404, -0.00004686) / xs
    w = 2.0 / xl
    p0 = _poly(w, 1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872, -0.00251540, 0.00053208)
    p1 = _poly(w, 1.25331414, 0.23498619, -0.03655620, 0.01504268, -0.00780353, 0.00325614, -0.00068245)
    big = x > 2.0
    k0, k1 = torch.where(big, p0, k0), torch.where(big, p1, k1)
    k2 = k0 + 2.0 * k1 / x
    return k0 / k2, k1 / k2


def _thermal(model, nu, ne, te, b, st, ct):
    """Thermal synchrotron fits (Pandya et al. or Dexter emission, Dexter's
    Faraday coefficients), invariant, in the magnetic basis."""
    if model.emission_type == _abi.FIT_DEXTER:
        x = nu / (3.0 * EE * b * st / (4.0 * math.pi * ME * CL) * te * te + 1.0)
        m13 = x ** (-1.0 / 3.0)
        shape = torch.exp(-1.8899 / m13)
        pref = ne * EE * EE * nu / (2.0 * math.sqrt(3.0) * CL * te * te)
        jI = pref * 2.5651 * (1.0 + 1.92 * m13 + 0.9977 * m13 * m13) * shape
        jQ = pref * 2.5651 * (1.0 + 0.93193 * m13 + 0.499873 * m13 * m13) * shape
        iv = (1.81384 / x + 3.42319 * m13 * m13 + 0.0292545 / torch.sqrt(x) + 2.03773 * m13) * shape
        jV = 2.0 * ne * EE * EE * nu * ct / (st * 3.0 * math.sqrt(3.0) * CL * te ** 3) * iv
    else:
        nu_c = EE * b / (2.0 * math.pi * ME * CL)
        x = nu / (2.0 / 9.0 * nu_c * st * te * te).clamp(min=TINY)
        pref = ne * EE * EE * nu_c / CL
        lin = pref * math.sqrt(2.0) * math.pi / 27.0 * st
        x13 = x ** (1.0 / 3.0)
        ex = torch.exp(-x13)
        bend = 1.8877486253633869933 * torch.sqrt(x13)
        jI = lin * (torch.sqrt(x) + bend) ** 2 * ex
        t = te ** 0.96
        jQ = lin * (torch.sqrt(x) + (7.0 * t + 35.0) / (10.0 * t + 75.0) * bend) ** 2 * ex
        shift = st * 0.4356824462767121 - ct * 0.9001004421765051
        jV = pref * (37.0 - 87.0 * shift) / (100.0 * (te + 1.0)) * (
            1.0 + (te ** 0.6 / 25.0 + 0.7) * x ** 0.36) ** (5.0 / 3.0) * ex
    jI, jQ, jV = (j / (nu * nu) for j in (jI, jQ, jV))
    jP = torch.sqrt(jQ * jQ / (jI * jI) + jV * jV / (jI * jI)) * jI
    cut = torch.where(jI < jP / model.max_pol_frac, jI / jP * model.max_pol_frac, torch.ones_like(jI))
    jQ, jV = jQ * cut, jV * cut
    xb = HPL * nu / (ME * CL * CL * te)
    expm1 = torch.where(xb < 2e-3, xb / 24.0 * (24.0 + xb * (12.0 + xb * (4.0 + xb))), torch.exp(xb) - 1.0)
    binv = 2.0 * HPL / expm1 / (CL * CL)
    om0, wp2, w = EE * b / (ME * CL), 4.0 * math.pi * ne * EE * EE / ME, 2.0 * math.pi * nu
    y = (te * torch.sqrt(math.sqrt(2.0) * st * 1e3 * om0 / w)).clamp(min=1e-12)
    r0, r1 = _bessel_ratios(1.0 / te)
    tail = (0.011 * torch.exp(-y / 47.2) - 369.69342869090815 * (y + 1e-16) ** (-8.0 / 3.0)) * (
        0.5 + 0.5 * torch.tanh((torch.log(y) - 4.787491742782046) / 0.1))
    jf = 2.011 * torch.exp(-(y ** 1.035) / 4.7) - torch.cos(y / 2.0) * torch.exp(
        -(y ** 1.2) / 2.73) - 0.011 * torch.exp(-y / 47.2) + tail
    rQ = math.pi * nu / CL * (jf * wp2 * om0 * om0 / w ** 4) * (r1 + 6.0 * te) * st * st * nu
    rV = 2.0 * math.pi * nu / CL * (wp2 * om0 / w ** 3) * r0 * (1.0 - 0.11 * torch.log(1.0 + 0.035 * y)) * ct * nu
    es, as_, fs = model.emission_scale, model.absorption_scale, model.faraday_scale
    return {"jI": es * jI, "jQ": es * jQ, "jV": es * jV, "aI": as_ * jI / binv, "aQ": as_ * jQ / binv,
            "aV": as_ * jV / binv, "rQ": fs * rQ, "rV": fs * rV}


# ---- FMKS with a GRMHD grid

class _Grmhd:
    def __init__(self, p, model, prims, times, t_obs, freqs, slow):
        self.p, self.model, self.freqs, self.slow = p, model, freqs, slow
        self.adaptive = bool(p.adaptive)
        self.prims, self.times, self.t_obs = prims, times, t_obs

    @staticmethod
    def radius(c, Y):
        return torch.exp(Y[:, 0, 1])

    def theta(self, x1, x2):
        """theta(x1, x2), its first and its second derivatives."""
        m = self.model
        al, xt, pn, sm = m.poly_alpha, m.poly_xt, m.poly_norm, m.mks_smooth
        y = 2.0 * x2 - 1.0
        z = y / xt
        ef = torch.exp(sm * (m.startx1 - x1))
        za = z.abs() ** al
        za1 = z.abs() ** (al - 1.0) * torch.sign(z)
        za2 = z.abs() ** (al - 2.0)
        s2, c2 = torch.sin(2.0 * math.pi * x2), torch.cos(2.0 * math.pi * x2)
        G = math.pi * x2 + 0.5 * (1.0 - m.hslope) * s2
        J = pn * y * (1.0 + za / (al + 1.0)) + 0.5 * math.pi
        dG = math.pi + (1.0 - m.hslope) * math.pi * c2
        dJ = 2.0 * pn * (1.0 + za / (al + 1.0)) + 2.0 * al * pn * y * za1 / ((al + 1.0) * xt)
        ddG = -2.0 * (1.0 - m.hslope) * math.pi ** 2 * s2
        ddJ = 4.0 * pn * al / (al + 1.0) * (2.0 * za1 / xt + y * (al - 1.0) * za2 / (xt * xt))
        t1 = -sm * ef * (J - G)
        return (G + ef * (J - G), t1, dG + ef * (dJ - dG), -sm * t1, -sm * ef * (dJ - dG), ddG + ef * (ddJ - ddG))

    def _native(self, x1, x2):
        """g_{mu nu} and g^{0 mu} of the native coordinates."""
        a = self.model.spin
        r = torch.exp(x1)
        th, t1, t2 = self.theta(x1, x2)[:3]
        s2, c2 = torch.sin(th) ** 2, torch.cos(th) ** 2
        rho = r * r + a * a * c2
        f = 2.0 * r / rho
        z = torch.zeros_like(r)
        rows = [[f - 1.0, f * r, z, -a * f * s2],
                [f * r, (1.0 + f) * r * r + rho * t1 * t1, rho * t1 * t2, -a * s2 * (1.0 + f) * r],
                [z, rho * t1 * t2, rho * t2 * t2, z],
                [-a * f * s2, -a * s2 * (1.0 + f) * r, z, s2 * (rho + a * a * s2 * (1.0 + f))]]
        g = torch.stack([torch.stack(q, -1) for q in rows], -2)
        return g, torch.stack([-(1.0 + f), f / r, -f * t1 / (r * t2), z], -1)

    def metric(self, c, Y):
        return self._native(Y[:, 0, 1], Y[:, 0, 2])[0]

    def rhs(self, c, Y):
        a = self.model.spin
        x1, x2 = Y[:, 0, 1], Y[:, 0, 2]
        th, t1, t2, t11, t12, t22 = self.theta(x1, x2)
        r = torch.exp(x1)
        sn, cs = torch.sin(th), torch.cos(th)
        s2, sc = sn * sn, 2.0 * sn * cs
        rho = r * r + a * a * cs * cs
        f = 2.0 * r / rho
        rho_t = -a * a * sc
        f_r, f_t = 2.0 * (rho - 2.0 * r * r) / (rho * rho), -2.0 * r * rho_t / (rho * rho)
        E = (slice(None), None)
        F0, F1 = (-a * (s2 * f_t + sc * f))[E], (-a * (sc * (1.0 + f) + s2 * f_t))[E]
        A, Bq, C = f_r[E], (-a * s2 * f_r)[E], (2.0 * r)[E]
        D = (s2 * (2.0 * r + a * a * s2 * f_r))[E]
        Ft = f_t[E]
        H = (sc * (rho + a * a * s2 * (1.0 + f)) + s2 * (rho_t + a * a * (sc * (1.0 + f) + s2 * f_t)))[E]
        re, t1e, t2e, rhoe, fe = r[E], t1[E], t2[E], rho[E], f[E]
        n = Y[:, 1:]
        q0, q1, q2, q3 = n[..., 0], re * n[..., 1], t1e * n[..., 1] + t2e * n[..., 2], n[..., 3]
        sig = q0 + q1
        rr = (A * sig + Bq * q3, A * sig + Bq * q3, C * q2, Bq * sig + D * q3)
        rt = (Ft * sig + F0 * q3, Ft * sig + F1 * q3, rho_t[E] * q2, F0 * q0 + F1 * q1 + H * q3)
        q = (q0, q1, q2, q3)
        k = tuple(v[:, :1] for v in q)
        kr, kt = tuple(v[:, :1] for v in rr), tuple(v[:, :1] for v in rt)
        t = [k[1] * rr[i] + q1 * kr[i] + k[2] * rt[i] + q2 * kt[i] for i in range(4)]
        t[1] = t[1] - sum(k[i] * rr[i] for i in range(4))
        t[2] = t[2] - sum(k[i] * rt[i] for i in range(4))
        dlt = (r * r - 2.0 * r + a * a)[E]
        h0 = 0.5 * (-(1.0 + fe) * t[0] + fe * t[1])
        h1 = 0.5 * (fe * t[0] + dlt / rhoe * t[1] + a / rhoe * t[3])
        h2 = 0.5 * t[2] / rhoe
        h3 = 0.5 * (a / rhoe * t[1] + t[3] / (rhoe * s2[E].clamp(min=TINY)))
        kn = n[:, :1]
        h1 = (h1 + re * kn[..., 1] * n[..., 1]) / re
        h2 = h2 + t11[E] * kn[..., 1] * n[..., 1] + t12[E] * (kn[..., 1] * n[..., 2] + kn[..., 2] * n[..., 1]) + \
            t22[E] * kn[..., 2] * n[..., 2]
        out = torch.empty_like(Y)
        out[:, 0] = Y[:, 1]
        out[:, 1:] = -torch.stack([h0, h1, (h2 - t1e * h1) / t2e, h3], -1)
        return out

    def rays(self):
        dev, p, m = _device(), self.p, self.model
        self.cells = [self._cells(torch.tensor(f, device=dev)) for f in self.prims]
        x1 = math.log(p.camera.radius)
        lo, hi = 0.0, 1.0
        for _ in range(64):
            mid = 0.5 * (lo + hi)
            th = self.theta(torch.tensor([x1], dtype=F64), torch.tensor([mid], dtype=F64))[0]
            lo, hi = (mid, hi) if float(th) < p.camera.inclination else (lo, mid)
        x = np.array([0.0, x1, 0.5 * (lo + hi), 0.0])
        g = self._native(torch.tensor([x[1]], dtype=F64), torch.tensor([x[2]], dtype=F64))[0][0].numpy()
        gi = np.linalg.inv(g)
        frame = _tetrad(g, -gi[:, 0], gi @ np.array([1.0, 1.0, 0.0, 0.0]), np.array([0.0, 0.0, 1.0, 0.0]),
                        np.ones(4))
        Y = _screen_rays(p, g, x, frame, dev)
        n = Y.shape[0]
        return Y, {**_pass_constants(p, n, dev),
                   **_frequency_constants(self.freqs, m.mbh_solar, len(self.freqs), n, dev)}

    def _four_vectors(self, g, gc, U, B):
        v2 = (U * (g[..., 1:, 1:] @ U[..., None])[..., 0]).sum(-1)
        fac = torch.sqrt(-1.0 / gc[..., 0] * (1.0 + v2.abs()))[..., None]
        u = torch.cat([-fac * gc[..., :1], U - fac * gc[..., 1:]], -1)
        ub = ((g @ u[..., None])[..., 1:, 0] * B).sum(-1, keepdim=True)
        b = torch.cat([ub, (B + u[..., 1:] * ub) / u[..., :1]], -1)
        return u, b, _dot(g, b, b).abs().clamp(min=1e-40)

    def _cells(self, prims):
        """[n1, n2, n3, 12]: the primitives and n_e, Theta_e, B, sigma of each cell."""
        m = self.model
        P = prims.to(F64).permute(1, 2, 3, 0).contiguous()
        i = torch.arange(m.n1, device=P.device, dtype=F64)
        j = torch.arange(m.n2, device=P.device, dtype=F64)
        x1, x2 = torch.meshgrid(m.startx1 + (i + 0.5) * m.dx1, m.startx2 + (j + 0.5) * m.dx2, indexing="ij")
        g, gc = self._native(x1, x2)
        g, gc = g[:, :, None].expand(-1, -1, m.n3, -1, -1), gc[:, :, None].expand(-1, -1, m.n3, -1)
        bsq = self._four_vectors(g, gc, P[..., 2:5], P[..., 5:8])[2]
        rho, uu = P[..., 0], P[..., 1]
        mp, me = 1.67262171e-24, 9.1093826e-28
        L = 6.67430e-8 * m.mbh_solar * 1.98847e33 / (CL * CL)
        unit = m.M_unit / L ** 3
        beta = (m.gam - 1.0) * uu / (0.5 * bsq)
        bs = (beta / m.beta_crit) ** 2
        trat = (m.trat_large * bs + m.trat_small) / (1.0 + bs)
        te = mp / me * (1.0 / 3.0) * (2.0 / 3.0) / (2.0 / 3.0 + trat / 3.0)
        return torch.cat([P, torch.stack([rho * unit / (mp + me) * m.ne_factor, (te * uu / rho).clamp(min=1e-3),
                                          torch.sqrt(bsq) * CL * math.sqrt(4.0 * math.pi * unit), bsq / rho], -1)],
                         -1).reshape(-1, 12)

    def _stencil(self, x1, x2, phi):
        m = self.model
        phi = phi - torch.floor(phi / (2.0 * math.pi)) * 2.0 * math.pi
        pos = [(x1 - m.startx1) / m.dx1 - 0.5, (x2 - m.startx2) / m.dx2 - 0.5, (phi - m.startx3) / m.dx3 - 0.5]
        base = [torch.floor(v).clamp(-1, n - 1) for v, n in zip(pos, (m.n1, m.n2, m.n3))]
        w = [(v - b).clamp(0.0, 1.0) for v, b in zip(pos, base)]
        cells, weights = [], []
        for bits in range(8):
            o = (bits & 1, bits >> 1 & 1, bits >> 2 & 1)
            i, j, k = (b.to(torch.int64) + d for b, d in zip(base, o))
            pole = (j < 0) | (j >= m.n2)
            k = (k + pole * (m.n3 // 2)) % m.n3
            cells.append((i.clamp(0, m.n1 - 1) * m.n2 + j.clamp(0, m.n2 - 1)) * m.n3 + k)
            fac = [v if d else 1.0 - v for v, d in zip(w, o)]
            weights.append(fac[0] * fac[1] * fac[2])
        return torch.stack(cells, -1), torch.stack(weights, -1)[..., None]

    def resident(self, Y):
        t = self.t_obs + Y[:, 0, 0]
        return (t >= self.times[0]) & (t <= self.times[-1])

    def coefficients(self, c, Y, inside):
        m = self.model
        x1, x2, phi = Y[:, 0, 1], Y[:, 0, 2], Y[:, 0, 3]
        r = torch.exp(x1)
        emits = inside & (r >= m.r_in) & (r < m.r_out) & (x1 >= m.startx1) & (x1 < m.startx1 + m.n1 * m.dx1) & \
            (x2 >= m.startx2) & (x2 < m.startx2 + m.n2 * m.dx2)
        at, w = self._stencil(x1, x2, phi)
        vals = [(cells[at] * w).sum(1) for cells in self.cells]
        if self.slow:
            t = self.t_obs + Y[:, 0, 0]
            v = vals[-1]
            for i in range(len(vals) - 2, -1, -1):
                fr = ((t - self.times[i]) / (self.times[i + 1] - self.times[i])).clamp(0.0, 1.0)[:, None]
                v = torch.where((t < self.times[i + 1])[:, None], (1.0 - fr) * vals[i] + fr * vals[i + 1], v)
        else:
            v = vals[0]
        emits = emits & (v[:, 0] > 0.0) & (v[:, 1] > 0.0)
        g, gc = self._native(x1, x2)
        u, b, _ = self._four_vectors(g, gc, v[:, 2:5], v[:, 5:8])
        sigma = v[:, 11]
        above = m.sigma_cut_high if m.sigma_cut_high > 0.0 else m.sigma_cut
        ramp = torch.cos(0.5 * math.pi / max(above - m.sigma_cut, TINY) * (sigma - m.sigma_cut))
        keep = torch.where(sigma < m.sigma_cut, torch.ones_like(r),
                           torch.where(sigma >= above, torch.zeros_like(r), ramp))
        ne = v[:, 8] * keep
        return _screen_coefficients(c, m, g, Y, u, b, False, ne, v[:, 9], v[:, 10], emits & (ne > 0.0), 1e-4)
