"""Workloads of the library, each through its public entry points, as a program
that uses it makes them: point-wise metric functors and curvature, curvature
grids, renders (FP64, mixed, several in one launch), ray arrays, the shadow
sweep and bisection, and a mix of requests to the server.

listed() names the fixed cases, draw(rng) gives one more of the same ranges,
prepare(case, seed) what the caller holds before the call, run(state) one call
with its whole outputs, work(case) the bytes and operations it cannot do
without, exact(case, seed) the outputs in 64-bit torch where they have a value
that does not come out of a numerical accident (a fixed step across a horizon).
"""
import math

import numpy as np
import torch

import geon_gb300 as geon

HALF_PI = math.pi / 2
B_C = 3.0 * math.sqrt(3.0)  # critical impact parameter over M
SCHW_ESCAPE = 100.0         # escape radius of the renders, in M

# kind of metric -> (constructor, observer of a render, forward sign)
METRICS = {
    "minkowski": (lambda: geon.Minkowski(), [0.0, 20.0, 0.0, 0.0], 1),
    "schwarzschild": (lambda: geon.Schwarzschild(1.0, 1.001, SCHW_ESCAPE), [0.0, 30.0, HALF_PI, 0.0], 1),
    "alcubierre": (lambda: geon.Alcubierre(2.0, 0.125, 0.5, 0.0), [0.0, -10.0, 0.0, 0.0], -1),
    "morris_thorne": (lambda: geon.MorrisThorne(1.0), [0.0, 10.0, HALF_PI, 0.0], 1),
}
FD_METRICS = ("alcubierre", "morris_thorne")
# operations of one RK4 step: the closed-form right-hand sides (mixed path), and
# the finite-difference fallback of the FP64 path with its structural zeros left out
STEP_FLOPS = {"minkowski": 104, "schwarzschild": 268, "alcubierre": 344, "morris_thorne": 132}
STEP_FLOPS_FD = {"alcubierre": 1412, "morris_thorne": 480}


def listed():
    return [
        # the smallest call: Gamma at a handful of points (a plot, a unit check)
        {"name": "christoffel_few", "family": "points", "op": "christoffel", "metric": "alcubierre", "n": 8},
        # the Schwarzschild vacuum check: R at 1e5 seeded points, r in [3, 50] M
        {"name": "vacuum_100k", "family": "points", "op": "ricci_scalar", "metric": "schwarzschild", "n": 100000},
        # a small curvature slab with device outputs (the slabs of the serving stream, ragged)
        {"name": "slab_dev", "family": "grid", "metric": "morris_thorne", "nx": 33, "ny": 31, "nz": 32, "nk": 16,
         "device": True, "k_out": True},
        # numerical curvature of the warp bubble on 128^3, into the caller's host arrays
        {"name": "grid_128", "family": "grid", "metric": "alcubierre", "nx": 128, "ny": 128, "nz": 128, "nk": 16,
         "device": False, "k_out": False},
        # the default render of the reference (FP64) at its 256^2 view
        {"name": "render_fp64", "family": "render", "metric": "schwarzschild", "precision": "fp64", "width": 256,
         "height": 256, "spa": 1, "u8": False, "stars": True, "fov": 60.0, "max_steps": 20000},
        # a thumbnail of the warp bubble at the default precision (finite-difference Gamma)
        {"name": "render_warp_fp64", "family": "render", "metric": "alcubierre", "precision": "fp64", "width": 96,
         "height": 54, "spa": 1, "u8": False, "stars": True, "fov": 90.0, "max_steps": 5000},
        # a black-hole frame for a video: mixed precision, 2x2 samples, bytes out
        {"name": "frame_mixed", "family": "render", "metric": "schwarzschild", "precision": "mixed", "width": 960,
         "height": 540, "spa": 2, "u8": True, "stars": True, "fov": 60.0, "max_steps": 20000},
        # both exotic images in one launch, every ray near the step cap
        {"name": "batch_exotic", "family": "batch", "width": 512, "height": 384, "fov": 90.0, "max_steps": 20000},
        # the shadow sweep: 2^20 equatorial rays, host arrays in and out
        {"name": "sweep_1m", "family": "sweep", "precision": "mixed", "n": 1 << 20, "r_obs": 20.0, "lo": 10.0,
         "hi": 20.0, "escape": 1000.0},
        # 64 bisections of the critical angle, 40 halvings each
        {"name": "bisect_64", "family": "bisect", "precision": "mixed", "nb": 64, "iters": 40, "r_obs": 20.0,
         "escape": 1000.0},
        # a light-deflection table: escaping rays of every orbit plane, final states out
        {"name": "lens_fast", "family": "lens", "precision": "fp64fast", "n": 36001, "r_obs": 30.0},
        # a burst of requests of every type to the server
        {"name": "serve_mix", "family": "serve", "renders": 5, "bisects": 4, "slabs": 3, "size": 192,
         "precision": "mixed"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["points", "points", "grid", "render", "render", "batch", "sweep", "bisect", "lens", "serve"])
    if family == "points":
        op = rng.choice(["g", "christoffel", "ricci_scalar", "einstein", "nec"])
        return {"family": family, "op": op, "metric": rng.choice(["schwarzschild", "alcubierre", "morris_thorne"]),
                "n": _log(rng, 1, 120000)}
    if family == "grid":
        return {"family": family, "metric": rng.choice(["alcubierre", "morris_thorne", "schwarzschild"]),
                "nx": _log(rng, 3, 128), "ny": _log(rng, 3, 128), "nz": _log(rng, 3, 128), "nk": rng.choice([1, 5, 16]),
                "device": rng.random() < 0.5, "k_out": rng.random() < 0.5}
    if family == "render":
        metric = rng.choice(list(METRICS))
        fov = rng.uniform(40.0, 90.0)
        if rng.random() < 0.5:  # mixed: up to a full frame
            spa = rng.choice([1, 1, 2])
            exotic = metric in FD_METRICS
            return {"family": family, "metric": metric, "precision": "mixed", "width": _log(rng, 16, 640 if exotic else 960),
                    "height": _log(rng, 16, 360 if exotic else 540), "spa": 1 if exotic else spa, "u8": rng.random() < 0.5,
                    "stars": rng.random() < 0.5, "fov": fov, "max_steps": 20000}
        if metric == "schwarzschild":
            return {"family": family, "metric": metric, "precision": rng.choice(["fp64", "fp64", "fp64fast", "adaptive"]),
                    "width": _log(rng, 16, 256), "height": _log(rng, 16, 256), "spa": 1, "u8": rng.random() < 0.5,
                    "stars": rng.random() < 0.5, "fov": fov, "max_steps": 20000}
        return {"family": family, "metric": metric, "precision": "fp64", "width": _log(rng, 9, 96),
                "height": _log(rng, 9, 54), "spa": 1, "u8": False, "stars": True, "fov": fov,
                "max_steps": _log(rng, 1000, 5000)}
    if family == "batch":
        return {"family": family, "width": _log(rng, 17, 512), "height": _log(rng, 17, 384), "fov": rng.uniform(40.0, 90.0),
                "max_steps": 20000}
    if family == "sweep":
        if rng.random() < 0.3:  # FP64: the escape radius of the renders keeps the path short
            return {"family": family, "precision": "fp64", "n": _log(rng, 1, 16384), "r_obs": 20.0, "lo": 10.0, "hi": 20.0,
                    "escape": 100.0}
        r_obs = rng.choice([20.0, 30.0])
        lo = 10.0 if r_obs == 20.0 else 5.0
        return {"family": family, "precision": "mixed", "n": _log(rng, 1, 1 << 20), "r_obs": r_obs, "lo": lo,
                "hi": lo + 10.0, "escape": 1000.0}
    if family == "bisect":
        mixed = rng.random() < 0.7
        return {"family": family, "precision": "mixed" if mixed else "fp64fast", "nb": _log(rng, 1, 64 if mixed else 16),
                "iters": rng.randint(20, 60 if mixed else 40), "r_obs": 20.0, "escape": 1000.0 if mixed else 60.0}
    if family == "lens":
        return {"family": family, "precision": rng.choice(["fp64", "fp64fast", "mixed"]), "n": _log(rng, 1, 36000),
                "r_obs": rng.choice([20.0, 30.0, 50.0])}
    return {"family": "serve", "renders": rng.randint(1, 6), "bisects": rng.randint(0, 5), "slabs": rng.randint(0, 3),
            "size": _log(rng, 32, 192), "precision": "mixed"}


# --- inputs ---------------------------------------------------------------------

def _points(metric, n, rng):
    """Points of the region of interest of a metric's chart."""
    x = np.zeros((n, 4))
    if metric in ("alcubierre", "minkowski"):
        x[:, 1:] = rng.uniform(-4.0, 4.0, (n, 3))
    else:
        x[:, 1] = rng.uniform(3.0, 50.0, n) if metric == "schwarzschild" else rng.uniform(-5.0, 5.0, n)
        x[:, 2] = rng.uniform(0.1, math.pi - 0.1, n)
        x[:, 3] = rng.uniform(0.0, 2.0 * math.pi, n)
    return x


def _grid_box(metric, rng):
    """lo, hi of a grid job: the configured box, moved a little by the seed."""
    if metric == "alcubierre":
        lo, hi = [-4.0] * 3, [4.0] * 3
    elif metric == "morris_thorne":
        lo, hi = [-5.0, 0.4, 0.0], [5.0, 2.7, 6.0]
    else:
        lo, hi = [4.0, 0.4, 0.0], [30.0, 2.7, 6.0]
    move = rng.uniform(-0.05, 0.05, 3)
    return [a + float(d) for a, d in zip(lo, move)], [b + float(d) for b, d in zip(hi, move)]


def _camera(metric, case, rng, width=None, height=None):
    """A view near the configured pose: the observer's distance moves with the seed."""
    _, obs, fs = METRICS[metric]
    obs = list(obs)
    obs[1] *= 1.0 + float(rng.uniform(0.0, 0.05))
    return geon.Camera(obs, case.get("fov", 60.0), width or case["width"], height or case["height"], forward_sign=fs)


def _lens_rays(case, rng):
    """Null rays from a static observer on the equator at r_obs, launch angle
    from the hole outside the shadow (1.05 b_c and more), any orbit plane."""
    n, r = case["n"], case["r_obs"]
    f = 1.0 - 2.0 / r
    a0 = math.asin(1.05 * B_C * math.sqrt(f) / r)
    alpha = rng.uniform(a0, 1.2, n)
    psi = rng.uniform(0.0, 2.0 * math.pi, n)
    # keep the planes away from the chart's poles, where a (theta, phi) step is
    # ill-conditioned: tilt of the plane up to 60 degrees
    psi = np.where(np.abs(np.sin(psi)) > 0.866, psi + HALF_PI, psi)
    y = np.zeros((n, 8))
    y[:, 1], y[:, 2] = r, HALF_PI
    y[:, 4] = 1.0 / math.sqrt(f)
    y[:, 5] = -np.cos(alpha) * math.sqrt(f)
    y[:, 6] = np.sin(alpha) * np.sin(psi) / r
    y[:, 7] = np.sin(alpha) * np.cos(psi) / r
    return y


def prepare(case, seed):
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 0x6E0])
    s = {"case": case}
    family = case["family"]
    if family == "points":
        s["metric"] = METRICS[case["metric"]][0]()
        s["x"] = _points(case["metric"], case["n"], rng)
        if case["op"] == "nec":
            s["k"] = rng.normal(size=(5, 4))  # five vectors shared by every point
    elif family == "grid":
        s["metric"] = METRICS[case["metric"]][0]()
        s["lo"], s["hi"] = _grid_box(case["metric"], rng)
        s["n"] = (case["nx"], case["ny"], case["nz"])
        s["seed"] = int(rng.integers(1 << 40))
        npts, nk = case["nx"] * case["ny"] * case["nz"], case["nk"]
        if case["device"]:
            s["ein"] = torch.empty((npts, 4, 4), dtype=torch.float64, device="cuda")
            s["nec"] = torch.empty((npts, nk), dtype=torch.float64, device="cuda")
            s["k"] = torch.empty((npts, nk, 4), dtype=torch.float64, device="cuda") if case["k_out"] else None
        else:
            # reused result arrays, written once as a program's warm-up call would
            s["ein"], s["nec"] = np.zeros((npts, 4, 4)), np.zeros((npts, nk))
            s["k"] = np.zeros((npts, nk, 4)) if case["k_out"] else None
            for a in (s["ein"], s["nec"], s["k"]):
                if a is not None:
                    a.fill(0.0)
    elif family == "render":
        s["metric"] = METRICS[case["metric"]][0]()
        s["cam"] = _camera(case["metric"], case, rng)
        # flat space: a coarser step, so that rays reach the escape radius within the cap
        step = 0.1 * (1.0 + float(rng.uniform(0.0, 0.05))) if case["metric"] == "minkowski" else 0.05
        s["cfg"] = geon.RenderConfig(step=step, max_steps=case["max_steps"], samples_per_axis=case["spa"],
                                     show_stars=case["stars"], precision=case["precision"])
    elif family == "batch":
        cfg = geon.RenderConfig(max_steps=case["max_steps"], show_stars=True, precision="mixed")
        s["items"] = [(METRICS[m][0](), _camera(m, case, rng), cfg) for m in FD_METRICS]
    elif family == "sweep":
        s["metric"] = geon.Schwarzschild(1.0, 1.001, case["escape"])
        s["alpha"] = np.radians(rng.uniform(case["lo"], case["hi"], case["n"]))
    elif family == "bisect":
        s["metric"] = geon.Schwarzschild(1.0, 1.001, case["escape"])
        s["lo"] = np.radians(rng.uniform(13.0, 14.0, case["nb"]))
        s["hi"] = np.radians(rng.uniform(14.5, 15.5, case["nb"]))
    elif family == "lens":
        s["metric"] = geon.Schwarzschild(1.0, 1.001, SCHW_ESCAPE)
        s["y0"] = _lens_rays(case, rng)
    else:
        s["server"] = geon.Server(2 << 30)
        s["requests"] = _requests(case, rng)
    return s


def _requests(case, rng):
    """A burst of requests: renders over the four metrics, bisections, curvature slabs."""
    out = []
    for i in range(case["renders"]):
        m = list(METRICS)[(1 + i) % 4]
        cam = _camera(m, {"fov": float(rng.uniform(40.0, 90.0))}, rng, case["size"], case["size"] * (8 - i) // 8)
        out.append(("render", METRICS[m][0](), cam, geon.RenderConfig(precision=case["precision"], show_stars=True)))
    for _ in range(case["bisects"]):
        out.append(("bisect", geon.Schwarzschild(1.0), math.radians(float(rng.uniform(13.0, 14.0))),
                    math.radians(float(rng.uniform(14.5, 15.5)))))
    for _ in range(case["slabs"]):
        lo, hi = _grid_box("alcubierre", rng)
        out.append(("slab", METRICS["alcubierre"][0](), lo, hi))
    return out


# --- one pass -------------------------------------------------------------------

def _stats(st):
    return {"captured": st.captured, "escaped": st.escaped, "diverged": st.diverged, "steps": st.total_steps,
            "max_null": st.max_null_residual, "avg_steps": st.avg_steps}


def run(s):
    case = s["case"]
    family = case["family"]
    if family == "points":
        op, m, x = case["op"], s["metric"], s["x"]
        if op in ("g", "christoffel"):
            return getattr(m, op)(x)
        if op == "nec":
            return geon.curvature.nec_contraction(m, x, s["k"])
        return getattr(geon.curvature, op)(m, x)
    if family == "grid":
        if case["device"]:
            geon.curvature.grid_dev(s["metric"], s["lo"], s["hi"], s["n"], s["ein"], s["nec"], nk=case["nk"],
                                    seed=s["seed"], k_out=s["k"], stream=torch.cuda.current_stream().cuda_stream)
        else:
            geon.curvature.grid_into(s["metric"], s["lo"], s["hi"], s["n"], s["ein"], s["nec"], s["k"], nk=case["nk"],
                                     seed=s["seed"])
        return {"einstein": s["ein"], "nec": s["nec"], "k": s["k"]}
    if family == "render":
        if case["u8"]:
            rgb8, rgb, st = geon.render_u8(s["metric"], s["cam"], s["cfg"], with_float=True)
            return {"rgb8": rgb8, "rgb": rgb, "stats": _stats(st)}
        rgb, st, cls, pst = geon.render(s["metric"], s["cam"], s["cfg"], with_classes=True)
        return {"rgb": rgb, "class": cls, "steps": pst, "stats": _stats(st)}
    if family == "batch":
        return [{"rgb": rgb, "class": cls, "steps": pst, "stats": _stats(st)}
                for rgb, st, cls, pst in geon.render_batch(s["items"])]
    if family == "sweep":
        term, steps = geon.shadow.classify(s["metric"], case["r_obs"], s["alpha"], precision=case["precision"])
        return {"term": term, "steps": steps}
    if family == "bisect":
        ac, lo, hi, steps = geon.shadow.bisect(s["metric"], case["r_obs"], s["lo"], s["hi"], iters=case["iters"],
                                               precision=case["precision"])
        return {"alpha_c": ac, "lo": lo, "hi": hi, "steps": steps}
    if family == "lens":
        r = geon.trace(s["metric"], s["y0"], 0.05, 20000, precision=case["precision"])
        return {"term": r.termination, "state": r.final_state, "steps": r.steps_taken, "resid": r.null_residual}
    srv, jobs = s["server"], []
    for q in s["requests"]:
        if q[0] == "render":
            jobs.append(srv.submit_render(q[1], q[2], q[3]))
        elif q[0] == "bisect":
            jobs.append(srv.submit_bisect(q[1], 20.0, q[2], q[3], iters=32, precision=case["precision"]))
        else:
            jobs.append(srv.submit_curvature(q[1], q[2], q[3], (32, 32, 32), nk=16, seed=77))
    out = {"render": [], "slab": [], "bisect": []}
    for q, j in zip(s["requests"], jobs):
        r = j.result()
        if q[0] == "render":
            st = r[1]
            r = {"rgb": r[0], "class": r[2], "steps": r[3],
                 "counts": np.array([st.captured, st.escaped, st.diverged, st.total_steps]), "null_and_avg": np.array([st.max_null_residual, st.avg_steps])}
        out[q[0]].append(r)
    out["bisect"] = {k: np.array([b[k] for b in out["bisect"]]) for k in ("alpha_c", "lo", "hi", "steps")}
    return out


# --- what a pass cannot do without ------------------------------------------------

def _trace_work(metric, precision, rays, max_steps, escape=SCHW_ESCAPE, r_obs=30.0, step=0.05):
    """Ray-steps of a view, and their operations."""
    if metric == "schwarzschild":
        steps = min(max_steps, (escape + r_obs) / step)
    elif metric == "minkowski":
        steps = min(max_steps, 1000.0 / step)
    else:
        steps = max_steps
    flops = STEP_FLOPS_FD[metric] if precision == "fp64" and metric in STEP_FLOPS_FD else STEP_FLOPS[metric]
    if precision == "adaptive":
        steps = steps / 50.0
        flops = 400
    return rays * steps * flops


GAMMA_FLOPS = {"minkowski": 1, "schwarzschild": 60, "alcubierre": 350, "morris_thorne": 120}


def work(case):
    family = case["family"]
    if family == "points":
        width = {"g": 16, "christoffel": 64, "ricci_scalar": 1, "einstein": 16, "nec": 5}[case["op"]]
        gam = GAMMA_FLOPS[case["metric"]]
        flops = {"g": 20, "christoffel": gam}.get(case["op"], 9 * gam + 1200)
        return {"bytes": 8 * case["n"] * (4 + width), "flops": case["n"] * flops}
    if family == "grid":
        n = case["nx"] * case["ny"] * case["nz"]
        per = 8 * (16 + case["nk"] * (5 if case["k_out"] else 1))
        flops = {"alcubierre": 10000, "morris_thorne": 5000, "schwarzschild": 3000}[case["metric"]]
        return {"bytes": n * per, "flops": n * (flops + case["nk"] * 80)}
    if family == "render":
        npix = case["width"] * case["height"]
        rays = npix * case["spa"] ** 2
        return {"bytes": npix * (15 if case["u8"] else 24),
                "flops": _trace_work(case["metric"], case["precision"], rays, case["max_steps"])}
    if family == "batch":
        npix = case["width"] * case["height"]
        return {"bytes": 2 * npix * 24,
                "flops": sum(_trace_work(m, "mixed", npix, case["max_steps"]) for m in FD_METRICS)}
    if family == "sweep":
        a_c = math.degrees(math.asin(B_C * math.sqrt(1.0 - 2.0 / case["r_obs"]) / case["r_obs"]))
        esc = (case["hi"] - a_c) / (case["hi"] - case["lo"])
        steps = esc * (case["escape"] + case["r_obs"]) / 0.01 + (1.0 - esc) * case["r_obs"] / 0.01
        return {"bytes": case["n"] * 20, "flops": case["n"] * steps * 268}
    if family == "bisect":
        return {"bytes": case["nb"] * 48, "flops": case["nb"] * case["iters"] * 2.0 * case["r_obs"] / 0.01 * 268}
    if family == "lens":
        return {"bytes": case["n"] * (64 + 84),
                "flops": _trace_work("schwarzschild", case["precision"], case["n"], 20000, r_obs=case["r_obs"])}
    rays = sum(case["size"] * (case["size"] * (8 - i) // 8) for i in range(case["renders"]))
    flops = sum(_trace_work(list(METRICS)[(1 + i) % 4], "mixed", case["size"] ** 2 * (8 - i) / 8, 20000)
                for i in range(case["renders"]))
    flops += case["bisects"] * 32 * 4000 * 268 + case["slabs"] * 32768 * 11000
    return {"bytes": rays * 24 + case["slabs"] * 32768 * 256 + case["bisects"] * 40, "flops": flops}


# --- 64-bit values in plain torch --------------------------------------------------

def _metric_jet(metric, x):
    """g, its first derivatives dg[a] and second derivatives ddg[a][b], in closed form."""
    n = x.shape[0]
    z = dict(dtype=torch.float64, device=x.device)
    g, dg, ddg = torch.zeros(n, 4, 4, **z), torch.zeros(n, 4, 4, 4, **z), torch.zeros(n, 4, 4, 4, 4, **z)
    g[:, 0, 0], g[:, 1, 1], g[:, 2, 2], g[:, 3, 3] = -1.0, 1.0, 1.0, 1.0
    if metric == "alcubierre":
        R, s, v = 2.0, 0.125, 0.5
        p = x[:, 1:]
        r = p.norm(dim=1)
        tp, tm = torch.tanh((r + R) / s), torch.tanh((r - R) / s)
        norm = 1.0 / (2.0 * math.tanh(R / s))
        sp, sm = 1.0 - tp * tp, 1.0 - tm * tm
        f = (tp - tm) * norm
        f1 = (sp - sm) * norm / s
        f2 = -2.0 * (tp * sp - tm * sm) * norm / s ** 2
        e = p / r[:, None]
        eye = torch.eye(3, **z)
        fi = f1[:, None] * e
        ee = e[:, :, None] * e[:, None, :]
        fij = f2[:, None, None] * ee + (f1 / r)[:, None, None] * (eye - ee)
        g[:, 0, 0] = -1.0 + v * v * f * f
        g[:, 0, 1] = g[:, 1, 0] = -v * f
        dg[:, 1:, 0, 0] = 2.0 * v * v * f[:, None] * fi
        dg[:, 1:, 0, 1] = dg[:, 1:, 1, 0] = -v * fi
        ddg[:, 1:, 1:, 0, 0] = 2.0 * v * v * (fi[:, :, None] * fi[:, None, :] + f[:, None, None] * fij)
        ddg[:, 1:, 1:, 0, 1] = ddg[:, 1:, 1:, 1, 0] = -v * fij
    elif metric == "morris_thorne":
        l, s, c = x[:, 1], torch.sin(x[:, 2]), torch.cos(x[:, 2])
        r2 = 1.0 + l * l
        g[:, 2, 2], g[:, 3, 3] = r2, r2 * s * s
        dg[:, 1, 2, 2], dg[:, 1, 3, 3], dg[:, 2, 3, 3] = 2.0 * l, 2.0 * l * s * s, 2.0 * r2 * s * c
        ddg[:, 1, 1, 2, 2], ddg[:, 1, 1, 3, 3] = 2.0, 2.0 * s * s
        ddg[:, 2, 2, 3, 3] = 2.0 * r2 * (c * c - s * s)
        ddg[:, 1, 2, 3, 3] = ddg[:, 2, 1, 3, 3] = 4.0 * l * s * c
    elif metric == "schwarzschild":
        r, s, c = x[:, 1], torch.sin(x[:, 2]), torch.cos(x[:, 2])
        f = 1.0 - 2.0 / r
        f1, f2 = 2.0 / r ** 2, -4.0 / r ** 3
        g[:, 0, 0], g[:, 1, 1], g[:, 2, 2], g[:, 3, 3] = -f, 1.0 / f, r * r, r * r * s * s
        dg[:, 1, 0, 0], dg[:, 1, 1, 1] = -f1, -f1 / f ** 2
        dg[:, 1, 2, 2], dg[:, 1, 3, 3], dg[:, 2, 3, 3] = 2.0 * r, 2.0 * r * s * s, 2.0 * r * r * s * c
        ddg[:, 1, 1, 0, 0], ddg[:, 1, 1, 1, 1] = -f2, -f2 / f ** 2 + 2.0 * f1 ** 2 / f ** 3
        ddg[:, 1, 1, 2, 2], ddg[:, 1, 1, 3, 3] = 2.0, 2.0 * s * s
        ddg[:, 2, 2, 3, 3] = 2.0 * r * r * (c * c - s * s)
        ddg[:, 1, 2, 3, 3] = ddg[:, 2, 1, 3, 3] = 4.0 * r * s * c
    return g, dg, ddg


def _curvature(metric, x):
    """Gamma, the Einstein tensor and R of a metric at points x, analytically."""
    g, dg, ddg = _metric_jet(metric, x)
    gi = torch.linalg.inv(g)
    low = 0.5 * (dg.permute(0, 2, 1, 3) + dg.permute(0, 2, 3, 1) - dg)        # Gamma_{s a b}
    dlow = 0.5 * (ddg.permute(0, 1, 3, 2, 4) + ddg.permute(0, 1, 3, 4, 2) - ddg)  # d_m Gamma_{s a b}
    gam = torch.einsum("nus,nsab->nuab", gi, low)
    dgi = -torch.einsum("nua,nmab,nbs->nmus", gi, dg, gi)
    dgam = torch.einsum("nmus,nsab->nmuab", dgi, low) + torch.einsum("nus,nmsab->nmuab", gi, dlow)
    ric = (torch.einsum("nccab->nab", dgam) - torch.einsum("nbcac->nab", dgam)
           + torch.einsum("ncab,ndcd->nab", gam, gam) - torch.einsum("ncad,ndbc->nab", gam, gam))
    rs = torch.einsum("nab,nab->n", gi, ric)
    return g, gam, ric - 0.5 * g * rs[:, None, None], rs


def _null_vectors(g, seed, nk, first):
    """The grid job's null vectors: splitmix64 directions in the static observer's tetrad."""
    n = g.shape[0]

    def mix(v):
        v = v + np.uint64(0x9E3779B97F4A7C15)
        v = (v ^ (v >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        v = (v ^ (v >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return v ^ (v >> np.uint64(31))

    idx = (np.arange(n * nk, dtype=np.uint64) + np.uint64(first * nk)) ^ np.uint64(seed)
    h = mix(idx)
    u = torch.from_numpy((h >> np.uint64(11)).astype(np.float64)).to(g.device).view(n, nk) * 2.0 ** -53
    w = torch.from_numpy((mix(h) >> np.uint64(11)).astype(np.float64)).to(g.device).view(n, nk) * 2.0 ** -53
    c = 2.0 * u - 1.0
    rho, phi = torch.sqrt(torch.clamp(1.0 - c * c, min=0.0)), 2.0 * math.pi * w
    dirs = torch.stack([torch.ones_like(c), rho * torch.cos(phi), rho * torch.sin(phi), c], dim=2)
    e = torch.zeros(n, 4, 4, dtype=torch.float64, device=g.device)
    e[:, 0, 0] = 1.0 / torch.sqrt(-g[:, 0, 0])
    for i in range(1, 4):
        v = torch.zeros(n, 4, dtype=torch.float64, device=g.device)
        v[:, i] = 1.0
        for j in range(i):
            gj = torch.einsum("nab,nb->na", g, e[:, j])
            v = v - ((gj * v).sum(1) / (gj * e[:, j]).sum(1))[:, None] * e[:, j]
        e[:, i] = v / torch.sqrt(torch.einsum("nab,na,nb->n", g, v, v))[:, None]
    return torch.einsum("nqa,nam->nqm", dirs, e)


def _exact_points(case, s):
    x = torch.from_numpy(s["x"]).cuda()
    metric, op = case["metric"], case["op"]
    flat = metric in ("minkowski", "schwarzschild")  # vacuum: the curvature is rounding noise about 0
    if flat and op in ("ricci_scalar", "einstein", "nec") or metric == "minkowski" and op == "christoffel":
        return None
    g, gam, ein, rs = _curvature(metric, x)
    if op == "nec":
        k = torch.from_numpy(s["k"]).cuda()
        return torch.einsum("nab,qa,qb->nq", ein, k, k) / (8.0 * math.pi)
    return {"g": g, "christoffel": gam, "ricci_scalar": rs, "einstein": ein}[op]


def _exact_grid(case, s):
    if case["metric"] == "schwarzschild":
        return None
    pts = torch.from_numpy(geon.curvature.grid_points(s["lo"], s["hi"], s["n"])).cuda()
    n, nk = pts.shape[0], case["nk"]
    ein, nec, ks = [], [], []
    for i in range(0, n, 1 << 18):
        g, _, e, _ = _curvature(case["metric"], pts[i:i + (1 << 18)])
        k = _null_vectors(g, s["seed"], nk, i)
        ein.append(e)
        nec.append(torch.einsum("nab,nqa,nqb->nq", e, k, k) / (8.0 * math.pi))
        if case["k_out"]:
            ks.append(k)
    return {"einstein": torch.cat(ein), "nec": torch.cat(nec), "k": torch.cat(ks) if ks else None}


def _schw_rhs(y):
    _, r, th, _, p0, p1, p2, p3 = y.unbind(1)
    s, c = torch.sin(th), torch.cos(th)
    f = 1.0 - 2.0 / r
    a = 1.0 / (r * r)
    k4 = -2.0 * (a / f) * p0 * p1
    k5 = -a * f * p0 * p0 + (a / f) * p1 * p1 + (r - 2.0) * (p2 * p2 + s * s * p3 * p3)
    k6 = -2.0 / r * p1 * p2 + s * c * p3 * p3
    k7 = -2.0 * p3 * (p1 / r + c / s * p2)
    return torch.stack([p0, p1, p2, p3, k4, k5, k6, k7], dim=1)


def _exact_lens(case, s):
    """Fixed-step RK4 of the same rays to the escape radius, in the chart."""
    if case["precision"] == "mixed":
        return None  # its final azimuth is the orbit frame's: no count of turns
    y = torch.from_numpy(s["y0"]).cuda()
    out, live = y.clone(), torch.arange(y.shape[0], device=y.device)
    h = 0.05
    for n in range(20000):
        if n % 16 == 0 or n > 2300:
            done = y[:, 1] > SCHW_ESCAPE
            if bool(done.any()):
                out[live[done]] = y[done]
                y, live = y[~done], live[~done]
                if y.shape[0] == 0:
                    break
        k1 = _schw_rhs(y)
        k2 = _schw_rhs(y + 0.5 * h * k1)
        k3 = _schw_rhs(y + 0.5 * h * k2)
        k4 = _schw_rhs(y + h * k3)
        step = y + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        y = torch.where((y[:, 1] > SCHW_ESCAPE)[:, None], y, step)
    return {"state": out}


def exact(case, seed):
    family = case["family"]
    if family in ("render", "batch", "sweep", "serve"):
        return None  # images, classes and counts
    if family == "bisect":
        r = case["r_obs"]
        a = math.asin(B_C * math.sqrt(1.0 - 2.0 / r) / r)
        return {"alpha_c": np.full(case["nb"], a)}
    s = prepare(case, seed)
    return {"points": _exact_points, "grid": _exact_grid, "lens": _exact_lens}[family](case, s)
