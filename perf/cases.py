"""Performance cases of the geodesic engine: the calls its users make, over the range of sizes.

A case is one call through the package's public entry points: `Engine.integrate` (host
pixels in, host records out), `Engine.integrate_async` (device buffers), `Engine.run` (a
whole adaptive run with its output files), `DeviceMesh.run` (the same with the mesh and the
results in device memory) or `Engine.positions` (the recorded positions of the rays).

Two kinds of screen appear. In plain r a ray from a camera at r = 1000 takes about 66,000
steps of the reference's step rule (0.03), in ln r about 700: the first is what the
benchmark runs, the second what the reference's shipped configurations run.
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

import foort_gb300
from foort_gb300 import abi, workloads

DEG = math.pi / 180.0
METRICS = {"kerr": abi.METRIC_KERR, "flat": abi.METRIC_FLAT, "johannsen": abi.METRIC_JOHANNSEN,
           "rasheed_larsen": abi.METRIC_RASHEED_LARSEN, "manko_novikov": abi.METRIC_MANKO_NOVIKOV}
INTEGRATORS = {"rk4": abi.INTEGRATOR_RK4, "verlet": abi.INTEGRATOR_VERLET}
PRECISIONS = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED, "fp64_analytic": abi.PREC_FP64_ANALYTIC}
# the reference's "Lorenzo" set of Rasheed-Larsen parameters (m, a, p, q)
LORENZO = (0.3556562853309941, 0.2969060968239216, 3.057664971085168, 0.942335028914832)
RESULT_WORDS = abi.RESULT_DTYPE.itemsize // 8
DIAGS = {"quadrant+passes": abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_EQUATORIAL_PASSES,
         "quadrant+radius": abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_CLOSEST_RADIUS,
         "passes+radius": abi.DIAG_EQUATORIAL_PASSES | abi.DIAG_CLOSEST_RADIUS,
         "all": abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_EQUATORIAL_PASSES | abi.DIAG_CLOSEST_RADIUS}


def _view(call, metric, precision, integrator, logr, side, a, inclination, half_width, **more):
    c = {"call": call, "metric": metric, "precision": precision, "integrator": integrator, "logr": logr,
         "side": side, "a": a, "inclination": inclination, "half_width": half_width,
         "alpha13": 0.0, "alpha3": 0.0, "tolerance": 0.001, "timeout": 10000 if logr else 100000,
         "diags": "quadrant+passes"}
    c.update(more)
    return c


def listed():
    return [
        # A first look at a view: the smallest screen, where launch and call costs count.
        dict(_view("integrate", "johannsen", "mixed", "rk4", True, 16, 0.7, 90.0, 6.0, alpha13=2.0), name="preview_16"),
        # An ordinary uniform screen (10,000 rays): too few to fill the GPU.
        dict(_view("integrate", "kerr", "mixed", "rk4", False, 100, 0.5, 80.0, 10.0), name="kerr_view_100"),
        # An adaptive run as a FOORT run makes it: 128 x 128 seed, three subdivisions,
        # host mesh, output files.
        dict(_view("run", "kerr", "mixed", "rk4", False, 128, 0.99, 60.0, 12.0, diags="quadrant+radius",
                   subdivide=3, iteration=800), name="kerr_adaptive_run"),
        # Many images in one launch on device buffers: a parameter study that fills the GPU.
        dict(_view("device", "kerr", "mixed", "rk4", False, 256, 0.5, 45.0, 12.5, images=8), name="kerr_batch_8"),
        # A deformed black hole on a large screen with the Verlet integrator.
        dict(_view("integrate", "johannsen", "mixed", "verlet", False, 384, 0.9, 30.0, 10.0, alpha13=0.4,
                   diags="passes+radius"), name="johannsen_verlet_384"),
        # A deep adaptive run (129 x 129 seed, six subdivisions, 4097 x 4097 grid) with the
        # mesh and the results in device memory.
        dict(_view("dmesh", "kerr", "mixed", "rk4", False, 129, 0.998, 17.0, 10.0, subdivide=6,
                   iteration=1 << 22), name="kerr_deep_device"),
        # The reference's shipped Test configuration, in its own precision.
        dict(_view("integrate", "johannsen", "fp64", "verlet", True, 250, 0.7, 5.0, 7.5, alpha13=2.0,
                   tolerance=-1.0), name="johannsen_fp64_250"),
        # The reference's algorithm on an odd-sized Kerr screen, RK4.
        dict(_view("integrate", "kerr", "fp64", "rk4", True, 101, 0.9, 60.0, 12.0), name="kerr_fp64_101"),
        # The reference's shipped debug configuration (RK4) in mixed precision.
        dict(_view("integrate", "johannsen", "mixed", "rk4", True, 250, 0.7, 90.0, 6.0, alpha13=2.0),
             name="johannsen_mixed_250"),
        # A string-theory black hole with the costliest generated right-hand side.
        dict(_view("integrate", "rasheed_larsen", "mixed", "rk4", True, 97, 0.0, 63.0, 12.0, diags="all"),
             name="rasheed_larsen_97"),
        # Recorded ray paths: a screen and about 25 positions kept of each of its rays.
        dict(_view("positions", "kerr", "mixed", "verlet", True, 60, 0.9, 70.0, 10.0, diags="quadrant+radius",
                   keep=25), name="kerr_positions_60"),
        # The all-FP64 run with analytic derivatives that accuracy is stated against.
        dict(_view("integrate", "kerr", "fp64_analytic", "rk4", True, 64, 0.99, 60.0, 12.0, diags="all"),
             name="kerr_analytic_64"),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "log", "log", "fp64", "fp64", "analytic", "batch", "adaptive", "positions"])
    a = round(rng.uniform(0.0, 0.998), 4)
    inclination = round(rng.uniform(5.0, 88.0), 2)
    half_width = round(rng.uniform(6.0, 15.0), 3)
    diags = rng.choice(sorted(DIAGS))
    if kind == "plain":  # benchmark-like screens, one ray to a full GPU
        metric, integrator = rng.choice([("kerr", "rk4"), ("kerr", "rk4"), ("kerr", "verlet"),
                                         ("johannsen", "verlet"), ("flat", "rk4")])
        return _view("integrate", metric, "mixed", integrator, False, _side(rng, 1, 300), a, inclination, half_width,
                     diags=diags, alpha13=round(rng.uniform(-1.0, 1.0), 3))
    if kind == "batch":
        return _view("device", "kerr", "mixed", "rk4", False, _side(rng, 40, 250), a, inclination, half_width,
                     diags=diags, images=rng.randint(2, 8))
    if kind == "adaptive":
        return _view(rng.choice(["run", "dmesh"]), "kerr", "mixed", "rk4", False, _side(rng, 33, 129),
                     a, inclination, half_width, diags=rng.choice(["quadrant+radius", "quadrant+passes"]),
                     subdivide=rng.randint(2, 4), iteration=rng.randint(100, 2000))
    if kind == "positions":
        return _view("positions", rng.choice(["kerr", "johannsen"]), rng.choice(["mixed", "fp64"]),
                     rng.choice(["rk4", "verlet"]), True, _side(rng, 8, 80), a, inclination, half_width, diags=diags,
                     alpha13=round(rng.uniform(-1.0, 1.0), 3), keep=rng.randint(10, 60))
    integrator = rng.choice(["rk4", "verlet"])
    if kind == "analytic":
        return _view("integrate", rng.choice(["kerr", "johannsen"]), "fp64_analytic", integrator, True,
                     _side(rng, 4, 80), a, inclination, half_width, diags=diags,
                     alpha13=round(rng.uniform(-1.0, 1.0), 3))
    metric = rng.choice(["kerr", "johannsen", "rasheed_larsen", "manko_novikov"])
    side = _side(rng, 4, 48 if metric == "manko_novikov" else 250 if kind == "log" else 110)
    return _view("integrate", metric, "mixed" if kind == "log" else "fp64", integrator, True, side,
                 min(a, 0.95) if metric == "manko_novikov" else a, inclination, half_width, diags=diags,
                 alpha13=round(rng.uniform(-1.0, 2.0), 3), alpha3=round(rng.uniform(1.0, 13.0), 2),
                 timeout=3000 if metric == "manko_novikov" else 10000,  # its deformed core traps rays
                 tolerance=rng.choice([-1.0, 0.001]))


def _params(case, a):
    if case["metric"] == "kerr":
        return (a,)
    if case["metric"] == "johannsen":
        return (a, case["alpha13"], 0.0, 0.0, 0.0)
    if case["metric"] == "rasheed_larsen":
        return LORENZO
    if case["metric"] == "manko_novikov":
        return (max(a, 0.05), case["alpha3"])
    return ()


def _images(case, seed):
    """(parameters, inclination, half-width, side) per image: the case's view, moved a
    little by the seed. The images of a batch spread over spins, inclinations and sides."""
    rng = random.Random(seed)
    out = []
    for k in range(case.get("images", 1)):
        side = case["side"] >> (k % 3)
        a, inc = case["a"], case["inclination"]
        if k:
            a, inc = (a + 0.37 * k) % 0.998, 5.0 + (inc + 31.0 * k) % 80.0
        a = min(a * (1.0 + rng.uniform(-0.02, 0.02)), 0.9985)
        inc = min(max(inc + rng.uniform(-1.0, 1.0), 2.0), 90.0)
        out.append((_params(case, a), inc * DEG, case["half_width"] * (1.0 + rng.uniform(-0.02, 0.02)), max(side, 2)))
    return out


def _horizon_eps(case, params):
    if case["logr"]:
        return 0.01
    return 0.01 / (1.0 + math.sqrt(1.0 - params[0] ** 2)) if params else 0.01


def _desc(case, views):
    d = workloads.base_desc(PRECISIONS[case["precision"]])
    d.metric_id, d.rlog = METRICS[case["metric"]], 1 if case["logr"] else 0
    d.integrator_id, d.verlet_tol = INTEGRATORS[case["integrator"]], case["tolerance"]
    d.timeout_max_steps = case["timeout"]
    d.diag_flags = DIAGS[case["diags"]]
    d.value_diag = abi.DIAG_EQUATORIAL_PASSES if case["diags"] == "passes+radius" else abi.DIAG_FOUR_COLOR_SCREEN
    d.horizon_eps = _horizon_eps(case, views[0][0])
    if case["logr"]:
        d.term_flags |= abi.TERM_THETA_SINGULARITY
        d.smallest_step = 1e-7
    if case["call"] == "positions":
        d.diag_flags |= abi.DIAG_GEODESIC_POSITION
        d.geopos_output_steps = case["keep"]
    ims = [abi.make_image(p, r=1000.0, theta=th, half_width=w, horizon_eps=_horizon_eps(case, p))
           for p, th, w, _ in views]
    return d, abi.attach_images(d, ims)


def prepare(case, seed):
    views = _images(case, seed)
    d, keep = _desc(case, views)
    st = {"case": case, "desc": d, "keep": keep, "engine": foort_gb300.Engine(d)}
    if case["call"] in ("run", "dmesh"):
        st["mesh"] = dict(max_pixels=0, initial_pixels=case["side"] ** 2, max_subdivide=case["subdivide"],
                          iteration_pixels=case["iteration"], initial_sub_to_final=0)
        if case["call"] == "run":
            st["dir"] = tempfile.TemporaryDirectory(prefix="foort_")
            st["files"] = np.zeros((2, 1 << 21), dtype=np.uint8)
        else:
            st["cap"] = 1 << 18
            st["out"] = torch.empty((st["cap"], RESULT_WORDS), dtype=torch.int64, device="cuda")
            st["records"] = torch.zeros_like(st["out"])
        return st
    st["px"] = np.concatenate([abi.square_pixels(v[3], image=i) for i, v in enumerate(views)])
    if case["call"] == "positions":
        st["points"] = np.zeros((2 * case["keep"] * len(st["px"]), 4))
    if case["call"] == "device":
        st["d_px"] = torch.from_numpy(st["px"].view(np.int64)).cuda()
        st["out"] = torch.empty((len(st["px"]), RESULT_WORDS), dtype=torch.int64, device="cuda")
    return st


def _records(r):
    return {name: r[name] for name in abi.RESULT_DTYPE.names}


def _device_records(words):
    """The 104-byte records of a device buffer: words 0, 1 and 11 hold the integers."""
    f = words.view(torch.float64)
    return {"whole": words[:, [0, 1, 11]], "state": f[:, 2:11], "closest_r": f[:, 12]}


def run(state):
    case, e = state["case"], state["engine"]
    if case["call"] == "integrate":
        return _records(e.integrate(state["px"]))
    if case["call"] == "device":
        e.integrate_async(state["d_px"].data_ptr(), len(state["px"]), state["out"].data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
        e.sync()
        return _device_records(state["out"])
    d = state["desc"]
    if case["call"] == "positions":
        first = e.integrate(state["px"])
        counts, points = e.positions(state["px"], first)
        state["points"][:len(points)] = points
        return {**_records(first), "counts": counts, "points": state["points"]}
    if case["call"] == "run":
        mesh = foort_gb300.Mesh("v2", d.diag_flags, d.value_diag, **state["mesh"])
        out = foort_gb300.Output(os.path.join(state["dir"].name, "run"), d.diag_flags, d.value_diag,
                                 first_line=mesh.first_line_info(d))
        geodesics, rounds = e.run([mesh], [out])
        out.close()
        mesh.close()
        for k, name in enumerate(sorted(os.listdir(state["dir"].name))):
            with open(os.path.join(state["dir"].name, name), "rb") as f:
                f.readinto(state["files"][k])
        return {"geodesics": geodesics, "rounds": rounds, "files": state["files"]}
    mesh = foort_gb300.DeviceMesh(d.diag_flags, d.value_diag, stream=torch.cuda.current_stream().cuda_stream,
                                  **state["mesh"])
    kept = [0]

    def on_round(d_px, d_res, n, rnd):  # the round's records go behind those of the rounds before
        state["records"][kept[0]:kept[0] + n] = state["out"][:n]
        kept[0] += n

    geodesics, rounds = mesh.run(e, state["out"].data_ptr(), state["cap"], on_round)
    mesh.close()
    return {"geodesics": geodesics, "rounds": rounds, **_device_records(state["records"])}


# Steps of a ray (r = 1000 camera) and operations of a step with analytic derivatives:
# right-hand sides, stage states, update and checks.
STEPS = {False: 66000, True: 700}
STEP_OPS = {("kerr", "rk4"): 1000, ("kerr", "verlet"): 330, ("flat", "rk4"): 450, ("flat", "verlet"): 180,
            ("johannsen", "rk4"): 2000, ("johannsen", "verlet"): 560, ("rasheed_larsen", "rk4"): 2800,
            ("rasheed_larsen", "verlet"): 800, ("manko_novikov", "rk4"): 6000, ("manko_novikov", "verlet"): 1600}


def work(case):
    n = sum(max(case["side"] >> (k % 3), 2) ** 2 for k in range(case.get("images", 1)))
    if case["call"] in ("run", "dmesh"):
        n = int(n * {2: 1.15, 3: 1.6, 4: 2.4, 6: 11.0}[case["subdivide"]])
    passes = 2 if case["call"] == "positions" else 1
    return {"bytes": (abi.PIXEL_DTYPE.itemsize + abi.RESULT_DTYPE.itemsize) * n * passes,
            "flops": float(n) * STEPS[case["logr"]] * STEP_OPS[case["metric"], case["integrator"]] * passes}


# ---- 64-bit values ------------------------------------------------------------------
# A ray-by-ray integration in torch doubles of the ln r screens of Kerr and Johannsen
# black holes: the metric as written, its derivatives by complex steps, the RK4 or Verlet
# step with the reference's step rule, its terminations and diagnostics.
PI = 3.1415926535  # the reference's constant


def _g_dd(p, x1, th):
    """g_tt, g_tphi, g_rr, g_thth, g_phiphi in (t, ln r, theta, phi)."""
    a, a13 = p[0], (p[1] if len(p) > 1 else 0.0)
    r, s2, c2 = torch.exp(x1), torch.sin(th) ** 2, torch.cos(th) ** 2
    rho2, delta = r * r + a * a * c2, r * r + a * a - 2.0 * r
    ra = (r * r + a * a) * (1.0 + a13 / r ** 3)
    den = ra - a * a * s2
    k = rho2 / (den * den)
    return torch.stack([-k * (delta - a * a * s2), -a * (ra - delta) * k * s2, rho2 / delta * r * r, rho2,
                        k * s2 * (ra * ra - a * a * delta * s2)])


def _inverse(g):
    det = g[0] * g[4] - g[1] * g[1]
    return torch.stack([g[4] / det, -g[1] / det, 1.0 / g[2], 1.0 / g[3], g[0] / det])


def _metric(p, x):
    """d_ln r g, d_theta g and the inverse metric at x."""
    tiny = 1e-30
    z = torch.zeros_like(x[1])
    x1 = torch.complex(torch.stack([x[1], x[1]]), torch.stack([z + tiny, z]))
    th = torch.complex(torch.stack([x[2], x[2]]), torch.stack([z, z + tiny]))
    g = _g_dd(p, x1, th)
    return g[:, 0].imag / tiny, g[:, 1].imag / tiny, _inverse(g[:, 0].real)


def _lower(d, u):
    return torch.stack([d[0] * u[0] + d[1] * u[3], d[2] * u[1], d[3] * u[2], d[1] * u[0] + d[4] * u[3]])


def _accel(m, u):
    d1, d2, gu = m
    w1, w2 = _lower(d1, u), _lower(d2, u)
    f = 2.0 * (u[1] * w1 + u[2] * w2)
    f[1] -= (u * w1).sum(0)
    f[2] -= (u * w2).sum(0)
    return -0.5 * torch.stack([gu[0] * f[0] + gu[1] * f[3], gu[2] * f[1], gu[3] * f[2], gu[1] * f[0] + gu[4] * f[3]])


def _start(p, theta, w, side, device):
    """Initial positions and velocities of the screen's rays (the camera's frame, its
    theta leg without the phi leg's part, then E = 1)."""
    r0 = 1000.0
    one = torch.ones((), dtype=torch.float64)
    g = _g_dd(p, math.log(r0) * one, theta * one)
    gi = _inverse(g)
    full = lambda c: torch.tensor([[c[0], 0, 0, c[1]], [0, c[2], 0, 0], [0, 0, c[3], 0], [c[1], 0, 0, c[4]]],  # noqa: E731
                                  dtype=torch.float64)
    G, U = full(g), full(gi)
    dot = lambda a, b: a @ G @ b  # noqa: E731
    e0 = U[0]
    s0 = -1.0 if dot(e0, e0) < 0 else 1.0
    e0 = s0 * e0 / torch.sqrt(s0 * dot(e0, e0))
    e3 = U[3] - e0 * (s0 * dot(U[3], e0))
    n3 = dot(e3, e3)
    s3 = -1.0 if n3 < 0 else 1.0
    e3 = e3 * (s3 * r0 * math.sin(theta)) / torch.sqrt(s3 * n3)
    e1 = U[1] - e0 * (s0 * dot(U[1], e0)) - e3 * (s3 * dot(U[1], e3))
    e1 = e1 / torch.sqrt(dot(e1, e1))
    e2 = U[2] - e0 * (s0 * dot(U[2], e0))
    e2 = e2 * r0 / torch.sqrt(dot(e2, e2))
    i = torch.arange(side * side, dtype=torch.float64)
    alpha = 2.0 * w * (torch.div(i, side, rounding_mode="floor") / (side - 1) - 0.5)
    beta = 2.0 * w * (torch.remainder(i, side) / (side - 1) - 0.5)
    den = torch.sqrt(r0 * r0 + alpha * alpha + beta * beta)
    pf = torch.stack([-torch.ones_like(den), -r0 / den, -beta / r0 / den, alpha / r0 / math.sin(theta) / den])
    v = torch.stack([e0, e1, e2, e3]).T @ pf
    v = v / (G[0] @ v)
    x = torch.tensor([0.0, math.log(r0), theta, 0.0], dtype=torch.float64)[:, None].expand(4, side * side).clone()
    return x.to(device), v.to(device)


def exact(case, seed):
    if not case["logr"] or case["call"] != "integrate" or case["metric"] not in ("kerr", "johannsen") \
            or case["side"] > 110:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    (p, theta, w, side), = _images(case, seed)
    rk4, tol, diags = case["integrator"] == "rk4", case["tolerance"], DIAGS[case["diags"]]
    horizon = (1.0 + math.sqrt(1.0 - p[0] * p[0])) * (1.0 + _horizon_eps(case, p))
    x, u = _start(p, theta, w, side, device)
    n = side * side
    out = {k: torch.zeros(n, dtype=torch.float64, device=device) for k in ("lam", "closest_r")}
    out.update({k: torch.zeros((n, 4), dtype=torch.float64, device=device) for k in ("pos", "vel")})
    ids = torch.arange(n, device=device)
    lam, rmin = torch.zeros(n, dtype=torch.float64, device=device), torch.exp(x[1])
    for step in range(1, case["timeout"] + 2):
        m = torch.minimum(PI - x[2], x[2])
        h = 1.0 / ((u[1].abs() + 1e-20) / 0.03 + (u[2].abs() + 1e-20) / (0.03 * m).abs() + (u[3] + 1e-20).abs() / 0.03)
        h = torch.clamp(h, min=1e-7)
        if rk4:
            k1 = _accel(_metric(p, x), u)
            u2 = u + 0.5 * h * k1
            k2 = _accel(_metric(p, x + 0.5 * h * u), u2)
            u3 = u + 0.5 * h * k2
            k3 = _accel(_metric(p, x + 0.5 * h * u2), u3)
            u4 = u + h * k3
            k4 = _accel(_metric(p, x + h * u3), u4)
            x, u = x + h / 6.0 * (u + 2.0 * u2 + 2.0 * u3 + u4), u + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        else:
            a0 = _accel(_metric(p, x), u)
            x = x + u * h + a0 * (0.5 * h * h)
            mt, v = _metric(p, x), u + a0 * h
            nv = u + 0.5 * h * (a0 + _accel(mt, v))
            while tol > 0.0:  # each ray iterates until its own velocity settles
                go = ((nv - v) ** 2).sum(0) > tol * tol * (nv ** 2).sum(0)
                if not bool(go.any()):
                    break
                v = torch.where(go, nv, v)
                nv = torch.where(go, u + 0.5 * h * (a0 + _accel(mt, v)), nv)
            u = nv
        lam = lam + h
        r = torch.exp(x[1])
        rmin = torch.minimum(rmin, r)
        hole = r < horizon
        done = hole | (r > 1000.0) | (step > case["timeout"]) | (x[2].abs() < 1e-5) | ((PI - x[2]).abs() < 1e-5)
        if bool(done.any()):
            k = ids[done]
            out["lam"][k], out["pos"][k], out["vel"][k] = lam[done], x[:, done].T, u[:, done].T
            out["closest_r"][k] = torch.where(hole, 0.0, rmin)[done]
            live = ~done
            ids, lam, rmin, x, u = ids[live], lam[live], rmin[live], x[:, live], u[:, live]
        if not len(ids):
            break
    if not diags & abi.DIAG_CLOSEST_RADIUS:
        out["closest_r"][:] = -1.0
    return {name: out[name].cpu().numpy() if name in out else None for name in abi.RESULT_DTYPE.names}
