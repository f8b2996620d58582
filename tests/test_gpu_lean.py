"""The lean mixed kernels (kernel_lean.cuh) against the general ones: the same records bit
for bit. FOORT_MIXED_FP64_DECISIONS takes the general kernel, whose decisions agree with
the float-float ones except within 2^-48 of a threshold, so no tolerance is needed."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from foort_gb300 import abi, workloads

ALL_DIAGS = abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_EQUATORIAL_PASSES | abi.DIAG_CLOSEST_RADIUS
LORENZO = (0.3556562853309941, 0.2969060968239216, 3.057664971085168, 0.942335028914832)


@pytest.fixture(scope="module")
def eng():
    import foort_gb300
    from foort_gb300 import build as engine_build
    engine_build.build()
    foort_gb300.check_layout()
    return foort_gb300


def describe(metric, params, rlog, inclination, integrator=abi.INTEGRATOR_RK4, timeout=None):
    d = workloads.base_desc(abi.PREC_MIXED)
    d.metric_id, d.rlog, d.integrator_id = metric, rlog, integrator
    d.timeout_max_steps = timeout or (10000 if rlog else 100000)
    d.diag_flags = ALL_DIAGS
    if rlog:
        d.term_flags |= abi.TERM_THETA_SINGULARITY
    keep = abi.attach_images(d, [abi.make_image(params, r=1000.0, theta=np.radians(inclination), half_width=9.0)])
    return d, keep


def same_records(a, b):
    for name in abi.RESULT_DTYPE.names:
        np.testing.assert_array_equal(a[name], b[name], err_msg=name)


# spins from none to near-extremal, views along the axis and from the equator (where every
# step is inside EquatorialPasses' threshold), a ray that ends after one step
@pytest.mark.gpu
@pytest.mark.parametrize("metric,params,rlog,inclination,side,timeout", [
    (abi.METRIC_KERR, (0.0,), 1, 63.0, 23, None),
    (abi.METRIC_KERR, (0.998,), 1, 17.0, 37, None),
    (abi.METRIC_KERR, (0.7,), 1, 90.0, 21, None),
    (abi.METRIC_KERR, (0.9,), 1, 2.0, 21, None),
    (abi.METRIC_KERR, (0.9,), 0, 80.0, 9, None),
    (abi.METRIC_KERR, (0.9,), 0, 60.0, 2, None),
    (abi.METRIC_KERR, (0.9,), 1, 60.0, 33, 0),
    (abi.METRIC_KERR, (0.9,), 1, 60.0, 33, 400),
    (abi.METRIC_FLAT, (), 0, 63.0, 7, None),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1), 1, 63.0, 33, None),
    (abi.METRIC_JOHANNSEN, (0.7, 2.0, 0.0, 0.0, 0.0), 1, 90.0, 21, None),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1), 0, 63.0, 3, 20000),
    (abi.METRIC_JOHANNSEN, (0.3, -0.9, 0.0, 0.0, 0.0), 1, 30.0, 33, None),
    (abi.METRIC_JOHANNSEN, (0.99, 0.0, 0.0, 0.0, 0.0), 1, 2.0, 17, None),
    (abi.METRIC_JOHANNSEN, (0.9, 0.4, 0.0, 0.0, 0.0), 0, 30.0, 9, None),
    (abi.METRIC_JOHANNSEN, (0.7, 2.0, 0.0, 0.0, 1e-3), 1, 90.0, 9, None),
    (abi.METRIC_RASHEED_LARSEN, LORENZO, 1, 63.0, 33, None),
    (abi.METRIC_RASHEED_LARSEN, LORENZO, 0, 63.0, 3, 20000),
])
def test_lean_kernels_give_the_general_kernels_records(eng, metric, params, rlog, inclination, side, timeout):
    px = abi.square_pixels(side)
    d, keep = describe(metric, params, rlog, inclination, timeout=timeout)
    got = {}
    for lanes in (1, 2):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[lanes] = e.integrate(px)
            counts = e.stats()
            assert counts["rhs_evals"] == 4 * counts["steps"] == 4 * int(got[lanes]["steps"].sum())
    d.mixed_options = abi.MIXED_FP64_DECISIONS
    with eng.Engine(d) as e:
        e.set_lanes(1)
        want = e.integrate(px)
    same_records(got[1], want)
    same_records(got[2], want)
    del keep


# tolerances: no velocity iterations, a few, many
@pytest.mark.gpu
@pytest.mark.parametrize("metric,params,rlog,inclination,side,timeout,tolerance", [
    (abi.METRIC_KERR, (0.9,), 1, 63.0, 33, None, -1.0),
    (abi.METRIC_KERR, (0.998,), 1, 17.0, 33, None, 0.001),
    (abi.METRIC_KERR, (0.0,), 1, 90.0, 17, None, 1e-5),
    (abi.METRIC_KERR, (0.7,), 0, 63.0, 5, 20000, 0.001),
    (abi.METRIC_FLAT, (), 0, 63.0, 7, 20000, 0.001),
    (abi.METRIC_FLAT, (), 0, 63.0, 5, 3000, 1e-7),
    (abi.METRIC_JOHANNSEN, (0.9, 0.4, 0.0, 0.0, 0.0), 1, 63.0, 33, None, -1.0),
    (abi.METRIC_JOHANNSEN, (0.3, -0.9, 0.0, 0.0, 0.0), 1, 2.0, 33, None, 1e-5),
    (abi.METRIC_JOHANNSEN, (0.9, 0.4, 0.0, 0.0, 0.0), 0, 30.0, 5, 20000, 0.001),
    (abi.METRIC_JOHANNSEN, (0.9, 0.4, 0.0, 0.0, 0.0), 1, 63.0, 2, 0, 0.001),
])
def test_lean_verlet_gives_the_general_kernels_records(eng, metric, params, rlog, inclination, side, timeout, tolerance):
    px = abi.square_pixels(side)
    d, keep = describe(metric, params, rlog, inclination, integrator=abi.INTEGRATOR_VERLET, timeout=timeout)
    d.verlet_tol = tolerance
    with eng.Engine(d) as e:
        got, counts = e.integrate(px), e.stats()
    d.mixed_options = abi.MIXED_FP64_DECISIONS
    with eng.Engine(d) as e:
        same_records(got, e.integrate(px))
        assert counts["rhs_evals"] == e.stats()["rhs_evals"] and counts["steps"] == e.stats()["steps"]
    del keep


@pytest.mark.gpu
def test_a_full_gpu_of_refilled_lanes_gives_the_general_kernels_records(eng):
    """More pixels than resident lanes, so that every lane is refilled, with two images of
    different spins side by side."""
    d, _ = describe(abi.METRIC_KERR, (0.9,), 1, 70.0)
    keep = abi.attach_images(d, [abi.make_image((a,), r=1000.0, theta=1.2, half_width=8.0) for a in (0.9, 0.2)])
    px = np.concatenate([abi.square_pixels(260, image=i) for i in (0, 1)])
    px = px[np.random.default_rng(5).permutation(len(px))]
    with eng.Engine(d) as e:
        got = e.integrate(px)
    d.mixed_options = abi.MIXED_FP64_DECISIONS
    with eng.Engine(d) as e:
        same_records(got, e.integrate(px))
    del keep


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_ANALYTIC])
@pytest.mark.parametrize("metric,params,rlog,side,timeout", [
    (abi.METRIC_KERR, (0.9,), 1, 17, None),
    (abi.METRIC_KERR, (0.0,), 1, 7, 0),
    (abi.METRIC_KERR, (0.99,), 0, 2, 3000),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1), 1, 17, None),
    (abi.METRIC_RASHEED_LARSEN, LORENZO, 1, 9, None),
    (abi.METRIC_FLAT, (), 0, 3, 3000),
])
def test_two_lanes_in_fp64_give_the_one_lane_results(eng, metric, params, rlog, side, timeout, precision):
    """The FP64 and FP64-analytic kernels on several lanes per geodesic (where they exist)
    against one lane."""
    px = abi.square_pixels(side)
    d, keep = describe(metric, params, rlog, 63.0, timeout=timeout)
    d.precision = precision
    got = {}
    for lanes in (1, 2):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[lanes] = e.integrate(px)
            counts = e.stats()
            assert counts["rhs_evals"] == 4 * counts["steps"] == 4 * int(got[lanes]["steps"].sum())
            assert counts["fp64_steps"] == (counts["steps"] if precision == abi.PREC_FP64_ANALYTIC else 0)
    same_records(got[2], got[1])
    del keep


@pytest.mark.gpu
def test_fp64_launches_in_every_block_size_give_the_same_records(eng):
    """FP64 launches take CTAs of 32 threads, four per SM, unless a shape is asked for."""
    px = abi.square_pixels(41)
    d, keep = describe(abi.METRIC_KERR, (0.9,), 1, 63.0, integrator=abi.INTEGRATOR_VERLET)
    d.precision = abi.PREC_FP64
    got = {}
    for block in (0, 32, 64, 128):
        with eng.Engine(d) as e:
            e.set_launch(block, 0)
            got[block] = e.integrate(px)
            assert e.stats()["block_size"] == (block or 32)
    for block in got:
        same_records(got[block], got[0])
    del keep


def test_packed_bodies_match_the_generator():
    """gen_packed.inc is what gen_packed.py prints for the committed gen_christoffel.inc."""
    gen = os.path.join(ROOT, "foort_gb300", "gen", "gen_packed.py")
    out = subprocess.run([sys.executable, gen], check=True, capture_output=True, text=True).stdout
    with open(os.path.join(ROOT, "foort_gb300", "csrc", "gen_packed.inc")) as f:
        assert f.read() == out


def several_lanes_and_one(eng, d, px, **run):
    got = {}
    for lanes in (1, 2):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[lanes] = e.integrate(px, **run)
            got[lanes, "counts"] = {k: e.stats()[k] for k in ("steps", "rhs_evals", "fp64_steps", "geodesics")}
    return got


# both integrators, no velocity iterations and many, radii to the horizon and through the
# theta singularity, rays that end after one step, pixel counts that leave a warp part-filled
@pytest.mark.gpu
@pytest.mark.parametrize("metric,params,rlog,inclination,side,timeout,integrator,tolerance", [
    (abi.METRIC_KERR, (0.998,), 1, 17.0, 33, None, abi.INTEGRATOR_VERLET, 1e-5),
    (abi.METRIC_KERR, (0.0,), 1, 90.0, 9, None, abi.INTEGRATOR_VERLET, -1.0),
    (abi.METRIC_KERR, (0.7,), 0, 63.0, 3, 3000, abi.INTEGRATOR_VERLET, 0.001),
    (abi.METRIC_KERR, (0.9,), 1, 2.0, 31, None, abi.INTEGRATOR_RK4, 0.001),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1), 1, 63.0, 33, None, abi.INTEGRATOR_VERLET, 1e-5),
    (abi.METRIC_JOHANNSEN, (0.7, 2.0, 0.0, 0.0, 0.0), 1, 90.0, 33, None, abi.INTEGRATOR_VERLET, -1.0),
    (abi.METRIC_JOHANNSEN, (0.3, -0.9, 0.0, 0.0, 0.0), 1, 2.0, 17, None, abi.INTEGRATOR_RK4, 0.001),
    (abi.METRIC_JOHANNSEN, (0.9, 0.4, 0.0, 0.0, 0.0), 0, 30.0, 2, 3000, abi.INTEGRATOR_RK4, 0.001),
    (abi.METRIC_JOHANNSEN, (0.9, 0.4, 0.0, 0.0, 0.0), 1, 30.0, 2, 0, abi.INTEGRATOR_VERLET, 0.001),
])
def test_shared_steps_in_fp64_give_the_one_lane_results(eng, metric, params, rlog, inclination, side, timeout,
                                                        integrator, tolerance):
    """The FP64 kernels that share a step between four or eight lanes write each rounding out as the
    one-lane kernel has it: the same records bit for bit, and the same counts."""
    d, keep = describe(metric, params, rlog, inclination, integrator=integrator, timeout=timeout)
    d.precision, d.verlet_tol = abi.PREC_FP64, tolerance
    got = several_lanes_and_one(eng, d, abi.square_pixels(side))
    same_records(got[2], got[1])
    assert got[2, "counts"] == got[1, "counts"]
    del keep


@pytest.mark.gpu
@pytest.mark.parametrize("metric,integrator,side,precision", [
    (abi.METRIC_KERR, abi.INTEGRATOR_RK4, 60, abi.PREC_FP64),        # eight lanes from the start
    (abi.METRIC_KERR, abi.INTEGRATOR_RK4, 100, abi.PREC_FP64),       # from two
    (abi.METRIC_KERR, abi.INTEGRATOR_RK4, 180, abi.PREC_FP64),       # from one
    (abi.METRIC_KERR, abi.INTEGRATOR_VERLET, 120, abi.PREC_FP64),    # from one
    (abi.METRIC_JOHANNSEN, abi.INTEGRATOR_RK4, 100, abi.PREC_FP64),
    (abi.METRIC_JOHANNSEN, abi.INTEGRATOR_VERLET, 100, abi.PREC_FP64),
    (abi.METRIC_JOHANNSEN, abi.INTEGRATOR_VERLET, 120, abi.PREC_FP64),
    (abi.METRIC_KERR, abi.INTEGRATOR_RK4, 40, abi.PREC_FP64_ANALYTIC),   # eight from the start
    (abi.METRIC_KERR, abi.INTEGRATOR_RK4, 120, abi.PREC_FP64_ANALYTIC),  # from two
])
def test_fp64_lanes_are_refilled_and_run_two_images(eng, metric, integrator, side, precision):
    """More pixels than the kernels with shared steps hold at a time, two images side by
    side: one lane, several lanes and the built-in choice give the same records, also where
    a step budget ends some of them."""
    d, _ = describe(metric, (0.9,), 1, 70.0, integrator=integrator, timeout=600)
    d.precision = precision
    pars = [(a,) if metric == abi.METRIC_KERR else (a, 0.5, 0.0, 0.0, 0.0) for a in (0.9, 0.2)]
    keep = abi.attach_images(d, [abi.make_image(p, r=1000.0, theta=1.2, half_width=8.0) for p in pars])
    px = np.concatenate([abi.square_pixels(side, image=i) for i in (0, 1)])
    px = px[np.random.default_rng(5).permutation(len(px))]
    got = several_lanes_and_one(eng, d, px)
    same_records(got[2], got[1])
    assert got[2, "counts"] == got[1, "counts"]
    with eng.Engine(d) as e:
        same_records(e.integrate(px), got[1])
        e.set_lanes(2)
        e.set_budget(50000)
        part = e.integrate(px, allow=(abi.FOORT_E_BUDGET,))
    stopped = (part["err"] & (abi.ERR_BUDGET | abi.ERR_UNFINISHED)) != 0
    assert stopped.any() and np.all(part["term"][stopped] == abi.TERMCODE_CONTINUE)
    same_records(part[~stopped], got[1][~stopped])
    del keep


# every step sampled, each third with the last, one kept position, all of them
@pytest.mark.gpu
@pytest.mark.parametrize("keep_steps,freq", [(25, (1, 1, 0)), (7, (3, 0, 1)), (1, (1, 0, 0)), (0, (1, 1, 1))])
@pytest.mark.parametrize("metric,params,rlog,side,integrator", [
    (abi.METRIC_KERR, (0.9,), 1, 17, abi.INTEGRATOR_RK4),
    (abi.METRIC_KERR, (0.9,), 1, 17, abi.INTEGRATOR_VERLET),
    (abi.METRIC_FLAT, (), 0, 5, abi.INTEGRATOR_RK4),
    (abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.0, 0.0, 0.0), 1, 17, abi.INTEGRATOR_VERLET),
    (abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.0, 0.0, 0.0), 1, 17, abi.INTEGRATOR_RK4),
    (abi.METRIC_RASHEED_LARSEN, LORENZO, 1, 9, abi.INTEGRATOR_RK4),
])
def test_lean_kernels_record_the_general_kernels_positions(eng, metric, params, rlog, side, integrator, keep_steps,
                                                          freq):
    px = abi.square_pixels(side)
    d, keep = describe(metric, params, rlog, 63.0, integrator=integrator, timeout=900)
    d.diag_flags |= abi.DIAG_GEODESIC_POSITION
    d.geopos_output_steps, d.geopos_freq = keep_steps, abi.UpdateFreq(*freq)
    got = {}
    for name, options, lanes in (("general", abi.MIXED_FP64_DECISIONS, 1), ("one lane", 0, 1), ("two lanes", 0, 2)):
        d.mixed_options = options
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[name] = e.positions(px, e.integrate(px))
    for name in ("one lane", "two lanes"):
        np.testing.assert_array_equal(got[name][0], got["general"][0])
        np.testing.assert_array_equal(got[name][1], got["general"][1])
    assert np.isfinite(got["general"][1]).all()
    del keep


# rays whose last step overflows FP32: a velocity iteration that diverges before the horizon,
# a step from the rotation axis that ends at an infinite theta
@pytest.mark.gpu
@pytest.mark.parametrize("view,seed,pixel", [
    (dict(integrator="verlet", side=82, a=0.0877, inclination=15.93, half_width=12.989, diags="all"), 89670267,
     (4468 // 82, 4468 % 82, 82)),
    (dict(integrator="rk4", side=42, a=0.0693, inclination=12.78, half_width=9.337, diags="quadrant+passes"), 855370547,
     (164, 326, 329)),
])
def test_lean_kernels_overflow_where_the_general_ones_do(eng, view, seed, pixel):
    import importlib.util
    spec = importlib.util.spec_from_file_location("performance_cases", os.path.join(ROOT, "perf", "cases.py"))
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    case = dict(call="integrate", metric="kerr", precision="mixed", logr=False, alpha13=0.0, alpha3=0.0, tolerance=0.001,
                timeout=100000)
    case.update(view)
    state = cases.prepare(case, seed)
    d, px = state["desc"], np.zeros(1, dtype=abi.PIXEL_DTYPE)
    px["row"], px["col"], px["grid"] = pixel
    got = {}
    for options in (0, abi.MIXED_FP64_DECISIONS):
        d.mixed_options = options
        with eng.Engine(d) as e:
            got[options] = e.integrate(px)
    assert got[0]["err"][0] & abi.ERR_NONFINITE
    same_records(got[0], got[abi.MIXED_FP64_DECISIONS])
