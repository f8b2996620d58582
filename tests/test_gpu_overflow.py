"""Rays whose state overflows: the specialised kernels (kernel_lean.cuh, kernel_fp64_split.cuh)
end them as the general kernels do, with the same codes, counts and bits. The screens look
along the rotation axis, or take coarse steps, so that some of their rays step past it or
inside the horizon and diverge there."""
import random

import numpy as np
import pytest

from foort_gb300 import abi, workloads


@pytest.fixture(scope="module")
def eng():
    import foort_gb300
    from foort_gb300 import build as engine_build
    engine_build.build()
    foort_gb300.check_layout()
    return foort_gb300


def describe(precision, metric, params, integrator, rlog, inclination, r, half_width, epsilon, smallest_step, timeout,
             boundary, tolerance, term_flags):
    d = workloads.base_desc(precision)
    d.metric_id, d.integrator_id, d.rlog = metric, integrator, rlog
    d.epsilon, d.smallest_step, d.timeout_max_steps = epsilon, smallest_step, timeout
    d.boundary_radius, d.verlet_tol, d.term_flags = boundary, tolerance, term_flags
    d.diag_flags = abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_CLOSEST_RADIUS
    keep = abi.attach_images(d, [abi.make_image(params, r=r, theta=np.radians(inclination), half_width=half_width)])
    return d, keep


def same_records(a, b):
    for name in abi.RESULT_DTYPE.names:
        if name != "equat_passes":
            np.testing.assert_array_equal(a[name], b[name], err_msg=name)


RK4, VERLET = abi.INTEGRATOR_RK4, abi.INTEGRATOR_VERLET
STOPS = abi.TERM_HORIZON | abi.TERM_BOUNDARY_SPHERE | abi.TERM_TIMEOUT
ALL_STOPS = STOPS | abi.TERM_THETA_SINGULARITY


# sums of the contraction between half the largest float and the largest one: the general
# kernels double them
@pytest.mark.gpu
@pytest.mark.parametrize("metric,params,integrator,rlog,view,side", [
    (abi.METRIC_FLAT, (), RK4, 0, (0.01, 5.0, 40.0, 0.03, 0.01, 50, 1000.0, 0.001, STOPS), 64),
    (abi.METRIC_KERR, (0.0,), RK4, 0, (0.01, 30.0, 0.5, 3.0, 1e-7, 900, 1e5, 0.001, STOPS), 64),
    (abi.METRIC_JOHANNSEN, (0.9563767844865592, 0.5064812267713692, 0.0, 0.0, 0.0), RK4, 0,
     (0.01, 5.0, 12.0, 10.0, 1e-12, 300, 1000.0, -1.0, ALL_STOPS), 64),
    (abi.METRIC_JOHANNSEN, (0.0, 0.408884871033909, 0.0, 0.0, 0.0), VERLET, 1,
     (0.01, 1000.0, 0.5, 1.0, 1e-7, 50, 1e12, 0.001, ALL_STOPS & ~abi.TERM_BOUNDARY_SPHERE), 64),
    (abi.METRIC_JOHANNSEN, (0.0, 1.0380233096005593, 0.0, 0.0, 0.001), RK4, 0,
     (2.0, 5.0, 40.0, 10.0, 1e-7, 1, 1000.0, 0.001, ALL_STOPS & ~abi.TERM_BOUNDARY_SPHERE), 7),
])
def test_lean_contractions_overflow_where_the_general_ones_do(eng, metric, params, integrator, rlog, view, side):
    """A diagnostic that does not update at each step takes the general kernel, with the same
    float-float decisions."""
    inclination, r, half_width, *rest = view
    d, keep = describe(abi.PREC_MIXED, metric, params, integrator, rlog, inclination, r, half_width, *rest)
    px = abi.square_pixels(side)
    got = []
    for lanes in (1, 2):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got.append((e.integrate(px), e.stats()["steps"]))
    d.diag_flags |= abi.DIAG_EQUATORIAL_PASSES
    d.equat_freq = abi.UpdateFreq(2, 0, 0)
    with eng.Engine(d) as e:
        e.set_lanes(1)
        want = e.integrate(px), e.stats()["steps"]
    assert (want[0]["err"] & abi.ERR_NONFINITE).any()
    for records, steps in got:
        same_records(records, want[0])
        assert steps == want[1]
    del keep


# g^tphi infinite beside finite derivatives: r and theta take no product with it
@pytest.mark.gpu
@pytest.mark.parametrize("integrator", [RK4, VERLET])
def test_shared_fp64_steps_end_where_one_lane_does(eng, integrator):
    d, keep = describe(abi.PREC_FP64, abi.METRIC_KERR, (0.0,), integrator, 1, 0.3, 30.0, 0.5, 100.0, 0.01, 1, 1e5, -1.0,
                       ALL_STOPS & ~abi.TERM_BOUNDARY_SPHERE)
    d.theta_eps = 0.01
    px = abi.square_pixels(33)
    got = {}
    for lanes in (1, 2):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[lanes] = e.integrate(px)
    assert (got[1]["err"] & abi.ERR_NONFINITE).any()
    same_records(got[2], got[1])
    del keep


# a finite difference across Delta = 0, where d_r g_rr is infinite
@pytest.mark.gpu
@pytest.mark.parametrize("integrator", [RK4, VERLET])
@pytest.mark.parametrize("side", [4, 90])
def test_shared_fp64_steps_cross_the_horizon_as_one_lane_does(eng, integrator, side):
    h = 2.0 ** -23
    d, keep = describe(abi.PREC_FP64, abi.METRIC_KERR, (0.0,), integrator, 0, 60.0, 2.0 - h, 0.5, 0.03, 1e-12, 3, 1e5, -1.0,
                       abi.TERM_BOUNDARY_SPHERE | abi.TERM_TIMEOUT)
    d.derivative_h = h
    px = abi.square_pixels(side)
    got = {}
    for lanes in (1, 2):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[lanes] = e.integrate(px)
    assert (got[1]["err"] & abi.ERR_NONFINITE).all()
    same_records(got[2], got[1])
    del keep


def random_setting(rng, precision):
    """Views, steps and limits from ordinary to absurd."""
    metric = rng.choice([abi.METRIC_KERR, abi.METRIC_KERR, abi.METRIC_FLAT, abi.METRIC_RASHEED_LARSEN,
                         abi.METRIC_JOHANNSEN, abi.METRIC_JOHANNSEN])
    a = rng.choice([0.0, 1e-3, rng.uniform(0.0, 1.0), 0.998])
    others = rng.choice([(0.0, 0.0, 0.0), (0.0, 0.0, 0.0), (0.3, 0.2, 0.1), (0.0, 0.0, 1e-3)])
    params = {abi.METRIC_KERR: (a,), abi.METRIC_FLAT: (),
              abi.METRIC_RASHEED_LARSEN: (0.3556562853309941, 0.2969060968239216, 3.057664971085168, 0.942335028914832),
              abi.METRIC_JOHANNSEN: (a, rng.uniform(-1.0, 2.0)) + others}[metric]
    rlog = 0 if metric == abi.METRIC_FLAT else rng.randint(0, 1)
    d, keep = describe(precision, metric, params, rng.choice([RK4, VERLET]), rlog,
                       rng.choice([0.01, 0.3, 2.0, rng.uniform(5.0, 90.0), 90.0]), rng.choice([1000.0, 30.0, 5.0]),
                       rng.choice([0.5, 6.0, 12.0, 40.0]), rng.choice([0.03, 0.1, 0.3, 1.0, 3.0, 10.0, 100.0]),
                       rng.choice([1e-12, 1e-7, 1e-2]), rng.choice([0, 1, 50, 300]), rng.choice([1e3, 1e3, 1e5, 1e12, 1e30]),
                       rng.choice([-1.0, 1e-3, 1e-6]), rng.choice([STOPS, ALL_STOPS, ALL_STOPS & ~abi.TERM_BOUNDARY_SPHERE]))
    d.theta_eps = rng.choice([1e-5, 1e-2, 0.0])
    return d, keep, abi.square_pixels(rng.choice([1, 2, 7, 33]) + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PREC_MIXED, abi.PREC_FP64, abi.PREC_FP64_ANALYTIC])
@pytest.mark.parametrize("seed", range(8))
def test_random_views_end_alike_in_every_kernel(eng, precision, seed):
    rng = random.Random(1000 * precision + seed)
    for _ in range(12):
        d, keep, px = random_setting(rng, precision)
        got = []
        for lanes in (0, 1, 2):
            with eng.Engine(d) as e:
                e.set_lanes(lanes)
                got.append((e.integrate(px), {k: e.stats()[k] for k in ("steps", "rhs_evals")}))
        d.diag_flags |= abi.DIAG_EQUATORIAL_PASSES
        d.equat_freq = abi.UpdateFreq(2, 0, 0)  # the general kernels
        with eng.Engine(d) as e:
            e.set_lanes(1)
            want = e.integrate(px), {k: e.stats()[k] for k in ("steps", "rhs_evals")}
        for records, counts in got:
            same_records(records, want[0])
            assert counts == want[1]
        del keep
