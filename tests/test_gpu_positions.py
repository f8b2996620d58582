"""Recorded positions (foort_gpu_positions) in FP64 and FP64-analytic: the second pass retraces the
first whichever kernels the two take, and the workspace that a context keeps serves calls
of any sizes."""
import numpy as np
import pytest

from foort_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

RK4, VERLET = abi.INTEGRATOR_RK4, abi.INTEGRATOR_VERLET
LORENZO = (0.3556562853309941, 0.2969060968239216, 3.057664971085168, 0.942335028914832)


@pytest.fixture(scope="module")
def eng():
    import foort_gb300
    from foort_gb300 import build as engine_build
    engine_build.build()
    foort_gb300.check_layout()
    return foort_gb300


def describe(precision, metric, params, integrator, rlog, timeout=300, keep_steps=20, epsilon=0.1):
    d = workloads.base_desc(precision)
    d.metric_id, d.integrator_id, d.rlog = metric, integrator, rlog
    d.timeout_max_steps, d.epsilon = timeout, epsilon
    d.diag_flags = abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_CLOSEST_RADIUS | abi.DIAG_GEODESIC_POSITION
    d.geopos_output_steps, d.geopos_freq = keep_steps, abi.UpdateFreq(1, 1, 0)
    if rlog:
        d.term_flags |= abi.TERM_THETA_SINGULARITY
    keep = abi.attach_images(d, [abi.make_image(params, r=1000.0, theta=1.1, half_width=9.0)])
    return d, keep


CASES = [
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_KERR, (0.9,), RK4, 1),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_KERR, (0.9,), VERLET, 1),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_KERR, (0.9,), RK4, 0),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_FLAT, (), RK4, 0),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_FLAT, (), VERLET, 0),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.0, 0.0, 0.0), RK4, 1),
    (abi.PREC_FP64, abi.METRIC_KERR, (0.9,), RK4, 1),
    (abi.PREC_FP64, abi.METRIC_KERR, (0.9,), VERLET, 1),
    (abi.PREC_FP64, abi.METRIC_KERR, (0.9,), VERLET, 0),
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.0, 0.0, 0.0), RK4, 1),
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.0, 0.0, 0.0), VERLET, 1),
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, (0.7, 1.5, 0.3, 0.2, 0.1), VERLET, 1),
    (abi.PREC_FP64, abi.METRIC_RASHEED_LARSEN, LORENZO, RK4, 1),
    (abi.PREC_FP64, abi.METRIC_FLAT, (), RK4, 0),
]


# few rays (the most lanes per geodesic), with a short timeout those that start with two lanes and
# with one
@pytest.mark.parametrize("precision,metric,params,integrator,rlog", CASES)
@pytest.mark.parametrize("side,timeout", [(13, 300), (130, 30), (250, 12)])
def test_every_lane_choice_records_the_one_lane_positions(eng, precision, metric, params, integrator, rlog, side,
                                                         timeout):
    px = abi.square_pixels(side)
    d, keep = describe(precision, metric, params, integrator, rlog, timeout)
    got = {}
    for lanes in (1, 2, 0):
        with eng.Engine(d) as e:
            e.set_lanes(lanes)
            got[lanes] = e.positions(px, e.integrate(px))
    for lanes in (2, 0):
        np.testing.assert_array_equal(got[lanes][0], got[1][0])
        np.testing.assert_array_equal(got[lanes][1], got[1][1])
    assert np.isfinite(got[1][1]).all() and len(got[1][1]) >= 2 * len(px)
    del keep


@pytest.mark.parametrize("precision,metric,params,integrator,rlog", [CASES[0], CASES[6], CASES[9]])
def test_part_of_a_screen_is_retraced_by_itself(eng, precision, metric, params, integrator, rlog):
    """Results of a large launch, positions of a few of its pixels: another number of
    geodesics, other kernels."""
    px = abi.square_pixels(120)
    d, keep = describe(precision, metric, params, integrator, rlog)
    with eng.Engine(d) as e:
        first = e.integrate(px)
        some = np.arange(5, len(px), 301)
        counts, points = e.positions(px[some], first[some])
    with eng.Engine(d) as e:
        e.set_lanes(1)
        want = e.positions(px[some], first[some])
    np.testing.assert_array_equal(counts, want[0])
    np.testing.assert_array_equal(points, want[1])
    del keep


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED, abi.PREC_FP64_ANALYTIC])
def test_one_context_records_screens_of_any_sizes(eng, precision):
    """Growing, shrinking, more than the 64 MiB that a context keeps, and a call that fails."""
    d, keep = describe(precision, abi.METRIC_KERR, (0.9,), RK4, 1, timeout=60, keep_steps=59)
    with eng.Engine(d) as e:
        for side in (9, 40, 5, 260, 9):
            px = abi.square_pixels(side)
            first = e.integrate(px)
            counts, points = e.positions(px, first)
            with eng.Engine(d) as other:
                want = other.positions(px, first)
            np.testing.assert_array_equal(counts, want[0])
            np.testing.assert_array_equal(points, want[1])
            assert np.isfinite(points).all()
            if side == 260:
                assert points.nbytes > 64 << 20
            wrong = first.copy()
            wrong["steps"][0] += 1
            with pytest.raises(eng.FoortError):
                e.positions(px, wrong)
    del keep
