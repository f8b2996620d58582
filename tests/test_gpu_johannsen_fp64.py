"""Johannsen in FP64 with alpha13 alone: the kernels without the zero terms (kernel_fp64_split.cuh)
give the general kernels' records bit for bit, at every start they have. A second image
with another deviation parameter, which no pixel uses, takes the general kernels."""
import numpy as np
import pytest

from foort_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

RK4, VERLET = abi.INTEGRATOR_RK4, abi.INTEGRATOR_VERLET


@pytest.fixture(scope="module")
def eng():
    import foort_gb300
    from foort_gb300 import build as engine_build
    engine_build.build()
    foort_gb300.check_layout()
    return foort_gb300


def describe(integrator, rlog, timeout, tolerance, general, a=0.7, alpha13=2.0, inclination=75.0):
    d = workloads.base_desc(abi.PREC_FP64)
    d.metric_id, d.integrator_id, d.rlog = abi.METRIC_JOHANNSEN, integrator, rlog
    d.timeout_max_steps, d.verlet_tol = timeout, tolerance
    d.diag_flags = abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_EQUATORIAL_PASSES | abi.DIAG_CLOSEST_RADIUS
    if rlog:
        d.term_flags |= abi.TERM_THETA_SINGULARITY
    params = [(a, alpha13, 0.0, 0.0, 0.0)] + ([(a, alpha13, 0.3, 0.0, 0.0)] if general else [])
    keep = abi.attach_images(d, [abi.make_image(p, r=1000.0, theta=np.radians(inclination), half_width=9.0) for p in params])
    return d, keep


def same_records(a, b):
    for name in abi.RESULT_DTYPE.names:
        np.testing.assert_array_equal(a[name], b[name], err_msg=name)


# whole rays on one lane: the reduced metric's one-lane kernel against the general one
@pytest.mark.parametrize("integrator,rlog,timeout,tolerance,a,alpha13,inclination,side", [
    (RK4, 1, 10000, 0.001, 0.7, 2.0, 75.0, 33),
    (RK4, 1, 10000, 0.001, 0.0, -0.8, 2.0, 17),
    (RK4, 0, 3000, 0.001, 0.9, 0.4, 30.0, 3),
    (VERLET, 1, 10000, -1.0, 0.7, 2.0, 5.0, 33),
    (VERLET, 1, 10000, 1e-5, 0.99, -0.5, 90.0, 33),
    (VERLET, 0, 3000, 0.001, 0.3, 1.0, 60.0, 3),
])
def test_one_lane_without_the_zero_terms(eng, integrator, rlog, timeout, tolerance, a, alpha13, inclination, side):
    px = abi.square_pixels(side)
    got = []
    for general in (False, True):
        d, keep = describe(integrator, rlog, timeout, tolerance, general, a, alpha13, inclination)
        with eng.Engine(d) as e:
            e.set_lanes(1)
            got.append((e.integrate(px), {k: e.stats()[k] for k in ("steps", "rhs_evals", "lanes_per_geodesic")}))
        del keep
    same_records(got[0][0], got[1][0])
    assert got[0][1] == got[1][1]


# geodesics per SM: a start with eight lanes (four in Verlet), two, one and a tail, and one to
# the end
@pytest.mark.parametrize("integrator", [RK4, VERLET])
@pytest.mark.parametrize("rlog", [0, 1])
@pytest.mark.parametrize("per_sm", [20, 200, 900, 1030])
def test_every_start_gives_the_general_one_lane_records(eng, integrator, rlog, per_sm):
    import torch
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 5
    px = abi.square_pixels(int(np.ceil(np.sqrt(n))))[:n]
    got = []
    for general in (False, True):
        d, keep = describe(integrator, rlog, 25, 0.001, general)
        d.epsilon = 0.3  # rays that reach the hole within the steps
        with eng.Engine(d) as e:
            e.set_lanes(1 if general else 0)
            got.append((e.integrate(px), {k: e.stats()[k] for k in ("steps", "rhs_evals")}))
        del keep
    same_records(got[0][0], got[1][0])
    assert got[0][1] == got[1][1]
