"""The kernel that a launch takes (foort_gpu_kernel_name), over the options that choose it."""
import re

import pytest

from foort_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

RK4, VERLET = abi.INTEGRATOR_RK4, abi.INTEGRATOR_VERLET
ALPHA13, FULL = (0.7, 1.0, 0.0, 0.0, 0.0), (0.7, 1.0, 0.3, 0.0, 0.0)
LEAN, MIXED, PAIR = "integrate_lean_kernel", "integrate_mixed_kernel", "integrate_mixed_pair_kernel"
FP64, FP64_PAIR, SPLIT = "integrate_fp64_kernel", "integrate_fp64_pair_kernel", "integrate_fp64_split_kernel"


@pytest.fixture(scope="module")
def eng():
    import foort_gb300
    from foort_gb300 import build as engine_build
    engine_build.build()
    foort_gb300.check_layout()
    return foort_gb300


def kernel(e):
    """(name, the number that the mangled template arguments end with, or None)"""
    name = e.kernel_name()
    last = re.search(r"ILi\d+ELb[01]ELi[01]ELi(\d)EE", name)  # metric, alpha13 alone, integrator, start
    return re.search(r"integrate_\w+?_kernel", name).group(), int(last.group(1)) if last else None


@pytest.mark.parametrize("precision,metric,params,integrator,lanes,options,every,want", [
    (abi.PREC_MIXED, abi.METRIC_KERR, (0.9,), RK4, 0, 0, 1, (LEAN, None)),
    (abi.PREC_MIXED, abi.METRIC_KERR, (0.9,), RK4, 0, 0, 2, (PAIR, None)),
    (abi.PREC_MIXED, abi.METRIC_KERR, (0.9,), VERLET, 0, abi.MIXED_FP64_DECISIONS, 1, (MIXED, None)),
    (abi.PREC_MIXED, abi.METRIC_JOHANNSEN, FULL, RK4, 0, 0, 1, (LEAN, None)),
    (abi.PREC_MIXED, abi.METRIC_JOHANNSEN, FULL, RK4, 1, 0, 1, (MIXED, None)),
    (abi.PREC_MIXED, abi.METRIC_JOHANNSEN, FULL, VERLET, 0, 0, 1, (MIXED, None)),
    (abi.PREC_MIXED, abi.METRIC_JOHANNSEN, ALPHA13, VERLET, 0, 0, 1, (LEAN, None)),
    (abi.PREC_FP64, abi.METRIC_KERR, (0.9,), RK4, 0, 0, 1, (SPLIT, 8)),
    (abi.PREC_FP64, abi.METRIC_KERR, (0.9,), VERLET, 2, 0, 1, (SPLIT, 4)),
    (abi.PREC_FP64, abi.METRIC_KERR, (0.9,), RK4, 1, 0, 1, (FP64, None)),
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, ALPHA13, RK4, 1, 0, 1, (SPLIT, 0)),  # one lane, no zero terms
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, ALPHA13, VERLET, 1, 0, 1, (SPLIT, 0)),
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, FULL, VERLET, 1, 0, 1, (FP64, None)),
    (abi.PREC_FP64, abi.METRIC_FLAT, (), RK4, 0, 0, 1, (FP64_PAIR, None)),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_KERR, (0.9,), RK4, 0, 0, 1, (LEAN, None)),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_JOHANNSEN, ALPHA13, RK4, 0, 0, 1, (MIXED, None)),
])
def test_options_choose_the_kernel(eng, precision, metric, params, integrator, lanes, options, every, want):
    d = workloads.base_desc(precision)
    d.metric_id, d.integrator_id, d.mixed_options = metric, integrator, options
    d.boundary_every, d.timeout_max_steps = every, 3
    d.diag_flags = abi.DIAG_FOUR_COLOR_SCREEN
    keep = abi.attach_images(d, [abi.make_image(params, r=1000.0, theta=1.1, half_width=9.0)])
    with eng.Engine(d) as e:
        assert e.kernel_name() == ""
        e.set_lanes(lanes)
        e.integrate(abi.square_pixels(9))
        assert kernel(e) == want
    del keep
