"""Launch shapes: what a caller asks for is what a launch takes."""
import numpy as np
import pytest

from foort_gb300 import abi, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    import foort_gb300
    from foort_gb300 import build as engine_build
    engine_build.build()
    foort_gb300.check_layout()
    return foort_gb300


@pytest.fixture(scope="module")
def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def describe(precision, metric=abi.METRIC_KERR, params=(0.9,), integrator=abi.INTEGRATOR_RK4, rlog=1, timeout=0):
    d = workloads.base_desc(precision)
    d.metric_id, d.integrator_id, d.rlog, d.timeout_max_steps = metric, integrator, rlog, timeout
    d.diag_flags = abi.DIAG_FOUR_COLOR_SCREEN | abi.DIAG_EQUATORIAL_PASSES | abi.DIAG_CLOSEST_RADIUS
    keep = abi.attach_images(d, [abi.make_image(params, r=1000.0, theta=1.1, half_width=9.0)])
    return d, keep


# a CTA size alone takes as many CTAs as fit, a cap alone CTAs of 128 threads, in every
# precision; 0 and 0 is the built-in shape
@pytest.mark.parametrize("precision", [abi.PREC_MIXED, abi.PREC_FP64, abi.PREC_FP64_ANALYTIC])
@pytest.mark.parametrize("integrator", [abi.INTEGRATOR_RK4, abi.INTEGRATOR_VERLET])
@pytest.mark.parametrize("lanes", [0, 1])
def test_a_forced_size_or_cap_leaves_the_other_as_documented(eng, sms, precision, integrator, lanes):
    d, keep = describe(precision, integrator=integrator)
    px = abi.square_pixels(316)
    with eng.Engine(d) as e:
        e.set_lanes(lanes)
        want = e.integrate(px)
        for block in (64, 96, 128):
            e.set_launch(block, 0)
            got, st = e.integrate(px), e.stats()
            assert st["block_size"] == block and st["n_blocks"] % sms == 0
            assert st["n_blocks"] * block >= 192 * sms  # every kernel here fits at least this many threads on an SM
            for name in abi.RESULT_DTYPE.names:
                np.testing.assert_array_equal(got[name], want[name], err_msg=name)
        for cap in (1, 2):
            e.set_launch(0, cap)
            e.integrate(px)
            st = e.stats()
            assert (st["block_size"], st["n_blocks"]) == (128, cap * sms)
    del keep


# two lanes per geodesic only where they are the faster kernel: on both sides of each limit
# (in geodesics per SM)
@pytest.mark.parametrize("metric,params,rlog,limit", [
    (abi.METRIC_KERR, (0.9,), 0, 64),
    (abi.METRIC_KERR, (0.9,), 1, 448),
    (abi.METRIC_FLAT, (), 0, 0),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1), 0, 256),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1), 1, 1792),
    (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.0, 0.0, 0.0), 0, 192),
])
def test_two_lanes_up_to_the_limit_of_each_metric(eng, sms, metric, params, rlog, limit):
    d, keep = describe(abi.PREC_MIXED, metric, params, rlog=rlog)
    n = limit * sms
    px = abi.square_pixels(int(np.ceil(np.sqrt(n + 2))))
    with eng.Engine(d) as e:
        for count, lanes in ((n, 2), (n + 1, 1)):
            if count:
                e.integrate(px[:count])
                assert e.stats()["lanes_per_geodesic"] == lanes
    del keep


@pytest.mark.parametrize("metric,params", [(abi.METRIC_KERR, (0.9,)), (abi.METRIC_JOHANNSEN, (0.8, 1.0, 0.5, 0.2, 0.1))])
def test_fp64_waves_in_plain_r_leave_few_lanes_idle(eng, sms, metric, params):
    """FP64-analytic Verlet fits twelve CTAs of 32 threads on an SM and takes eight, unless
    twelve make fewer waves of threads."""
    d, keep = describe(abi.PREC_FP64_ANALYTIC, metric, params, abi.INTEGRATOR_VERLET, rlog=0)
    px = abi.square_pixels(int(np.ceil(np.sqrt(600 * sms))))
    with eng.Engine(d) as e:
        for per_sm, threads in ((100, 100), (250, 250), (256, 256), (300, 300), (384, 384), (400, 256), (600, 384)):
            n = per_sm * sms
            e.integrate(px[:n])
            st = e.stats()
            assert (st["block_size"], st["n_blocks"]) == (32, -(-threads * sms // 32))
    del keep


# more pixels than a search times: the sample runs in the whole launch's kernel and shape
@pytest.mark.parametrize("precision,metric,params,integrator", [
    (abi.PREC_FP64, abi.METRIC_JOHANNSEN, (0.7, 1.0, 0.0, 0.0, 0.0), abi.INTEGRATOR_VERLET),
    (abi.PREC_FP64_ANALYTIC, abi.METRIC_KERR, (0.9,), abi.INTEGRATOR_RK4),
])
def test_tuned_fp64_shapes_are_launched_as_they_were_timed(eng, sms, precision, metric, params, integrator):
    import torch
    d, keep = describe(precision, metric, params, integrator, timeout=12)
    px = abi.square_pixels(int(np.ceil(np.sqrt(1100 * sms))))
    eng.tune_clear()
    with eng.Engine(d) as e:
        want = e.integrate(px)
        d_px = torch.from_numpy(px.view(np.uint8).copy()).cuda()
        d_out = torch.zeros(len(px) * abi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        best = e.autotune(d_px.data_ptr(), len(px), d_out.data_ptr())
        shapes = {(s["block_size"], s["blocks_per_sm"], s["lanes"]) for s in eng.tune_candidates(precision, True)}
        assert (best["block_size"], best["blocks_per_sm"], best["lanes"]) in shapes
        got, st = e.integrate(px), e.stats()
        assert st["block_size"] == best["block_size"] and st["lanes_per_geodesic"] == best["lanes"]
        if best["blocks_per_sm"]:
            assert st["n_blocks"] <= best["blocks_per_sm"] * sms
        e.set_launch(96, 0)  # a forced size takes no cap that was found for another
        e.integrate(px)
        assert e.stats()["n_blocks"] * 96 >= 192 * sms
    eng.tune_clear()
    for name in abi.RESULT_DTYPE.names:
        np.testing.assert_array_equal(got[name], want[name], err_msg=name)
        np.testing.assert_array_equal(d_out.cpu().numpy().view(abi.RESULT_DTYPE)[name], want[name], err_msg=name)
    del keep
