"""The autotuner's candidates and cache keys. None of this needs a GPU."""
import pytest

import foort_gb300 as fg
from foort_gb300 import abi


@pytest.fixture(autouse=True)
def lib(engine_lib):
    return engine_lib


@pytest.mark.parametrize("several", [0, 1])
@pytest.mark.parametrize("precision", [abi.PREC_MIXED, abi.PREC_FP64, abi.PREC_FP64_ANALYTIC])
def test_candidates_vary_what_the_built_in_rule_varies(precision, several):
    """Every CTA size filled to what fits, and in FP64 the built-in rule's own shapes."""
    got = fg.tune_candidates(precision, several)
    want = [(32, 0), (64, 0), (128, 0)]
    if precision != abi.PREC_MIXED:
        want = [(32, 4), (32, 8)] + want
    for lanes in (1, 2):
        assert [(s["block_size"], s["blocks_per_sm"]) for s in got if s["lanes"] == lanes] == \
            (want if lanes == 1 or several else [])
    assert all(s["refill_steps"] == 1 and s["poll_steps"] == 512 for s in got)
    part = (abi.LaunchShape * 2)()  # no more than there is room for
    assert fg.load().foort_tune_candidates(precision, several, part, 1) == len(got)
    assert part[0].as_dict() == got[0] and part[1].block_size == 0


def johannsen_key(*deviations, precision=abi.PREC_MIXED, options=0):
    d = abi.default_desc()
    d.metric_id, d.precision, d.mixed_options = abi.METRIC_JOHANNSEN, precision, options
    keep = abi.attach_images(d, [abi.make_image((0.9, 0.4, *p)) for p in deviations])
    key = fg.tune_key(d, 152, 3000)
    del keep
    return key


def test_keys_tell_johannsens_kernels_apart():
    """alpha13 alone has kernels of its own, in mixed precision and FP64; the FP64-analytic ones and
    those with FP64 decisions are the same either way."""
    for precision in (abi.PREC_MIXED, abi.PREC_FP64):
        plain = johannsen_key((0.0, 0.0, 0.0), precision=precision)
        assert plain == f"sm152:m3:i0:p{precision}:r0:d0:f0:b11"
        full = johannsen_key((0.0, 0.0, 0.1), precision=precision)
        assert full == f"sm152:m3:i0:p{precision}:r0:d0:f0:j1:b11"
        assert johannsen_key((0.0, 0.0, 0.0), (0.2, 0.0, 0.0), precision=precision) == full
        assert johannsen_key((0.0, 0.0, 0.0), (0.0, 0.0, 0.0), precision=precision) == plain
    for precision, options in ((abi.PREC_FP64_ANALYTIC, 0), (abi.PREC_MIXED, abi.MIXED_FP64_DECISIONS)):
        assert johannsen_key((0.3, 0.0, 0.0), precision=precision, options=options) == \
            johannsen_key((0.0, 0.0, 0.0), precision=precision, options=options)


@pytest.mark.parametrize("field,used", [
    ("horizon_every", ("term_flags", abi.TERM_HORIZON)), ("boundary_every", ("term_flags", abi.TERM_BOUNDARY_SPHERE)),
    ("timeout_every", ("term_flags", abi.TERM_TIMEOUT)), ("theta_every", ("term_flags", abi.TERM_THETA_SINGULARITY)),
    ("equat_freq", ("diag_flags", abi.DIAG_EQUATORIAL_PASSES)), ("closest_freq", ("diag_flags", abi.DIAG_CLOSEST_RADIUS))])
def test_keys_tell_lean_and_general_kernels_apart(field, used):
    """An update that is used and not made at each step takes the general kernels, in mixed precision
    and FP64-analytic; flat space has no horizon."""
    for precision in (abi.PREC_MIXED, abi.PREC_FP64, abi.PREC_FP64_ANALYTIC):
        for metric in (abi.METRIC_KERR, abi.METRIC_FLAT):
            d = abi.default_desc()
            d.metric_id, d.precision = metric, precision
            base = f"sm152:m{metric}:i0:p{precision}:r0:d0:f0"
            setattr(d, field, abi.UpdateFreq(3, 0, 0) if field.endswith("freq") else 3)
            setattr(d, used[0], getattr(d, used[0]) & ~used[1])
            assert fg.tune_key(d, 152, 3000) == base + ":b11"
            setattr(d, used[0], getattr(d, used[0]) | used[1])
            general = precision != abi.PREC_FP64 and not (field == "horizon_every" and metric == abi.METRIC_FLAT)
            assert fg.tune_key(d, 152, 3000) == base + (":u1" if general else "") + ":b11"
            d.mixed_options = abi.MIXED_FP64_DECISIONS
            assert fg.tune_key(d, 152, 3000) == base.replace(":d0", ":d1") + ":b11"
