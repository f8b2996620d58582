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
