"""laph_solver_footprint counts the one-kernel filter pass's plan (2 MiB after rounding) only for batches that run it:
filter_kernel 2 never does, and has the same allocations otherwise."""
import pytest

import laph_eigsys_b200 as lb

PLAN = 2 << 20


def _bytes(probs, **kw):
    return lb.solver_footprint(probs, guard=16, deg=24, **kw)


@pytest.mark.parametrize("probs,kw,plan", [
    ([(32, 120)] * 2, {}, 0),                              # 1e7 site-columns
    ([(48, 220)], {}, 0),
    ([(8, 60)] * 16, {}, PLAN),
    ([(8, 60)] * 16, {"block": 16, "filter_tile": 128}, PLAN),
    ([(8, 60)] * 16, {"block": 32}, 0),                    # a request for the step kernels
    ([(8, 60)] * 16, {"filter_tile": 64}, 0),
    ([(5, 12), (6, 12), (7, 12), (8, 12)], {}, PLAN),
    ([(5, 12), (6, 12), (7, 12), (8, 12), (9, 12)], {}, 0),  # five extents
])
def test_plan_is_counted_where_it_is_allocated(probs, kw, plan):
    assert _bytes(probs, **kw) - _bytes(probs, filter_kernel=2, **kw) == plan
