"""The one-kernel filter pass of small batches (csrc/filter_pass.cu) against the step kernels (variant 2, which always
runs step by step): the same arithmetic per site and column, so the same eigenpairs to the last bit.  Extents at the
edges of its tiles (27 sites, one CTA; 256 sites a CTA at 8^3; ragged tiles and odd column strides at 5, 7 and 11), several
extents in one batch, more extents than it takes at once, BF16 links, and a cap of degree 2, whose pass is a single step."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu


def _solve(gpu, probs, variant, **kw):
    s = gpu.Solver(probs, guard=8, tol=1e-10, smear_kind=gpu.SMEAR_STOUT, smear_p1=0.1, smear_iters=2,
                   filter_kernel=variant, **kw)
    for i, (L, _) in enumerate(probs):
        s.set_links(i, random_links(L, 0.35, 4100 + 10 * L + i))
    st, res = s.run()
    out = [s.get(i) for i in range(len(probs))]
    steps, launches = s.counters()[:2]
    s.close()
    return st, [r["iters"] for r in res], out, steps, launches


@pytest.mark.parametrize("probs,kw", [
    ([(3, 8)], dict(deg=8, max_it=300)),
    ([(5, 20)], dict(deg=12, max_it=300)),
    ([(8, 24)], dict(deg=16, max_it=300)),
    ([(11, 50), (11, 20), (11, 50)], dict(deg=24, max_it=300)),
    ([(7, 30), (8, 40), (12, 24), (10, 50), (7, 12)], dict(deg=16, max_it=300)),
    ([(5, 12), (6, 12), (7, 12), (8, 12), (9, 12)], dict(deg=16, max_it=300)),
    ([(8, 40), (12, 60)], dict(deg=20, max_it=300, link_prec=1)),
    ([(6, 12)], dict(deg=2, max_it=12)),
], ids=["27 sites", "5", "8", "three of 11", "four extents", "five extents", "bf16", "degree 2"])
def test_pass_kernel_is_bitwise_the_step_kernels(gpu, probs, kw):
    a = _solve(gpu, probs, 1, **kw)
    b = _solve(gpu, probs, 2, **kw)
    assert a[0] == b[0] and a[1] == b[1]
    assert a[3] == b[3]
    for (ea, va, pa), (eb, vb, pb) in zip(a[2], b[2]):
        assert np.array_equal(ea, eb) and np.array_equal(va, vb) and np.array_equal(pa, pb)
    if len({L for L, _ in probs}) <= 4 and kw["deg"] > 3:
        assert a[4] < b[4], "the batch did not take the one-kernel pass"
