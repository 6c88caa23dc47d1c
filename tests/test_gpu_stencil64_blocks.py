"""The FP64 block stencils (A W and the residual) at every width of their column blocks: the solver takes narrower blocks
for smaller batches, each thread 1, 2 or 4 columns a trip, with the same arithmetic and the same sums per column -- so a
problem solved alone, in the narrowest blocks, and as the first of ever larger batches has the same bits.  343 sites: two
full tiles and a ragged one; 27 sites: a single ragged tile."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu


def _solve(gpu, L, nev, n):
    s = gpu.Solver([(L, nev)] * n, guard=16, tol=1e-10, deg=12, max_it=300, smear_kind=gpu.SMEAR_STOUT, smear_p1=0.1,
                   smear_iters=2)
    for i in range(n):
        s.set_links(i, random_links(L, 0.35, 9000 + 100 * L + i))
    st, res = s.run()
    out = s.get(0)
    s.close()
    return st, res[0], out


# 32 columns: 3 n (or n) tiles; the blocks halve below 148 CTAs, so these are 2, 4, 8, 16 and 32 columns wide
@pytest.mark.parametrize("L,nev,batches", [(7, 11, (1, 8, 13, 25, 50)), (3, 8, (1, 149))], ids=["343 sites", "27 sites"])
def test_blocks_of_every_width_have_the_same_bits(gpu, L, nev, batches):
    st, res, (ev, V, ph) = _solve(gpu, L, nev, batches[0])
    assert st == 0 and res["max_resid"] <= 1e-10
    for n in batches[1:]:
        st, r, (e, v, p) = _solve(gpu, L, nev, n)
        assert st == 0 and r["iters"] == res["iters"] and r["max_resid"] == res["max_resid"]
        assert np.array_equal(e, ev) and np.array_equal(v, V) and np.array_equal(p, ph)
