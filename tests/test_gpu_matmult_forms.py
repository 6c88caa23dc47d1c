"""The three forms of the one-launch MatShell product (csrc/stencil64.cu) at their edges, against the oracle's tv_iter: one
cluster of 16 CTAs (27 sites, most CTAs empty; 12^3, its largest), one CTA per SM (13^3; 33^3, the largest with a site per
thread), and grid-stride (34^3); degrees 2 and 3 (T_1 alone is another path) to 12, one context used twice."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,deg", [(3, 2), (3, 9), (8, 8), (12, 3), (12, 12), (13, 12), (33, 4), (34, 3)])
def test_forms_against_tv_iter(gpu, orc, L, deg):
    U = random_links(L, 0.4, 4700 + L)
    c = gpu.Context(L, 11.8, 0.6, deg)
    c.set_links(U)
    rng = np.random.default_rng(L)
    for _ in range(2):
        x = rng.normal(size=3 * L ** 3) + 1j * rng.normal(size=3 * L ** 3)
        ref = orc.tv_iter(U, L, 11.8, 0.6, deg, x)
        assert np.linalg.norm(c.matmult(x) - ref) <= 1e-13 * np.linalg.norm(ref)
    c.close()
