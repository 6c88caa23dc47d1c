"""The Gram of small batches (k_gram_split, csrc/dense.cu) where its staging can go wrong: fewer rows than one 16-row stage
past a multiple (3^3: 81 rows), one row short of a ring's worth, a second row chunk of a few stages (14^3: 8232 rows in
chunks of 8192), one tile pair and several, diagonal and off-diagonal.  A wrong Gram or projected matrix shows in the
returned block: it would not be orthonormal, or its Ritz pairs would not satisfy the operator (checked with the
context's own stencil)."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nev,n", [(3, 8, 1), (4, 40, 2), (5, 70, 1), (7, 24, 3), (14, 24, 1), (14, 60, 2)])
def test_blocks_are_orthonormal_eigenvectors(gpu, L, nev, n):
    tol = 1e-10
    s = gpu.Solver([(L, nev)] * n, guard=8, tol=tol, deg=16, max_it=400)
    links = [random_links(L, 0.4, 4300 + L + i) for i in range(n)]
    for i, U in enumerate(links):
        s.set_links(i, U)
    st, _ = s.run()
    assert st == 0
    for i, U in enumerate(links):
        ev, V, _ = s.get(i)
        assert np.abs(V.conj().T @ V - np.eye(nev)).max() <= 1e-10
        c = gpu.Context(L)
        c.set_links(U)
        r = [np.linalg.norm(c.apply_neglap(V[:, j]) + ev[j] * V[:, j]) for j in range(nev)]
        c.close()
        assert max(r) <= 2.0 * tol * 12.0
    s.close()
