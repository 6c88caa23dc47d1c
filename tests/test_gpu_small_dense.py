"""The small dense step of the Rayleigh-Ritz (csrc/small.cu) at the block widths where its paths change: 32 (one tile,
one pair per CTA), 224 and 256 (the last width whose Jacobi runs on 8 CTAs, and one on 16), 320 and 352 (the last in
shared memory, and one in global memory), 384 and 416 (the Cholesky's panel in shared memory and not), 512; and one, two
and three Jacobi sweeps, which split into launches of two (one where the matrix is in global memory)."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu

L = 8


@pytest.fixture(scope="module")
def dense(orc):
    U = random_links(L, 0.4, 1301)
    A = orc.neglap_dense(U, L)
    return U, A, np.linalg.eigvalsh(A)


@pytest.mark.parametrize("nev,sweeps", [(12, 2), (12, 1), (200, 2), (240, 2), (240, 3), (304, 2), (330, 2), (330, 3),
                                        (368, 2), (390, 2), (490, 1), (490, 2)])
def test_block_widths(gpu, dense, nev, sweeps):
    """Eigenvalues to 1e-10 of lambda_max (the residual bound 1e-10 makes them far better where gaps exceed it, and never
    worse than the residual itself), residuals to the solver's tolerance, and an orthonormal block."""
    U, A, w = dense
    s = gpu.Solver([(L, nev)], guard=16, tol=1e-10, deg=16, max_it=300, jacobi_sweeps=sweeps)
    s.set_links(0, U)
    st, res = s.run()
    ev, V, _ = s.get(0)
    s.close()
    assert st == 0 and res[0]["nconv"] == nev
    assert np.abs(-ev - w[:nev]).max() <= 1e-10 * 12.0
    assert np.linalg.norm(A @ V + V * ev[None, :], axis=0).max() <= 2e-10 * 12.0
    assert np.abs(V.conj().T @ V - np.eye(nev)).max() <= 1e-10
