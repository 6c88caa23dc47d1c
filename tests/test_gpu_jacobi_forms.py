"""The Jacobi of the small dense step (csrc/small.cu) off its default form: blocks whose cluster the device has no room
for run in global memory, with the same bits (limited by hand here: no clusters at all, and none of 16 CTAs); the widths
where the kernels around it change (128 | 160 split threads, 160 | 192 and 256 | 288 rows of the rotations' product); and
narrow problems beside one too wide for shared memory, which sets the form of the batch."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu


def _solve(gpu, probs, limit=None, sweeps=2, tol=1e-10):
    s = gpu.Solver(probs, guard=16, tol=tol, deg=16, max_it=300, jacobi_sweeps=sweeps)
    if limit is not None:
        gpu.check(gpu.lib.laph_solver_limit_jacobi(s._h, limit), "laph_solver_limit_jacobi")
    for i, (L, _) in enumerate(probs):
        s.set_links(i, random_links(L, 0.4, 1301 + 7 * i))
    st, res = s.run()
    out = [s.get(i) for i in range(len(probs))]
    s.close()
    assert st == 0 and all(r["nconv"] == nev for r, (_, nev) in zip(res, probs))
    return out


# widths 32, 128, 224 (clusters of 8), 256 and 320 (of 16); at six sweeps the last launches find the matrix diagonal and
# only bring the rows into Ritz order, in place
@pytest.mark.parametrize("nev,limit,sweeps", [(12, 0, 2), (112, 0, 2), (112, 0, 3), (208, 0, 2), (240, 224, 2), (240, 0, 3),
                                              (304, 224, 2),
                                              (40, 0, 6), (208, 0, 6)])
def test_without_room_for_clusters_the_bits_are_the_same(gpu, nev, limit, sweeps):
    a, b = (_solve(gpu, [(8, nev)], limit=l, sweeps=sweeps) for l in (None, limit))
    assert all(np.array_equal(x, y) for x, y in zip(a[0], b[0]))


def _check(gpu, orc, probs, out, tol):
    for i, ((L, nev), (ev, V, _)) in enumerate(zip(probs, out)):
        A = orc.neglap_dense(random_links(L, 0.4, 1301 + 7 * i), L)
        w = np.linalg.eigvalsh(A)
        assert np.abs(-ev - w[:nev]).max() <= 1e-10 * 12.0
        assert np.linalg.norm(A @ V + V * ev[None, :], axis=0).max() <= 2.0 * tol * 12.0
        assert np.abs(V.conj().T @ V - np.eye(nev)).max() <= 1e-10


@pytest.mark.parametrize("nev", [112, 144, 176, 272])
def test_widths_where_the_kernels_change(gpu, orc, nev):
    probs = [(8, nev)]
    _check(gpu, orc, probs, _solve(gpu, probs), 1e-10)


@pytest.mark.parametrize("probs", [[(6, 12), (8, 330), (7, 40)], [(6, 12), (8, 240), (8, 100)]],
                         ids=["beside 352", "beside 256"])
def test_narrow_problems_beside_a_wide_one(gpu, orc, probs):
    _check(gpu, orc, probs, _solve(gpu, probs), 1e-10)


def test_the_limit_is_refused_where_it_cannot_apply(gpu):
    s = gpu.Solver([(4, 8)], guard=8, tol=1e-8, deg=8)
    assert gpu.lib.laph_solver_limit_jacobi(s._h, -1) == gpu._lib.LAPH_EINVAL
    assert gpu.lib.laph_solver_limit_jacobi(None, 0) == gpu._lib.LAPH_EINVAL
    s.close()
