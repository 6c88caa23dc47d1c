"""The 10-step Lanczos upper estimate of each problem's spectrum (laph_solver_features, `bound`) against the same ten steps
on the host: the oracle's assembled -Delta, the same start vector, NumPy's eigensolver on the tridiagonal.  Then a free
field, whose Krylov space ends after seven steps (seven distinct eigenvalues at 4^3): the estimate is the top, 12."""
import ctypes

import numpy as np
import pytest

from conftest import random_links, unit_links

pytestmark = pytest.mark.gpu

STEPS = 10


def _start(dim, p):
    """The kernel's start vector for problem p: a counter hash."""
    u = np.uint64
    z = np.arange(dim, dtype=u) * u(0x9E3779B97F4A7C15) + u(0x632BE59BD9B4E019) + u((p * 0xD1B54A32D192ED03) % 2 ** 64)
    z = (z ^ (z >> u(30))) * u(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> u(27))) * u(0x94D049BB133111EB)
    z = z ^ (z >> u(31))
    a = (z >> u(11)).astype(float) / 2.0 ** 53 - 0.5
    b = ((z * u(0x9E3779B97F4A7C15)) >> u(11)).astype(float) / 2.0 ** 53 - 0.5
    return a + 1j * b


def _lanczos_bound(A, p):
    v = _start(A.shape[0], p)
    v /= np.linalg.norm(v)
    prev, beta = np.zeros_like(v), 0.0
    al, be = [], []
    for _ in range(STEPS):
        w = A @ v - beta * prev
        al.append(np.vdot(v, w).real)
        w -= al[-1] * v
        beta = np.linalg.norm(w)
        be.append(beta)
        prev, v = v, w / beta
    theta, q = np.linalg.eigh(np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1))
    return theta[-1] + abs(be[-1] * q[-1, -1])


def _bounds(gpu, probs, links):
    s = gpu.Solver(probs, guard=8, tol=1e-3, deg=8, max_it=2)
    for i, U in enumerate(links):
        s.set_links(i, U)
    s.run()
    bound = np.empty(len(probs))
    gpu.check(gpu.lib.laph_solver_features(s._h, None, ctypes.c_void_p(bound.ctypes.data)), "laph_solver_features")
    s.close()
    return bound


def test_bound_is_the_lanczos_estimate(gpu, orc):
    probs = [(8, 12), (5, 8), (7, 12), (8, 12)]
    links = [random_links(L, eps, 5800 + i) for i, ((L, _), eps) in enumerate(zip(probs, (0.25, 0.4, 0.3, 0.45)))]
    got = _bounds(gpu, probs, links)
    for p, ((L, _), U) in enumerate(zip(probs, links)):
        A = orc.neglap_dense(U, L)
        # sums of 1536 terms round at 1e-13 of 12, and ten steps in which no Ritz pair converges add them up
        assert abs(got[p] - _lanczos_bound(A, p)) <= 1e-10, p
        assert got[p] <= 12.5 and got[p] >= np.linalg.eigvalsh(A)[-1] - 0.5


def test_bound_of_an_invariant_subspace(gpu):
    got = _bounds(gpu, [(4, 8)], [unit_links(4)])
    assert abs(got[0] - 12.0) <= 1e-8
