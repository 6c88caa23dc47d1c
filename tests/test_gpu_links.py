"""Links in and out of a context and a solver (the tiled reorder of csrc/links.cu, staged in chunks by csrc/capi_ctx.cu):
every layout in, every layout out, bit for bit, at sizes below one 32-site tile (27 sites), of ragged tiles, at one staging
chunk and at several with a short last one; a non-finite entry is refused wherever it falls, names its site, and leaves
the context's links as they were."""
import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu


def _boundary(U, layout, gpu):
    """U (V3, 3, 3, 3) as the layout's host array."""
    if layout == gpu.LAYOUT_EIGEN:
        return np.ascontiguousarray(np.swapaxes(U, 2, 3))  # column-major 3x3 memory
    if layout == gpu.LAYOUT_CONF:
        c = np.zeros((U.shape[0], 4, 3, 3), dtype=np.complex128)
        c[:, 0] = np.eye(3)
        c[:, 1:] = U
        return c
    return U


@pytest.mark.parametrize("L", [3, 4, 7, 10, 11, 21])
def test_round_trip_of_every_layout(gpu, L):
    U = random_links(L, 0.5, 4400 + L)
    layouts = (gpu.LAYOUT_ROWMAJOR, gpu.LAYOUT_EIGEN, gpu.LAYOUT_CONF)
    c = gpu.Context(L)
    for a in layouts:
        c.set_links(_boundary(U, a, gpu), a)
        for b in layouts:
            assert np.array_equal(c.get_links(b), _boundary(U, b, gpu)), (a, b)
    c.close()


@pytest.mark.parametrize("L,site", [(4, 63), (11, 0), (11, 1023), (11, 1024), (11, 1330), (21, 9260)])
def test_non_finite_links_are_refused_and_change_nothing(gpu, L, site):
    U = random_links(L, 0.5, 4500 + L)
    c = gpu.Context(L)
    c.set_links(U)
    for value in (np.nan, np.inf):
        bad = 2.0 * U
        bad[site, 2, 1, 0] = value
        with pytest.raises(gpu.LaphError, match=f"site {site}"):
            c.set_links(bad)
        assert np.array_equal(c.get_links(), U)
    c.close()


def test_solver_takes_every_layout(gpu):
    L = 5
    U = random_links(L, 0.4, 4600)
    out = []
    for layout in (gpu.LAYOUT_ROWMAJOR, gpu.LAYOUT_EIGEN, gpu.LAYOUT_CONF):
        s = gpu.Solver([(L, 12)], guard=16, tol=1e-10, deg=12)
        s.set_links(0, _boundary(U, layout, gpu), layout)
        assert s.run()[0] == 0
        out.append(s.get(0))
        s.close()
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], o))
