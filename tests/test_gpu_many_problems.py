"""A batch of more problems than a grid has rows (65535): the small dense step and the plaquette values run it in groups.
The batch repeats two timeslices, so every problem has to come out as one of two solved in a small batch: its plaquette
features bit for bit, its eigenvalues to the tolerance (on both sides of a group's edge), and all converged."""
import ctypes

import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu

L, NEV, N = 3, 8, 65535 + 5


def _solve(gpu, n, links):
    # block 32 keeps the filter of the small batch on the step kernels that the large one takes
    s = gpu.Solver([(L, NEV)] * n, guard=8, tol=1e-8, deg=8, max_it=60, block=32)
    for i in range(n):
        s.set_links_device(i, links[i % 2].data_ptr())
    st, res = s.run()
    feats = np.empty((n, 16), np.float32)
    gpu.check(gpu.lib.laph_solver_features(s._h, ctypes.c_void_p(feats.ctypes.data), None), "laph_solver_features")
    ev = {i: s.get(i, vectors=False)[0] for i in (0, 1, n // 2, n - 6, n - 5, n - 4, n - 1) if 0 <= i < n}
    s.close()
    return st, res, feats, ev


def test_more_problems_than_grid_rows(gpu):
    import torch
    links = [torch.from_numpy(random_links(L, 0.4, 5600 + i)).cuda() for i in range(2)]
    torch.cuda.synchronize()
    st, _, f2, e2 = _solve(gpu, 2, links)
    assert st == 0
    st, res, f, e = _solve(gpu, N, links)
    assert st == 0 and all(r["nconv"] == NEV for r in res)
    assert np.array_equal(f[0::2, :4], np.broadcast_to(f2[0, :4], f[0::2, :4].shape))
    assert np.array_equal(f[1::2, :4], np.broadcast_to(f2[1, :4], f[1::2, :4].shape))
    for i, ev in e.items():
        # each problem has its own random start block: equal to the residual bound, 1e-8 of 12
        assert np.abs(ev - e2[i % 2]).max() <= 1e-8 * 12.0, i
