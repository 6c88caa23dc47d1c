"""The autotuner times the kernels that the tuned solve will run: a sample's solver takes the forms of its whole batch
(csrc/batch_form.h), settings tuned for one form are not read back for another, and a batch whose filter runs whole
passes as one kernel has no block and no tile to tune."""
import ctypes

import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu

L, NEV = 8, 20
KW = dict(guard=16, tol=1e-10, deg=24, max_it=300)


class _Sample:
    """A solver over `probs` as the sample of `batch` (laph_solver_create_for, the autotuner's own)."""

    def __new__(cls, gpu, probs, batch, **kw):
        from laph_eigsys_b200 import _lib
        arrays = [(_lib.laph_problem * len(p))(*[_lib.laph_problem(*q) for q in p]) for p in (probs, batch)]
        o = gpu.solve_opts(**kw)
        h = ctypes.c_void_p()
        gpu.check(gpu.lib.laph_solver_create_for(ctypes.byref(h), arrays[0], len(probs), ctypes.byref(o), 0, arrays[1],
                                                 len(batch)), "laph_solver_create_for")
        s = object.__new__(gpu.Solver)
        s.problems, s.opts, s._h = list(probs), o, h
        return s


def _run(s, probs):
    for i, (l, _) in enumerate(probs):
        s.set_links(i, random_links(l, 0.4, 5300 + i))
    assert s.run()[0] == 0
    out, launches = [s.get(i) for i in range(len(probs))], s.counters()[1]
    s.close()
    return out, launches


# 200 x 8^3 x 64 columns: 6.6e6 site-columns, past the one-kernel pass; five extents: more than it takes
@pytest.mark.parametrize("batch", [[(L, NEV)] * 200, [(L, NEV)] * 2 + [(5, 8), (6, 8), (7, 8), (9, 8)]],
                         ids=["large batch", "five extents"])
def test_a_sample_runs_the_kernels_of_its_batch(gpu, batch):
    probs = [(L, NEV)] * 2
    ref, steps = _run(gpu.Solver(probs, filter_kernel=2, **KW), probs)
    alone, pass_launches = _run(gpu.Solver(probs, **KW), probs)
    out, launches = _run(_Sample(gpu, probs, batch, **KW), probs)
    assert pass_launches < steps and launches == steps
    for a, b, c in zip(ref, alone, out):  # the forms differ in no bit
        assert all(np.array_equal(x, y) and np.array_equal(x, z) for x, y, z in zip(a, b, c))


def test_settings_belong_to_the_form_they_were_tuned_for(gpu, tmp_path):
    cache = tmp_path / "tune.txt"
    links = [random_links(L, 0.4, 5400 + i) for i in range(2)]
    kw = dict(KW, deg=40, window=gpu.WINDOW_LANCZOS)

    def tune(n):
        return gpu.autotune([(L, NEV)] * n, links, nsample=2, cache=cache, **kw)

    opts, small = tune(2)
    # deg (8) and guard (2 more) only; the batch keeps its pass
    assert small["from_cache"] == 0 and small["trials"] <= 10
    assert (small["block"], small["tile"]) == (opts.block, opts.filter_tile) == (16, 128)
    _, large = tune(200)
    assert large["from_cache"] == 0 and large["trials"] > 10
    assert tune(2)[1]["from_cache"] == 1 and tune(201)[1]["from_cache"] == 1
    opts, again = tune(3)  # still a pass: the line of two
    assert again["from_cache"] == 1 and opts.block == 16
