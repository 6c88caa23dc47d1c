"""Which kernels the default filter runs (csrc/solver.cu): a small batch takes the one-kernel pass, and a column block or
a tile other than such a batch's own (16 columns, 128 sites) takes the kernels that run step by step, which alone have
them.  The step kernels then stay covered on small lattices: every tile with both link types, the staged and the brick
variant, and the bounds-checked build, all bit for bit."""
import ctypes
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import random_links

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _solve(gpu, probs, seed=5100, **kw):
    s = gpu.Solver(probs, guard=16, tol=1e-10, deg=24, smear_kind=gpu.SMEAR_STOUT, smear_p1=0.1, smear_iters=2, **kw)
    for i, (L, _) in enumerate(probs):
        s.set_links(i, random_links(L, 0.35, seed + 10 * L + i))
    st, _ = s.run()
    assert st == 0
    out, launches = [s.get(i) for i in range(len(probs))], s.counters()[1]
    s.close()
    return out, launches


def _same(a, b):
    return all(np.array_equal(x, y) for p, q in zip(a, b) for x, y in zip(p, q))


PROBS = [(10, 24), (12, 30)]


def _form(gpu, probs, **kw):
    s = gpu.Solver(probs, **kw)
    block, one = ctypes.c_int(), ctypes.c_int()
    gpu.check(gpu.lib.laph_solver_form(s._h, ctypes.byref(block), ctypes.byref(one)), "laph_solver_form")
    s.close()
    return block.value, one.value


def test_a_solver_says_which_form_it_runs(gpu):
    assert _form(gpu, PROBS) == (16, 1)
    assert _form(gpu, PROBS, block=16, filter_tile=128) == (16, 1)
    assert _form(gpu, PROBS, filter_tile=64) == (16, 0)
    assert _form(gpu, PROBS, block=8) == (8, 0)
    assert _form(gpu, PROBS, filter_kernel=2) == (16, 0)
    assert _form(gpu, [(32, 120)]) == (16, 0)  # 4.5e6 site-columns
    assert _form(gpu, [(32, 120)] * 2) == (32, 0)


def test_own_block_and_tile_keep_the_one_kernel_pass(gpu):
    ref, steps = _solve(gpu, PROBS, filter_kernel=2)
    for kw in ({}, {"block": 16}, {"filter_tile": 128}, {"block": 16, "filter_tile": 128}):
        out, launches = _solve(gpu, PROBS, **kw)
        assert launches < steps and _same(out, ref), kw


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("kw", [{"filter_tile": 64}, {"filter_tile": 256}, {"block": 32}, {"block": 32, "filter_tile": 128},
                                {"block": 8}, {"block": 16, "filter_tile": 256}])
def test_other_blocks_and_tiles_run_step_by_step(gpu, kw, prec):
    lp = gpu.LINKS_BF16 if prec == "bf16" else gpu.LINKS_FP32
    ref, steps = _solve(gpu, PROBS, filter_kernel=2, link_prec=lp)
    out, launches = _solve(gpu, PROBS, link_prec=lp, **kw)
    assert launches == steps and _same(out, ref)


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
def test_staged_and_brick_variants_match_the_step_kernel(gpu, prec):
    lp = gpu.LINKS_BF16 if prec == "bf16" else gpu.LINKS_FP32
    probs = [(16, 40), (32, 24), (16, 20)]
    ref, steps = _solve(gpu, probs, block=32, link_prec=lp)
    for variant in (3, 4):
        out, launches = _solve(gpu, probs, filter_kernel=variant, link_prec=lp)
        assert launches == steps and _same(out, ref), variant


def _checked(out_path):
    """The step kernels' solve in a process with the checked library; its eigenpairs go to out_path."""
    import laph_eigsys_b200 as lb
    assert lb.check_enabled()
    lb.check_report(reset=True)
    arrays = {}
    for tile in (64, 128, 256):
        out, launches = _solve(lb, PROBS, block=32, filter_tile=tile)
        for i, (ev, V, _) in enumerate(out):
            arrays[f"ev{tile}_{i}"], arrays[f"v{tile}_{i}"] = ev, V
        arrays[f"launches{tile}"] = np.array(launches)
    np.savez(out_path, **arrays)
    print(json.dumps(lb.check_report()))


def test_step_kernels_under_the_checked_build(gpu, tmp_path):
    path = tmp_path / "checked.npz"
    code = f"import sys; sys.path.insert(0, {HERE!r}); import test_gpu_filter_forms as t; t._checked({str(path)!r})"
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, LAPH_GPU_LIB="check"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-3000:]
    assert json.loads(p.stdout.strip().splitlines()[-1]) == {"count": 0}
    got = np.load(path)
    ref, steps = _solve(gpu, PROBS, filter_kernel=2)
    for tile in (64, 128, 256):
        assert int(got[f"launches{tile}"]) == steps
        for i, (ev, V, _) in enumerate(ref):
            # the same source compiled with the checks: eigenvalues to rounding (of 12), vectors up to their phase
            assert np.abs(got[f"ev{tile}_{i}"] - ev).max() <= 1e-10 * 12.0
            overlap = np.abs(got[f"v{tile}_{i}"].conj().T @ V)
            assert np.abs(np.linalg.norm(overlap, axis=0) - 1.0).max() <= 1e-6


@pytest.mark.parametrize("loop", [0, 1], ids=["device loop", "host loop"])
@pytest.mark.parametrize("prec,lbytes", [("fp32", 216), ("bf16", 112)])
def test_filter_bytes_count_the_links_the_form_reads(gpu, prec, lbytes, loop):
    """One filter pass (after the first Rayleigh-Ritz) over 32 unlocked columns of 8^3: the same steps in both forms,
    whose links are read once, or per step and block of 16 columns."""
    got = {}
    for name, kw in (("pass", {}), ("steps", {"block": 16, "filter_tile": 64})):
        s = gpu.Solver([(8, 20)], guard=12, tol=1e-10, deg=12, max_it=2, host_loop=loop,
                       link_prec=gpu.LINKS_BF16 if prec == "bf16" else gpu.LINKS_FP32, **kw)
        s.set_links(0, random_links(8, 0.4, 5700))
        s.run()
        got[name] = s.counters()[0], s.filter_bytes()
        s.close()
    assert got["pass"][0] == got["steps"][0] and got["pass"][0] % (8 ** 3 * 32) == 0
    steps = got["pass"][0] // (8 ** 3 * 32)
    assert steps >= 1
    for a, b in zip(got["steps"][1], got["pass"][1]):
        assert a - b == 8 ** 3 * lbytes * (2 * steps - 1)
