"""The source shape's persistent tile kernel (k_ss_tile) where its pieces change: one
ragged tile, tiles cut by the last row, eigenvector counts that do not fill a ring
stage, several tiles per CTA, and lattices whose bins do not fit shared memory --
against the definition psi(r) = sum_x ||V_{x+r} V_x^dag||_F."""
import ctypes
import itertools

import numpy as np
import pytest

import laph_eigsys_b200 as lb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
EPS = 2.0 ** -53


# (L, nev): 1 and 8 sites per parity class, 27 and 125 (ragged tiles), 7 ragged tiles
# (224 tile pairs), 1088 pairs; 4913 bins, past shared memory
@pytest.mark.parametrize("L,nev", [(2, 1), (4, 3), (6, 8), (10, 9), (12, 5), (16, 17), (34, 4)])
def test_tiles(L, nev):
    gen = torch.Generator("cuda").manual_seed(100 * L + nev)
    v = torch.randn(nev, L, L, L, 3, dtype=torch.complex128, device="cuda", generator=gen)
    torch.cuda.synchronize()
    psi = np.full((L // 2) ** 3, np.nan)
    lb.check(lb.lib.laph_sourceshape(ctypes.c_void_p(v.data_ptr()), L, nev, None, 1,
                                     ctypes.c_void_p(psi.ctypes.data), 0), "laph_sourceshape")
    V = v.permute(1, 2, 3, 4, 0).contiguous()  # [x, y, z, colour, n]
    rs = list(itertools.product(range(L // 2), repeat=3))
    if len(rs) > 64:
        rs = rs[:2] + rs[-2:] + [rs[i] for i in np.random.default_rng(L).choice(len(rs), 60, replace=False)]
    for r in rs:
        W = torch.roll(V, shifts=[-2 * d for d in r], dims=(0, 1, 2))  # W(x) = V(x + r)
        ref = float(torch.linalg.matrix_norm(W @ V.conj().transpose(-1, -2)).sum())
        # products: nev terms whose sum is ~sqrt(nev) smaller than its terms' magnitude;
        # then a sum of L^3 positive norms; both sides round
        tol = 4 * (nev ** 1.5 + L ** 3) * EPS
        got = psi[(r[0] * (L // 2) + r[1]) * (L // 2) + r[2]]
        assert abs(got - ref) <= tol * ref, (r, got, ref)
