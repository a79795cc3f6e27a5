"""GPU test of the reference-layout list build at the edges of its rules: 2 to 6 cells per
side (one image per stencil cell is used from 5 on), cells above and below the counting
sort's size, an odd and an even number of atoms, coordinates outside the box, which the
binning takes into the edge cells, and coordinates on a grid of 0.01 A, where many pairs lie
at exactly the list radius and every product has to round by itself.  Rows equal the oracle's entry by entry."""
import numpy as np
import pytest

from helpers import ref_params
from molecular_simulation_code_b200 import nonbond as nb
from molecular_simulation_code_b200.system import make_system
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut,side", [(17.0, 2), (10.0, 3), (8.5, 4), (7.0, 5), (5.5, 6)])
@pytest.mark.parametrize("n_wat,outside,grid", [(1400, False, False), (1401, True, False),
                                                (1400, False, True)])
def test_list_rows_exact(ctx, cut, side, n_wat, outside, grid):
    s = make_system(40, n_wat, 2)
    p = ref_params(s, cut=cut, pad=1.0)
    op = O.params(p.alpha, p.box, p.cut_coul, p.rcut, p.neighbor_pad)
    _, nt, nd = O.cell_grid(op)
    assert nd == side
    pos = s.position_aos()
    if grid:
        pos[:, :3] = np.round(pos[:, :3], 2)
        pos[:, :3] = np.minimum(pos[:, :3], s.box)
    if outside:
        rng = np.random.default_rng(3)
        hi, lo = rng.permutation(s.np_atoms)[:80].reshape(2, 40)
        pos[hi, rng.integers(0, 3, 40)] += np.float32(1.3) * s.box
        pos[lo, rng.integers(0, 3, 40)] = -rng.uniform(0.1, 3.0, 40).astype(np.float32)
    tt, ttb, st, en, ab = O.bin_sort(op, pos)
    ps = np.ascontiguousarray(pos[ttb - 1])
    sb = np.zeros_like(s.specbond)
    for new in range(s.np_atoms):
        o = ttb[new] - 1
        sb[new, :s.num3bond[o]] = tt[s.specbond[o, :s.num3bond[o]] - 1]
    n3 = np.ascontiguousarray(s.num3bond[ttb - 1])
    alloc = 9600  # a box of two cells per side lists pairs twice
    onl, onn, mx = O.build_neighbor_sorted(op, ps, ab, st, en, O.stencil(nt, nd), sb, n3, alloc)
    assert mx <= alloc
    nl, nn, na = nb.neighbor_wrapper(ctx, ps, sb, n3, p, neigh_alloc=alloc)
    assert na == alloc and np.array_equal(nn, onn)
    used = np.arange(alloc)[None, :] < nn[:, None]
    assert np.array_equal(nl.reshape(-1, alloc)[used], onl.reshape(-1, alloc)[used])


@pytest.mark.parametrize("cut,side", [(17.0, 2), (13.0, 3), (10.0, 4), (9.0, 5)])
@pytest.mark.parametrize("n_wat", [3866, 3867])  # 11,998 and 12,001 atoms
@pytest.mark.parametrize("outside", [False, True])
def test_list_rows_exact_at_chunk_sizes(ctx, cut, side, n_wat, outside):
    """Chunks of 4 atoms below 12,000 atoms and of 8 from there on, coordinates on the grid."""
    s = make_system(40, n_wat, 2)
    p = ref_params(s, cut=cut, pad=1.0)
    op = O.params(p.alpha, p.box, p.cut_coul, p.rcut, p.neighbor_pad)
    _, nt, nd = O.cell_grid(op)
    assert nd == side
    pos = s.position_aos()
    pos[:, :3] = np.minimum(np.round(pos[:, :3], 2), s.box)
    if outside:
        pos[::97, 0] += np.float32(1.3) * s.box
        pos[5::97, 1] = -2.5
    tt, ttb, st, en, ab = O.bin_sort(op, pos)
    ps = np.ascontiguousarray(pos[ttb - 1])
    sb = np.zeros_like(s.specbond)
    for new in range(s.np_atoms):
        o = ttb[new] - 1
        sb[new, :s.num3bond[o]] = tt[s.specbond[o, :s.num3bond[o]] - 1]
    n3 = np.ascontiguousarray(s.num3bond[ttb - 1])
    alloc = 9600  # a box of two cells per side lists pairs twice
    onl, onn, mx = O.build_neighbor_sorted(op, ps, ab, st, en, O.stencil(nt, nd), sb, n3, alloc)
    assert mx <= alloc
    nl, nn, na = nb.neighbor_wrapper(ctx, ps, sb, n3, p, neigh_alloc=alloc)
    assert na == alloc and np.array_equal(nn, onn)
    used = np.arange(alloc)[None, :] < nn[:, None]
    assert np.array_equal(nl.reshape(-1, alloc)[used], onl.reshape(-1, alloc)[used])
