"""GPU test of the pair kernels' row split: 4, 2 or 1 warps per list row by system size.

Sizes on each side of the rule (4 warps, 2 warps, 1 warp per row in the mixed path; 4, 2, 1
in FP64), and long rows (a 13 A cut-off: more 32-entry batches than energy slots).
Bars as in test_gpu_mixed_path: FP64 within 1e-10 of the oracle's FP64 list forces, mixed
force RMS error at most 1e-6, energies of the mixed path within 1e-6 of FP64's.
"""
import numpy as np
import pytest

from molecular_simulation_code_b200 import mixed as M
from molecular_simulation_code_b200.system import make_system
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_gly,n_wat,cut", [(20, 780, 10.0), (150, 2500, 10.0), (150, 2500, 13.0),
                                             (400, 4000, 10.0), (600, 11500, 10.0)])
def test_row_split_matches_oracle(ctx, n_gly, n_wat, cut):
    s = make_system(n_gly, n_wat, 5)
    p = O.params(0.2, s.box, cut, cut, 1.0)
    # the O(N^2) list: the cell list counts pairs twice in a box of two cells per side
    nl, nn = O.neighbor_n2(p, s.position_aos(), s.specbond, s.num3bond, 2048)
    _, ref, pot, ec, vir = O.force_dsf(p, s.position_aos(), s.q, (s.lj1, s.lj2, s.lj3, s.lj4),
                                       s.ntypes, nl, nn, 2048)
    m = M.System(ctx, s, cut=cut, skin=1.0)
    m.set_state(s.xyz.astype(np.float64))
    for precision, ftol, etol in ((M.FP64, 1e-10, 1e-10), (M.MIXED, 1e-6, 1e-6)):
        e = m.compute(precision, rebuild=True)
        f = m.get_state()[2]
        err = M.force_max_rel(f, ref) if precision == M.FP64 else M.force_rms_rel(f, ref)
        assert err <= ftol
        assert abs(e[0] - pot) <= etol * abs(pot) and abs(e[1] - ec) <= etol * abs(ec)
        assert np.abs(e[2:] - vir).max() <= 10 * etol * np.abs(vir).max()
        m.compute(precision, energy=False)  # the force-only kernel: the same bits
        assert np.array_equal(m.get_state()[2], f)
    m.close()
