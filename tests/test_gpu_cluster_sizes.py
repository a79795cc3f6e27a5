"""GPU test of the largest-cluster analysis at the edges of its launches: molecule counts
around the warp and block sizes (1, 33, 1024, 1025, 2500) and cell grids of one, two and
more cells per side (repeated cells count again, as in the reference).  Whole numbers and
the updated ``ptta_full`` equal the oracle's."""
import numpy as np
import pytest

from molecular_simulation_code_b200 import nonbond as nb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_gly,box,densmin", [(1, 10.0, 0), (33, 17.0, 4), (33, 26.0, 3),
                                               (1024, 80.0, 2), (1025, 60.0, 4),
                                               (2500, 90.0, 3)])
@pytest.mark.parametrize("greatest_in", [0, 3])
def test_cluster_analysis_sizes(ctx, n_gly, box, densmin, greatest_in):
    rng = np.random.default_rng(n_gly)
    apg, box = 3, np.float32(box)
    centres = rng.uniform(0, float(box), (n_gly, 1, 3))
    x = np.mod(centres + rng.normal(0, 0.7, (n_gly, apg, 3)), float(box)).reshape(-1, 3)
    n = n_gly * apg + 5  # five atoms of something else
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = np.concatenate([x, rng.uniform(0, float(box), (5, 3))]).astype(np.float32)
    perm = rng.permutation(n)
    pos, gid = np.ascontiguousarray(pos[perm]), (perm + 1).astype(np.int32)
    ptta0 = rng.uniform(0, float(box), (n_gly * apg, 3))
    ibox = np.float32(1.0 / np.float64(box))
    vol = np.float32(np.float32(box * box) * box)
    pt_o, pt_g = ptta0.copy(), ptta0.copy()
    want = O.greatest_cluster(pos, gid, n_gly, apg, box, ibox, vol, 9.0, 6.0, densmin, pt_o,
                              greatest_in)
    if want[2].max() > 256:  # more than a density list holds (one cell seen 27 times): refused
        with pytest.raises(nb.SofiaError, match="density list overflow"):
            nb.get_greatest_cluster(ctx, pos, gid, n_gly, apg, box, 9.0, 6.0, densmin, pt_g,
                                    greatest_in)
        return
    got = nb.get_greatest_cluster(ctx, pos, gid, n_gly, apg, box, 9.0, 6.0, densmin, pt_g,
                                  greatest_in)
    assert got[:2] == want[:2]
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[3], want[3])
    assert np.array_equal(pt_g, pt_o)
