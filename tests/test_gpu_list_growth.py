"""GPU test of captured work that outlives its lists: a force evaluation that grows the row
capacity frees the lists which the system's captured MD steps were made with.  The next
segment is bit for bit that of a system which never had the small lists."""
import dataclasses

import numpy as np
import pytest

from molecular_simulation_code_b200 import mixed as M
from molecular_simulation_code_b200.system import make_system

pytestmark = pytest.mark.gpu


def test_md_graphs_after_list_growth(ctx):
    s = make_system(20, 780, 6)
    # a droplet in a box of 64 times its volume: rows sized for 1/64 of its density
    box = np.float32(4.0 * float(s.box))
    drop = dataclasses.replace(s, box=box)
    compact, spread = s.xyz.astype(np.float64), 4.0 * s.xyz.astype(np.float64)
    rest = np.zeros_like(compact)

    def system():
        m = M.System(ctx, drop, cut=10.0, skin=2.0)
        m.md_setup(drop, dt=1.0, gamma=0.0, seed=4, terms=0, shake=False)
        return m

    m = system()
    m.set_state(spread, rest)
    m.md_run(2)  # captured on the lists of the spread atoms
    small = m.stats()["jcap"]
    m.set_state(compact, rest)
    m.compute()
    assert m.stats()["jcap"] > small
    m.md_run(6)
    got = m.get_state()[:2]
    m.close()
    lone = system()
    lone.set_state(compact, rest)
    lone.compute()
    lone.md_run(6)
    want = lone.get_state()[:2]
    lone.close()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
