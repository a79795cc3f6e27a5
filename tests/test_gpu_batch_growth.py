"""GPU test of a batch whose membership crosses the row-split rule: 4, 2 and 1 warps per list
row in either precision, growing and shrinking, so that graphs of every split are captured
and taken again.  Every replica follows its lone trajectory and energies, bit for bit."""
import numpy as np
import pytest

from molecular_simulation_code_b200 import mixed as M
from molecular_simulation_code_b200.batch import Batch
from molecular_simulation_code_b200.system import make_system

pytestmark = pytest.mark.gpu

# mixed: 4 warps per row to about 9,100 atoms, 2 to 36,500; FP64: to 4,500 and 9,100
SIZES = [(20, 640), (30, 1000), (60, 5200), (80, 5600)]
RUNS = [[0], [0, 1], [0, 1, 2], [0, 1, 2, 3], [0], [1, 2], [0, 1, 2, 3], [1]]
STEPS = 4


@pytest.fixture(scope="module")
def replicas():
    return [make_system(g, w, 40 + g) for g, w in SIZES]


def _system(ctx, s, k, precision):
    m = M.System(ctx, s, cut=8.0, skin=2.0, precision=precision)
    m.set_state(s.xyz.astype(np.float64), s.velocity.astype(np.float64))
    m.md_setup(s, dt=1.0, gamma=0.01, seed=60 + k)
    return m


@pytest.mark.parametrize("precision", [M.MIXED, M.FP64])
def test_growing_batch_equals_alone(ctx, replicas, precision):
    want = []
    for k, s in enumerate(replicas):
        m = _system(ctx, s, k, precision)
        e = [m.md_run(STEPS, energy_every=STEPS) for r in RUNS if k in r]
        want.append((e,) + m.get_state()[:2])
        m.close()
    systems = [_system(ctx, s, k, precision) for k, s in enumerate(replicas)]
    got = [[] for _ in systems]
    b = None
    for r in RUNS:
        members = [systems[k] for k in r]
        if b is None:
            b = Batch(ctx, members)
            b.set_segment(STEPS)
        else:
            b.set_systems(members)
        for k, e in zip(r, b.run(STEPS, energy_every=STEPS)):
            got[k].append(e)
    for k, m in enumerate(systems):
        x, v, _ = m.get_state()
        assert np.array_equal(x, want[k][1]) and np.array_equal(v, want[k][2]), k
        assert got[k] == want[k][0], k
    b.close()
    for m in systems:
        m.close()
