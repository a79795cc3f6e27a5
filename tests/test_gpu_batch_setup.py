"""GPU test of a batch whose members are set up anew between two runs, without another
set_systems: the RATTLE stage and the LJ shift are part of the captured steps.  The runs
after it are those of the replicas alone, bit for bit, and members that no longer agree are
refused as set_systems refuses them."""
import numpy as np
import pytest

from molecular_simulation_code_b200 import mixed as M
from molecular_simulation_code_b200._lib import SOFIA_EINVAL, SofiaError
from molecular_simulation_code_b200.batch import Batch
from molecular_simulation_code_b200.system import make_system

pytestmark = pytest.mark.gpu


def _setup(m, s, **md):
    m.md_setup(s, dt=1.0, gamma=0.01, seed=8, **md)


def _system(ctx, s):
    m = M.System(ctx, s, cut=8.0, skin=2.0)
    m.set_state(s.xyz.astype(np.float64), s.velocity.astype(np.float64))
    _setup(m, s)
    return m


@pytest.mark.parametrize("md", [dict(rattle=True), dict(lj_shift=True),
                                dict(rattle=True, lj_shift=True)])
def test_members_set_up_between_runs(ctx, md):
    data = [make_system(6, 700, 31), make_system(12, 1100, 32)]
    want = []
    for s in data:
        m = _system(ctx, s)
        m.md_run(5)
        _setup(m, s, **md)
        e = m.md_run(5, energy_every=5)
        want.append((e,) + m.get_state()[:2])
        m.close()
    systems = [_system(ctx, s) for s in data]
    b = Batch(ctx, systems)
    b.set_segment(5)
    b.run(5)
    _setup(systems[0], data[0], **md)
    if "lj_shift" in md:  # one of two: the pair constants differ
        with pytest.raises(SofiaError) as err:
            b.run(5)
        assert err.value.code == SOFIA_EINVAL
    _setup(systems[1], data[1], **md)
    e = b.run(5, energy_every=5)
    for k, m in enumerate(systems):
        x, v, _ = m.get_state()
        assert e[k] == want[k][0], k
        assert np.array_equal(x, want[k][1]) and np.array_equal(v, want[k][2]), k
    b.close()
    for m in systems:
        m.close()
