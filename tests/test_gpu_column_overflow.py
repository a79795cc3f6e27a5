"""GPU test of a refused list build: more than 2,048 atoms in one xy column.

Every call that needs the list is refused, the second one as the first (there is no list
to go on with), and a valid state afterwards gives what it gave before, bit for bit."""
import dataclasses

import numpy as np
import pytest

from molecular_simulation_code_b200 import mixed as M
from molecular_simulation_code_b200._lib import SOFIA_EINVAL, SofiaError
from molecular_simulation_code_b200.batch import Batch
from molecular_simulation_code_b200.system import make_system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def states():
    s = make_system(20, 780, 6)  # 2,540 atoms
    good = s.xyz.astype(np.float64)
    column = good.copy()
    column[:, :2] = 0.05 + good[:, :2] / float(s.box)  # 1 A wide, the columns are 4.3 A
    return s, good, column


def _system(ctx, s):
    m = M.System(ctx, s, cut=8.0, skin=2.0)
    m.md_setup(s, dt=1.0, gamma=0.01, seed=4, terms=0, shake=False)
    return m


def _refused(call):
    for _ in range(2):
        with pytest.raises(SofiaError) as e:
            call()
        assert e.value.code == SOFIA_EINVAL


@pytest.mark.parametrize("first", ["new", "after a list"])
def test_refused_build_leaves_no_list(ctx, states, first):
    s, good, column = states
    m = _system(ctx, s)
    m.set_state(good)
    m.compute(rebuild=True)
    want = m.get_state()[2]
    if first == "new":
        m.close()
        m = _system(ctx, s)
    m.set_state(column)
    _refused(lambda: m.compute())
    _refused(lambda: m.compute(energy=False))
    m.set_state(good)
    m.compute()
    assert np.array_equal(m.get_state()[2], want)
    m.close()


def test_refused_call_on_reference_records(ctx, states):
    s, good, column = states
    m = _system(ctx, s)
    pos = s.position_aos()
    m.forces_dropin(pos)
    want = m.forces_dropin(pos)[0]
    bad = dataclasses.replace(s, xyz=column.astype(np.float32)).position_aos()
    _refused(lambda: m.forces_dropin(bad))
    assert np.array_equal(m.forces_dropin(pos)[0], want)
    m.close()


@pytest.mark.parametrize("graph", [True, False])
def test_refused_md_segment(ctx, states, graph):
    s, good, column = states
    v = s.velocity.astype(np.float64)
    m = _system(ctx, s)
    m.set_state(good, v)
    m.md_run(5, use_graph=graph)
    want = m.get_state()[0]
    m.set_state(column, np.zeros_like(v))
    with pytest.raises(SofiaError):
        m.md_run(1, use_graph=graph)
    # the same again without a new state, the atoms still in their column
    m.set_state(column, np.zeros_like(v))
    with pytest.raises(SofiaError):
        m.compute()
    with pytest.raises(SofiaError):
        m.md_run(1, use_graph=graph)
    m.set_state(good, v)
    m.set_md_step(0)
    m.md_run(5, use_graph=graph)
    assert np.array_equal(m.get_state()[0], want)
    m.close()


def test_refused_batch_member(ctx, states):
    s, good, column = states
    v = s.velocity.astype(np.float64)
    lone = _system(ctx, s)
    lone.set_state(good, v)
    lone.md_run(5)
    want = lone.get_state()[0]
    lone.close()
    two = [_system(ctx, s), _system(ctx, s)]
    b = Batch(ctx, two)
    for m, x in zip(two, (column, good)):
        m.set_state(x, 0.0 * v)
    with pytest.raises(SofiaError):
        b.run(1)
    for m in two:
        m.set_state(good, v)
        m.set_md_step(0)
    b.run(5)
    for m in two:
        assert np.array_equal(m.get_state()[0], want)
    b.close()
    for m in two:
        m.close()
