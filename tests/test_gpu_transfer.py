"""GPU test of the host copies: array sizes around the driver's small-copy limit (64 KB), a
pinned slot (1 MB) and the threads' shares, pageable and pinned, through a gather whose
result is known exactly; the state arrays round trip; and two contexts in two threads, which
share the pinned slots."""
import threading

import numpy as np
import pytest

from helpers import small_system
from molecular_simulation_code_b200 import mixed as M
from molecular_simulation_code_b200 import nonbond as nb

pytestmark = pytest.mark.gpu

SIZES = [1, 16384, 16385, 262143, 262144, 262145, 393216, 524289, 1310721, 2621447]


def _gather(ctx, n, seed, pinned=False):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 2 ** 31, n, dtype=np.int32)
    order = rng.permutation(n).astype(np.int32)
    if pinned:
        import torch
        t = torch.empty(n, dtype=torch.int32, pin_memory=True)
        t.copy_(torch.from_numpy(a))
        a = t.numpy()
    return np.array_equal(nb.sort_posit(ctx, order + 1, a), a[order])


@pytest.mark.parametrize("n", SIZES)
def test_host_copies_sizes(ctx, n):
    assert _gather(ctx, n, n) and _gather(ctx, n, n + 1, pinned=True)


@pytest.mark.parametrize("n_gly,n_wat", [(10, 300), (100, 5000), (2000, 9000)])
def test_state_round_trip(ctx, n_gly, n_wat):
    s = small_system(10, 300)
    n = 10 * n_gly + 3 * n_wat
    rng = np.random.default_rng(n)
    # positions and velocities only pass through; any topology of n atoms will do
    import dataclasses
    reps = -(-n // s.np_atoms)
    big = dataclasses.replace(
        s, types=np.tile(s.types, reps)[:n], q=np.tile(s.q, reps)[:n],
        specbond=np.zeros((n, 12), np.int32), num3bond=np.zeros(n, np.int32),
        box=np.float32((10.0 * n) ** (1 / 3)))
    m = M.System(ctx, big, cut=6.0, skin=1.0)
    x, v = rng.uniform(-1e3, 1e3, (n, 3)), rng.normal(size=(n, 3))
    m.set_state(x, v)
    x1, v1, _ = m.get_state()
    assert np.array_equal(x1, x) and np.array_equal(v1, v)
    m.close()


def test_two_contexts_in_two_threads():
    bad = []

    def work(seed):
        with nb.Context(0) as c:
            for k, n in enumerate(SIZES[3:] * 2):
                if not _gather(c, n, 1000 * seed + k):
                    bad.append((seed, n))

    threads = [threading.Thread(target=work, args=(t,)) for t in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
