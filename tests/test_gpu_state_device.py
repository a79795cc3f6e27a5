"""GPU test of sofia_system_set_state / get_state on device arrays: on this GPU and (where
there is one) on another, written by work still queued on the default stream and
overwritten as soon as the call returns.  Values only pass through: exact."""
import numpy as np
import pytest
import torch

from helpers import small_system
from molecular_simulation_code_b200 import mixed as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [0, 1])
def test_state_device_arrays(ctx, device):
    if device >= torch.cuda.device_count():
        pytest.skip("needs a second GPU")
    s = small_system()
    m = M.System(ctx, s, cut=6.0, skin=1.0)
    rng = np.random.default_rng(device)
    want = [rng.normal(size=(m.n, 3)) for _ in range(2)]
    with torch.cuda.device(device):
        src = [torch.from_numpy(w).cuda() for w in want]
        a = [torch.zeros_like(t) for t in src]
        torch.cuda.synchronize()
        if device == 0:
            torch.cuda._sleep(20_000_000)  # about 10 ms: the copies below are still queued
        for t, w in zip(a, src):
            t.copy_(w)
        if device != 0:
            torch.cuda.synchronize()  # the context's default stream is another GPU's
        ctx.check(ctx._lib.sofia_system_set_state(m.handle, a[0].data_ptr(), a[1].data_ptr()))
        for t in a:
            t.fill_(7.0)
        torch.cuda.synchronize()
        ctx.check(ctx._lib.sofia_system_get_state(m.handle, a[0].data_ptr(), a[1].data_ptr(),
                                                  None))
        assert all(torch.equal(t, w) for t, w in zip(a, src))
    x, v, _ = m.get_state()
    assert np.array_equal(x, want[0]) and np.array_equal(v, want[1])
    m.close()
