"""Device arrays at addresses that are no multiple of a float's size, as byte
buffers hold them: a box's state set from and read back to them equals that of
aligned arrays, bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

from cuco_gb300 import Box, BoxConfig, ics
from cuco_gb300.engine import MODE_FIXED, MODE_PLAIN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_FIXED])
@pytest.mark.parametrize("offset", [1, 2, 4])
def test_byte_offsets(mode, offset):
    n, L = 3001, 1000.0
    rng = np.random.default_rng(offset)
    state = [rng.uniform(0, L, (n, 3)).astype(np.float32), rng.normal(0, 50, (n, 3)).astype(np.float32)]
    box = Box(BoxConfig(n=n, pm_grid=32, cell_grid=16, boxsize=L, mass=1.0, G=ics.G_INTERNAL, softening=1.0, mode=mode))
    box.set_state(*state)
    box.forces()
    want = box.get_state()
    shifted = [torch.zeros(12 * n + 16, dtype=torch.uint8, device="cuda:0") for _ in range(4)]
    for t, a in zip(shifted, state):
        t[offset:offset + 12 * n] = torch.from_numpy(a.view(np.uint8).reshape(-1))
    torch.cuda.synchronize()
    at = [t.data_ptr() + offset for t in shifted]
    box.set_state_device(at[0], at[1])
    box.forces()
    assert box.lib.cuco_box_get_state(box.h, *[ctypes.c_void_p(a) for a in at], 1) == 0
    for t, w in zip(shifted, want):
        got = t[offset:offset + 12 * n].cpu().numpy().view(np.float32).reshape(n, 3)
        assert np.array_equal(got, w)
        assert not t[:offset].any() and not t[offset + 12 * n:].any()
    box.close()
