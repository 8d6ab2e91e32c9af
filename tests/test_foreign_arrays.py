"""Device arrays a box's kernels must not touch themselves - another GPU's, or at
an odd address - on the stand-in CUDA runtime: every access to them is a copy;
arrays of the box's own GPU are read and written by kernels, without copies."""
import pytest

from fake_host import run


@pytest.mark.parametrize("mode", ["MODE_PLAIN", "MODE_FIXED"])
@pytest.mark.parametrize("device,odd,copied", [(0, 0, False), (1, 0, True), (0, 2, True)])
def test_set_and_get(tmp_path, mode, device, odd, copied):
    run(tmp_path, f"""
n = 1000
box = Box(config(n, 32, mode={mode}))
arrays = [fake.fake_alloc(12 * n + 4, {device}) + {odd} for _ in range(4)]
p = [ctypes.c_void_p(a) for a in arrays]
fake.fake_reset()
box.set_state_device(arrays[0], arrays[1])
assert lib.cuco_box_get_state(box.h, *p, 1) == 0
seen = [(what, int(at, 16)) for what, at in log() if int(at, 16) in arrays]
assert {{at for _, at in seen}} >= set(arrays[:2])
for what, at in seen:
    assert what.startswith("copy") == {copied}, (what, hex(at))
written = {{at for what, at in seen if what == "copy to"}}
assert written == (set(arrays) if {copied} else set())
""")
