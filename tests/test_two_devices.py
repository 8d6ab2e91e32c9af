"""A process that uses two GPUs, on a stand-in CUDA runtime that keeps a
kernel's dynamic shared-memory limit per device, as the real one does: the
sorts and the transforms that need more than the default limit run on the
second device after the first, and on the first after a failed attempt."""
import pytest

from fake_host import run


@pytest.mark.parametrize("n", [20000, 40000])
def test_sort(tmp_path, n):
    run(tmp_path, f"""
buf = [fake.fake_alloc(4 * {n}, 0) for _ in range(2)]
cudart = ctypes.CDLL(None)
for device in (0, 1, 0):
    assert cudart.cudaSetDevice(device) == 0
    status = lib.cuco_radix_sort_noalloc(ctypes.c_void_p(buf[0]), ctypes.c_void_p(buf[1]), {n}, 18, None)
    assert status == 0, (device, lib.cuco_last_error())
""")


@pytest.mark.parametrize("M", [200, 256, 512])
def test_box(tmp_path, M):
    run(tmp_path, f"""
for device in (0, 1):
    box = Box(config(20000, {M}, device=device))
    box.set_state(np.zeros((20000, 3), np.float32))
    box.forces()
    box.sync()
    box.close()
""")


def test_ensemble(tmp_path):
    run(tmp_path, """
for device in (0, 1):
    ens = Ensemble([config(3000, 128, device=device), config(3000, 216, device=device)])
    ens.set_state(0, np.zeros((3000, 3), np.float32))
    ens.set_state(1, np.zeros((3000, 3), np.float32))
    ens.forces()
    ens.close()
""")


def test_failed_attempt_is_not_kept(tmp_path):
    run(tmp_path, """
buf = [fake.fake_alloc(4 * 20000, 0) for _ in range(2)]
sort = lambda: lib.cuco_radix_sort_noalloc(ctypes.c_void_p(buf[0]), ctypes.c_void_p(buf[1]), 20000, 18, None)
fake.fake_fail_attributes(1)
assert sort() != 0
assert sort() == 0
""")
