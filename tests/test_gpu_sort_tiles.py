"""The radix sort at the edges of its tile sizes (1024, 2048 and 4096 keys, one
tile, a partial last tile, the counts where the tile size changes), through
the call that may take any tile (cuco_radix_sort_noalloc), the reference-named
call whose counters limit it, and keys only; and the cell bounds' conversion
at the edges of its blocks."""
import numpy as np
import pytest

from cuco_gb300 import _native
from test_gpu_capi import dev_alloc, from_dev, to_dev

pytestmark = pytest.mark.gpu

SIZES = [1, 255, 1023, 1024, 1025, 4095, 4096, 4097, 5120, 8191, 65537, 622591, 622592, 1048576]


def keys_of(n, bits, kind):
    rng = np.random.default_rng(n + bits)
    if kind == "equal":
        return np.full(n, (1 << bits) - 1, dtype=np.uint32)
    k = rng.integers(0, 1 << bits, size=n, dtype=np.uint32)
    return np.sort(k) if kind == "sorted" else k


@pytest.mark.parametrize("kind", ["random", "equal", "sorted"])
@pytest.mark.parametrize("n", SIZES)
def test_pairs_any_tile(n, kind):
    lib = _native.load()
    bits = 18 if n % 2 else 21
    k = keys_of(n, bits, kind)
    v = np.random.default_rng(n).integers(0, 1 << 32, size=n, dtype=np.uint32)
    d_k, d_v = to_dev(lib, k), to_dev(lib, v)
    assert lib.cuco_radix_sort_noalloc(d_k, d_v, n, bits, None) == 0
    order = np.argsort(k, kind="stable")
    assert np.array_equal(from_dev(lib, d_k, n, np.uint32), k[order])
    assert np.array_equal(from_dev(lib, d_v, n, np.uint32), v[order])
    for d in (d_k, d_v):
        lib.freeArray(d)


@pytest.mark.parametrize("bits", [4, 18, 30, 32])
@pytest.mark.parametrize("n", [1025, 4097, 622593, 1245184, 1245185, 2490369, 3000001])
def test_reference_call(n, bits):
    """counters holds 32 words per 1024 keys and no more."""
    lib = _native.load()
    k = keys_of(n, bits, "random")
    nb = (n + 1023) // 1024
    guard = np.full(32 * nb + 64, 0xA5A5A5A5, dtype=np.uint32)
    v = np.arange(n, dtype=np.uint32)
    d = [to_dev(lib, k), to_dev(lib, v), dev_alloc(lib, 4 * n), dev_alloc(lib, 4 * n), to_dev(lib, guard)]
    lib.radixSort(d[0], d[1], d[2], d[3], d[4], None, None, 0, n, bits, False)
    order = np.argsort(k, kind="stable").astype(np.uint32)
    assert np.array_equal(from_dev(lib, d[0], n, np.uint32), k[order])
    assert np.array_equal(from_dev(lib, d[1], n, np.uint32), order)
    assert np.all(from_dev(lib, d[4], guard.size, np.uint32)[32 * nb:] == 0xA5A5A5A5)
    d_k = to_dev(lib, k)
    lib.radixSortKeysOnly(d_k, d[2], d[4], None, None, 0, n, bits, False)
    assert np.array_equal(from_dev(lib, d_k, n, np.uint32), k[order])
    for p in d + [d_k]:
        lib.freeArray(p)
