"""GPU: the radix sort at the edges of its launch shapes (one block up to 4,096 and 8,192 keys, tiles of 2,048 / 4,096 / 8,192
keys, counts summed in place up to 64 tiles), against numpy's stable sort: whole numbers, exact."""
import ctypes as C

import numpy as np
import pytest

from pcisph_gb300 import RadixSort, _lib

pytestmark = pytest.mark.gpu


def _dev(a):
    torch = pytest.importorskip("torch")
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _keys(n, bits, kind):
    rng = np.random.default_rng(n + bits)
    if kind == "random":
        return rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    k = (np.arange(n, dtype=np.uint64) // 8 * 8 * (1 << bits) // n).astype(np.uint32)
    if kind == "swapped":
        i = rng.integers(0, n, max(1, n // 17))
        k[i] = k[i[::-1]]
    return k


@pytest.mark.parametrize("n", [1, 31, 33, 511, 4095, 4096, 4097, 8191, 8192, 8193, 65535, 65536, 65537, 131072, 262144,
                               262145, 524287, 524288, 524289, 600001])
@pytest.mark.parametrize("bits,kind,digit_bits", [(32, "random", 8), (13, "random", 8), (17, "swapped", 10),
                                                  (9, "sorted", 4), (21, "random", 11)])
def test_sort_shapes(n, bits, kind, digit_bits):
    torch = pytest.importorskip("torch")
    keys = _keys(n, bits, kind)
    vals = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    order = np.argsort(keys, kind="stable")
    k, v = _dev(keys), _dev(vals)
    RadixSort(0, digit_bits=digit_bits).enqueue(k, v, n, max_bits=bits)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint32), keys[order])
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])
    k, v = _dev(keys), _dev(vals)  # the same sort without allocations (and without raised shared-memory limits)
    rc = _lib.load().pcisph_radixsort_enqueue_noalloc(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n, bits, None)
    assert rc == _lib.OK
    torch.cuda.synchronize()
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint32), keys[order])
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])


def _bucket_keys(x, h, buckets):
    """The reference's bucket of each position (grid_utils.cl:9-19), whole numbers in wrapping 32-bit arithmetic."""
    c = np.floor(x / np.float32(h)).astype(np.int64).astype(np.uint32)
    with np.errstate(over="ignore"):
        k = (c[:, 0] * np.uint32(19349663)) ^ (c[:, 1] * np.uint32(73856093)) ^ (c[:, 2] * np.uint32(83492791))
        v = (k << np.uint32(6)) + (c[:, 0] & np.uint32(63)) + np.uint32(4) * (c[:, 1] & np.uint32(63)) + np.uint32(16) * (c[:, 2] & np.uint32(63))
    return (v & np.uint32(0x7FFFFFFF)) % np.uint32(buckets)


# A step sorts by the bits of its bucket count: digits narrower than the sorter's, tiles of 2,048 keys up to 65,536 particles
# where these leave room for the counts, matches instead of ballots in the first pass. From shuffled particles, and again in the
# order that the first sort left
@pytest.mark.parametrize("n", [1, 2, 127, 4096, 4097, 8192, 8193, 10241, 16384, 16385, 20000, 32768, 33000, 40000, 65535, 65536,
                               65537, 131072, 140001, 262144, 300000, 524288, 700001, 1048577])
def test_a_steps_sort(oracle, n):
    from gpu_util import fluid_like
    d = 0.02
    p = oracle.derive_params(0.5 * d, 1000.0, n, 0, 1e-3, -9.81, 0.2 * d ** 3, 0.5)
    f = fluid_like(p, spatial_order=0)
    x = (np.random.default_rng(n).random((n, 3)) * 2 * d * (n / 8) ** (1 / 3)).astype(np.float32)
    for _ in range(2):
        keys = _bucket_keys(x, p.cell_size, p.bucket_count)
        order = np.argsort(keys, kind="stable")
        f.set_fluid_state(x)
        f.run_stage("sort")
        np.testing.assert_array_equal(f.get_field("keys"), keys[order])
        np.testing.assert_array_equal(f.get_field("src"), order.astype(np.uint32))
        x = x[order]
    f.close()
