"""The bitonic sorters at the edges of their tiles, against the network replay
(bit for bit): one CTA (2^12 elements), a cluster of eight (2^15), stages with
global passes over clusters and over one-CTA tiles, sizes that leave whole
tiles of padding, and data whose order is not total."""
import numpy as np
import pytest

import oracle
from inputs import keys_of_type

pytestmark = pytest.mark.gpu

TYPES = [(0, np.int8), (3, np.uint16), (8, np.float16), (4, np.int32), (9, np.float32),
         (7, np.uint64), (10, np.float64)]


def _bits(a):
    return a.view(f"u{a.dtype.itemsize}")


def _specials(a):
    """NaN, both zeros and infinities at every 37th place of a float array."""
    if np.issubdtype(a.dtype, np.floating):
        pat = np.array([0.0, -0.0, np.nan, np.inf, -np.inf, -0.0, 1.0, np.nan], dtype=a.dtype)
        a[::37] = np.resize(pat, a[::37].size)
    return a


def _check(clops, ctx, queue, algo, code, a, offset=0):
    """Out of place at an element offset into both buffers; the input stays."""
    es = a.dtype.itemsize
    bi = clops.Buffer.from_array(ctx, queue, np.concatenate([a[:offset], a]))
    bo = clops.Buffer(ctx, (a.size + offset + 1) * es)
    guard = np.full(a.size + offset + 1, 77, dtype=a.dtype)
    bo.write(queue, guard)
    wi = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, bi.ptr + offset * es, a.nbytes)
    wo = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, bo.ptr + offset * es, a.nbytes)
    s = clops.Sorter(ctx, algo, code)
    clops.wait(clops.call(clops.lib.clo_sort_with_device_data, s.h, queue.h, None, wi, wo,
                          a.size, 0))
    got = bo.read(queue, a.dtype, a.size + offset + 1)
    ref = oracle.bitonic_sort_threaded(a, code)
    np.testing.assert_array_equal(_bits(got[offset:-1]), _bits(ref))
    np.testing.assert_array_equal(got[:offset], guard[:offset])
    assert got[-1] == guard[-1]
    np.testing.assert_array_equal(_bits(bi.read(queue, a.dtype, a.size + offset)[offset:]),
                                  _bits(a))
    s.destroy()
    for w in (wi, wo):
        clops.lib.ccl_buffer_destroy(w)
    bi.destroy()
    bo.destroy()


@pytest.mark.parametrize("code,dt", TYPES)
@pytest.mark.parametrize("n", [31, 4095, 4096, 4097, 8200, 32767, 32769, 70001, 1 << 17])
def test_tile_edges_out_of_place(clops, ctx, queue, code, dt, n):
    a = keys_of_type(900 + n, n, dt)
    _check(clops, ctx, queue, "abitonic", code, a)
    _check(clops, ctx, queue, "sbitonic", code, _specials(a), offset=1)


# The last size of the clusters and the first beyond (2^20 or 2^19 elements
# for 8-byte types), each with whole tiles of padding.
@pytest.mark.parametrize("code,dt", [(4, np.int32), (8, np.float16), (10, np.float64)])
@pytest.mark.parametrize("n", [(1 << 19) - 40001, (1 << 19) + 1, (1 << 20) + 70001])
def test_cluster_limit(clops, ctx, queue, code, dt, n):
    a = keys_of_type(901, n, dt)
    _check(clops, ctx, queue, "abitonic", code, a)
    # Special values in one tile only.
    a[-30000:] = _specials(a[-30000:].copy())
    _check(clops, ctx, queue, "sbitonic", code, a, offset=3)


def test_two_wraps_of_one_buffer(clops, ctx, queue):
    n = 40000
    a = keys_of_type(902, n + 8, np.float32)
    b = clops.Buffer.from_array(ctx, queue, a)
    wi = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, b.ptr, n * 4)
    wo = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, b.ptr, n * 4)
    s = clops.Sorter(ctx, "abitonic", 9)
    clops.wait(clops.call(clops.lib.clo_sort_with_device_data, s.h, queue.h, None, wi, wo, n, 0))
    np.testing.assert_array_equal(b.read(queue, np.float32, n), oracle.bitonic_sort(a[:n], 9))
    s.destroy()
    for w in (wi, wo):
        clops.lib.ccl_buffer_destroy(w)
    b.destroy()
