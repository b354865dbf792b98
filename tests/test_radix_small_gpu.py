"""Radix sorts in one CTA and in one cluster, and one-byte keys by their
histogram: sizes around each limit (4096 and 8192 keys, 16384 with values) and
at uneven slices, constant digits, keys narrower than their elements; against
the oracle's stable sort, exactly."""
import numpy as np
import pytest

import oracle
from inputs import keys_of_type, splitmix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kcode,kdt", [(1, np.uint8), (3, np.uint16), (5, np.uint32), (7, np.uint64)])
@pytest.mark.parametrize("vcode,vdt", [(5, np.uint32), (7, np.uint64)])
@pytest.mark.parametrize("n", [2, 511, 513, 4095, 4096, 4097, 8192, 8193, 12289, 16383, 16384, 16385])
@pytest.mark.parametrize("mask", [(1 << 64) - 1, 0xFF00FF, 0])
def test_small_pairs(clops, ctx, queue, kcode, kdt, vcode, vdt, n, mask):
    bits = 8 * np.dtype(kdt).itemsize
    k = keys_of_type(n, n, kdt) & np.array(mask & ((1 << bits) - 1), dtype=np.uint64).astype(kdt)
    v = np.arange(n).astype(vdt)
    s = clops.Sorter(ctx, "satradix", kcode)
    kb = clops.Buffer.from_array(ctx, queue, k)
    vb = clops.Buffer.from_array(ctx, queue, v)
    clops.wait(s.sort_kv_device(queue, kb, vb, vcode, n))
    rk, rv = oracle.radix_sort(k, v)
    np.testing.assert_array_equal(kb.read(queue, kdt, n), rk)
    np.testing.assert_array_equal(vb.read(queue, vdt, n), rv)
    for x in (kb, vb, s):
        x.destroy()


# Keys of the low half of the element: the other bits travel with it, so the
# order of equal keys shows.
@pytest.mark.parametrize("ecode,edt,kcode", [(5, np.uint32, 3), (7, np.uint64, 5), (7, np.uint64, 1),
                                             (3, np.uint16, 1)])
@pytest.mark.parametrize("n", [1000, 4097, 9000, 16385, 40000])
def test_small_partial_keys(clops, ctx, queue, ecode, edt, kcode, n):
    a = keys_of_type(n + ecode, n, edt)
    s = clops.Sorter(ctx, "satradix", ecode, key_type=kcode)
    bi = clops.Buffer.from_array(ctx, queue, a)
    bo = clops.Buffer(ctx, a.nbytes)
    clops.wait(s.sort_device(queue, bi, n, buf_out=bo))
    low = a & np.array((1 << (8 * {1: 1, 3: 2, 5: 4}[kcode])) - 1, dtype=edt)
    np.testing.assert_array_equal(bo.read(queue, edt, n), a[np.argsort(low, kind="stable")])
    for x in (bi, bo, s):
        x.destroy()


@pytest.mark.parametrize("code,dt", [(1, np.uint8), (0, np.int8)])
@pytest.mark.parametrize("n", [8193, 100001, (1 << 22) + 5])
@pytest.mark.parametrize("kind", ["uniform", "one", "two"])
@pytest.mark.parametrize("offset", [0, 3])
def test_bytes(clops, ctx, queue, code, dt, n, kind, offset):
    a = (splitmix64(n, n) >> np.uint64(56)).astype(np.uint8)
    if kind != "uniform":
        a = np.where(a < (256 if kind == "one" else 200), 255 if kind == "one" else 7, 0).astype(np.uint8)
    s = clops.Sorter(ctx, "satradix", code)
    b = clops.Buffer(ctx, n + offset + 1)
    b.write(queue, np.concatenate([np.full(offset, 9, np.uint8), a, [9]]).astype(np.uint8))
    w = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, b.ptr + offset, n)
    clops.wait(clops.call(clops.lib.clo_sort_with_device_data, s.h, queue.h, None, w, None, n, 0))
    got = b.read(queue, np.uint8, n + offset + 1)
    np.testing.assert_array_equal(got[offset:-1], np.sort(a))
    assert got[-1] == 9 and np.all(got[:offset] == 9)
    clops.lib.ccl_buffer_destroy(w)
    b.destroy()
    s.destroy()


@pytest.mark.parametrize("code,dt", [(3, np.uint16), (2, np.int16)])
@pytest.mark.parametrize("n", [(5 << 18) - 1, 5 << 18, (5 << 18) + 77, 5 * (1 << 20) + 3])
@pytest.mark.parametrize("kind", ["uniform", "one", "ends", "mostly_one", "spread"])
@pytest.mark.parametrize("offset", [0, 1])
def test_two_byte_keys(clops, ctx, queue, code, dt, n, kind, offset):
    """From 5 x 2^18 two-byte keys the output comes from the 65536-bin histogram:
    counters that pass 2^15 and 2^16 in one CTA, runs of empty bins, bins of
    one key."""
    r = splitmix64(n, n) >> np.uint64(48)
    a = {"uniform": r, "one": np.full(n, 0xFFFF), "ends": np.where(r < 40000, 0, 0xFFFF),
         "mostly_one": np.where(np.arange(n) < 65536, np.arange(n), 513),
         "spread": np.arange(n) % 65536}[kind].astype(np.uint16)
    s = clops.Sorter(ctx, "satradix", code)
    b = clops.Buffer(ctx, 2 * (n + offset + 1))
    b.write(queue, np.concatenate([np.full(offset, 9), a, [9]]).astype(np.uint16))
    w = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, b.ptr + 2 * offset, 2 * n)
    clops.wait(clops.call(clops.lib.clo_sort_with_device_data, s.h, queue.h, None, w, None, n, 0))
    got = b.read(queue, np.uint16, n + offset + 1)
    np.testing.assert_array_equal(got[offset:-1], np.sort(a))
    assert got[-1] == 9 and np.all(got[:offset] == 9)
    clops.lib.ccl_buffer_destroy(w)
    b.destroy()
    s.destroy()


@pytest.mark.parametrize("code,dt,n", [(5, np.uint32, 50000), (5, np.uint32, 1 << 17),
                                       (4, np.int32, (1 << 17) + 1), (7, np.uint64, (1 << 18) - 3),
                                       (7, np.uint64, (1 << 18) + 1)])
def test_whole_keys_around_the_bitonic_limit(clops, ctx, queue, code, dt, n):
    a = keys_of_type(n, n, dt)
    s = clops.Sorter(ctx, "satradix", code)
    bi = clops.Buffer.from_array(ctx, queue, a)
    bo = clops.Buffer(ctx, a.nbytes)
    clops.wait(s.sort_device(queue, bi, n, buf_out=bo))
    np.testing.assert_array_equal(bo.read(queue, dt, n), oracle.radix_sort(a))
    np.testing.assert_array_equal(bi.read(queue, dt, n), a)
    for x in (bi, bo, s):
        x.destroy()
