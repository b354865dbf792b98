"""Radix sorts whose passes are planned on the device: constant digits at
every place (odd and even numbers of passes left, none at all), in place, out
of place and with values, and sizes around each tile shape's limit of one
tile per SM; against the oracle's stable sort, exactly."""
import numpy as np
import pytest

import oracle
from inputs import keys_of_type, splitmix64

pytestmark = pytest.mark.gpu

MASKS = [0, 0xFF, 0xFF00, 0xFF000000, 0xFF00FF, 0xFFFFFF, 0xFF00FF00FF00FF, 0xFF << 56,
         0xFFFFFF0000000000, (1 << 64) - 1]


def _keys(n, dt, mask):
    a = keys_of_type(3 + n, n, dt)
    fill = np.array(0x5A5A5A5A5A5A5A5A).astype(dt)
    m = np.array(mask & ((1 << (8 * a.itemsize)) - 1), dtype=np.uint64).astype(dt)
    return (a & m) | (fill & ~m)


@pytest.mark.parametrize("code,dt", [(1, np.uint8), (3, np.uint16), (5, np.uint32), (7, np.uint64)])
@pytest.mark.parametrize("mask", MASKS)
@pytest.mark.parametrize("n", [2, 5000, 200003])
def test_constant_digits(clops, ctx, queue, code, dt, mask, n):
    a = _keys(n, dt, mask)
    ref = oracle.radix_sort(a)
    s = clops.Sorter(ctx, "satradix", code)
    bi = clops.Buffer.from_array(ctx, queue, a)
    bo = clops.Buffer(ctx, a.nbytes)
    clops.wait(s.sort_device(queue, bi, n, buf_out=bo))
    np.testing.assert_array_equal(bo.read(queue, dt, n), ref)
    np.testing.assert_array_equal(bi.read(queue, dt, n), a)
    # The same in a replayed graph, in place.
    g = clops.Graph(queue)
    g.begin()
    s.sort_device(queue, bi, n)
    g.end()
    for _ in range(2):
        bi.write(queue, a)
        g.launch()
        queue.finish()
        np.testing.assert_array_equal(bi.read(queue, dt, n), ref)
    g.destroy()
    for x in (bi, bo, s):
        x.destroy()


@pytest.mark.parametrize("code,dt", [(1, np.uint8), (5, np.uint32), (7, np.uint64)])
@pytest.mark.parametrize("mask", MASKS)
def test_constant_digits_pairs(clops, ctx, queue, code, dt, mask):
    n = 70001
    k = _keys(n, dt, mask)
    v = np.arange(n, dtype=np.uint32)
    s = clops.Sorter(ctx, "satradix", code)
    kb = clops.Buffer.from_array(ctx, queue, k)
    vb = clops.Buffer.from_array(ctx, queue, v)
    clops.wait(s.sort_kv_device(queue, kb, vb, 5, n))
    rk, rv = oracle.radix_sort(k, v)
    np.testing.assert_array_equal(kb.read(queue, dt, n), rk)
    np.testing.assert_array_equal(vb.read(queue, np.uint32, n), rv)
    for x in (kb, vb, s):
        x.destroy()


# One tile per SM of each eighth of the large tile (60 keys a thread for
# 32-bit keys, 28 for (u64, u32) pairs), and one key more: 152 SMs; 640 large
# tiles of pairs, the last that look back by groups.
@pytest.mark.parametrize("kpt", [7, 15, 30, 45, 60])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_tile_shape_limits(clops, ctx, queue, kpt, extra):
    n = 152 * 256 * kpt + extra
    a = (splitmix64(kpt, n) >> np.uint64(33)).astype(np.uint32)
    s = clops.Sorter(ctx, "satradix", 5)
    b = clops.Buffer.from_array(ctx, queue, a)
    clops.wait(s.sort_device(queue, b, n))
    np.testing.assert_array_equal(b.read(queue, np.uint32, n), np.sort(a))
    b.destroy()
    s.destroy()


@pytest.mark.parametrize("n", [152 * 256 * 7 + 1, 152 * 256 * 21, 152 * 256 * 28 + 1,
                               640 * 7168, 640 * 7168 + 1])
def test_tile_shape_limits_pairs(clops, ctx, queue, n):
    k = splitmix64(9, n) & np.uint64(0xFFFF00000000FFFF)
    v = np.arange(n, dtype=np.uint32)
    s = clops.Sorter(ctx, "satradix", 7)
    kb = clops.Buffer.from_array(ctx, queue, k)
    vb = clops.Buffer.from_array(ctx, queue, v)
    clops.wait(s.sort_kv_device(queue, kb, vb, 5, n))
    order = np.argsort(k, kind="stable")
    np.testing.assert_array_equal(kb.read(queue, np.uint64, n), k[order])
    np.testing.assert_array_equal(vb.read(queue, np.uint32, n), order.astype(np.uint32))
    for x in (kb, vb, s):
        x.destroy()
