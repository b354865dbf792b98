"""Radix passes that run as resident CTAs taking tile after tile (three waves of
two tiles an SM, 152 SMs: 912 tiles) and the sizes below, with whole and partial
last tiles, constant digits (skipped passes, a copied one in place), and keys
that are not 16-byte aligned; against a stable sort, exactly."""
import numpy as np
import pytest

from inputs import splitmix64

pytestmark = pytest.mark.gpu

ALL = (1 << 64) - 1
TILE = {(4, 0): 15360, (8, 0): 10240, (4, 4): 10240, (8, 4): 7168, (8, 8): 5120, (4, 8): 7168}


def _keys(n, dt, mask):
    a = splitmix64(n, n) & np.uint64(mask)
    return a.astype(dt)


@pytest.mark.parametrize("code,dt", [(5, np.uint32), (7, np.uint64)])
@pytest.mark.parametrize("mask", [ALL, 0, 0xFFFFFF, 0xFF00FF])
@pytest.mark.parametrize("tiles,extra", [(911, 0), (911, 1), (912, 0), (2000, 12345)])
def test_keys(clops, ctx, queue, code, dt, mask, tiles, extra):
    n = tiles * TILE[np.dtype(dt).itemsize, 0] + extra
    a = _keys(n, dt, mask)
    ref = np.sort(a)
    s = clops.Sorter(ctx, "satradix", code)
    bi = clops.Buffer.from_array(ctx, queue, a)
    bo = clops.Buffer(ctx, a.nbytes)
    clops.wait(s.sort_device(queue, bi, n, buf_out=bo))
    np.testing.assert_array_equal(bo.read(queue, dt, n), ref)
    clops.wait(s.sort_device(queue, bi, n))
    np.testing.assert_array_equal(bi.read(queue, dt, n), ref)
    for x in (bi, bo, s):
        x.destroy()


@pytest.mark.parametrize("kcode,kdt,vcode,vdt", [(5, np.uint32, 5, np.uint32), (7, np.uint64, 5, np.uint32),
                                                 (7, np.uint64, 7, np.uint64), (5, np.uint32, 7, np.uint64),
                                                 (3, np.uint16, 5, np.uint32)])
@pytest.mark.parametrize("mask", [ALL, 0xFFFFFF])
@pytest.mark.parametrize("tiles,extra", [(912, 0), (1000, 77)])
def test_pairs(clops, ctx, queue, kcode, kdt, vcode, vdt, mask, tiles, extra):
    size = (max(4, np.dtype(kdt).itemsize), np.dtype(vdt).itemsize)
    n = tiles * TILE[size] + extra
    k = _keys(n, kdt, mask)
    v = np.arange(n, dtype=vdt)
    s = clops.Sorter(ctx, "satradix", kcode)
    kb = clops.Buffer.from_array(ctx, queue, k)
    vb = clops.Buffer.from_array(ctx, queue, v)
    clops.wait(s.sort_kv_device(queue, kb, vb, vcode, n))
    order = np.argsort(k, kind="stable")
    np.testing.assert_array_equal(kb.read(queue, kdt, n), k[order])
    np.testing.assert_array_equal(vb.read(queue, vdt, n), order.astype(vdt))
    for x in (kb, vb, s):
        x.destroy()


@pytest.mark.parametrize("code,dt", [(5, np.uint32), (7, np.uint64)])
@pytest.mark.parametrize("mask", [ALL, 0xFFFFFF])
def test_unaligned(clops, ctx, queue, code, dt, mask):
    """Buffers one element off: tiles loaded lane by lane, the copy by elements."""
    n = 930 * TILE[np.dtype(dt).itemsize, 0] + 5
    a = _keys(n + 1, dt, mask)
    size = a.itemsize
    s = clops.Sorter(ctx, "satradix", code)
    b = clops.Buffer.from_array(ctx, queue, a)
    w = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, b.ptr + size, n * size)
    clops.wait(clops.call(clops.lib.clo_sort_with_device_data, s.h, queue.h, None, w, w, n, 0))
    np.testing.assert_array_equal(b.read(queue, dt, n + 1),
                                  np.concatenate([a[:1], np.sort(a[1:])]))
    clops.lib.ccl_buffer_destroy(w)
    for x in (b, s):
        x.destroy()
