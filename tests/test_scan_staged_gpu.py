"""Scans around the sizes where the staged kernel takes over from the register
rows, by types and alignment, whole and partial tiles; the no-allocation scan
of the same arrays; against the serial scan, exactly."""
import ctypes as C

import numpy as np
import pytest

import oracle
from inputs import splitmix64

pytestmark = pytest.mark.gpu

M = 1 << 20
CASES = [
    (1, np.uint8, 1, np.uint8, 8 * M, 0), (3, np.uint16, 1, np.uint8, 8 * M, 0),
    (2, np.int16, 2, np.int16, 8 * M, 0), (5, np.uint32, 1, np.uint8, M, 0),
    (4, np.int32, 3, np.uint16, M, 0), (7, np.uint64, 5, np.uint32, 8 * M, 0),
    (6, np.int64, 0, np.int8, 8 * M, 0), (1, np.uint8, 7, np.uint64, 16 * M, 0),
    (2, np.int16, 6, np.int64, 16 * M, 0),
    (5, np.uint32, 7, np.uint64, M // 2, 1), (7, np.uint64, 7, np.uint64, M // 2, 1),
    (0, np.int8, 4, np.int32, M // 2, 1), (1, np.uint8, 3, np.uint16, 8192, 1),
    (7, np.uint64, 5, np.uint32, 8192, 1),
]


@pytest.mark.parametrize("it,idt,ot,odt,line,off", CASES)
@pytest.mark.parametrize("past", [0, 1, 8192 * 3 + 1000])
def test_around_the_line(clops, ctx, queue, it, idt, ot, odt, line, off, past):
    n = line + past
    a = splitmix64(n, n).astype(np.uint64).astype(idt)
    ref = oracle.scan(a, it, odt)
    es, os_ = a.itemsize, np.dtype(odt).itemsize
    bi = clops.Buffer.from_array(ctx, queue, np.concatenate([a[:off], a]))
    guard = np.full(n + off + 1, 99, dtype=odt)
    bo = clops.Buffer.from_array(ctx, queue, guard)
    wi = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, bi.ptr + off * es, a.nbytes)
    wo = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, bo.ptr + off * os_, n * os_)
    sc = clops.Scanner(ctx, it, ot)
    noalloc = clops.lib.clo_scan_blelloch_noalloc
    noalloc.restype = C.c_uint32
    noalloc.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_size_t,
                        C.POINTER(C.POINTER(clops.GError))]
    for plain in (True, False):
        bo.write(queue, guard)
        if plain:
            clops.wait(clops.call(clops.lib.clo_scan_with_device_data, sc.h, queue.h, None, wi, wo,
                                  n, 0))
        else:
            clops.call(noalloc, queue.h, it, ot, bi.ptr + off * es, bo.ptr + off * os_, n)
            queue.finish()
        got = bo.read(queue, odt, n + off + 1)
        assert got[-1] == 99 and np.all(got[:off] == 99)
        np.testing.assert_array_equal(got[off:-1], ref)
    for w in (wi, wo):
        clops.lib.ccl_buffer_destroy(w)
    for x in (bi, bo, sc):
        x.destroy()
