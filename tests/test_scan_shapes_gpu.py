"""Scans at the edges of each launch shape (one tile of 8192, 4096-element
tiles up to 2^20 elements, 8192- and 16384-element tiles beyond), with whole
and partial warps, and arrays at 16-byte, 32-byte and no vector alignment;
against the serial scan, exactly."""
import numpy as np
import pytest

import oracle
from inputs import splitmix64

pytestmark = pytest.mark.gpu

PAIRS = [(5, np.uint32, 7, np.uint64), (5, np.uint32, 5, np.uint32), (4, np.int32, 6, np.int64),
         (1, np.uint8, 5, np.uint32), (0, np.int8, 7, np.uint64), (7, np.uint64, 7, np.uint64),
         (7, np.uint64, 1, np.uint8), (3, np.uint16, 3, np.uint16), (7, np.uint64, 5, np.uint32)]
SIZES = [1, 33, 1023, 1024, 1025, 8191, 8192, 8193, 12288, 16385, (1 << 20) - 1, (1 << 20) + 1,
         3000017]


def _scan_at(clops, ctx, queue, a, in_type, sum_type, sum_dt, off_in, off_out):
    """Scans a from byte offset off_in of one buffer to off_out of another."""
    n = a.size
    bi = clops.Buffer(ctx, a.nbytes + off_in)
    wi = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, bi.ptr + off_in, a.nbytes)
    clops.call(clops.lib.ccl_buffer_enqueue_write, wi, queue.h, 1, 0, a.nbytes, clops.np_ptr(a),
               None)
    es = np.dtype(sum_dt).itemsize
    out = np.full(n + off_out // es + 1, 99, dtype=sum_dt)
    bo = clops.Buffer.from_array(ctx, queue, out)
    wo = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, bo.ptr + off_out, n * es)
    sc = clops.Scanner(ctx, in_type, sum_type)
    clops.wait(clops.call(clops.lib.clo_scan_with_device_data, sc.h, queue.h, None, wi, wo, n, 0))
    got = bo.read(queue, sum_dt, out.size)
    assert got[-1] == 99 and np.all(got[:off_out // es] == 99)
    for w in (wi, wo):
        clops.lib.ccl_buffer_destroy(w)
    for x in (bi, bo, sc):
        x.destroy()
    return got[off_out // es:-1]


@pytest.mark.parametrize("in_type,in_dt,sum_type,sum_dt", PAIRS)
@pytest.mark.parametrize("n", SIZES)
def test_shape_edges(clops, ctx, queue, in_type, in_dt, sum_type, sum_dt, n):
    a = splitmix64(60 + n, n).astype(np.uint64).astype(in_dt)
    ref = oracle.scan(a, in_type, sum_dt)
    # Vector widths of 32 and 16 bytes, and element by element.
    for off_in, off_out in ((0, 0), (16, 32), (0, 16), (a.itemsize, 0)):
        got = _scan_at(clops, ctx, queue, a, in_type, sum_type, sum_dt, off_in, off_out)
        np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("segments", [1, 1023, 1024, 4096, 4097])
@pytest.mark.parametrize("code,dt", [(5, np.uint32), (7, np.uint64)])
def test_segment_counts_around_the_one_cta_classification(clops, ctx, queue, segments, code, dt):
    """Segments of every class (and one long enough for several tiles) by
    number: one CTA classifies up to 4096; the buffer is small enough for the
    quarter-size tiles of the long segments."""
    lens = (splitmix64(segments, segments) % np.uint64(70)).astype(np.int64)
    lens[:: max(1, segments // 7)] = 3000
    lens[0] = 30000
    lens[-1] = max(lens[-1], 9001)
    off = np.zeros(segments + 1, dtype=np.uint64)
    off[1:] = np.cumsum(lens).astype(np.uint64)
    n = int(off[-1])
    a = splitmix64(5, n).astype(dt)
    s = clops.Sorter(ctx, "satradix", code)
    b = clops.Buffer.from_array(ctx, queue, a)
    ob = clops.Buffer.from_array(ctx, queue, off)
    clops.wait(s.sort_segmented_device(queue, b, ob, segments))
    got = b.read(queue, dt, n)
    seg = np.repeat(np.arange(segments), lens)
    np.testing.assert_array_equal(got, a[np.lexsort((a, seg))])
    for x in (b, ob, s):
        x.destroy()
