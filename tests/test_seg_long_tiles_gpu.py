"""Segmented sorts on either side of the buffer size from which the
long-segment pass takes the shape's own tiles (one for every SM; smaller
buffers take quarter-size ones whatever the shape): segments at the edges of
those tiles, and of whole tiles at every 16-byte phase with the last one ending
at the buffer's end; against the oracle, exactly."""
import numpy as np
import pytest

import oracle
from inputs import keys_of_type, offsets_of
from test_segmented_gpu import EDGE_LENS, SHAPES, _seg_sort

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


# (shape, key type, its long tile, the quarter-size tile)
TILES = [(0, 5, np.uint32, 14336, 3584), (SHAPES[2], 5, np.uint32, 12288, 3584),
         (SHAPES[3], 4, np.int32, 10240, 3584), (0, 7, np.uint64, 8192, 2048),
         (SHAPES[2], 6, np.int64, 7168, 2048), (SHAPES[3], 7, np.uint64, 6144, 2048),
         (0, 1, np.uint8, 14336, 3584), (SHAPES[3], 3, np.uint16, 10240, 3584)]


@pytest.mark.parametrize("variant,code,dt,tile,small", TILES)
@pytest.mark.parametrize("own", [True, False])
def test_edges_at_the_limit(clops, ctx, queue, variant, code, dt, tile, small, own):
    edges = [17000, tile - 1, tile, tile + 1, 2 * tile - 1, 2 * tile + 1, 3 * tile] if own else \
        [5 * small - 1, 5 * small, 5 * small + 1, 8 * small - 1, 8 * small + 1]
    lens = EDGE_LENS + edges
    before, after = 5, 7
    limit = _sms() * tile
    fill = limit - sum(lens) - before - after - (0 if own else 1)
    off = offsets_of(lens[:20] + [fill] + lens[20:], start=before)
    n = int(off[-1]) + after
    assert (n >= limit) == own and abs(n - limit) <= 1
    a = keys_of_type(300 + code, n, dt)
    got = _seg_sort(clops, ctx, queue, code, a, off, options=f"segvariant={variant}")
    np.testing.assert_array_equal(got, oracle.seg_sort(a, off))
    np.testing.assert_array_equal(got[:before], a[:before])
    np.testing.assert_array_equal(got[-after:], a[-after:])


@pytest.mark.parametrize("variant,code,dt,tile,small", TILES[:6])
@pytest.mark.parametrize("own", [True, False])
def test_whole_tiles_at_every_phase_to_the_buffer_end(clops, ctx, queue, variant, code, dt, tile,
                                                      small, own):
    t = tile if own else 8 * small  # long enough for the long-segment pass
    # The filler (a multiple of 16 bytes) keeps the phases 1, 2, 3, 0 of the
    # starts after it.
    fill = (_sms() * tile - 10 * t - 4) // 4 * 4 + (4 if own else -4)
    lens = [fill, 2 * t, 1, 2 * t, 1, 3 * t, 1, t, 2 * t]
    off = offsets_of(lens, start=1)
    n = int(off[-1])
    assert (n >= _sms() * tile) == own
    a = keys_of_type(77 + code, n, dt)
    got = _seg_sort(clops, ctx, queue, code, a, off, options=f"segvariant={variant}")
    np.testing.assert_array_equal(got, oracle.seg_sort(a, off))
    np.testing.assert_array_equal(got[:1], a[:1])


@pytest.mark.parametrize("kind", ["equal", "sorted", "reverse", "distinct16"])
@pytest.mark.parametrize("code,dt,tile", [(5, np.uint32, 14336), (7, np.uint64, 8192)])
def test_low_entropy_in_the_long_tiles(clops, ctx, queue, kind, code, dt, tile):
    half = _sms() * tile // 2
    off = offsets_of([half + 3, 40000, 1, half - 5, 30000])
    a = keys_of_type(51, int(off[-1]), dt)
    if kind == "equal":
        a[:] = 0x9E3779B9
    elif kind == "distinct16":
        a = a & np.array(0xF000000F, dtype=dt)
    else:
        a = np.sort(a)[::1 if kind == "sorted" else -1].copy()
    got = _seg_sort(clops, ctx, queue, code, a, off)
    np.testing.assert_array_equal(got, oracle.seg_sort(a, off))
