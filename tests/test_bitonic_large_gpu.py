"""The bitonic sorters' other tiles, against the network replay (bit for bit):
8-byte elements at the sizes that take tiles of 2^13 (doubles beyond 2^22,
with and without values whose order is not total, integers beyond 2^24; whole
tiles of padding one element past them); the limit of
the one-launch cluster (2^15); sbitonic at the sizes of the global passes."""
import numpy as np
import pytest

import oracle
from inputs import keys_of_type
from test_bitonic_tiles_gpu import _check, _specials

pytestmark = pytest.mark.gpu

ALL = [(0, np.int8), (1, np.uint8), (2, np.int16), (3, np.uint16), (4, np.int32), (5, np.uint32),
       (6, np.int64), (7, np.uint64), (8, np.float16), (9, np.float32), (10, np.float64)]


@pytest.mark.parametrize("code,dt,special", [
    (10, np.float64, "none"), (10, np.float64, "everywhere"), (10, np.float64, "one_tile"),
    (6, np.int64, "none"), (7, np.uint64, "none")])
@pytest.mark.parametrize("n", [(1 << 22) + 1, 1 << 23])
@pytest.mark.parametrize("offset", [0, 1])
def test_eight_byte_large_tiles(clops, ctx, queue, code, dt, special, n, offset):
    a = keys_of_type(903 + code, n, dt)
    if special == "everywhere":
        a = _specials(a)
    elif special == "one_tile":
        a[70000:75000] = _specials(a[70000:75000].copy())
    _check(clops, ctx, queue, "abitonic", code, a, offset=offset)


@pytest.mark.parametrize("code,dt", [(6, np.int64), (7, np.uint64)])
@pytest.mark.parametrize("n", [1 << 24, (1 << 24) + 1])
def test_integers_at_the_line(clops, ctx, queue, code, dt, n):
    _check(clops, ctx, queue, "abitonic", code, keys_of_type(907, n, dt), offset=n & 1)


@pytest.mark.parametrize("code,dt", [(10, np.float64), (6, np.int64)])
def test_eight_byte_large_tiles_in_place(clops, ctx, queue, code, dt):
    for n in ((1 << 22) + 1, 1 << 23):
        a = _specials(keys_of_type(904, n, dt))
        s = clops.Sorter(ctx, "abitonic", code)
        b = clops.Buffer.from_array(ctx, queue, a)
        clops.wait(s.sort_device(queue, b, n))
        np.testing.assert_array_equal(b.read(queue, np.uint64, n),
                                      oracle.bitonic_sort_threaded(a, code).view(np.uint64))
        b.destroy()
        s.destroy()


@pytest.mark.parametrize("code,dt", ALL)
@pytest.mark.parametrize("n", [(1 << 15) - 1, 1 << 15, (1 << 15) + 1])
def test_one_launch_cluster_limit(clops, ctx, queue, code, dt, n):
    a = keys_of_type(905 + n, n, dt)
    _check(clops, ctx, queue, "abitonic", code, a)
    a[-5000:] = _specials(a[-5000:].copy())
    _check(clops, ctx, queue, "sbitonic", code, a, offset=3)


@pytest.mark.parametrize("code,dt", ALL)
@pytest.mark.parametrize("n", [40001, 65536, 131075, (1 << 21) + 3])
def test_sbitonic_global_passes(clops, ctx, queue, code, dt, n):
    _check(clops, ctx, queue, "sbitonic", code, keys_of_type(906 + code, n, dt))
