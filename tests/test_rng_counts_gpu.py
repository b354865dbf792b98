"""Fills whose count decides the states per thread: around the counts from
which a thread takes four, and counts and outputs that rule the vectors out;
against the oracle's draw loop, exactly."""
import numpy as np
import pytest

import oracle
from inputs import splitmix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,count", [
    ("parkmiller", (1 << 18) - 4), ("parkmiller", 1 << 18), ("parkmiller", (1 << 18) + 1),
    ("mwc64x", (1 << 21) - 4), ("mwc64x", 1 << 21), ("xorshift128", (1 << 21) + 4),
    ("lcg", (1 << 21) + 3), ("xorshift64", 257)])
@pytest.mark.parametrize("skip", [0, 1])
def test_fill_counts(clops, ctx, queue, name, count, skip):
    draws = 5
    size = clops.RNG_SEED_SIZE[name]
    seeds = splitmix64(7, count * size // 8 + 1).view(np.uint8)[:count * size].copy()
    if name == "parkmiller":
        w = seeds.view(np.uint32)
        w[:] = w % 2147483646 + 1
    rng = clops.Rng(ctx, queue, name, clops.CLO_RNG_SEED_EXT_HOST, count, seeds=seeds)
    ob = clops.Buffer(ctx, (draws * count + 1) * 4)
    wo = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, ob.ptr + 4 * skip, draws * count * 4)
    clops.wait(clops.call(clops.lib.clo_rng_fill, rng.h, queue.h, wo, draws, 32, 0))
    ref, st = oracle.rng_fill(name, seeds, count, draws)
    got = ob.read(queue, np.uint32, draws * count + 1)[skip:skip + draws * count]
    np.testing.assert_array_equal(got, np.asarray(ref).reshape(-1))
    np.testing.assert_array_equal(rng.states(queue), np.asarray(st).view(np.uint8).reshape(-1))
    clops.lib.ccl_buffer_destroy(wo)
    ob.destroy()
    rng.destroy()
