"""Fills around the counts and numbers of draws from which a thread takes four
states (2^23; with 16-byte states 2^21 from 32 draws on); against the oracle's
draw loop, exactly."""
import numpy as np
import pytest

import oracle
from inputs import splitmix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,count,draws", [
    ("lcg", (1 << 23) - 4, 2), ("lcg", 1 << 23, 2), ("xorshift64", 1 << 23, 3),
    ("mwc64x", (1 << 23) + 4, 2), ("xorshift128", 1 << 21, 31), ("xorshift128", 1 << 21, 32),
    ("tauslcg", (1 << 21) - 4, 32), ("tauslcg", (1 << 21) + 4, 33), ("tauslcg", 1 << 23, 2)])
def test_fill_lines(clops, ctx, queue, name, count, draws):
    size = clops.RNG_SEED_SIZE[name]
    seeds = splitmix64(8, count * size // 8).view(np.uint8).copy()
    rng = clops.Rng(ctx, queue, name, clops.CLO_RNG_SEED_EXT_HOST, count, seeds=seeds)
    ob = clops.Buffer(ctx, draws * count * 4)
    clops.wait(clops.call(clops.lib.clo_rng_fill, rng.h, queue.h, ob.h, draws, 32, 0))
    ref, st = oracle.rng_fill(name, seeds, count, draws)
    np.testing.assert_array_equal(ob.read(queue, np.uint32, draws * count), np.asarray(ref).reshape(-1))
    np.testing.assert_array_equal(rng.states(queue), np.asarray(st).view(np.uint8).reshape(-1))
    ob.destroy()
    rng.destroy()
