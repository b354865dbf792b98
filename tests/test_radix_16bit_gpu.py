"""Two-byte keys with more than three steps of 32760 keys a CTA: counters that
pass 2^15 at several steps and move to the 32-bit ones, in either half of a
word, and threads and warps whose keys are all one value; against NumPy's
sort, exactly."""
import numpy as np
import pytest

from inputs import splitmix64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [512, 513])
@pytest.mark.parametrize("kind", ["one", "ends", "mostly_one", "runs"])
@pytest.mark.parametrize("offset", [0, 1])
def test_counters_past_2_15(clops, ctx, queue, value, kind, offset):
    sms = 152
    n = max((1 << 24) + 3, 3 * 32760 * sms + 32760 * sms // 2 + 3)
    r = splitmix64(n, n) >> np.uint64(48)
    a = {"one": np.full(n, value), "ends": np.where(r < 40000, value - 512, 65023 + value - 512),
         "mostly_one": np.where(r < 3000, r, value),
         "runs": np.arange(n) // 1021 % 3 + value}[kind].astype(np.uint16)
    s = clops.Sorter(ctx, "satradix", clops.CLO_USHORT)
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
