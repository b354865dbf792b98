"""Device-to-device buffer copies around the size up to which they are
kernels, aligned and not, with odd tails; the bytes around stay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [0, 1, 15, 16, 4097, (4 << 20) - 1, 4 << 20, (4 << 20) + 16])
@pytest.mark.parametrize("src_off,dst_off", [(0, 0), (16, 32), (3, 0), (0, 8)])
def test_copy_sizes(clops, ctx, queue, size, src_off, dst_off):
    rng = np.random.RandomState(size % 1000 + src_off)
    a = rng.randint(0, 256, size + 64).astype(np.uint8)
    b = rng.randint(0, 256, size + 64).astype(np.uint8)
    sb, db = clops.Buffer.from_array(ctx, queue, a), clops.Buffer.from_array(ctx, queue, b)
    clops.call(clops.lib.ccl_buffer_enqueue_copy, sb.h, db.h, queue.h, src_off, dst_off, size, None)
    queue.finish()
    b[dst_off:dst_off + size] = a[src_off:src_off + size]
    np.testing.assert_array_equal(db.read(queue, np.uint8, b.size), b)
    np.testing.assert_array_equal(sb.read(queue, np.uint8, a.size), a)
    sb.destroy()
    db.destroy()
