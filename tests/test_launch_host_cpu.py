"""Which kernels the library's calls launch, over a CUDA runtime that launches
nothing."""
import ctypes as C

import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.load(tmp_path_factory.mktemp("fake"))


def _names(fake, call):
    fake.lib.fake_reset(0)
    call()
    return [x[0] for x in fake_cuda.launches(fake)]


# Sums of one or two bytes or narrower than the input, 8-byte sums of one or
# two bytes and unaligned arrays leave the register rows where those are slow
# (some of them took twice the time there).
U8, U16, U32, U64 = 1, 3, 5, 7
M = 1 << 20


@pytest.mark.parametrize("i,o,offset,n,staged", [
    (U32, U64, 0, 1 << 28, False), (U32, U32, 0, 1 << 28, False), (U64, U64, 0, 1 << 28, False),
    (U8, U32, 0, 1 << 28, False), (U16, U32, 0, 1 << 28, False),
    (U8, U8, 0, 8 * M, False), (U8, U8, 0, 8 * M + 1, True), (U16, U16, 0, 1 << 28, True),
    (U32, U8, 0, M, False), (U32, U16, 0, M + 1, True), (U64, U32, 0, 1 << 26, True),
    (U8, U64, 0, 16 * M, False), (U8, U64, 0, 16 * M + 1, True), (U16, U64, 0, 1 << 28, True),
    (U32, U64, 8, M // 2, False), (U32, U64, 8, M // 2 + 1, True), (U8, U32, 4, 1 << 26, True),
    (U64, U32, 8, 5000, True), (U64, U64, 16, 1 << 26, False),
])
def test_scan_route(fake, i, o, offset, n, staged):
    ctx = fake.Context(0)
    q = fake.Queue(ctx)
    sc = fake.Scanner(ctx, i, o)
    wrap = lambda at: fake.call(fake.lib.ccl_buffer_new_wrap, ctx.h, at, 8 * n)
    a, b = wrap(1 << 40), wrap((1 << 41) + offset)
    names = _names(fake, lambda: fake.call(fake.lib.clo_scan_with_device_data, sc.h, q.h, None, a,
                                           b, n, 0))
    scans = [x for x in names if "clear" not in x]
    assert len(scans) == 1 and ("scan_staged" in scans[0]) == staged, names
    for x in (a, b):
        fake.lib.ccl_buffer_destroy(x)
    for x in (sc, q, ctx):
        x.destroy()


# The per-kernel timing names kernels by the sorter that was called, whichever
# kernels it takes.
@pytest.mark.parametrize("algo,code,n,names", [
    ("satradix", U32, 1000, {"satradix_tile_sort": 1}),
    ("satradix", U64, 1 << 16, {"satradix_tile_sort": 1, "satradix_global_steps": 5,
                                "satradix_tile_finish": 5}),
    ("satradix", U32, 1 << 20, {"satradix_upsweep": 1, "satradix_onesweep": 4}),
    ("sbitonic", U32, 1000, {"sbitonic_tile_sort": 1}),
    ("sbitonic", U32, 1 << 13, {"sbitonic_tile_sort": 1}),
    ("abitonic", U32, 1 << 16, {"abitonic_tile_sort": 1, "abitonic_global_steps": 4,
                                "abitonic_tile_finish": 4}),
])
def test_timing_names(fake, algo, code, n, names):
    ctx = fake.Context(0)
    q = fake.Queue(ctx)
    s = fake.Sorter(ctx, algo, code)
    a, b = fake.Buffer(ctx, 8 * n), fake.Buffer(ctx, 8 * n)
    fake.lib.clo_gb300_timing_enable(1)
    fake.lib.clo_gb300_timing_reset()
    s.sort_device(q, a, n, buf_out=b)
    got = {f"{x}_{k}": fake.kernel_timing(f"{x}_{k}")[2]
           for x in ("satradix", "sbitonic", "abitonic")
           for k in ("tile_sort", "global_steps", "tile_finish", "upsweep", "onesweep")}
    fake.lib.clo_gb300_timing_enable(0)
    assert {k: v for k, v in got.items() if v} == names
    for x in (s, a, b, q, ctx):
        x.destroy()


# The radix sort's launcher refuses what its passes would corrupt: values with
# the keys going to another buffer, odd numbers of passes in place.
@pytest.mark.parametrize("n", [5000, 100000, 1 << 24])
@pytest.mark.parametrize("src,dst,vb,bits,ok", [
    (0, 0, 4, 32, True), (0, 1, 0, 32, True), (0, 1, 0, 24, True), (0, 0, 0, 8, True),
    (0, 0, 8, 64, True), (0, 1, 4, 32, False), (0, 1, 8, 16, False), (0, 0, 0, 24, False),
    (0, 0, 4, 40, False), (0, 0.5, 0, 24, False)])
def test_radix_sort_refusals(fake, n, src, dst, vb, bits, ok):
    ctx = fake.Context(0)
    q = fake.Queue(ctx)
    f = fake.lib["_ZN3clo10radix_sortEPKvPvS2_miiiP11ccl_contextP11CUstream_stPP7_GError"]
    f.restype = C.c_int
    f.argtypes = [C.c_void_p] * 3 + [C.c_size_t] + [C.c_int] * 3 + [C.c_void_p] * 3
    at = lambda x: int(1 << 40) + int(x * 8 * n) // 8 * 8
    e = fake.err_ptr()
    fake.lib.fake_reset(0)
    # (The host memory that stands for the buffers is never touched.)
    r = f(at(src), at(dst), (1 << 41) if vb else None, n, 8, vb, bits, ctx.h, None, C.addressof(e))
    assert (r == 0) == ok and bool(e) != ok
    if ok:
        assert fake.lib.fake_launches() > 0
    else:
        assert fake.lib.fake_launches() == 0 and e.contents.code == fake.CLO_ERROR_ARGS
        fake.lib.clo_error_free(e)
    q.destroy()
    ctx.destroy()


# Sorts of one tile an SM (one-word keys; 4.2 tiles with more) look back by
# groups, whatever the number of SMs. (The last number in the kernel's name is
# how it takes its tiles: 1 by groups.)
@pytest.mark.parametrize("sms", [148, 152, 160])
@pytest.mark.parametrize("values,tile,fifths", [(0, 15360, 5), (U32, 10240, 21)])
def test_grouped_lookback_limit(fake, sms, values, tile, fifths):
    fake.lib.fake_set_sms(sms)
    ctx = fake.Context(0)
    fake.lib.fake_set_sms(152)
    q = fake.Queue(ctx)
    s = fake.Sorter(ctx, "satradix", U32)
    limit = sms * fifths // 5 * tile
    a, b = fake.Buffer(ctx, 4 * limit + 4), fake.Buffer(ctx, 4 * limit + 4)
    for n, grouped in ((limit, True), (limit + 1, False)):
        names = _names(fake, (lambda: s.sort_kv_device(q, a, b, values, n)) if values else
                       (lambda: s.sort_device(q, a, n, buf_out=b)))
        passes = [x for x in names if "radix_pass_tiles" in x]
        assert len(passes) == 4
        assert all(("ELi1EEE" in x) == grouped for x in passes), (n, passes[0])
    for x in (s, a, b, q, ctx):
        x.destroy()
