"""The tensor-core u8 stencil against the CPU oracle where its tiles, bands and
windows can go wrong: every pair of contraction step counts, widths and
heights around the tile edges (256 bytes, 32 and 64 rows), the smallest
images, aligned, 4-byte aligned and unaligned rows, all borders, full-range
pixels, weights above 256 and the arbitrary-size path's right-border lanes.
The outputs are integers: they must be equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import device_image, device_output, read_output  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()
FIXED = (kcv.REPLICATE, kcv.REFLECT, kcv.WRAP, kcv.REVERSE)


def _check(call, oracle_call, rng, w, h, c, pad, offset, saturated):
    host = rng.integers(0, 256, (h, w * c + pad), dtype=np.uint8)
    if saturated:
        host[:] = 255
    sbuf, sptr, sstride = device_image(torch, host, offset)
    dbuf, dptr, dstride = device_output(torch, h, w * c, np.uint8, pad_elems=pad, offset=offset)
    ctx = kcv.Context.for_torch(0)
    werr, want = oracle_call(host)
    assert call(sptr, sstride, dptr, dstride, ctx) == werr
    assert ctx.synchronize() == kcv.OK
    ctx.close()
    if werr == kcv.OK:
        got, pad_ok = read_output(dbuf, h, w * c, np.uint8, dstride, offset)
        assert pad_ok
        assert np.array_equal(got, want), f"{int((got != want).sum())} bytes differ"


def _gaussian(rng, w, h, c, k, sigma, border, pad=0, offset=0, ext=False, saturated=False):
    bv = 17

    def call(sp, ss, dp, ds, ctx):
        return kcv.gaussian_blur_u8(sp, ss, dp, ds, w, h, c, k, k, sigma, sigma, border, ctx,
                                    border_value=bv if ext else None)

    _check(call, lambda host: oracle.gaussian_blur_u8(host, w, h, c, k, sigma, border, ext=ext, border_value=bv),
           rng, w, h, c, pad, offset, saturated)


# (kernel size, channels): each instantiated pair of step counts and the run-time ones.
STEPS = [(3, 1), (5, 3), (7, 3), (9, 4), (15, 1), (15, 2), (15, 3), (15, 4), (21, 1), (21, 4), (31, 1), (33, 1),
         (35, 2), (63, 3), (255, 1), (255, 4)]


@pytest.mark.parametrize("k,c", STEPS)
@pytest.mark.parametrize("edge", [-1, 0, 1])
def test_tile_edges(k, c, edge):
    rng = np.random.default_rng(1000 * k + 10 * c + edge)
    least = k // 2 + (k // 2 + 7) // 8 * 8  # the arbitrary sizes' smallest width
    w = max(512 // c + edge, least)
    for n, h in enumerate((64 + edge, 32 + edge, k - 1)):
        border = kcv.REPLICATE if k > 9 and k not in (15, 21) else FIXED[(n + edge + c) % 4]
        pad = (0, -w * c % 16, 4 - w * c % 4)[(n + edge) % 3]
        _gaussian(rng, w, max(h, k - 1), c, k, 0.3 * k, border, pad=pad, offset=(0, 4, 7)[n] if pad == 0 else 0)


@pytest.mark.parametrize("k,c,sigma", [(11, 1, 2.0), (13, 3, 9.0), (31, 3, 5.0), (31, 4, 30.0), (63, 2, 12.0)])
@pytest.mark.parametrize("border", [kcv.CONSTANT, kcv.WRAP, kcv.REVERSE])
def test_arbitrary_sizes_with_extended_borders(k, c, sigma, border):
    rng = np.random.default_rng(k + c)
    for saturated in (False, True):
        _gaussian(rng, 3 * k + 5, k + 40, c, k, sigma, border, pad=3, ext=True, saturated=saturated)


@pytest.mark.parametrize("k", [3, 5, 7, 15, 21])
def test_smallest_images_and_many_tiles(k):
    rng = np.random.default_rng(k)
    for border in FIXED:
        _gaussian(rng, k - 1, k - 1, 3, k, 1.1, border, pad=1)
    # Several tiles per CTA, whole and ragged, in both staging buffers.
    _gaussian(rng, 3001, 1100, 3, k, 1.7, kcv.REFLECT)
    _gaussian(rng, 4096, 1088, 2, k, 1.7, kcv.CONSTANT, ext=True, saturated=True)


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("taps", [([0, 1, 0, 1, 0], [0, 0, 1, 0, 0]), ([255] * 5, [255] * 5), ([3, 0, 1, 0, 9], [1, 2, 0, 0, 50])])
def test_separable_u8(c, taps):
    rng = np.random.default_rng(c)
    kx, ky = (np.array(t, np.uint8) for t in taps)
    for n, (w, h) in enumerate(((4, 4), (256 // c, 33), (700, 65))):
        for border in FIXED + (kcv.CONSTANT,):
            ext = border == kcv.CONSTANT

            def call(sp, ss, dp, ds, ctx):
                return kcv.separable_filter_2d("u8", sp, ss, dp, ds, w, h, c, taps[0], 5, taps[1], 5, border, ctx,
                                               border_value=17 if ext else None)

            _check(call, lambda host: oracle.separable_filter_2d(host, w, h, c, kx, ky, border, ext=ext,
                                                                 border_value=17),
                   rng, w, h, c, (0, 5, -w * c % 16)[n], 0, False)


@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("c", [1, 2, 3, 4])
def test_binomial(k, c):
    """Smaller images (any alignment) and larger ones on unaligned rows; the
    last is large and aligned, which stays on the tiled stencil."""
    rng = np.random.default_rng(10 * k + c)
    for n, (w, h, pad) in enumerate([(k - 1, k - 1, 0), (256 // c, 32, 0), (256 // c + 1, 33, 1), (700, 65, 3),
                                     (2049 // c, 2100, 1), (4096 // c, 1100, -(4096 // c) * c % 16)]):
        for saturated in (False, True):
            _gaussian(rng, w, h, c, k, 0.0, (FIXED + (kcv.CONSTANT,))[(n + c) % 5], pad=pad,
                      ext=(n + c) % 5 == 4, saturated=saturated)


def test_in_place_arbitrary_size_keeps_its_result():
    rng = np.random.default_rng(9)
    w, h, c, k = 300, 90, 3, 31
    host = rng.integers(0, 256, (h, w * c), dtype=np.uint8)
    img = torch.from_numpy(host).cuda()
    ctx = kcv.Context.for_torch(0)
    assert kcv.gaussian_blur_u8(img.data_ptr(), w * c, img.data_ptr(), w * c, w, h, c, k, k, 4.0, 4.0,
                                kcv.REPLICATE, ctx) == kcv.OK
    assert ctx.synchronize() == kcv.OK
    ctx.close()
    assert np.array_equal(img.cpu().numpy(), oracle.gaussian_blur_u8(host, w, h, c, k, 4.0, kcv.REPLICATE)[1])


def test_batch_runs_of_tiles():
    """A plan whose jobs hold one tile, several and more than a CTA's run, of
    every instantiation, twice (the second launch replays the graph)."""
    rng = np.random.default_rng(77)
    items, reqs = [], []
    for n, (k, c) in enumerate([s for s in STEPS if s[0] <= 15] * 3):
        w, h = ((2500 // c, 700), (20, 15), (256 // c + 1, 129))[n % 3]
        host = rng.integers(0, 256, (h, w * c + n % 5), dtype=np.uint8)
        sbuf, sptr, sstride = device_image(torch, host)
        dbuf, dptr, dstride = device_output(torch, h, w * c, np.uint8, pad_elems=n % 4)
        border = FIXED[n % 4]
        reqs.append(kcv.make_request(kcv.OP_GAUSSIAN_BLUR_U8, sptr, sstride, dptr, dstride, w, h, c, k, k, 1.4, 1.4,
                                     border_type=border))
        items.append((sbuf, dbuf, dstride, w, h, c, oracle.gaussian_blur_u8(host, w, h, c, k, 1.4, border)[1]))
    ctx = kcv.Context.for_torch(0)
    plan = kcv.BatchPlan(reqs, ctx)
    assert plan.statuses == [kcv.OK] * len(reqs)
    for _ in range(2):
        for it in items:
            it[1].fill_(0xA5)
        assert plan.launch(True) == kcv.OK
        assert ctx.synchronize() == kcv.OK
        for _, dbuf, dstride, w, h, c, want in items:
            got, pad_ok = read_output(dbuf, h, w * c, np.uint8, dstride)
            assert pad_ok and np.array_equal(got, want), (w, h, c)
    plan.close()
    ctx.close()
