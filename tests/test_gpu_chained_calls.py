"""Calls that follow one another without synchronisation, each reading what the
call before it has just written and writing what an earlier one read, against
the same chain on the CPU oracle.  The images are small, so that the grids of
several calls are resident together (programmatic dependent launch).  Integers:
the outputs must be equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import pyr_sizes  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()
LENGTHS = (1, 2, 3, 4, 5, 8)


def _gauss(k, sigma, border):
    def call(src, dst, w, h, c, ctx):
        return kcv.gaussian_blur_u8(kcv.ptr(src), kcv.stride(src), kcv.ptr(dst), kcv.stride(dst), w, h, c, k, k,
                                    sigma, sigma, border, ctx)

    return call, lambda img, w, h, c: oracle.gaussian_blur_u8(img, w, h, c, k, sigma, border)[1]


def _sep(dtype, kx, ky):
    def call(src, dst, w, h, c, ctx):
        return kcv.separable_filter_2d(dtype, kcv.ptr(src), kcv.stride(src), kcv.ptr(dst), kcv.stride(dst), w, h, c,
                                       kx, 5, ky, 5, kcv.WRAP, ctx)

    dt = {"u8": np.uint8, "u16": np.uint16, "s16": np.int16}[dtype]
    return call, lambda img, w, h, c: oracle.separable_filter_2d(img, w, h, c, np.array(kx, dt), np.array(ky, dt),
                                                                 kcv.WRAP)[1]


def _median(dtype, k):
    def call(src, dst, w, h, c, ctx):
        return kcv.median_blur(dtype, kcv.ptr(src), kcv.stride(src), kcv.ptr(dst), kcv.stride(dst), w, h, c, k, k,
                               kcv.WRAP, ctx)

    return call, lambda img, w, h, c: oracle.median_blur(img, w, h, c, k, kcv.WRAP)


# Shifts (one unit tap per axis) keep every element, so that a stale one stays visible.
SHIFT = ([0, 0, 0, 1, 0], [1, 0, 0, 0, 0])
CHAINS = {
    "binomial5_unaligned": (_gauss(5, 0.0, kcv.REFLECT), "u8", 61, 37, 1),
    "binomial5_aligned": (_gauss(5, 0.0, kcv.REFLECT), "u8", 64, 50, 1),
    "binomial9_unaligned": (_gauss(9, 0.0, kcv.WRAP), "u8", 131, 75, 1),
    "generated7_unaligned": (_gauss(7, 0.6, kcv.REVERSE), "u8", 67, 90, 3),
    "generated7_rgba": (_gauss(7, 0.6, kcv.REVERSE), "u8", 67, 90, 4),
    "arbitrary31": (_gauss(31, 1.1, kcv.REPLICATE), "u8", 333, 70, 1),
    "u8_shift": (_sep("u8", *SHIFT), "u8", 75, 61, 3),
    "u16_shift_unaligned": (_sep("u16", *SHIFT), "u16", 253, 77, 1),
    "u16_shift_aligned": (_sep("u16", *SHIFT), "u16", 256, 77, 1),
    "s16_shift_unaligned": (_sep("s16", *SHIFT), "s16", 253, 77, 1),
    "s16_shift_3_channels": (_sep("s16", *SHIFT), "s16", 85, 40, 3),
    "median3": (_median("u8", 3), "u8", 61, 53, 3),
    "median5": (_median("u8", 5), "u8", 131, 53, 1),
    "median7_u16": (_median("u16", 7), "u16", 75, 41, 1),
    "median9": (_median("u8", 9), "u8", 61, 33, 1),
}


def _random(rng, dtype, h, row):
    info = np.iinfo(dtype)
    return rng.integers(info.min, int(info.max) + 1, (h, row), dtype=dtype)


def _upload(host):
    return torch.from_numpy(host.view(np.int16) if host.dtype == np.uint16 else host).cuda()


@pytest.mark.parametrize("name", sorted(CHAINS))
def test_ping_pong(name):
    (call, want), dtype, w, h, c = CHAINS[name]
    dt = {"u8": np.uint8, "u16": np.uint16, "s16": np.int16}[dtype]
    rng = np.random.default_rng(len(name))
    ctx = kcv.Context.for_torch(0)
    hosts = [_random(rng, dt, h, w * c) for _ in range(6)]
    sources = [_upload(x) for x in hosts]
    pair = [torch.zeros_like(sources[0]) for _ in range(2)]
    results = []
    for n in LENGTHS:
        for src in sources:
            pair[0].copy_(src)
            for i in range(n):
                assert call(pair[i % 2], pair[(i + 1) % 2], w, h, c, ctx) == kcv.OK
            results.append(pair[n % 2].clone())
    assert ctx.synchronize() == kcv.OK
    chains = [[x] for x in hosts]
    for chain in chains:
        for _ in range(LENGTHS[-1]):
            chain.append(want(chain[-1], w, h, c).reshape(h, w * c))
    for k, got in enumerate(results):
        n, i = LENGTHS[k // len(sources)], k % len(sources)
        assert np.array_equal(got.cpu().numpy().view(dt), chains[i][n]), (n, i)
    ctx.close()


@pytest.mark.parametrize("c", [1, 3])
def test_pyramid_and_derivatives_of_a_changing_image(c):
    """Pyramids into the same level buffers and derivatives of an image that a
    Gaussian rewrites between them."""
    rng = np.random.default_rng(c)
    w, h, levels = 173, 121, 4
    sizes = pyr_sizes(w, h, levels)
    ctx = kcv.Context.for_torch(0)
    host = _random(rng, np.uint8, h, w * c)
    outs = [torch.zeros((oh, ow * c), dtype=torch.uint8, device="cuda") for ow, oh in sizes]
    dx = torch.zeros((h, w * c), dtype=torch.int16, device="cuda")
    source = _upload(host)
    pair = [torch.zeros_like(source) for _ in range(2)]
    blur, blur_want = _gauss(3, 0.6, kcv.REFLECT)
    rounds = []
    for n in (1, 2, 3, 6, 7):
        pair[0].copy_(source)
        for i in range(n):
            a, b = pair[i % 2], pair[(i + 1) % 2]
            assert blur(a, b, w, h, c, ctx) == kcv.OK
            assert kcv.build_pyramid_u8(kcv.ptr(b), kcv.stride(b), w, h, c, [kcv.ptr(o) for o in outs],
                                        [kcv.stride(o) for o in outs], kcv.REVERSE, ctx) == kcv.OK
            assert kcv.sobel_3x3_horizontal_s16_u8(kcv.ptr(b), kcv.stride(b), kcv.ptr(dx), kcv.stride(dx), w, h, c,
                                                   ctx) == kcv.OK
        rounds.append((n, [o.clone() for o in outs], dx.clone()))
    assert ctx.synchronize() == kcv.OK
    blurred = [host]
    for _ in range(7):
        blurred.append(blur_want(blurred[-1], w, h, c).reshape(h, w * c))
    for n, got_levels, got_dx in rounds:
        img, iw, ih = blurred[n], w, h
        for (ow, oh), got in zip(sizes, got_levels):
            img = oracle.blur_and_downsample_u8(img, iw, ih, c, kcv.REVERSE)[1]
            iw, ih = ow, oh
            assert np.array_equal(got.cpu().numpy(), img), (n, ow)
        want_dx = oracle.sobel_3x3_s16_u8(blurred[n], w, h, c, True)[1]
        assert np.array_equal(got_dx.cpu().numpy(), want_dx[:, : w * c]), n
    ctx.close()
