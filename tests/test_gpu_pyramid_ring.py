"""blur_and_downsample_u8 and pyramids where the ring of staged rows can go
wrong, against the CPU oracle: heights around multiples of the ring's groups
(4 source rows), of the ring (16) and of a band (32 destination rows), widths
around a strip, aligned and unaligned rows, every border, 1 to 4 channels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import device_image, device_output, pyr_sizes, read_output  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()
BORDERS = (kcv.REPLICATE, kcv.REFLECT, kcv.WRAP, kcv.REVERSE, kcv.CONSTANT)


@pytest.mark.parametrize("c", [1, 2, 3, 4])
@pytest.mark.parametrize("h", [4, 5, 7, 16, 17, 35, 63, 64, 66, 131, 2500])
def test_heights(c, h):
    rng = np.random.default_rng(10 * h + c)
    ctx = kcv.Context.for_torch(0)
    for n, w in enumerate((4, 256 // c + 1, 520) if h < 1000 else (41,)):
        for pad, offset in ((-w * c % 16, 0), (1, 3)):
            border = BORDERS[(n + h + pad) % 5]
            ext = border == kcv.CONSTANT
            host = rng.integers(0, 256, (h, w * c + pad), dtype=np.uint8)
            sbuf, sptr, sstride = device_image(torch, host, offset)
            ow, oh = (w + 1) // 2, (h + 1) // 2
            dbuf, dptr, dstride = device_output(torch, oh, ow * c, np.uint8, pad_elems=pad, offset=offset)
            assert kcv.blur_and_downsample_u8(sptr, sstride, w, h, dptr, dstride, c, border, ctx,
                                              border_value=9 if ext else None) == kcv.OK
            assert ctx.synchronize() == kcv.OK
            want = oracle.blur_and_downsample_u8(host, w, h, c, border, ext=ext, border_value=9)[1]
            got, pad_ok = read_output(dbuf, oh, ow * c, np.uint8, dstride, offset)
            assert pad_ok and np.array_equal(got, want), (w, pad)
    ctx.close()


def test_levels_follow_each_other():
    """Every level reads the one before it, launched right behind it: repeated
    builds of changing images."""
    rng = np.random.default_rng(3)
    w, h, c, levels = 1201, 903, 3, 7
    sizes = pyr_sizes(w, h, levels)
    ctx = kcv.Context.for_torch(0)
    outs = [torch.zeros((oh, ow * c), dtype=torch.uint8, device="cuda") for ow, oh in sizes]
    for _ in range(5):
        host = rng.integers(0, 256, (h, w * c), dtype=np.uint8)
        src = torch.from_numpy(host).cuda()
        assert kcv.build_pyramid_u8(kcv.ptr(src), kcv.stride(src), w, h, c, [kcv.ptr(o) for o in outs],
                                    [kcv.stride(o) for o in outs], kcv.REVERSE, ctx) == kcv.OK
        assert ctx.synchronize() == kcv.OK
        img, iw, ih = host, w, h
        for (ow, oh), out in zip(sizes, outs):
            img = oracle.blur_and_downsample_u8(img, iw, ih, c, kcv.REVERSE)[1]
            iw, ih = ow, oh
            assert np.array_equal(out.cpu().numpy(), img), (ow, oh)
    ctx.close()
