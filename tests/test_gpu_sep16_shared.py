"""16-bit filters whose unaligned source and destination lie in one buffer,
against the CPU oracle.  Images that share no byte need no copy of the source,
so they take nothing from the pool."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import device_image  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()
TAPS = {"u16": ([0, 1, 2, 1, 0], [3, 0, 3, 0, 1]), "s16": ([-1, -2, 0, 2, 1], [1, 4, 6, 4, 1])}


def _call(dtype, src, src_stride, dst, dst_stride, w, h, ctx):
    kx, ky = TAPS[dtype]
    return kcv.separable_filter_2d(dtype, src, src_stride, dst, dst_stride, w, h, 1, kx, 5, ky, 5, kcv.REFLECT, ctx)


def _want(dtype, host, w, h):
    kx, ky = TAPS[dtype]
    dt = np.dtype("uint16" if dtype == "u16" else "int16")
    return oracle.separable_filter_2d(np.ascontiguousarray(host), w, h, 1, np.array(kx, dt), np.array(ky, dt),
                                      kcv.REFLECT)[1]


def _arbitrary(ctx):
    """A call that takes pool memory (or the injected failure of taking some)."""
    img = torch.zeros((64, 64), dtype=torch.uint8, device="cuda")
    out = torch.zeros_like(img)
    err = kcv.gaussian_blur_u8(img.data_ptr(), 64, out.data_ptr(), 64, 64, 64, 1, 31, 31, 0.0, 0.0, kcv.REPLICATE, ctx)
    assert ctx.synchronize() == kcv.OK
    return err


# name -> rows of the buffer per image row, then for source and destination:
# first buffer row, rows between rows, right of the other image or not.
LAYOUTS = {
    "side_by_side": (1, (0, 1, False), (0, 1, True)),
    "destination_first": (1, (0, 1, True), (0, 1, False)),
    "row_by_row": (2, (0, 2, False), (1, 2, False)),
    "different_strides": (4, (0, 2, False), (1, 4, False)),
    "overlapping_columns_other_rows": (2, (1, 2, True), (0, 2, False)),
}


@pytest.mark.parametrize("dtype", ["u16", "s16"])
@pytest.mark.parametrize("w,h", [(151, 47), (1023, 521)])
@pytest.mark.parametrize("layout", sorted(LAYOUTS))
def test_images_that_share_no_byte(dtype, w, h, layout):
    rng = np.random.default_rng(w + len(layout))
    dt = np.dtype("uint16" if dtype == "u16" else "int16")
    info = np.iinfo(dt)
    rows_per, *places = LAYOUTS[layout]
    pitch = 2 * w + 7
    host = rng.integers(info.min, int(info.max) + 1, (rows_per * h, pitch), dtype=dt)
    buf, base, stride = device_image(torch, host, 2)
    (s0, sstep, sright), (d0, dstep, dright) = places

    def view(first, step, right):
        x = w + 3 if right else 1
        return host[first:first + (h - 1) * step + 1:step, x:x + w], base + first * stride + 2 * x, step * stride

    source, sptr, sstride = view(s0, sstep, sright)
    dest, dptr, dstride = view(d0, dstep, dright)
    want = _want(dtype, source, w, h)
    ctx = kcv.Context.for_torch(0)
    ctx.fail_next_allocations(1)
    assert _call(dtype, sptr, sstride, dptr, dstride, w, h, ctx) == kcv.OK
    assert ctx.synchronize() == kcv.OK
    dest[:] = want  # and nothing else of the buffer changes
    got = buf.cpu().numpy()[2:2 + host.nbytes].view(dt).reshape(host.shape)
    assert np.array_equal(got, host), int((got != host).sum())
    assert _arbitrary(ctx) == kcv.ALLOCATION  # the failure is still to come
    ctx.close()


@pytest.mark.parametrize("dtype", ["u16", "s16"])
@pytest.mark.parametrize("w,h", [(151, 47), (1023, 521)])
def test_in_place_without_room_is_refused(dtype, w, h):
    """A call in place needs a copy of its source: without one it is refused and
    the image stays as it is."""
    rng = np.random.default_rng(w)
    dt = np.dtype("uint16" if dtype == "u16" else "int16")
    info = np.iinfo(dt)
    host = rng.integers(info.min, int(info.max) + 1, (h, w), dtype=dt)
    buf, ptr, stride = device_image(torch, host, 2)

    def image():
        return buf.cpu().numpy()[2:2 + host.nbytes].view(dt).reshape(h, w)

    capped = kcv.Context(0, torch.cuda.current_stream().cuda_stream, pool_limit=1024)
    assert _call(dtype, ptr, stride, ptr, stride, w, h, capped) == kcv.ALLOCATION
    assert capped.synchronize() == kcv.OK
    capped.close()
    ctx = kcv.Context.for_torch(0)
    ctx.fail_next_allocations(1)
    assert _call(dtype, ptr, stride, ptr, stride, w, h, ctx) == kcv.ALLOCATION
    assert ctx.synchronize() == kcv.OK
    assert np.array_equal(image(), host)
    assert _call(dtype, ptr, stride, ptr, stride, w, h, ctx) == kcv.OK
    assert ctx.synchronize() == kcv.OK
    assert np.array_equal(image(), _want(dtype, host, w, h))
    ctx.close()
