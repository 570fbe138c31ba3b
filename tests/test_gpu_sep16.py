"""The 16-bit streaming filter on rows that are not 16-byte aligned, against
the CPU oracle: every misalignment of source and destination rows, widths
around a lane's 8 elements and a strip's 240, heights around a band's 15 rows,
all borders, u16 (saturating) and s16.  Integers: the outputs must be equal."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import device_image, device_output, read_output  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()
BORDERS = (kcv.REPLICATE, kcv.REFLECT, kcv.WRAP, kcv.REVERSE, kcv.CONSTANT)
TAPS = {"u16": ([0, 1, 2, 1, 0], [300, 0, 3, 0, 1]), "s16": ([-1, -2, 0, 2, 1], [1, 4, 6, 4, 1])}


@pytest.mark.parametrize("dtype", ["u16", "s16"])
@pytest.mark.parametrize("w,h", [(4, 4), (9, 5), (16, 15), (239, 16), (241, 31), (250, 14), (487, 61), (1921, 700)])
def test_unaligned_rows(dtype, w, h):
    rng = np.random.default_rng(w * h)
    dt = np.dtype("uint16" if dtype == "u16" else "int16")
    info = np.iinfo(dt)
    kx, ky = TAPS[dtype]
    ctx = kcv.Context.for_torch(0)
    for n in range(8):
        pad, offset = n % 5, 2 * n
        border = BORDERS[(n + w) % 5]
        ext = border == kcv.CONSTANT
        host = rng.integers(info.min, int(info.max) + 1, (h, w + pad), dtype=dt)
        if n % 2:
            host = (host % 50).astype(dt)
        sbuf, sptr, sstride = device_image(torch, host, offset)
        doff = 2 * ((n * 3) % 8)
        dbuf, dptr, dstride = device_output(torch, h, w, dt, pad_elems=(n * 2) % 7, offset=doff)
        err = kcv.separable_filter_2d(dtype, sptr, sstride, dptr, dstride, w, h, 1, kx, 5, ky, 5, border, ctx,
                                      border_value=17 if ext else None)
        werr, want = oracle.separable_filter_2d(host, w, h, 1, np.array(kx, dt), np.array(ky, dt), border,
                                                ext=ext, border_value=17)
        assert err == werr == kcv.OK
        assert ctx.synchronize() == kcv.OK
        got, pad_ok = read_output(dbuf, h, w, dt, dstride, doff)
        assert pad_ok, n
        assert np.array_equal(got, want), (n, int((got != want).sum()))
    ctx.close()


@pytest.mark.parametrize("dtype", ["u16", "s16"])
@pytest.mark.parametrize("w,h", [(1023, 521), (1921, 700)])
def test_unaligned_in_place(dtype, w, h):
    """Source and destination are one unaligned image: every row is read as it was before the call."""
    rng = np.random.default_rng(w * h + 1)
    dt = np.dtype("uint16" if dtype == "u16" else "int16")
    info = np.iinfo(dt)
    kx, ky = TAPS[dtype]
    ctx = kcv.Context.for_torch(0)
    host = rng.integers(info.min, int(info.max) + 1, (h, w), dtype=dt)
    buf, ptr, stride = device_image(torch, host, 2)
    for _ in range(2):  # filtered twice
        werr, want = oracle.separable_filter_2d(host, w, h, 1, np.array(kx, dt), np.array(ky, dt), kcv.REFLECT)
        err = kcv.separable_filter_2d(dtype, ptr, stride, ptr, stride, w, h, 1, kx, 5, ky, 5, kcv.REFLECT, ctx)
        assert err == werr == kcv.OK
        assert ctx.synchronize() == kcv.OK
        got, _ = read_output(buf, h, w, dt, stride, 2)
        assert np.array_equal(got, want), int((got != want).sum())
        host = want
    ctx.close()
