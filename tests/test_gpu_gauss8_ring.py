"""The four-channel streaming Gaussian where its ring of staged rows can go
wrong, against the CPU oracle: heights around multiples of the copy groups, of
the rings (9, 20 and 14 rows) and of the bands (24, 14 and 48 rows), single calls and a plan
(whose shares make the tallest bands), aligned, 4-byte aligned and border
rows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import device_image, device_output, read_output  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()
BORDERS = (kcv.REPLICATE, kcv.REFLECT, kcv.WRAP, kcv.REVERSE, kcv.CONSTANT)


@pytest.mark.parametrize("k", [3, 5, 7])
def test_single_calls_and_plan(k):
    rng = np.random.default_rng(k)
    ctx = kcv.Context.for_torch(0)
    reqs, items = [], []
    for n, (w, h) in enumerate([(6, 6), (121, 15), (240, 22), (119, 42), (500, 48), (241, 49), (360, 97), (64, 1500),
                                (3840, 700), (1203, 2160)]):
        pad, offset = ((-4 * w) % 16, 0) if n % 2 else (4 * (n % 3), 4)
        border = BORDERS[n % 5]
        ext = border == kcv.CONSTANT
        host = rng.integers(0, 256, (h, 4 * w + pad), dtype=np.uint8)
        sbuf, sptr, sstride = device_image(torch, host, offset)
        dbuf, dptr, dstride = device_output(torch, h, 4 * w, np.uint8, pad_elems=pad, offset=offset)
        assert kcv.gaussian_blur_u8(sptr, sstride, dptr, dstride, w, h, 4, k, k, 1.3, 1.3, border, ctx,
                                    border_value=7 if ext else None) == kcv.OK
        assert ctx.synchronize() == kcv.OK
        want = oracle.gaussian_blur_u8(host, w, h, 4, k, 1.3, border, ext=ext, border_value=7)[1]
        got, pad_ok = read_output(dbuf, h, 4 * w, np.uint8, dstride, offset)
        assert pad_ok and np.array_equal(got, want), (w, h)
        dbuf.fill_(0xA5)
        reqs.append(kcv.make_request(kcv.OP_GAUSSIAN_BLUR_U8, sptr, sstride, dptr, dstride, w, h, 4, k, k, 1.3, 1.3,
                                     border_type=border, border_value=7, allow_extensions=ext))
        items.append((sbuf, dbuf, dstride, offset, w, h, want))
    plan = kcv.BatchPlan(reqs, ctx)
    assert plan.launch(True) == kcv.OK
    assert ctx.synchronize() == kcv.OK
    for _, dbuf, dstride, offset, w, h, want in items:
        got, pad_ok = read_output(dbuf, h, 4 * w, np.uint8, dstride, offset)
        assert pad_ok and np.array_equal(got, want), (w, h)
    plan.close()
    ctx.close()
