"""The register-streaming Sobel kernel at its edges, against the CPU oracle:
widths around a thread's 8 elements and its word window, heights around its
four rows, every alignment of source rows, 2-, 4- and 16-byte aligned
destinations, and a larger aligned image, which takes the tiled stencil."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from gpu_harness import device_image, device_output, read_output  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()


@pytest.mark.parametrize("c", [1, 2, 3, 4])
def test_edges(c):
    rng = np.random.default_rng(c)
    ctx = kcv.Context.for_torch(0)
    shapes = [(w, 2 + w % 7) for w in range(2, 27)] + [(1024 // c + 1, 33), (2500 // c, 1700), (4096 // c, 1100)]
    for n, (w, h) in enumerate(shapes):
        spad = -w * c % 16 if n == len(shapes) - 1 else n % 4
        soff, dpad, doff = (0, -w * c % 8, 0) if n == len(shapes) - 1 else (n % 5, n % 3, 2 * (n % 4))
        host = rng.integers(0, 256, (h, w * c + spad), dtype=np.uint8)
        sbuf, sptr, sstride = device_image(torch, host, offset=soff)
        for horizontal in (True, False):
            dbuf, dptr, dstride = device_output(torch, h, w * c, np.int16, pad_elems=dpad, offset=doff)
            fn = kcv.sobel_3x3_horizontal_s16_u8 if horizontal else kcv.sobel_3x3_vertical_s16_u8
            assert fn(sptr, sstride, dptr, dstride, w, h, c, ctx) == kcv.OK
            assert ctx.synchronize() == kcv.OK
            want = oracle.sobel_3x3_s16_u8(host, w, h, c, horizontal)[1]
            got, pad_ok = read_output(dbuf, h, w * c, np.int16, dstride, offset=doff)
            assert pad_ok and np.array_equal(got, want[:, : w * c]), (w, h, horizontal)
    ctx.close()
