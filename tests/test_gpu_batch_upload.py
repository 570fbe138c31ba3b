"""A batch plan is built while the context's stream is busy: its tables go up
through the pinned ring without a wait for the stream's earlier work, whatever
the number of tables, and they are complete when the plan runs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import __graft_entry__ as ge  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

kcv = ge.package()


def _requests(rng):
    """Requests of many kernel sizes and channel counts (a table or two for each kind)."""
    images, reqs = [], []
    for c in (1, 2, 3, 4):
        for k, sigma in ((3, 0.0), (3, 0.8), (5, 0.0), (5, 1.2), (7, 1.5), (9, 2.0), (15, 2.5), (9, 0.0)):
            w, h = int(rng.integers(64, 200)), int(rng.integers(40, 120))
            host = rng.integers(0, 256, (h, w * c), dtype=np.uint8)
            src = torch.from_numpy(host).cuda()
            dst = torch.zeros_like(src)
            images.append((host, src, dst, w, h, c, k, sigma))
            reqs.append(kcv.make_request(kcv.OP_GAUSSIAN_BLUR_U8, kcv.ptr(src), kcv.stride(src), kcv.ptr(dst),
                                         kcv.stride(dst), w, h, c, k, k, sigma, sigma, border_type=kcv.REFLECT))
    return images, reqs


def test_plan_creation_does_not_wait_for_the_stream():
    images, reqs = _requests(np.random.default_rng(7))
    ctx = kcv.Context.for_torch(0)
    for _ in range(9):  # every kernel loaded, every buffer of the ring grown
        kcv.BatchPlan(reqs, ctx).close()
        assert ctx.synchronize() == kcv.OK
    w, h = 3840, 2160
    src = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    dst = torch.zeros_like(src)
    for _ in range(600):  # tens of milliseconds
        assert kcv.gaussian_blur_u8(kcv.ptr(src), w, kcv.ptr(dst), w, w, h, 1, 255, 255, 0.0, 0.0, kcv.REPLICATE,
                                    ctx) == kcv.OK
    earlier = torch.cuda.Event()
    earlier.record()
    plan = kcv.BatchPlan(reqs, ctx)
    assert not earlier.query()
    assert plan.launch(False) == kcv.OK
    assert ctx.synchronize() == kcv.OK
    for host, _, out, iw, ih, c, k, sigma in images:
        want = oracle.gaussian_blur_u8(host, iw, ih, c, k, sigma, kcv.REFLECT)[1]
        assert np.array_equal(out.cpu().numpy(), want), (iw, ih, c, k, sigma)
    plan.close()
    ctx.close()
