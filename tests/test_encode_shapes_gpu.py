"""The encoder wavefront at the edges of its shapes and ranges against the
oracle's encoder: pictures of one unit, one row or column of units, every CTU
size and chroma format, noise between the sample limits (the largest
residuals and coefficients), and source samples above the bit depth, which
the interface does not reject."""
import numpy as np
import pytest

from test_encode_gpu import OPT_CCLM, OPT_DBF, OPT_DQ, OPT_FULL, _check_picture, _coded_planes, _desc

pytestmark = pytest.mark.gpu


def noise_planes(pkg, rng, w, h, cf, top):
    cw, ch = pkg.chroma_dims(w, h, cf)
    coarse = lambda hh, ww: np.kron(rng.integers(0, 2, (hh // 8, ww // 8)), np.ones((8, 8), np.int64))  # noqa: E731
    y = np.where(rng.random((h, w)) < 0.5, coarse(h, w) * top, rng.integers(0, top + 1, (h, w))).astype(np.uint16)
    if not cf:
        return y, None, None
    return y, rng.integers(0, top + 1, (ch, cw)).astype(np.uint16), (coarse(ch, cw) * top).astype(np.uint16)


@pytest.mark.parametrize("cf", [0, 1, 2, 3])
@pytest.mark.parametrize("bd,qp,dq,top", [(8, 0, True, 255), (10, 22, True, 1023), (12, 4, False, 4095),
                                          (12, 30, True, 4095), (12, 0, True, 4095), (8, 10, True, 65535),
                                          (10, 26, False, 40000)])
def test_encoder_shapes(ctx, pkg, orc, cf, bd, qp, dq, top):
    rng = np.random.default_rng([bd, qp, cf, top])
    opts = OPT_FULL | OPT_CCLM | OPT_DBF | (OPT_DQ if dq else 0)
    pics, srcs, want = [], [], []
    for w, h, ctu_log2 in ((32, 32, 5), (128, 32, 5), (32, 96, 5), (128, 64, 6), (128, 128, 7)):
        planes = noise_planes(pkg, rng, w, h, cf, top)
        pics.append(_desc(pkg, w, h, bd, qp, ctu_log2, opts, cf))
        srcs.append(planes)
        want.append(orc.encode_frame(*planes, bd, qp, ctu_log2, opts, cf=cf))
    cus, levels = ctx.encode_batch(np.array(pics), srcs)
    recs = ctx.download(_coded_planes(ctx, pkg, pics))
    at = 0
    for i, p in enumerate(pics):
        n = (int(p["width"]) // 32) * (int(p["height"]) // 32)
        _check_picture(i, p, cus[at:at + n], levels, recs[i], *want[i])
        at += n
