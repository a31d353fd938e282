"""P pictures whose reference slots hold samples above 8 bits: the clipped sum
of prediction and residual, against the sum of the two 16-bit numbers in more
bits. Transform-skip levels at QP 4 are the residual itself, over the whole
16-bit range; whole-sample motion copies the reference samples unclipped."""
import numpy as np
import pytest

from test_p_picture_wide_gpu import predict

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top", [255, 256, 5000, 30000, 65535])
def test_p_sum_of_any_reference_samples_and_residual(pkg, top):
    from rustmpeg_next_b200 import tables

    luma = tables.table("kLumaTaps8").reshape(16, 8).astype(np.int64)
    chroma = tables.table("kChromaTaps4").reshape(32, 4).astype(np.int64)
    rng = np.random.default_rng([top, 1])
    w, h = 96, 64
    ref = [rng.integers(0, top + 1, s).astype(np.uint16) for s in ((h, w), (h // 2, w // 2), (h // 2, w // 2))]
    n = (w // 32) * (h // 32)
    off = 1536 * np.arange(n)[:, None] + np.array([0, 1024, 1280])
    levels = rng.integers(-32768, 32768, 1536 * n)
    small = rng.random(len(levels)) < 0.5
    levels[small] = rng.integers(-300, 301, int(small.sum()))
    levels = levels.astype(np.int16)
    cus = np.zeros(n, pkg.INTER_CU_DTYPE)
    cus["ref_idx"], cus["inter_dir"], cus["bcw_idx"] = (0, -1), 1, 2
    cus["cbf"], cus["tu_tools"], cus["level_off"] = 7, 7, off
    mv = 32 * rng.integers(-20, 21, (n, 2))  # whole samples of every component
    mv[n - 2:] += 5                          # fractional: predictions clipped to 8 bits
    cus["mv"][:, 0] = mv
    pics = np.zeros(1, pkg.P_PIC_DTYPE)
    pics["width"], pics["height"], pics["qp"], pics["num_refs"], pics["out_slot"] = w, h, 4, 1, 1
    with pkg.Context(0) as ctx:
        ctx.dpb_reserve(2, w, h)
        ctx.dpb_upload(0, ref)
        ctx.decode_p_batch(pics, cus, levels)
        got = ctx.dpb_download(1)
    for k in range(n):
        x, y = 32 * (k % (w // 32)), 32 * (k // (w // 32))
        mx, my = int(mv[k, 0]), int(mv[k, 1])
        for c in range(3):
            s, px, py = (32, x, y) if c == 0 else (16, x // 2, y // 2)
            if c == 0:
                pred = predict(ref[0], px, py, s, luma, mx & 15, my & 15, mx >> 4, my >> 4)
            else:
                pred = predict(ref[c], px, py, s, chroma, mx & 31, my & 31, mx >> 5, my >> 5)
            res = levels[off[k, c]:off[k, c] + s * s].reshape(s, s).astype(np.int64)
            assert (got[c][py:py + s, px:px + s] == np.clip(pred + res, 0, 255)).all(), (k, c)
