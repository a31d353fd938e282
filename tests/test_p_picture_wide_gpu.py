"""P pictures whose reference slots hold samples above 8 bits (uploads do not
reject them): the prediction of each 32x32 unit without residual against the
8-bit filters written out here, whose window and horizontal sums are 16-bit
numbers; and the same units on 8-bit references, which take the packed path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def predict(ref, x0, y0, n, taps, fx, fy, dx, dy):
    """One n x n block at (x0, y0): reference reads clamped to the plane."""
    nt, half = taps.shape[1], taps.shape[1] // 2 - 1
    h, w = ref.shape
    ys = np.clip(np.arange(y0 + dy - half, y0 + dy - half + n + nt - 1), 0, h - 1)
    xs = np.clip(np.arange(x0 + dx - half, x0 + dx - half + n + nt - 1), 0, w - 1)
    win = ref[np.ix_(ys, xs)].astype(np.int16).astype(np.int64)
    hor = sum(taps[fx, k] * win[:, k:k + n] for k in range(nt))
    if fx == 0 and fy == 0:
        return win[half:half + n, half:half + n]
    if fy == 0:
        return np.clip((hor[half:half + n] + 32) >> 6, 0, 255)
    if fx == 0:
        v = sum(taps[fy, k] * win[k:k + n, half:half + n] for k in range(nt))
        return np.clip((v + 32) >> 6, 0, 255)
    t = hor.astype(np.int16).astype(np.int64)
    return np.clip((sum(taps[fy, k] * t[k:k + n] for k in range(nt)) + 2048) >> 12, 0, 255)


@pytest.mark.parametrize("top", [255, 256, 3000])
def test_p_prediction_of_any_reference_samples(pkg, top):
    from rustmpeg_next_b200 import tables

    luma = tables.table("kLumaTaps8").reshape(16, 8).astype(np.int64)
    chroma = tables.table("kChromaTaps4").reshape(32, 4).astype(np.int64)
    rng = np.random.default_rng(top)
    w, h = 96, 64
    ref = [rng.integers(0, top + 1, s).astype(np.uint16) for s in ((h, w), (h // 2, w // 2), (h // 2, w // 2))]
    n = (w // 32) * (h // 32)
    cus = np.zeros(n, pkg.INTER_CU_DTYPE)
    cus["ref_idx"], cus["inter_dir"], cus["bcw_idx"], cus["level_off"] = (0, -1), 1, 2, -1
    mv = rng.integers(-300, 301, (n, 2))
    mv[0] &= ~15
    mv[1, 0] &= ~31
    mv[2, 1] &= ~31
    cus["mv"][:, 0] = mv
    pics = np.zeros(1, pkg.P_PIC_DTYPE)
    pics["width"], pics["height"], pics["qp"], pics["num_refs"], pics["out_slot"] = w, h, 30, 1, 1
    with pkg.Context(0) as ctx:
        ctx.dpb_reserve(2, w, h)
        ctx.dpb_upload(0, ref)
        ctx.decode_p_batch(pics, cus, np.zeros(0, np.int16))
        got = ctx.dpb_download(1)
    for k in range(n):
        x, y = 32 * (k % (w // 32)), 32 * (k // (w // 32))
        mx, my = int(mv[k, 0]), int(mv[k, 1])
        want = [predict(ref[0], x, y, 32, luma, mx & 15, my & 15, mx >> 4, my >> 4)]
        want += [predict(ref[c], x // 2, y // 2, 16, chroma, mx & 31, my & 31, mx >> 5, my >> 5) for c in (1, 2)]
        for c in range(3):
            s, px, py = (32, x, y) if c == 0 else (16, x // 2, y // 2)
            # a residual-free unit stores the clipped prediction
            assert (got[c][py:py + s, px:px + s] == np.clip(want[c], 0, 255)).all(), (k, c, mx, my)

