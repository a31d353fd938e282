"""Motion compensation at the edges of its tiles against the oracle: block
sizes around the 32x16 tile and its runs, planes whose rows or base do not
allow whole-group loads, windows on and across every edge, odd output offsets,
and reference samples above the bit depth, which the interface does not
reject."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 3), (4, 16), (7, 17), (8, 8), (12, 4), (24, 15), (31, 33), (32, 16), (33, 16), (40, 5), (64, 64),
         (100, 20)]


@pytest.mark.parametrize("bd,top,width,shift", [(10, 1023, 160, 0), (12, 4095, 157, 0), (8, 255, 160, 1),
                                                (10, 65535, 160, 0), (12, 65535, 160, 3)])
@pytest.mark.parametrize("chroma", [0, 1, 3])
def test_mc_shapes(ctx, pkg, orc, bd, top, width, shift, chroma):
    import torch

    rng = np.random.default_rng([bd, top, width, chroma])
    h = 90
    flat = torch.from_numpy(rng.integers(0, top + 1, h * width + shift).astype(np.uint16).view(np.int16)).cuda()
    ref = flat[shift:].view(h, width)
    host = ref.cpu().numpy().view(np.uint16)
    blocks = np.zeros(8 * len(SIZES), pkg.MC_BLOCK_DTYPE)
    off = 1
    for i, b in enumerate(blocks):
        bw, bh = SIZES[i % len(SIZES)]
        b["w"], b["h"] = bw, bh
        b["x"] = int(rng.choice([-bw - 9, -3, 0, 1, 5, width - bw - 5, width - 2, width + 9]))
        b["y"] = int(rng.choice([-bh - 9, -3, 0, 7, h - bh - 4, h - 1, h + 20]))
        b["mv_x"], b["mv_y"] = rng.integers(-90, 91, 2) & rng.choice([-1, ~15])
        if i % 3 == 0:
            b["mv_y"] &= ~31
        if i % 3 == 1:
            b["mv_x"] &= ~31
        b["flags"] = rng.integers(0, 2 if chroma else 8)
        b["out_offset"] = off
        off += bw * bh + int(rng.integers(0, 2))
    out = torch.full((off,), -7, dtype=torch.int32, device="cuda")
    dev = torch.from_numpy(blocks.view(np.uint8).reshape(-1).copy()).cuda()
    if chroma:
        ctx.mc_chroma(ref, bd, chroma, dev, out)
    else:
        ctx.mc_luma(ref, bd, dev, out)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for b in blocks:
        x, y, bw, bh, mx, my, f = (int(b[k]) for k in ("x", "y", "w", "h", "mv_x", "mv_y", "flags"))
        if chroma:
            want = orc.mc_chroma(host, bd, x, y, bw, bh, mx, my, bi=bool(f & 1), cf=chroma)
        else:
            want = orc.mc_luma(host, bd, x, y, bw, bh, mx, my, bi=bool(f & 1), affine=bool(f & 2),
                               alt_hpel=bool(f & 4))
        o = int(b["out_offset"])
        assert (got[o:o + bw * bh].reshape(bh, bw) == want).all(), b
