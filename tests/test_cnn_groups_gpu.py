"""GPU: two blocks in flight per CTA in the CNN forward pass, at block counts
around the multiples of the CTA count (one group idle, one a block ahead) and
with blocks outside the plane among them: every block's result equals that of
the block alone, bit by bit, and the fp32 reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-147, 0, 1, 148, 149, 297])
def test_cnn_blocks_in_flight(ctx, pkg, extra):
    import torch
    from rustmpeg_next_b200 import cnn, synth

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = max(2, sms + extra)
    w, h = 160, 128
    y, _, _ = synth.value_noise_frame(w, h, 10, frame=9)
    plane = np.ascontiguousarray(y.astype(np.uint16))
    rng = np.random.default_rng(n)
    xy = np.stack([rng.integers(0, w - 31, n), rng.integers(0, h - 31, n)], axis=1).astype(np.int32)
    out = np.zeros(n, bool)
    out[1::7] = True
    xy[out] = [[w - 31, 0], [0, h - 31], [-1, 0], [0, 1 << 20]][n % 4]
    params = cnn.init_params(5)
    p = torch.from_numpy(params).cuda()
    pl = torch.from_numpy(plane.view(np.int16)).cuda()
    logits, gap, acts = ctx.cnn_forward(pl, 10, torch.from_numpy(xy).cuda(), p, 27, want_acts=True, sync=False)
    torch.cuda.synchronize()
    logits, gap, acts = logits.cpu(), gap.cpu(), acts.cpu()
    assert torch.isnan(logits[out]).all() and not torch.isnan(logits[~out]).any()
    ok = np.nonzero(~out)[0]
    blocks = np.stack([plane[yy:yy + 32, xx:xx + 32] for xx, yy in xy[ok]]).astype(np.float32)
    ref_logits, ref_gap, _ = cnn.reference_forward(blocks, 10, params, 27)
    assert torch.allclose(gap[ok], ref_gap, rtol=2e-2, atol=2e-3)
    assert torch.allclose(logits[ok], ref_logits, rtol=2e-2, atol=2e-2)
    for i in ok[::max(1, len(ok) // 16)]:
        one = ctx.cnn_forward(pl, 10, torch.from_numpy(xy[i:i + 1]).cuda(), p, 27, want_acts=True)
        for a, b in zip(one, (logits, gap, acts)):
            assert torch.equal(a.cpu()[0], b[i])
