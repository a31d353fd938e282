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


@pytest.mark.parametrize("extra", [-146, 1, 148, 300])
def test_cnn_gradients_with_skipped_blocks(ctx, pkg, extra):
    """Blocks outside the plane or with labels out of range are left out of
    the sums wherever they fall among a CTA's blocks (its first, one whose
    activations were to be fetched ahead, its last)."""
    import torch
    from rustmpeg_next_b200 import cnn, synth

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = max(2, sms + extra)
    w, h = 160, 128
    y, _, _ = synth.value_noise_frame(w, h, 10, frame=4)
    plane = np.ascontiguousarray(y.astype(np.uint16))
    rng = np.random.default_rng(n)
    xy = np.stack([rng.integers(0, w - 31, n), rng.integers(0, h - 31, n)], axis=1).astype(np.int32)
    labels = np.stack([rng.integers(0, 67, n), rng.integers(0, 6, n)], axis=1).astype(np.uint8)
    xy[0::5] = [w - 31, 0]
    labels[1::9, 0] = 67
    labels[4::11, 1] = 6
    ok = (xy[:, 0] <= w - 32) & (labels[:, 0] < 67) & (labels[:, 1] < 6)
    params = cnn.init_params(6)
    p = torch.from_numpy(params).cuda()
    pl = torch.from_numpy(plane.view(np.int16)).cuda()
    loss, grads = ctx.cnn_train_step(pl, 10, 27, torch.from_numpy(xy).cuda(), torch.from_numpy(labels).cuda(), p,
                                     sync=False)
    torch.cuda.synchronize()
    if not ok.any():
        assert float(loss.item()) == 0.0 and not grads.any()
        return
    blocks = np.stack([plane[yy:yy + 32, xx:xx + 32] for xx, yy in xy[ok]]).astype(np.float32)
    ref_loss, ref = cnn.reference_loss_and_grads(blocks, labels[ok], 10, params, 27)
    part = ok.sum() / n  # the mean runs over all n
    assert abs(float(loss.item()) - ref_loss * part) <= 1e-3 * max(1.0, abs(ref_loss))
    g = grads.cpu().numpy()
    groups = [(cnn.OFF_W1, 576), (cnn.OFF_B1, 32), (cnn.OFF_WI, 67 * 32), (cnn.OFF_BI, 67), (cnn.OFF_WS, 192),
              (cnn.OFF_BS, 6)] + [(cnn.off_w(l), 9216) for l in (2, 3, 4)] + [(cnn.off_b(l), 32) for l in (2, 3, 4)]
    for off, cnt in groups:
        a, b = g[off:off + cnt], ref[off:off + cnt] * part
        assert np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12) < 3e-2, off
