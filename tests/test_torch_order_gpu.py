"""Calls that synchronise take tensors that torch has only queued work on: its
stream is kept busy while the tensors are filled, and each call on the
context's own stream still sees them and keeps its results."""
import numpy as np
import pytest

from test_txsearch_gpu import _blocks

pytestmark = pytest.mark.gpu


def _luma_tx_search(pkg, ctx, late, rng):
    recs, pred, src, total = _blocks(60, 7)
    reqs = np.array(recs, dtype=pkg.TXS_REQ_DTYPE)
    lv, sm = late(np.zeros(total, np.int16)), late(np.zeros(total, np.int16))
    res = ctx.luma_tx_search(reqs, late(pred), late(src), lv, sm)
    return [res.tobytes(), lv.cpu().numpy().tobytes(), sm.cpu().numpy().tobytes()]


def _ctu_search(pkg, ctx, late, rng):
    reqs = np.zeros(4, pkg.CTU_SEARCH_REQ_DTYPE)
    reqs["x"], reqs["split_mask"] = np.arange(4) * 32, 0x3F
    plane = rng.integers(0, 1024, (64, 128)).astype(np.int16)
    return [ctx.ctu_search(late(plane), 10, 300, reqs).tobytes()]


def _plane_metrics(pkg, ctx, late, rng):
    a, b = rng.integers(0, 1024, (2, 64, 128)).astype(np.int16)
    return list(ctx.plane_metrics(late(a), late(b)))


def _qt_mtt_split(pkg, ctx, late, rng):
    reqs = np.zeros(2, pkg.SPLIT_REQ_DTYPE)
    reqs["x"], reqs["w"], reqs["h"], reqs["min_cb"], reqs["qp"] = (0, 64), 64, 64, 8, 22
    plane = np.kron([[100, 900, 900, 900], [500, 300, 100, 100]], np.ones((32, 32))).astype(np.int16)
    return [ctx.qt_mtt_split(late(plane), 10, reqs).tobytes()]


@pytest.mark.parametrize("call", [_luma_tx_search, _ctu_search, _plane_metrics, _qt_mtt_split])
def test_call_waits_for_queued_tensors(ctx, pkg, call):
    import torch

    big = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")

    def ready(a):
        t = torch.from_numpy(a).cuda()
        torch.cuda.synchronize()
        return t

    def late(a):  # holds its values only when torch's stream has passed the fills
        t, v = torch.full(a.shape, 5, dtype=torch.from_numpy(a).dtype, device="cuda"), ready(a)
        for _ in range(8):
            big.fill_(1)
        t.copy_(v)
        return t

    want = call(pkg, ctx, ready, np.random.default_rng(1))
    assert call(pkg, ctx, late, np.random.default_rng(1)) == want
