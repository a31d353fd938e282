"""The CTU search on source samples above the bit depth (nothing rejects
them): residuals, the Hadamard sums along the rows and nothing else are 16-bit
numbers that wrap. Around the CTU every sample is the same valid one, so each
mode's prediction of the unsplit block is that sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _satd(res):
    """32x32 residuals by 8x8 tiles: rows, wrapped to 16 bits, then columns."""
    had = np.ones((1, 1), np.int64)
    for _ in range(3):
        had = np.block([[had, had], [had, -had]])
    d = res.astype(np.int16).astype(np.int64).reshape(4, 8, 4, 8).transpose(0, 2, 1, 3)
    rows = (d @ had).astype(np.int16).astype(np.int64)
    return int(((np.abs(had @ rows).sum((2, 3)) + 2) >> 2).sum())


@pytest.mark.parametrize("bd", [8, 10, 12])
@pytest.mark.parametrize("top", [4095, 20000, 65535])
def test_ctu_search_of_samples_above_the_depth(ctx, pkg, bd, top):
    import torch

    rng = np.random.default_rng([bd, top])
    flat = 100
    src = np.full((96, 96), flat, np.uint16)
    src[32:64, 32:64] = rng.integers(0, top + 1, (32, 32))
    src[32:64, 32:40] = top  # rows whose sum leaves 16 bits first along one direction
    src[40:44, 40:64] = top
    modes = [0, 1, 2, 10, 18, 26, 33, 34, 42, 50, 58, 66]
    reqs = np.zeros(len(modes), pkg.CTU_SEARCH_REQ_DTYPE)
    reqs["x"], reqs["y"], reqs["split_mask"], reqs["n_cand"] = 32, 32, 1, 1
    reqs["cand"][:, 0] = modes
    got = ctx.ctu_search(torch.from_numpy(src.view(np.int16)).cuda(), bd, 0, reqs)
    want = _satd(src[32:64, 32:64].astype(np.int64) - flat)
    assert got["split_cost"][:, 0].tolist() == [want] * len(modes)
    assert got["cu_mode"].tolist() == modes
