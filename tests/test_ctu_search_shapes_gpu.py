"""The CTU search at the edges of its packed arithmetic against the oracle:
checkerboards and noise between the sample limits (the largest Hadamard sums
of 8, 10 and 12 bits), CTUs at odd positions and against every edge of a plane
of odd size, and repeated candidates."""
import numpy as np
import pytest

from test_ctu_search_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bd,top", [(8, 255), (10, 1023), (12, 4095)])
def test_ctu_search_extremes(ctx, pkg, orc, bd, top):
    rng = np.random.default_rng([bd, top])
    w, h = 139, 101
    yy, xx = np.mgrid[0:h, 0:w]
    kind = rng.integers(0, 4, (h // 16 + 1, w // 16 + 1))[yy // 16, xx // 16]
    noise = rng.integers(0, top + 1, (h, w))
    src = np.select([kind == 0, kind == 1, kind == 2], [((xx + yy) & 1) * top, ((yy >> 1) & 1) * top,
                                                        rng.integers(0, 2, (h, w)) * top], noise).astype(np.uint16)
    pos = [(0, 0), (w - 32, 0), (0, h - 32), (w - 32, h - 32), (1, 3), (33, 7), (77, 30), (w - 33, 50)]
    reqs = np.zeros(2 * len(pos), pkg.CTU_SEARCH_REQ_DTYPE)
    for i, q in enumerate(reqs):
        q["x"], q["y"] = pos[i % len(pos)]
        q["split_mask"] = 0x3F
        if i >= len(pos):
            q["n_cand"] = 1 + i % 6
            q["cand"] = rng.choice([0, 1, 2, 18, 19, 34, 49, 50, 51, 66], 6)
    _check(ctx, pkg, orc, src, bd, 30, reqs)
