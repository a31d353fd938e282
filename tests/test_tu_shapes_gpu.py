"""Transform units at the edges of the warp path against the oracle: every
shape 1x2..64x64 with every tool it may carry (BDPCM also after a transform,
and on 64x64 transform-skip units), levels and residuals over the whole 16-bit
range (where the forward first stage leaves 16 bits), extreme QPs, and inputs
that start at odd offsets."""
import numpy as np
import pytest

from test_tu_gpu import _run

pytestmark = pytest.mark.gpu


def records(pkg, forward, bit_depth, rng):
    bd_dirs = (pkg.TU_BDPCM_HOR, pkg.TU_BDPCM_VER)
    rows = []
    for a in range(7):
        for b in range(7):
            if a + b == 0:
                continue
            flags = [0, pkg.TU_DEP_QUANT, pkg.TU_IMPLICIT_MTS, pkg.TU_DEP_QUANT | pkg.TU_IMPLICIT_MTS,
                     pkg.TU_TRANSFORM_SKIP]
            flags += [pkg.TU_INTER] if forward else [pkg.TU_TRANSFORM_SKIP | d for d in bd_dirs] + list(bd_dirs) + \
                [pkg.TU_DEP_QUANT | d for d in bd_dirs]
            rows += [(a, b, f, 0, 0) for f in flags]
            if 2 <= a <= 5 and 2 <= b <= 5:
                rows += [(a, b, f, m, 0) for m in range(1, 5) for f in (0, pkg.TU_DEP_QUANT)]
            if a >= 2 and b >= 2:
                rows += [(a, b, f, 0, k) for k in (1, 2) for f in (0, pkg.TU_DEP_QUANT)]
    recs = np.zeros(len(rows), pkg.TU_DTYPE)
    r = np.array(rows)
    for k, f in enumerate(("log2_w", "log2_h", "flags", "mts_idx", "lfnst_idx")):
        recs[f] = r[:, k]
    recs["bit_depth"] = bit_depth
    recs["qp"] = rng.choice([0, 4, 22, 37, 63, 87], len(rows))
    recs["lfnst_mode"] = rng.integers(0, 95, len(rows))
    return recs


@pytest.mark.parametrize("forward", [False, True])
@pytest.mark.parametrize("bit_depth", [8, 10, 12])
@pytest.mark.parametrize("kind", ["full", "sparse", "edge"])
@pytest.mark.parametrize("odd", [0, 1])
def test_tu_shapes(ctx, pkg, orc, forward, bit_depth, kind, odd):
    rng = np.random.default_rng([int(forward), bit_depth, len(kind), odd])
    recs = records(pkg, forward, bit_depth, rng)
    size = 1 << (recs["log2_w"].astype(np.int64) + recs["log2_h"])
    offs = np.cumsum(size + odd) - size
    recs["in_off"] = recs["out_off"] = offs
    total = int(offs[-1] + size[-1]) + 8
    if kind == "full":
        data = rng.integers(-32768, 32768, total)
    elif kind == "sparse":
        data = np.where(rng.random(total) < 0.06, rng.integers(-40, 41, total), 0)
    else:
        data = rng.choice([-32768, 32767, 0], total)
    data = data.astype(np.int16)
    got = _run(ctx, pkg, recs, data, total, forward)
    keep = np.zeros(total, bool)
    for o, n in zip(offs, size):
        keep[o:o + n] = True
    got[~keep] = -7
    _, want = orc.tu_batch(recs, data, total, forward=forward)
    want = np.where(keep, want, -7)
    bad = np.nonzero(got != want)[0]
    if bad.size:
        i = int(np.searchsorted(offs, bad[0], side="right") - 1)
        raise AssertionError(f"{bad.size} values differ; first in unit {i}: {recs[i]}")
