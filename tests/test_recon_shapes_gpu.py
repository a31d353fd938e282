"""The reconstruction wavefront at the edges of its shapes: each chroma
format alone (its own CTA shape) and all of them in one batch (the largest
shape for every picture), pictures of one CTU, one CTU row or column, every
CTU size, and every luma mode value with every chroma mode value, against the
oracle, sample for sample."""
import numpy as np
import pytest

from test_recon_gpu import assert_same, oracle_outputs

pytestmark = pytest.mark.gpu

SIZES = [(32, 32, 5), (96, 32, 5), (32, 96, 5), (160, 128, 5), (64, 64, 6), (192, 128, 6), (256, 128, 7)]


def records(pkg, formats, bit_depth, seed):
    from rustmpeg_next_b200 import synth

    spec = [dict(width=w, height=h, bit_depth=bit_depth, chroma_format=cf, ctu_log2=c, qp=30)
            for cf in formats for w, h, c in SIZES]
    pics, cus, levels, ctus, aps = synth.random_records(spec, seed=seed, tools=0)
    rng = np.random.default_rng(seed)
    # every luma mode (and one past the range), every chroma mode and CCLM
    cus["luma_mode"] = rng.permutation(np.arange(len(cus)) % 68)
    chroma = np.concatenate([np.arange(70), [81, 82, 83] * 12])
    cus["chroma_mode"] = np.where(np.repeat(pics["chroma_format"], [(w // 32) * (h // 32) for _ in formats
                                                                     for w, h, _ in SIZES]) > 0,
                                  chroma[rng.integers(0, len(chroma), len(cus))], 0)
    return pics, cus, levels, ctus, aps


@pytest.mark.parametrize("formats,bit_depth", [((0,), 8), ((1,), 10), ((2,), 12), ((3,), 8), ((0, 1, 2, 3), 10)])
def test_recon_shapes(ctx, pkg, orc, formats, bit_depth):
    for seed in range(3):
        pics, cus, levels, ctus, aps = records(pkg, formats, bit_depth, seed)
        out = ctx.decode_batch(pkg.Batch(pics, cus, levels, ctus, aps))
        assert_same(out, oracle_outputs(orc, pics, cus, levels, ctus, aps))
