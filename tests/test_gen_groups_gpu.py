"""The persistent reconstruction of the general picture pass: groups whose
blocks are not one coding unit (several units merged in decode order, more
blocks than a CTA fetches ahead), which are done block by block, beside
ordinary groups; and a wait that gives up, which is reported and leaves the
context usable."""
import numpy as np
import pytest

from test_gen_picture_gpu import SPECS, _check, _parts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [2, 5, 40])
def test_merged_groups_match_the_oracle(ctx, pkg, orc, longest):
    from rustmpeg_next_b200 import synth

    rng = np.random.default_rng(longest)
    parts = _parts(synth, SPECS)
    merged = []
    for p in parts:
        sizes, out, k = p[2], [], 0
        while k < len(sizes):
            n = int(rng.integers(1, longest + 1)) if rng.random() < 0.5 else 1
            out.append(int(sizes[k:k + n].sum()))
            k += n
        merged.append(p[:2] + (np.array(out, np.uint32),) + p[3:])
    got = ctx.decode_general(pkg.GenBatch(**synth.general_batch(merged)))
    _check(orc, parts, got)


def test_level_wait_gives_up_and_context_stays_usable(pkg, orc):
    from rustmpeg_next_b200 import synth

    parts = _parts(synth, SPECS[:2])
    batch = pkg.GenBatch(**synth.general_batch(parts))
    with pkg.Context(0, spin_limit=1) as c:
        with pytest.raises(pkg.Timeout):
            c.decode_general(batch)
        with pytest.raises(pkg.Timeout):
            c.decode_general(batch)
    with pkg.Context(0) as c:
        _check(orc, parts, c.decode_general(batch))
