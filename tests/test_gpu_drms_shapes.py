"""DRMS kernel at the edges of its split (remc_post_drms): frames that do not
fill a group, molecules shorter than a warp, frames too large for shared
memory, one part and many, against the oracle's loop-order sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,frames", [
    ([1, 1], 1), ([1, 40, 3], 3), ([33, 31], 4), ([20] * 5, 5), ([150] * 4, 9), ([30] * 3, 303),
    ([2500, 2400], 2),  # 4 frames of 4900 beads exceed a CTA's shared memory
])
def test_drms_shapes(built_lib, lengths, frames):
    from oracle import bindings as ob
    from remcdockingsimulator_b200 import post
    rng = np.random.default_rng(sum(lengths) + frames)
    ms = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    n = int(ms[-1])
    ref = rng.normal(scale=12.0, size=(n, 3)).astype(np.float32)
    x = (ref[None] + rng.normal(scale=2.0, size=(frames, n, 3))).astype(np.float32)
    for reverse in ([False, True] if len(set(lengths)) == 1 else [False]):
        d, nat, rec, bind = post.drms(x, ref, ms, reverse=reverse)
        for f in range(frames):
            want, cnt = ob.post_drms(x[f], ref, ms, reverse, 12.0, 15.0)
            # FP64 sums of the same FP32 terms in another order
            assert abs(d[f] - want) <= 1e-12 * abs(want), (f, d[f], want)
            assert (nat[f], rec[f], bind[f]) == tuple(cnt)
