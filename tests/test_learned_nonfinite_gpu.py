"""The fp32 learned decoder on LLRs that leave the ordinary range: infinite by
hard decision at random positions, half of them wrong, so that inf - inf
makes NaN; NaN in the input; all but one edge of a row NaN; subnormal. A frame's
outputs are the oracle's, whose rule is that a NaN is no minimum and that an
edge with no other minimum gets no message (oracle/wldpc_oracle.c), and do not depend on whether the
batch is small or goes to the large-batch kernels (units of one warp, of
several, of two frames, rows of 6 to 20 edges). Equality; a NaN equals a NaN."""
import numpy as np
import pytest

import inputs
from test_learned_oracle import random_weights

pytestmark = pytest.mark.gpu

REPEATS = 500   # of the distinct frames in the large batch


def nonfinite_frames(oracle, rate, z, seed):
    rs, cols, shifts = oracle.code_blocks(rate, z)
    rng = np.random.default_rng(seed)
    _, _, llr = inputs.frames(oracle, rate, z, 60, inputs.SWEEP_EBNO[rate] - 2.0, seed)
    inf, n = np.float32(np.inf), llr.shape[1]
    for f in range(60):
        kind = f % 6
        if kind < 3:      # 30, 60 and 90% infinite
            at = rng.random(n) < 0.3 * (kind + 1)
            llr[f, at] = np.where(llr[f, at] > 0, inf, -inf)
        elif kind == 3:
            llr[f, rng.random(n) < 0.1] = np.nan
        elif kind == 4:   # all edges of some rows NaN but the first
            for row in range(0, z, 5):
                i = row % (len(rs) - 1)
                for b in range(rs[i] + 1, rs[i + 1]):
                    llr[f, cols[b] * z + (row + shifts[b]) % z] = np.nan
        else:
            llr[f] *= np.float32(1e-44 if f % 4 == 1 else 1e-38)
    return llr


@pytest.mark.parametrize("rate,z", [(0, 28), (0, 44), (2, 52), (2, 24), (4, 68), (5, 60), (1, 96)])
@pytest.mark.parametrize("scale", [None, 0.0, -0.5])
def test_outputs_follow_the_oracle_at_every_batch_size(wl, cuda, oracle, rate, z, scale):
    llr = nonfinite_frames(oracle, rate, z, 900 + 10 * z + rate)
    weights = random_weights(oracle, rate, z, 8, 33)[0]
    if scale is not None:
        weights[0] = scale
    post, hard, it, fail = oracle.learned_decode(rate, z, 8, weights, llr, cap=6)
    nan = np.isnan(post).any(1)
    assert nan[3::6].all() and nan.sum() >= (20 if scale is None else 10)
    post = np.where(np.isnan(post), np.float32(np.nan), post).view(np.int32)
    small = None
    for repeats in (1, REPEATS):
        d_llr = cuda.from_numpy(llr).cuda().repeat(repeats, 1)
        out = cuda.empty_like(d_llr)
        bits = cuda.empty(d_llr.shape, dtype=cuda.int8, device="cuda")
        status = cuda.empty(60 * repeats, dtype=cuda.int32, device="cuda")
        wl.LearnedDecoder(rate, z, 8, weights, 6).decode_device(d_llr, bits, out, status)
        out = cuda.where(cuda.isnan(out), cuda.full_like(out, float("nan")), out).view(cuda.int32)
        got = [x.view(repeats, 60, -1) for x in (out, bits, status)]
        small = small or got
        for x, y, ref in zip(got, small, (post, hard, (it | fail << 16)[:, None])):
            assert (x == y).all()
            assert (x == cuda.from_numpy(ref).cuda()).all()
