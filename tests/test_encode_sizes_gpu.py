"""The lane-per-frame encoder takes 4 or 8 frames per warp, by the code's z and
the batch: against the oracle at both sides of the line, with a last warp of
one frame, chunks of 16 and 8 bytes and bytes other than 0 and 1."""
import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,z", [(0, 24), (3, 28), (5, 56), (1, 60), (0, 96)])
@pytest.mark.parametrize("frames", [1, 4736, 4737, 4745])
def test_batches_match_oracle(wl, cuda, oracle, rate, z, frames):
    enc = wl.Encoder(rate, z)
    u = inputs.info_bits(500 + rate + z, frames, enc.k)
    cw = cuda.full((frames, enc.n), 9, dtype=cuda.uint8, device="cuda")
    enc.encode_device(cuda.from_numpy(u).cuda(), cw)
    assert (cw.cpu().numpy() == oracle.encode(rate, z, u)).all()
    u[:, ::3] *= 7   # any non-zero byte is a 1, and passes through
    enc.encode_device(cuda.from_numpy(u).cuda(), cw)
    out = cw.cpu().numpy()
    assert (out[:, :enc.k] == u).all()
    assert (out[:, enc.k:] == oracle.encode(rate, z, (u != 0).astype(np.uint8))[:, enc.k:]).all()
