"""decode(float*) of one frame, which the kernel stages from and writes to the
decoder's pinned host block: equal to the oracle bit for bit where a CTA has
room for one frame, several and eight, for the three min-sum flavours, with
another frame in the block from the call before."""
import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,z", [(0, 24), (3, 28), (5, 44), (1, 60), (2, 64), (4, 92), (0, 96)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_single_frame_matches_oracle(wl, cuda, oracle, rate, z, mode):
    llr = np.concatenate([inputs.frames(oracle, rate, z, 1, inputs.SWEEP_EBNO[rate] + db, 77 + k)[2]
                          for k, db in enumerate((-2.0, 0.5, 9.0))])
    po, do, ret, it, _ = oracle.decode(rate, z, llr, 6, mode)
    dec = wl.Decoder(rate, z, 6, mode)
    for f in range(3):
        post, hard, failed, iterations = dec.decode(llr[f])
        assert (post.view(np.uint32) == po[f].view(np.uint32)).all() and (hard == do[f]).all()
        assert failed == ret[f] and iterations == it[f]
