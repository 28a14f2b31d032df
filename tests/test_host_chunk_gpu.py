"""Host batches of pinned, pageable and mixed buffers, which are cut into
different chunks, with a last chunk of one frame and of some: equal to the
oracle whatever memory they are in."""
import numpy as np
import pytest

import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,z,frames", [(0, 96, 1025), (3, 36, 8193), (5, 24, 3100)])
@pytest.mark.parametrize("pinned", [(0, 0, 0), (1, 1, 1), (1, 0, 1), (0, 1, 1), (1, 1, 0)])
def test_every_memory_gives_the_oracles_frames(wl, cuda, oracle, rate, z, frames, pinned):
    _, _, llr = inputs.frames(oracle, rate, z, frames, inputs.SWEEP_EBNO[rate], 41)
    po, do, ret, it, fail = oracle.decode(rate, z, llr, 5)

    def buffer(like, pin):
        return cuda.empty(like.shape, dtype=cuda.from_numpy(like).dtype, pin_memory=bool(pin))
    status = (it | fail << 16).astype(np.int32)
    x, hard, st = (buffer(a, p) for a, p in zip((llr, do, status), pinned))
    errors = buffer(status, pinned[2])
    dec = wl.Decoder(rate, z, 5)
    for statuses in (st, None):
        x.copy_(cuda.from_numpy(llr))
        hard.fill_(7)
        dec.decode_host_hard_into(x, hard, errors, statuses)
        assert (hard.numpy() == do).all() and (errors.numpy() == ret).all()
        assert statuses is None or (statuses.numpy() == status).all()
        hard.fill_(7)
        dec.decode_host_into(x, hard, errors, statuses)
        assert (hard.numpy() == do).all() and (x.numpy().view(np.uint32) == po.view(np.uint32)).all()
