"""A staging wait that runs out in the large-batch decoders: units of one warp,
of several, and of two, three and four frames, plain, learned and binary16.
Every wait gives up at once (a limit that the host sets to 0; the copies
themselves land, and the kernel drains them), the caller of decode_device
learns of it from synchronize(), and the next decode is clean and exact."""
import numpy as np
import pytest

from test_learned16_gpu import random_weights
from test_unit_decode_gpu import check, handle, mixed_quality, reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,rate,z,frames", [
    ("plain", 0, 44, 2000), ("plain", 1, 24, 15000), ("plain", 0, 84, 333), ("learned", 0, 28, 500),
    ("learned", 4, 44, 6001), ("learned", 0, 52, 333), ("half", 4, 28, 401), ("half", 0, 36, 6001), ("half", 0, 84, 65)])
def test_expired_waits_are_reported(wl, cuda, oracle, kind, rate, z, frames):
    weights = None if kind == "plain" else random_weights(oracle, rate, z, 8, 5)[0]
    llr = mixed_quality(oracle, rate, z, frames, 8)
    dec = handle(wl, kind, rate, z, 7, weights)
    d_llr = cuda.from_numpy(llr).cuda()
    hard = cuda.empty(llr.shape, dtype=cuda.int8, device="cuda")
    dec.set_wait_limit(0)
    dec.decode_device(d_llr, hard)
    with pytest.raises(wl.LdpcError) as e:
        dec.synchronize()
    assert e.value.code == wl.ERR_TIMEOUT
    dec.synchronize()   # reported once
    dec.set_wait_limit(wl.WAIT_LIMIT_DEFAULT_US)
    check(cuda, dec, llr, reference(oracle, kind, rate, z, 7, weights, llr))
    dec.synchronize()
    dec.decode_host(llr[:70])   # nothing left for a later host batch to report


def test_small_learned_batches_report_too(wl, cuda, oracle):
    llr = mixed_quality(oracle, 0, 96, 20, 8)
    dec = handle(wl, "learned", 0, 96, 7, random_weights(oracle, 0, 96, 8, 5)[0])
    hard = cuda.empty(llr.shape, dtype=cuda.int8, device="cuda")
    dec.set_wait_limit(0)
    dec.decode_device(cuda.from_numpy(llr).cuda(), hard)
    with pytest.raises(wl.LdpcError) as e:
        dec.synchronize()
    assert e.value.code == wl.ERR_TIMEOUT
