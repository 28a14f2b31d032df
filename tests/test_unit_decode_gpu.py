"""The large-batch decoders (messages in tensor memory, persistent units): bit
for bit against the oracle at the batch sizes where they take over and around
them, for every shape of a unit -- one warp (z = 28, 32), whole warps (64, 96),
idle lanes (60, 84), two and three frames per unit (44, 40, 36) and four with
refill (24), 20 instead of 24 warps (rate 3/4B) and rows of 6 to 20 edges --
with frames that stop at the initial check, after some iterations and at the
cap, a last ticket of one frame of a pair, posteriors written over the LLRs,
caps 0 and 1, and a staging wait that gives up. Equality, tolerance 0."""
import numpy as np
import pytest

import inputs
from test_learned16_gpu import random_weights

pytestmark = pytest.mark.gpu

# decoder, rate, z, frames
CASES = [("plain", 0, 28, 64), ("plain", 0, 28, 63), ("plain", 1, 24, 15000), ("plain", 0, 36, 6001),
         ("plain", 0, 44, 1800), ("plain", 0, 40, 6003), ("plain", 4, 60, 65), ("plain", 2, 52, 641),
         ("plain", 0, 84, 333), ("plain", 1, 96, 6000), ("plain", 0, 64, 6000), ("plain", 5, 60, 2500),
         ("learned", 1, 24, 1800), ("learned", 2, 32, 67), ("learned", 2, 36, 1801), ("learned", 5, 36, 6000),
         ("learned", 4, 44, 6001), ("learned", 3, 60, 300), ("learned", 1, 96, 6000), ("learned", 4, 68, 1800),
         ("half", 0, 24, 401), ("half", 0, 32, 6001), ("half", 0, 36, 6001), ("half", 2, 44, 6000),
         ("half", 4, 28, 64), ("half", 5, 60, 2500), ("half", 0, 92, 129), ("half", 0, 96, 1801), ("half", 0, 84, 64)]


def mixed_quality(oracle, rate, z, frames, seed):
    """noise from none (valid codewords) to more than the code corrects"""
    parts = [inputs.frames(oracle, rate, z, frames // 4 + 4, inputs.SWEEP_EBNO[rate] + db, seed + k)[2]
             for k, db in enumerate((-1.5, -0.25, 0.5, 9.0))]
    return np.ascontiguousarray(np.stack(parts, 1).reshape(-1, parts[0].shape[1])[:frames])


def handle(wl, kind, rate, z, cap, weights):
    if kind == "plain":
        return wl.Decoder(rate, z, cap)
    return wl.LearnedDecoder(rate, z, 8, weights, cap, wl.LMS_F16X2 if kind == "half" else wl.LMS_F32)


def reference(oracle, kind, rate, z, cap, weights, llr):
    if kind == "plain":
        post, hard, _, it, fail = oracle.decode(rate, z, llr, cap)
        return post, hard, it, fail
    decode = oracle.learned16_decode if kind == "half" else oracle.learned_decode
    return decode(rate, z, 8, weights, llr, cap=cap)


def check(cuda, dec, llr, ref, in_place=False):
    d_llr = cuda.from_numpy(llr).cuda()
    hard = cuda.full(llr.shape, 7, dtype=cuda.int8, device="cuda")
    post = d_llr if in_place else cuda.empty_like(d_llr)
    status = cuda.full((llr.shape[0],), -1, dtype=cuda.int32, device="cuda")
    dec.decode_device(d_llr, hard, post, status)
    cuda.cuda.synchronize()
    po, do, it, fail = ref
    st = status.cpu().numpy()
    assert (st & 0xFFFF == it).all() and (st >> 16 == fail).all()
    assert (hard.cpu().numpy() == do).all()
    assert (post.cpu().numpy().view(np.uint32) == po.view(np.uint32)).all()


@pytest.mark.parametrize("kind,rate,z,frames", CASES)
def test_unit_decoders_match_oracle(wl, cuda, oracle, kind, rate, z, frames):
    weights = None if kind == "plain" else random_weights(oracle, rate, z, 8, 70 + rate + z)[0]
    llr = mixed_quality(oracle, rate, z, frames, 4000 + 10 * z + rate)
    for cap, in_place in ((7, False), (1, True)):
        ref = reference(oracle, kind, rate, z, cap, weights, llr)
        check(cuda, handle(wl, kind, rate, z, cap, weights), llr, ref, in_place)
        if cap == 7:
            assert ref[2].min() == 0 and ref[2].max() == 7 and len(set(ref[2].tolist())) > 3


def test_unit_decoder_with_cap_zero_and_expired_waits(wl, cuda, oracle):
    rate, z = 0, 28
    llr = mixed_quality(oracle, rate, z, 500, 5)
    check(cuda, wl.Decoder(rate, z, 0), llr, reference(oracle, "plain", rate, z, 0, None, llr))
    dec = wl.Decoder(rate, z, 10)
    d_llr = cuda.from_numpy(llr).cuda()
    hard = cuda.empty(llr.shape, dtype=cuda.int8, device="cuda")
    dec.set_wait_limit(0)
    dec.decode_device(d_llr, hard)
    with pytest.raises(wl.LdpcError) as e:
        dec.synchronize()
    assert e.value.code == wl.ERR_TIMEOUT
    dec.set_wait_limit(wl.WAIT_LIMIT_DEFAULT_US)
    check(cuda, dec, llr, reference(oracle, "plain", rate, z, 10, None, llr))
    dec.synchronize()


@pytest.mark.parametrize("kind,scale", [("plain", None), ("learned", None), ("learned", 0.0), ("learned", -0.5),
                                        ("half", None), ("half", 0.0)])
def test_unit_decoders_on_infinite_llrs(wl, cuda, oracle, kind, scale):
    """known bits as infinite LLRs: a third of them in every other frame, all in every third (with
    a scale that is not positive their messages are 0, otherwise only frames without infinite errors)"""
    rate, z, frames = 2, 52, 640
    weights = None if kind == "plain" else random_weights(oracle, rate, z, 8, 9)[0]
    if scale is not None:
        weights[0] = scale
    elif weights is not None:
        weights[0] = np.abs(weights[0]) + np.float32(0.125)
    llr = mixed_quality(oracle, rate, z, frames, 77)
    n = llr.shape[1]
    inf = np.float32(np.inf)
    llr[::2, : n // 3] = np.where(llr[::2, : n // 3] > 0, inf, -inf)
    rows = np.arange(0, frames, 3) if scale is not None else np.arange(3, frames, 4)
    llr[rows] = np.where(llr[rows] > 0, inf, -inf)
    check(cuda, handle(wl, kind, rate, z, 7, weights), llr, reference(oracle, kind, rate, z, 7, weights, llr))
