"""The mixed decoder without a tuning of the caller's own: it sizes its work
items by the batch. At both sides of every line the decoded batch equals the
(rate, z)-specialised decoders' (equality); a tuning that was set stays."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 600, 601, 12001, 45001])
def test_untuned_batches_match_specialised_decoders(wl, cuda, frames):
    from wimax_ldpc_lib_b200.mixed_batch import build_batch, decode_by_code
    variants, offsets, llr, _, groups = build_batch(frames, seed=frames)
    ref_hard = cuda.zeros(llr.numel(), dtype=cuda.int8, device="cuda")
    ref_status = cuda.zeros(frames, dtype=cuda.int32, device="cuda")
    decode_by_code(groups, llr, ref_hard, ref_status)
    mixed = wl.MixedDecoder(10)
    hard = cuda.zeros_like(ref_hard)
    status = cuda.full((frames,), -1, dtype=cuda.int32, device="cuda")
    mixed.decode_device(variants, offsets, llr, hard, None, status)
    mixed.synchronize()
    assert cuda.equal(hard, ref_hard) and cuda.equal(status, ref_status)


def test_a_set_tuning_is_not_replaced(wl, cuda):
    from wimax_ldpc_lib_b200.mixed_batch import build_batch
    variants, offsets, llr, _, _ = build_batch(700, seed=9)
    hard = cuda.zeros(llr.numel(), dtype=cuda.int8, device="cuda")
    mixed = wl.MixedDecoder(10)
    mixed.set_config(96, 5)
    mixed.decode_device(variants, offsets, llr, hard)
    mixed.synchronize()
    assert mixed.tuning() == (96, wl.MIXED_MSG_REGISTERS, 5, wl.MIXED_CONCURRENT)
