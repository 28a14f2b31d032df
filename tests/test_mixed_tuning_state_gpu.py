"""What one call leaves behind in a mixed decoder must not decide how later
batches are cut into work items, unless the caller chose it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batches(wl, cuda):
    """a batch that needs short items and one that needs longer ones, and the choice for it"""
    from wimax_ldpc_lib_b200.mixed_batch import build_batch
    out = {}
    for frames in (300, 13000):
        variants, offsets, llr, _, _ = build_batch(frames, seed=frames)
        out[frames] = (variants, offsets, llr, cuda.zeros(llr.numel(), dtype=cuda.int8, device="cuda"))
    fresh = wl.MixedDecoder(10)
    fresh.decode_device(*out[13000])
    fresh.synchronize()
    out["untuned"] = fresh.tuning()
    out["hard"] = out[13000][3].clone()
    return out


def holds_the_untuned_choice(cuda, mixed, batches):
    batches[13000][3].zero_()
    mixed.decode_device(*batches[13000])
    mixed.synchronize()
    assert mixed.tuning() == batches["untuned"]
    assert cuda.equal(batches[13000][3], batches["hard"])


@pytest.mark.parametrize("rows", [1, 2])
def test_rows_per_thread_after_a_small_batch(wl, cuda, batches, rows):
    mixed = wl.MixedDecoder(10)
    mixed.decode_device(*batches[300])
    mixed.set_rows_per_thread(rows)
    holds_the_untuned_choice(cuda, mixed, batches)
    assert mixed.rows_per_thread() == rows


@pytest.mark.parametrize("what", ["misaligned", "null", "bad code"])
def test_an_autotune_that_fails_chooses_nothing(wl, cuda, batches, what):
    mixed = wl.MixedDecoder(10)
    variants, offsets, llr, hard = batches[300]
    if what == "misaligned":
        llr = llr[1:]
    elif what == "null":
        llr = None
    else:
        variants = variants.clone()
        variants[7] = 114
    with pytest.raises(wl.LdpcError) as e:
        mixed.autotune(variants, offsets, llr, hard, repeats=1)
    assert e.value.code == wl.ERR_ARG
    holds_the_untuned_choice(cuda, mixed, batches)


def test_an_autotune_that_fails_keeps_a_set_tuning(wl, cuda, batches):
    mixed = wl.MixedDecoder(10)
    mixed.set_tuning(96, wl.MIXED_MSG_SHARED, 3, wl.MIXED_SERIAL)
    variants, offsets, llr, hard = batches[300]
    with pytest.raises(wl.LdpcError):
        mixed.autotune(variants, offsets, llr[1:], hard, repeats=1)
    mixed.decode_device(*batches[300])
    mixed.synchronize()
    assert mixed.tuning() == (96, wl.MIXED_MSG_SHARED, 3, wl.MIXED_SERIAL)
