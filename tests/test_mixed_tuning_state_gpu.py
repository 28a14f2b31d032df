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


def test_autotuning_a_small_batch_does_not_slow_it_down(wl, cuda, batches):
    """300 frames of 114 codes need items of one frame, a chunk that the autotuner's
    fixed ones (8 and more, twice the time) do not hold"""
    def fastest(mixed):
        times = []
        for _ in range(20):
            a, b = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            mixed.decode_device(*batches[300])
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    untuned = fastest(wl.MixedDecoder(10))
    mixed = wl.MixedDecoder(10)
    mixed.autotune(*batches[300], repeats=5)
    assert fastest(mixed) <= 1.3 * untuned
    fixed = wl.MixedDecoder(10)
    fixed.set_tuning(192, wl.MIXED_MSG_REGISTERS, 8)
    assert fastest(fixed) > 1.3 * untuned   # or this test shows nothing
    batches[13000][3].zero_()
    mixed.decode_device(*batches[13000])
    mixed.synchronize()
    assert cuda.equal(batches[13000][3], batches["hard"])
    assert mixed.tuning()[0::2] == batches["untuned"][0::2]
