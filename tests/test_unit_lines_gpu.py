"""The large-batch decoders at batch sizes from which a code goes to them
(unit_launch.cuh) and one below, for rows of 6 to 20 edges and units of one
warp and several: bit for bit against the oracle."""
import numpy as np
import pytest

from test_learned16_gpu import random_weights
from test_unit_decode_gpu import check, handle, mixed_quality, reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,rate,z,line", [
    ("plain", 1, 32, 15000), ("plain", 2, 72, 6000), ("plain", 3, 88, 1800), ("learned", 1, 24, 15000),
    ("learned", 4, 92, 1800), ("learned", 5, 76, 6000), ("learned", 1, 60, 400), ("half", 4, 28, 400),
    ("half", 3, 36, 15000), ("half", 5, 44, 6000)])
def test_both_sides_of_a_line(wl, cuda, oracle, kind, rate, z, line):
    weights = None if kind == "plain" else random_weights(oracle, rate, z, 8, 70 + rate + z)[0]
    llr = mixed_quality(oracle, rate, z, line, 6000 + 10 * z + rate)
    ref = reference(oracle, kind, rate, z, 6, weights, llr)
    dec = handle(wl, kind, rate, z, 6, weights)
    check(cuda, dec, llr, ref)
    check(cuda, dec, llr[:-1], tuple(np.ascontiguousarray(a[:-1]) for a in ref), in_place=True)
