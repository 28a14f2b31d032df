"""The training kernel where it can go wrong: rows whose minimum is infinite
(known bits) under a scale that cuts the message off; batches of more frames
than CTAs, which add up several; one, two and three iterations, whose first and
last are not checkpointed. Loss and gradient against
the oracle, which takes the same decisions in fp32 and accumulates in double, at
the tolerances of test_learned_gpu.py."""
import numpy as np
import pytest

import inputs
from test_learned_oracle import random_weights

pytestmark = pytest.mark.gpu


def check(wl, oracle, rate, z, T, w, llr, cw):
    loss_o, g_o = oracle.learned_loss_grad(rate, z, T, w, llr, cw)
    loss_g, g_g = wl.LearnedDecoder(rate, z, T, weights=w).loss_grad(llr, cw)
    g_o = g_o.reshape(g_g.shape)
    assert np.isfinite(loss_o) and np.isfinite(g_o).all()
    assert abs(loss_g - loss_o) <= 1e-5 * abs(loss_o)
    assert np.linalg.norm(g_g - g_o) <= 1e-4 * np.linalg.norm(g_o)
    return g_g


@pytest.mark.parametrize("rate,z", [(0, 28), (0, 96), (2, 40), (2, 64)])
@pytest.mark.parametrize("scale", [-0.5, 0.0])
def test_a_message_cut_off_at_an_infinite_minimum_has_no_gradient(wl, cuda, oracle, rate, z, scale):
    """all bits of layer 0's rows known, so that its minima are infinite"""
    T = 8
    w, rs, cols = random_weights(oracle, rate, z, T, 11)
    w[0, :, 0] = scale
    w[1, 1::2, 0] *= -1   # offsets of both signs
    _, cw, llr = inputs.frames(oracle, rate, z, 24, 1.75, seed=90)
    for c in cols[:rs[1]]:
        known = slice(c * z, (c + 1) * z)
        llr[:, known] = np.where(cw[:, known] == 1, np.float32(np.inf), np.float32(-np.inf))
    g = check(wl, oracle, rate, z, T, w, llr, cw)
    assert (g[:, :, 0] == 0).all()


@pytest.mark.parametrize("rate,z,T,frames", [(0, 24, 1, 4000), (0, 96, 2, 2000), (5, 60, 3, 3000), (3, 36, 8, 3600),
                                             (4, 28, 1, 1), (0, 96, 3, 5), (1, 52, 2, 7)])
def test_several_frames_per_cta_and_few_iterations(wl, cuda, oracle, rate, z, T, frames):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    assert frames < 32 or frames > 24 * sms // ((z + 31) // 32)   # twice the warps that fit an SM
    w = random_weights(oracle, rate, z, T, 19 + T)[0]
    _, cw, llr = inputs.frames(oracle, rate, z, frames, 1.75, seed=91)
    check(wl, oracle, rate, z, T, w, llr, cw)
