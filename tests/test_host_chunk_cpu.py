"""How host-buffer batches are cut (host_batch.h): pageable buffers, whose copies
overlap with nothing, in chunks of 8192 frames, pinned ones in up to eight."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def chunks(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_chunk") / "chunk")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include",
                           f"-I{ROOT}/wimax_ldpc_lib_b200/csrc", f"{ROOT}/tests/cpp/host_chunk.cc", "-o", exe])

    def ask(cases):
        args = [str(int(x)) for c in cases for x in c]
        return [int(x) for x in subprocess.check_output([exe] + args).split()]
    return ask


FRAMES = [1, 2, 1023, 1024, 1025, 1500, 2605, 3100, 8191, 8192, 8193, 12000, 65535, 65536, 65537, 10**6]
CODES = [24 * z for z in (24, 48, 60, 96)]


def test_pageable_batches_are_not_cut_below_8192_frames(chunks):
    cases = [(f, n, False, post) for f in FRAMES for n in CODES for post in (False, True)]
    assert chunks(cases) == [min(f, 8192) for f, _, _, _ in cases]


def test_pinned_batches(chunks):
    cases = [(f, n, True, post) for f in FRAMES for n in CODES for post in (False, True)]
    for (f, n, _, post), chunk in zip(cases, chunks(cases)):
        assert 1 <= chunk <= min(f, 8192)
        if chunk < f:   # cut: at most eight chunks up to 65,536 frames, none too short to pay for itself
            assert -(-f // chunk) <= 8 or chunk == 8192
            assert chunk >= 1024 and f * n * 4 >= 6000000
            assert post or chunk * n * 4 > 7000000 - n * 4
        else:
            assert f <= 1024 or f * n * 4 <= 7000000 + n * 4
