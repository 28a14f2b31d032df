"""The ordering that units of the large-batch decoders rely on (unit_sync.cuh),
on a host model of a warp's votes and of asynchronous tensor memory."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("unit_sync") / "model")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-w", f"-I{ROOT}/wimax_ldpc_lib_b200/csrc",
                           f"{ROOT}/tests/cpp/unit_sync_model.cc", "-o", exe])
    return exe


@pytest.mark.parametrize("what", ["votes", "clear"])
def test_nothing_out_of_order(model, what):
    r = subprocess.run([model, what], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
