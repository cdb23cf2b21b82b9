"""The coefficient matrices of the group solves and their reverse sweeps
(ysg_group.cuh) against the same expressions in extended precision, on the
CPU, from 0.1 to 128 mHz: tests/device_on_host/group_coef_check.cpp compiles
the device headers as host C++ and states the bounds.  At low frequencies the
terms of an entry differ in size by more than ten, so an entry formed with a
term that is taken out again loses digits that a comparison of traces at
1e-9 does not see."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import GOLDEN, ROOT

SRC = Path(__file__).resolve().parent / "device_on_host"
LIBDIR = ROOT / "yspec_b200" / "lib"
CUDA_INC = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers missing")
    out = tmp_path_factory.mktemp("group_coef") / "group_coef_check"
    res = subprocess.run([gxx, "-std=c++17", "-O1", "-w", "-ffp-contract=off", f"-I{CUDA_INC}",
                          f"-I{ROOT / 'yspec_b200' / 'csrc'}", f"-I{ROOT / 'include'}",
                          str(SRC / "group_coef_check.cpp"), "-o", str(out), f"-L{LIBDIR}", "-lyspec_b200",
                          f"-Wl,-rpath,{LIBDIR}"], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
    return out


@pytest.mark.parametrize("lowest", ["0.1", "1.0"])
@pytest.mark.parametrize("deck", ["model200.deck", "model200_ocean.deck", "model200_fic.deck", "model400.deck",
                                  "examples/prem.200"])
def test_entries(checker, deck, lowest):
    res = subprocess.run([str(checker), str(GOLDEN / deck), lowest], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
