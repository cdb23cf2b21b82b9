"""The group kernels of the solves and of the reverse sweeps on the CPU, a
thread at a time, with every index checked (address and undefined-behaviour
sanitizers) and uninitialised locals filled with a pattern: no access outside
the arrays a launch is given nor outside a block's shared memory, no thread that
waits for ever, and the numbers of the single-pair solves and sweeps to
rounding.  The kernels' device code is taken from their files up to the launch
code; static shared arrays become static ones."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import GOLDEN, ROOT
from yspec_b200 import workloads as W

SRC = Path(__file__).resolve().parent / "device_on_host"
CSRC = ROOT / "yspec_b200" / "csrc"
LIBDIR = ROOT / "yspec_b200" / "lib"
CUDA_INC = Path("/usr/local/cuda/include")
BUILDS = {"solve": ("k_solve_group.cu", "using GroupFn"), "adjoint": ("k_group_adjoint.cu", "using AdjFn")}


@pytest.fixture(scope="module")
def checkers(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers missing")
    out = tmp_path_factory.mktemp("group_kernels")
    running = {}
    for name, (src, end) in BUILDS.items():
        text = (CSRC / src).read_text()
        assert end in text
        part = out / f"{name}_device.cuh"
        part.write_text(text[:text.index(end)].replace("    __shared__ ", "    static ")
                        + "}  // namespace\n}  // inline namespace\n}  // namespace ysg\n")
        running[name] = subprocess.Popen(
            [gxx, "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-fpermissive", "-ftrivial-auto-var-init=pattern",
             "-fsanitize=address,undefined", "-fno-sanitize-recover=undefined", f'-DGROUP_KERNELS="{part}"',
             f"-I{SRC}", f"-I{CUDA_INC}", f"-I{CSRC}", f"-I{ROOT / 'include'}", str(SRC / f"group_{name}_check.cpp"),
             "-o", str(out / name), f"-L{LIBDIR}", "-lyspec_b200", f"-Wl,-rpath,{LIBDIR}"],
            stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)
    for name, p in running.items():
        _, err = p.communicate()
        assert p.returncode == 0, (name, err[-2000:])
    return out


CASES = [dict(grav=g, model_file=d, depth_s=s, depth_r=r, out=2, cor=1)
         for g, d, s, r in [(0, "model200.deck", 100.0, 0.0), (1, "model200_ocean.deck", 20.0, 250.0),
                            (2, "model200_fic.deck", 2880.0, 3.0), (2, "model200_ocean.deck", 3.0, 3.0),
                            (0, "model200_fic.deck", 20.0, 250.0), (1, "model200.deck", 150.0, 150.0),
                            (2, "examples/prem.200", 600.0, 400.0)]]


@pytest.mark.parametrize("name", sorted(BUILDS))
@pytest.mark.parametrize("i", range(len(CASES)))
def test_on_the_cpu(checkers, tmp_path, name, i):
    kw = dict(CASES[i], model_file=str(GOLDEN / CASES[i]["model_file"]))
    p = W.config("c1", seed=5, nrec=1, fmax=2.5, f21=1.5, f22=2.0, ats=1, lmin=0, lmax=70, dt=40.0, **kw)[0]
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0:detect_stack_use_after_return=0")
    res = subprocess.run([str(checkers / name), str(p.write(tmp_path / "e.in"))], capture_output=True, text=True,
                         timeout=900, env=env)
    assert res.returncode == 0, res.stdout + res.stderr[-3000:]
