"""Tables of the time stage (k_time_tables of k_ifft.cu) to half a unit in the
last place: the functions they are formed with, compiled as host C++, against
extended precision (tests/device_on_host/tables_check.cpp states the bound),
and e^{eps t} as the device writes it, seen through the time series of a
constant row: a single bin at zero frequency passes every butterfly
unchanged, and the scale dt n is a power of two."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import ROOT
from yspec_b200 import native as N

SRC = Path(__file__).resolve().parent / "device_on_host"
CUDA_INC = Path("/usr/local/cuda/include")


def test_functions(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not (CUDA_INC / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers missing")
    exe = tmp_path / "tables_check"
    res = subprocess.run([gxx, "-std=c++17", "-O1", "-w", "-ffp-contract=off", f"-I{CUDA_INC}",
                          f"-I{ROOT / 'yspec_b200' / 'csrc'}", str(SRC / "tables_check.cpp"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 1024, 16384, 65536, 131072])
@pytest.mark.parametrize("total", [0.5, -3.0, 11.7])
def test_exponentials(n, total):
    import torch

    dt = 0.5
    t = N.YsgTime(nt=n, i1=1, i2=1, nr=1, df=0.01, dt=dt, ep=total / (n * dt), tout=2.0 * dt * n, t_norm=1.0,
                  amp_norm=1.0)
    d = torch.tensor([[1.0, 0.0]], dtype=torch.float64, device="cuda")
    az = torch.zeros(1, dtype=torch.float64, device="cuda")
    out = torch.full((1, 4, n), float("nan"), dtype=torch.float64, device="cuda")
    m = C.c_int()
    rc = N.lib().ysg_traces_noalloc(C.byref(t), d.data_ptr(), d.data_ptr(), d.data_ptr(), az.data_ptr(),
                                    out.data_ptr(), C.byref(m), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and m.value == n
    torch.cuda.synchronize()
    got = out[0, 1].cpu().numpy() * (dt * n)
    want = np.exp((t.ep * (np.arange(n) * dt)).astype(np.longdouble))
    ulp = np.spacing(want.astype(np.float64))
    assert np.max(np.abs(got.astype(np.longdouble) - want) / ulp) <= 0.502
