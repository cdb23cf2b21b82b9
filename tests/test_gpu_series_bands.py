"""Time series of narrow bands and of several chunks of receivers.

A band that ends below an eighth of the row takes a first round of its own
(first_round of k_ifft.cu): bands whose last bin is the last one below that
line, the first one on it (the general round) and well below it, for every row
length from one thread's worth to tiles of 8192 in clusters of 8.  Rows beyond
65536 go through the compiled-in array in chunks of receivers, which take the
taper and e^{eps t} in turn: two receivers per chunk at 131072, one at 262144.
Restatement and tolerance as in test_gpu_series.py."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_series import expected
from yspec_b200 import native as N

pytestmark = pytest.mark.gpu


def _check(n, i1, i2, nr, taper, part):
    import torch

    rng = np.random.default_rng(n + i2 + taper)
    t = N.YsgTime(nt=n, i1=i1, i2=i2, nr=nr, df=0.01, dt=0.7, ep=0.5 / n, tout=0.7 * part * n, t_norm=3.0, amp_norm=0.25)
    if taper:
        t.f11, t.f12, t.f21, t.f22 = 0.01, 0.03, 0.01 * (0.6 * i2), 0.01 * (0.9 * i2 + 0.5)
    spec = rng.standard_normal((3, nr, i2 - i1 + 1)) + 1j * rng.standard_normal((3, nr, i2 - i1 + 1))
    az = rng.uniform(0, 2 * np.pi, nr)
    nout = N.lib().ysg_trace_rows(C.byref(t))
    d = torch.from_numpy(np.stack([spec.real, spec.imag], -1)).cuda()
    d_az = torch.from_numpy(az).cuda()
    out = torch.full((nr, 4, nout), float("nan"), dtype=torch.float64, device="cuda")
    m = C.c_int()
    rc = N.lib().ysg_traces_noalloc(C.byref(t), d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d_az.data_ptr(),
                                    out.data_ptr(), C.byref(m), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and m.value == nout
    torch.cuda.synchronize()
    got, want = out.cpu().numpy(), expected(t, spec, az, nout)
    np.testing.assert_array_equal(got[:, 0], want[:, 0])
    for k in range(nr):
        for c in range(1, 4):
            assert np.linalg.norm(got[k, c] - want[k, c]) <= 1e-13 * np.linalg.norm(want[k, c]), (k, c)


@pytest.mark.parametrize("n", [16, 32, 64, 128, 512, 2048, 4096, 8192, 16384, 32768, 65536])
@pytest.mark.parametrize("band", ["below", "at", "narrow", "lowest"])
def test_narrow_bands(n, band):
    i2 = {"below": n // 8, "at": n // 8 + 1, "narrow": max(1, n // 20), "lowest": 1}[band]
    _check(n, min(2, i2), i2, 3, band == "narrow" and n >= 512, 0.43 if band == "below" else 2.0)


@pytest.mark.parametrize("n,nr", [(131072, 5), (262144, 2)])
@pytest.mark.parametrize("taper", [False, True])
def test_chunks_of_receivers(n, nr, taper):
    _check(n, 2, n // 10, nr, taper, 0.7)
