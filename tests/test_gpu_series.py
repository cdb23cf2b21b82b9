"""The time-series kernels (k_ifft.cu) against a plain restatement of the
reference's radix-2 network (module_fourier.f90:7-50, single-precision pi in
the twiddle angles) over the transform lengths: a row per thread group (8 and
up), one tile per block, clusters of 2, 4 and 8 blocks, tiles of 8192, and the
two passes beyond 65536; full and narrow bands, with and without a taper,
traces cut short of the row and rows of one or several receivers.

Tolerance: 18 stages of complex multiply-adds at 1.1e-16 each, and the
post-processing, give some 1e-14 relative to a row's norm; 1e-13 is asked for.
"""
import ctypes as C

import numpy as np
import pytest

from yspec_b200 import native as N

pytestmark = pytest.mark.gpu

PI_D = float(np.float32(3.14159265358979323846))


def network(x):
    n = x.shape[-1]
    p = n.bit_length() - 1
    idx = np.arange(n)
    rev = np.zeros(n, dtype=int)
    for b in range(p):
        rev |= ((idx >> b) & 1) << (p - 1 - b)
    d = x[..., rev].copy()
    mh = 1
    while mh < n:
        w = np.exp(1j * (np.arange(mh) * (PI_D / mh)))
        v = d.reshape(d.shape[:-1] + (n // (2 * mh), 2, mh))
        a, b = v[..., 0, :].copy(), v[..., 1, :] * w
        v[..., 0, :] = a + b
        v[..., 1, :] = a - b
        mh *= 2
    return d


def expected(t, spec, az, nout):
    n, nr = t.nt, t.nr
    filt = np.ones(n // 2 + 1)
    if t.f22 != 0.0:
        w = np.arange(n // 2 + 1) * t.df
        filt = np.where(w < t.f11, 0.0, np.where(w < t.f12, 0.5 * (1 - np.cos(PI_D * (w - t.f11) / (t.f12 - t.f11))),
                        np.where(w < t.f21, 1.0, np.where(w < t.f22, 0.5 * (1 - np.cos(PI_D * (t.f22 - w) / (t.f22 - t.f21))), 0.0))))
    row = np.zeros((3, nr, n), dtype=complex)
    for b in range(t.i1 - 1, t.i2):
        if b <= n // 2:
            row[:, :, b] = spec[:, :, b - t.i1 + 1] * filt[b]
            if 0 < b < n - b:
                row[:, :, n - b] = np.conj(row[:, :, b])
    y = network(row)[..., :nout].real / (t.dt * n)
    tt = np.arange(nout) * t.dt
    y = y * np.exp(t.ep * tt) * t.amp_norm
    out = np.empty((nr, 4, nout))
    ca, sa = np.cos(az)[:, None], np.sin(az)[:, None]
    out[:, 0] = tt * t.t_norm
    out[:, 1] = y[0]
    out[:, 2] = -(y[1] * ca) + y[2] * sa
    out[:, 3] = y[1] * sa + y[2] * ca
    return out


@pytest.mark.parametrize("taper", [False, True])
@pytest.mark.parametrize("n", [8, 16, 32, 64, 512, 1024, 2048, 4096, 8192, 16384, 32768, 65536, 131072, 262144])
def test_against_network(n, taper):
    import torch

    rng = np.random.default_rng(n + taper)
    dev = torch.device("cuda", 0)
    i1, i2 = (2, n // 2 + 1) if not taper else (2, max(3, n // 5))
    nr = 1 if n > 100000 else 5
    t = N.YsgTime(nt=n, i1=i1, i2=i2, nr=nr, df=0.01, dt=0.7, ep=0.5 / n, tout=0.7 * (0.43 if taper else 2.0) * n,
                  t_norm=3.0, amp_norm=0.25)
    if taper:
        t.f11, t.f12, t.f21, t.f22 = 0.01, 0.03, 0.01 * (0.6 * i2), 0.01 * (0.9 * i2 + 0.5)
    spec = rng.standard_normal((3, nr, i2 - i1 + 1)) + 1j * rng.standard_normal((3, nr, i2 - i1 + 1))
    az = rng.uniform(0, 2 * np.pi, nr)
    nout = N.lib().ysg_trace_rows(C.byref(t))
    d = torch.from_numpy(np.stack([spec.real, spec.imag], -1)).to(dev)
    d_az = torch.from_numpy(az).to(dev)
    out = torch.full((nr, 4, nout), float("nan"), dtype=torch.float64, device=dev)
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
