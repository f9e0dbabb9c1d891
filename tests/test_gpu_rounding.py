"""Rounding error of the full transforms, axis by axis.

Random fields on grids with one long axis (the others have 8 points), forward
and inverse, against 80-bit transforms on the host.  The bound is the error
that the table-driven radix-8 passes have on the same fields (relative RMS, 48
fields each, below), and 1% more: the two radix plans of a length differ by
less than that, and the sampling error of an RMS over 48 fields is 0.3%.
Twiddles formed as products of table entries raise it by 2 to 10%, a factor
and a sum rounded apart in the small transforms by 1 to 4%, twiddles inside
the 6-point transform by 2%.
"""
import numpy as np
import pytest

from _util import to_host

FIELDS = 48
# precision, axis -> length -> error of the forward, of the inverse transform
BOUND = {
    (0, 0): {48: (2.035e-16, 2.036e-16), 64: (2.097e-16, 2.017e-16), 96: (2.107e-16, 2.128e-16),
             128: (2.239e-16, 2.143e-16), 192: (2.244e-16, 2.216e-16), 256: (2.388e-16, 2.285e-16),
             384: (2.372e-16, 2.310e-16), 512: (2.506e-16, 2.370e-16)},
    (0, 1): {48: (2.030e-16, 1.988e-16), 64: (2.098e-16, 1.998e-16), 96: (2.103e-16, 2.080e-16),
             128: (2.241e-16, 2.129e-16), 192: (2.243e-16, 2.161e-16), 256: (2.396e-16, 2.271e-16),
             384: (2.372e-16, 2.260e-16), 512: (2.508e-16, 2.355e-16)},
    (1, 0): {48: (1.099e-07, 1.072e-07), 64: (1.074e-07, 1.076e-07), 96: (1.190e-07, 1.135e-07),
             128: (1.167e-07, 1.177e-07), 192: (1.269e-07, 1.202e-07), 256: (1.193e-07, 1.188e-07),
             384: (1.262e-07, 1.215e-07), 512: (1.283e-07, 1.268e-07)},
    (1, 1): {48: (1.097e-07, 1.080e-07), 64: (1.071e-07, 1.082e-07), 96: (1.195e-07, 1.145e-07),
             128: (1.169e-07, 1.177e-07), 192: (1.274e-07, 1.207e-07), 256: (1.193e-07, 1.195e-07),
             384: (1.263e-07, 1.224e-07), 512: (1.284e-07, 1.274e-07)},
    (0, 2): {48: (2.089e-16, 2.039e-16), 64: (2.162e-16, 2.084e-16), 96: (2.165e-16, 2.146e-16),
             128: (2.297e-16, 2.221e-16), 192: (2.304e-16, 2.243e-16), 256: (2.378e-16, 2.299e-16),
             384: (2.434e-16, 2.353e-16), 512: (2.535e-16, 2.460e-16)},
    (1, 2): {48: (1.125e-07, 1.102e-07), 64: (1.099e-07, 1.105e-07), 96: (1.192e-07, 1.156e-07),
             128: (1.163e-07, 1.168e-07), 192: (1.236e-07, 1.210e-07), 256: (1.216e-07, 1.218e-07),
             384: (1.294e-07, 1.262e-07), 512: (1.271e-07, 1.269e-07)},
}


@pytest.mark.gpu
@pytest.mark.parametrize("precision,axis,n", [(p, a, n) for (p, a), t in BOUND.items() for n in t])
def test_transform_rounding(torch_cuda, precision, axis, n):
    import scipy.fft
    import gnss_b200 as G
    torch = torch_cuda
    shape = [8, 8, 8]
    shape[axis] = n
    nx, ny, nz = shape
    real, cplx = (np.float64, np.complex128) if precision == 0 else (np.float32, np.complex64)
    u = np.random.default_rng(axis * 1000 + n).standard_normal((FIELDS, nx, ny, nz)).astype(real)
    spec = np.fft.rfftn(u.astype(np.float64), axes=(1, 2, 3)).astype(cplx)
    want_f = scipy.fft.rfftn(u.astype(np.longdouble), axes=(1, 2, 3)).transpose(0, 2, 1, 3)
    t = scipy.fft.ifftn(spec.astype(np.clongdouble), axes=(1, 2))
    t[..., 0].imag = 0
    t[..., -1].imag = 0
    want_i = scipy.fft.irfft(t, n=nz, axis=3)
    got_f, got_i = [], []
    with G.Context(nx=nx, ny=ny, nz=nz, precision=precision) as ctx:
        for a, s in zip(u, spec):
            buf = np.zeros((nx, ny, 2 * (nz // 2 + 1)), dtype=real)
            buf[..., :nz] = a
            f = torch.from_numpy(buf.reshape(-1).view(cplx).reshape(ny, nx, nz // 2 + 1)).cuda()
            ctx.forward_transform(f)
            got_f.append(to_host(f))
            f = torch.from_numpy(np.ascontiguousarray(s.transpose(1, 0, 2))).cuda()
            ctx.inverse_transform(f)
            got_i.append(to_host(f).reshape(-1).view(real).reshape(nx, ny, -1)[..., :nz])
    for got, want, bound in zip((got_f, got_i), (want_f, want_i), BOUND[precision, axis][n]):
        got = np.array(got)
        err = float(np.sqrt((np.abs(got - want) ** 2).sum() / (np.abs(want) ** 2).sum()))
        assert err <= 1.01 * bound


# right-hand side (u, v, w, s) of a step on such fields with every transform's twiddles exact or one product away
STEP_BOUND = {
    (64, 64, 64, 0): (4.443e-16, 4.487e-16, 4.367e-16, 3.895e-16),
    (64, 64, 512, 0): (4.562e-16, 4.526e-16, 4.454e-16, 3.947e-16),
    (64, 64, 256, 1): (2.628e-07, 2.645e-07, 2.565e-07, 2.464e-07),
    (64, 64, 512, 1): (2.882e-07, 2.859e-07, 2.850e-07, 2.707e-07),
}


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,precision", list(STEP_BOUND))
def test_step_rounding(torch_cuda, nx, ny, nz, precision):
    """The history after an Euler step (the projected nonlinear term) against 80-bit floats."""
    import scipy.fft
    import gnss_b200 as G
    torch = torch_cuda
    cplx = np.complex128 if precision == 0 else np.complex64
    rng = np.random.default_rng(nx * 1000003 + ny * 1009 + nz)
    kx = np.fft.fftfreq(nx, 1 / nx)[None, :, None]
    ky = np.fft.fftfreq(ny, 1 / ny)[:, None, None]
    kz = np.arange(nz // 2 + 1.0)[None, None, :]
    k2 = kx * kx + ky * ky + kz * kz
    keep = k2 <= (2 / 3 * nx / 2) ** 2
    st = [np.where(keep, np.fft.rfftn(rng.standard_normal((nx, ny, nz))).transpose(1, 0, 2) * (1 + k2 / 64) ** -1.4,
                   0).astype(cplx) for _ in range(4)]
    with G.Context(nx=nx, ny=ny, nz=nz, precision=precision, re=500.0, dt=1e-3) as ctx:
        dev = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in st]
        hist = [torch.zeros_like(t) for t in dev]
        ctx.solver_ps(dev, hist, euler=True)
        got = [to_host(t) for t in hist]

    def phys(f):
        t = scipy.fft.ifftn(f.transpose(1, 0, 2), axes=(0, 1))
        t[..., 0].imag = 0
        t[..., -1].imag = 0
        return scipy.fft.irfft(t, n=nz, axis=2)

    def spec(p):
        return scipy.fft.rfftn(p).transpose(1, 0, 2)

    u, v, w, s = (f.astype(np.clongdouble) for f in st)
    up, vp, wp = phys(u), phys(v), phys(w)
    o1, o2, o3 = (phys(1j * t) for t in (ky * w - kz * v, kz * u - kx * w, kx * v - ky * u))
    n = [spec(o2 * wp - o3 * vp), spec(o3 * up - o1 * wp), spec(o1 * vp - o2 * up)]
    pr = (kx * n[0] + ky * n[1] + kz * n[2]) / np.maximum(k2, 1).astype(np.longdouble)
    want = [k * pr - f for k, f in zip((kx, ky, kz), n)]
    want.append(-spec(up * phys(1j * kx * s) + vp * phys(1j * ky * s) + wp * phys(1j * kz * s)))
    for g, x, bound in zip(got, want, STEP_BOUND[nx, ny, nz, precision]):
        x = np.where(keep, x, 0)
        x[0, 0, 0] = 0
        err = float(np.sqrt((np.abs(g - x) ** 2).sum() / (np.abs(x) ** 2).sum()))
        assert err <= 1.01 * bound
