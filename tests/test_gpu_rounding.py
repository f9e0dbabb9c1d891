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
