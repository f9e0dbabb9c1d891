"""The spectral sums of gnss_stats and gnss_turb_stats (k_stats_partial,
k_turb_partial, k_sums_final) and the mean profiles (k_yprof), against numpy,
on states with every mode of the spectrum present or only a few.

Sizes: fewer modes than the grid has threads, a few modes more than one and
two rounds of it, several rounds; the shortest and the longest y axis.  The
sums are of non-negative FP64 terms (about 10 roundings each) with fewer than
200 uncompensated additions after the per-thread sums: 1e-13 relative, also for
an FP32 state, whose values enter exactly.  A profile value is a compensated sum
of ny terms: 1e-15 of the sum of their magnitudes, 1e-7 with FP32 twiddles.
"""
import numpy as np
import pytest

from _util import to_dev

CASES = [
    # shape, precision, n_scalars, modes left in (None: all)
    ((8, 8, 8), 0, 1, None),
    ((48, 128, 32), 0, 2, None),     # 104 448 modes: less than one round
    ((96, 64, 48), 1, 2, None),      # 153 600: one round and a part
    ((64, 512, 24), 0, 1, 5),        # 425 984, the longest profile, a handful of modes
    ((128, 12, 384), 1, 1, None),    # 296 448
    ((512, 16, 128), 0, 2, None),    # 532 480: several rounds
]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,precision,ns,few", CASES,
                         ids=[f"{'x'.join(map(str, c[0]))}_{'fp64' if c[1] == 0 else 'fp32'}_s{c[2]}"
                              f"{'_sparse' if c[3] else ''}" for c in CASES])
def test_sums_and_profiles_against_numpy(torch_cuda, shape, precision, ns, few):
    import gnss_b200 as G
    torch = torch_cuda
    nx, ny, nz = shape
    nz2 = nz // 2 + 1
    rng = np.random.default_rng(nx + 7 * ny + nz)
    cdt = np.complex128 if precision == 0 else np.complex64
    f = [(rng.standard_normal((ny, nx, nz2)) + 1j * rng.standard_normal((ny, nx, nz2))).astype(cdt)
         for _ in range(3 + ns)]
    if few:
        keep = np.zeros(ny * nx * nz2, bool)
        keep[rng.integers(0, keep.size, few)] = True
        keep[[0, keep.size - 1]] = True
        for a in f:
            a[~keep.reshape(a.shape)] = 0
    k = [np.fft.fftfreq(n, 1.0 / n) for n in (nx, ny)]
    kz = np.arange(nz2, dtype=float)
    kz[-1] = -kz[-1]
    ksq = k[0][None, :, None] ** 2 + k[1][:, None, None] ** 2 + kz[None, None, :] ** 2
    wt = np.full(nz2, 2.0)
    wt[[0, -1]] = 1.0
    m = [np.abs(a.astype(np.complex128)) ** 2 for a in f]
    e = m[0] + m[1] + m[2]
    n2 = float(nx * ny * nz) ** 2
    with G.Context(nx=nx, ny=ny, nz=nz, re=100.0, sc=0.5, sc_c=2.0, n_scalars=ns, precision=precision) as ctx:
        L = 2 * np.pi
        assert abs(ctx.cfg.lx - L) < 1e-12 and abs(ctx.cfg.ly - L) < 1e-12 and abs(ctx.cfg.lz - L) < 1e-12
        st = [to_dev(torch, a) for a in f]
        stats = list(ctx.stats(st).values())
        got, prof = ctx.turb_stats(st)
    nu = 1.0 / 100.0
    ke, eps = (wt * e).sum() / n2 / 2, nu * (wt * ksq * e).sum() / n2
    chi = [2 * nu / sc * (wt * ksq * a).sum() / n2 for sc, a in zip((0.5, 2.0), m[3:])]
    var = [((wt * a).sum() - a[0, 0, 0]) / n2 for a in m[3:]]
    want = [ke, ke * 2 / 3, eps, chi[0], chi[1] if ns == 2 else 0.0, var[0], var[1] if ns == 2 else 0.0]
    np.testing.assert_allclose(stats, want, rtol=1e-13)
    with np.errstate(divide="ignore"):
        integral = (wt * np.where(ksq > 0, e / (2 * np.sqrt(ksq)), 0.0)).sum() / n2
    np.testing.assert_allclose([got["ke"], got["epsilon"], got["chi"], got["l"]],
                               [ke, eps, chi[0], 3 * np.pi / 4 * integral / ke], rtol=1e-13)
    tol = 1e-15 if precision == 0 else 1e-7
    for q, a in enumerate(f):
        line = a[:, 0, 0].astype(np.complex128)
        ref = np.fft.ifft(line).real * ny / (nx * ny * nz)
        assert np.abs(prof[q] - ref).max() <= tol * np.abs(line).sum() / (nx * ny * nz) + 1e-300, q
    assert not prof[3 + ns:].any()
