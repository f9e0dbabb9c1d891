"""The fused z kernels (k_zpipe FP32, k_zws FP64) at the edges of their packing.

Every z length they serve (odd and even elements per lane), with truncations
that keep the z Nyquist plane, all modes but it, and few modes; one and two
scalars and the drift term; and the FP64 512-point lines whose staging does
not fit (drift term; all modes kept with two scalars).  Two steps against the
staged z kernel (k_zphys); the bounds are those of the kernel variants (1e-13
FP64, 2e-6 FP32).
"""
import numpy as np
import pytest

from _util import rel_l2, to_dev, to_host

CASES = [
    # nx, ny, nz, scalars, alpha, alias
    (64, 16, 64, 1, 0.0, 1.0),       # kz = nz/2 kept
    (96, 16, 96, 2, 0.05, 1.0),
    (128, 8, 192, 2, 0.0, 2 / 3),    # few modes along z
    (256, 16, 128, 1, 0.0, 1.0),     # every mode along z
    (256, 8, 256, 2, 0.0, 1.0),
    (64, 48, 512, 1, 0.0, 2 / 3),
    (512, 8, 512, 2, 0.0, 1.0),      # FP64: lines read from global memory
    (384, 12, 512, 2, 0.05, 2 / 3),  # FP64: likewise
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny,nz,ns,alpha,alias", CASES)
def test_z_kernels_match_staged(torch_cuda, nx, ny, nz, ns, alpha, alias, precision):
    import gnss_b200 as G
    torch = torch_cuda
    dt = np.complex128 if precision == 0 else np.complex64
    rng = np.random.default_rng(5)
    init = G.jet_initial_state(nx, ny, nz, n_scalars=ns, seed=2, noise_kmax=3.0)
    init = [(f + np.fft.rfftn(1e-2 * rng.standard_normal((nx, ny, nz))).transpose(1, 0, 2)).astype(dt) for f in init]
    out = []
    for variant in (G.GNSS_VARIANT_REGISTER, G.GNSS_VARIANT_STAGED):
        with G.Context(nx=nx, ny=ny, nz=nz, re=500.0, dt=5e-4, n_scalars=ns, alpha=alpha, alias_filter=alias,
                       precision=precision) as ctx:
            ctx.set_option(G.GNSS_OPT_ZVARIANT, variant)
            assert ctx.get_option(G.GNSS_OPT_ZKERNEL) == variant
            st = [to_dev(torch, a) for a in init]
            hi = [torch.zeros_like(st[0]) for _ in st]
            ctx.de_alias(st)
            for s in range(2):
                ctx.solver_ps(st, hi, euler=(s == 0))
            ctx.check()
            out.append([to_host(t) for t in st + hi])
    tol = 1e-13 if precision == 0 else 2e-6
    for a, b in zip(*out):
        assert np.isfinite(a.view(a.real.dtype)).all()
        assert rel_l2(a, b) <= tol
