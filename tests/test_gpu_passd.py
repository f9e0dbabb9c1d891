"""The direct x / y passes (k_passd) at the edges of what they serve.

Steps on grids whose x and y lengths take every radix plan (48 .. 512, two and
three stages, last radix 8, 6, 4 and 3), cubic and mixed, with the dealiasing
sphere inside the box and with kept Nyquist rows, FP64 (8 columns per tile)
and FP32 (16, packed pairs), one and two scalars and the drift term's
Laplacian: two steps against the staged passes (k_pass).  The scratch of the
direct run is filled with NaN first: what lies outside the sphere is neither
written nor read.  Two steps differ by round-off only; the bounds are those of
the kernel variants (1e-13 FP64, 2e-6 FP32).

Whole transforms (odd row pitch: 8-byte copies in FP32) against numpy:
forward and inverse, 1e-14 FP64, 1e-6 FP32 (three passes of about
eps sqrt(log2 n) each).
"""
import numpy as np
import pytest

from _util import buffer_to_phys, phys_to_buffer, rel_l2, to_dev, to_host

STEPS = [
    # nx, ny, nz, precision, scalars, alpha, alias
    (48, 384, 32, 0, 1, 0.0, 2 / 3),
    (384, 48, 64, 1, 2, 0.0, 2 / 3),     # kept ky Nyquist row
    (96, 192, 48, 0, 2, 0.05, 2 / 3),
    (192, 96, 48, 1, 2, 0.05, 2 / 3),
    (64, 128, 16, 1, 1, 0.0, 15 / 16),
    (128, 256, 24, 0, 1, 0.0, 2 / 3),
    (512, 512, 16, 0, 2, 0.0, 2 / 3),
    (256, 512, 12, 1, 1, 0.0, 1.0),
    (64, 32, 64, 0, 1, 0.0, 2 / 3),      # y on the staged pass
    (32, 64, 32, 1, 1, 0.0, 2 / 3),      # x on the staged pass
]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,precision,ns,alpha,alias", STEPS)
def test_direct_passes_match_staged(torch_cuda, nx, ny, nz, precision, ns, alpha, alias):
    import gnss_b200 as G
    torch = torch_cuda
    dt = np.complex128 if precision == 0 else np.complex64
    rng = np.random.default_rng(7)
    init = G.jet_initial_state(nx, ny, nz, n_scalars=ns, seed=3, noise_kmax=6.0, dtype=np.complex128)
    shape = init[0].shape
    init = [(f + np.fft.rfftn(1e-2 * rng.standard_normal((nx, ny, nz))).transpose(1, 0, 2)).astype(dt) for f in init]
    out = []
    for variant in (G.GNSS_VARIANT_AUTO, G.GNSS_VARIANT_STAGED):
        ctx = G.Context(nx=nx, ny=ny, nz=nz, re=500.0, dt=1e-3, n_scalars=ns, alpha=alpha, alias_filter=alias,
                        precision=precision)
        ctx.set_option(G.GNSS_OPT_PVARIANT, variant)
        scratch = torch.full((int(ctx.lib.gnss_scratch_bytes(ctx._h)) // 4 + 64,), float("nan"), dtype=torch.float32,
                             device="cuda")
        assert ctx.lib.gnss_attach_scratch(ctx._h, scratch.data_ptr(), scratch.numel() * 4) == 0
        st = [to_dev(torch, a) for a in init]
        hi = [torch.zeros_like(st[0]) for _ in st]
        ctx.de_alias(st)
        for s in range(2):
            ctx.solver_ps(st, hi, euler=(s == 0))
        ctx.check()
        out.append([to_host(t) for t in st + hi])
        ctx.close()
    assert out[0][0].shape == shape
    tol = 1e-13 if precision == 0 else 2e-6
    for a, b in zip(*out):
        assert np.isfinite(a.view(a.real.dtype)).all()
        assert rel_l2(a, b) <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz", [(48, 96, 16), (192, 64, 12), (384, 128, 8), (256, 512, 24)])
@pytest.mark.parametrize("precision", [0, 1])
def test_transforms_match_numpy(torch_cuda, nx, ny, nz, precision):
    import gnss_b200 as G
    torch = torch_cuda
    dt = np.complex128 if precision == 0 else np.complex64
    u = np.random.default_rng(11).standard_normal((nx, ny, nz))
    tol = 1e-14 if precision == 0 else 1e-6
    spec = np.fft.rfftn(u).transpose(1, 0, 2)
    with G.Context(nx=nx, ny=ny, nz=nz, precision=precision) as ctx:
        f = to_dev(torch, phys_to_buffer(u, dt))
        ctx.forward_transform(f)
        assert rel_l2(to_host(f), spec) <= tol
        f = to_dev(torch, np.ascontiguousarray(spec.astype(dt)))
        ctx.inverse_transform(f)
        assert rel_l2(buffer_to_phys(to_host(f), (nx, ny, nz)), u) <= tol
