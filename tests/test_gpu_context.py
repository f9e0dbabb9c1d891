"""Contexts: cost of their introspection calls, and their reuse by the server.

A server hands the context of an ended request to the next request of its
geometry.  Nothing of the first run may show in the second: every result is
bit-identical to the jet run alone, as in the ensemble and server tests.
"""
import math
import time

import numpy as np
import pytest


@pytest.mark.gpu
def test_stage_bytes_is_cheap(torch_cuda):
    """The byte counts come from the bounds of the kept columns (0.1 ms at 512^3), not from a walk over the modes of
    the kept box, of which there are 20 million."""
    import gnss_b200 as G
    with G.Context(512) as ctx:
        best = min(_timed(ctx.stage_bytes) for _ in range(5))
    assert best < 5e-3


def _timed(call):
    t = time.perf_counter()
    call()
    return time.perf_counter() - t


def _requests(G, precision, n, n_scalars):
    """Requests run one after the other: the same geometry with other parameters and states, then neighbours of it that
    must not take its context over (box, dealiasing, scheme, drift on or off), then the first geometry again."""
    base = dict(nx=n, ny=n, nz=n, re=600.0, sc=0.7, sc_c=1.0, dt=1e-3, n_scalars=n_scalars, precision=precision)
    alpha = 0.05 if n_scalars == 2 else 0.0
    variants = [
        dict(alpha=alpha), dict(alpha=2 * alpha, re=2500.0, sc=2.0, sc_c=0.5, dt=4e-4, nu_stats=1.0 / 2500.0),
        dict(alpha=alpha, lx=4.0 * math.pi), dict(alpha=alpha, alias_filter=15.0 / 32.0),
        dict(alpha=alpha, scheme=G.GNSS_SCHEME_RK3IF), dict(alpha=0.0, dt=5e-4), dict(alpha=alpha, re=900.0),
    ]
    return [G.make_config(**{**base, **v}) for v in variants]


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n,n_scalars", [(1, 32, 1), (1, 64, 2), (0, 96, 2)])   # 96: a state of 36 MB
def test_reused_contexts_leave_no_trace(torch_cuda, precision, n, n_scalars):
    import gnss_b200 as G
    cplx = np.complex64 if precision else np.complex128
    cfgs = _requests(G, precision, n, n_scalars)
    init = [G.pack_state(G.jet_initial_state(n, n, n, n_scalars=n_scalars, seed=i, noise_kmax=4.0, amp=0.05,
                                             dtype=cplx)) for i in range(len(cfgs))]
    with G.Server(budget_bytes=8 << 30, max_active=2, steps_per_launch=5) as srv:
        for i, (cfg, a) in enumerate(zip(cfgs, init)):
            if i == 1:   # goes on from the first one's result: an FP64 mean line left over would round to this state
                a = got
            rid = srv.submit(cfg, a, 12)
            srv.wait(rid)
            got, stats, _ = srv.result(rid)
            kw = {k: getattr(cfg, k) for k, _ in G.GnssConfig._fields_ if k not in ("nx", "ny", "nz")}
            with G.Context(nx=n, ny=n, nz=n, **kw) as ctx:
                want, rows = np.empty_like(a), np.zeros((12, G.GNSS_NSTATS))
                ctx.run_host(a, want, 12, True, rows)
            assert np.array_equal(got, want), f"request {i}"
            for x, y in zip(stats.values(), rows[-1]):
                assert math.isclose(x, y, rel_tol=1e-12, abs_tol=0.0), f"request {i}"
