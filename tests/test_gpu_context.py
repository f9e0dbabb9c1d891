"""Contexts: cost of their introspection calls."""
import time

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
