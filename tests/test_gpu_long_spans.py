"""Inside and outside passes on bands wider than 512 spans, where the
pipelined inside kernel deals the rows of every diagonal pair over the CTAs
again and a lane takes more than sixteen split points: the same bits as the
plain wavefront (7 CTAs, one CTA), Z within 1e-6 of the FP64 oracle."""
import numpy as np
import pytest

from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,W", [(530, 529), (700, 699), (1203, 640)])
def test_long_spans_bit_identical_on_any_grid(L, W, monkeypatch):
    from messi_gb300 import api
    rng = np.random.default_rng(L)
    u = rng.uniform(-30.0, -8.0, L)
    p = u[:, None] + u[None, :] + rng.normal(-2.0, 2.5, (L, L))
    k = np.arange(L)[None, :] - np.arange(L)[:, None]
    p[(k < 1) | (k > W)] = -np.inf
    p = np.asfortranarray(np.maximum(p, p.T))
    got = []
    for ctas in (0, 7, 1):
        if ctas:
            monkeypatch.setenv("MESSI_WAVE_CTAS", str(ctas))
        ctx = api.Context(0)
        try:
            got.append((api.computeinsideKH99(u, p, zonly=False, ctx=ctx),) + api.computeposteriors(u, p, ctx=ctx))
        finally:
            ctx.close()
    for other in got[1:]:
        for a, b in zip(other, got[0]):
            np.testing.assert_array_equal(a, b)
    ref = co.inside_banded_Z(u, p, W)
    assert abs(got[0][1] - ref) <= 1e-6 * abs(ref)
