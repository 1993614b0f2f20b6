"""The inside pass whose CTAs wait for one another's cells: the smallest
alignments, cells per CTA around the 64 and 512 that are finished at a time,
and scores that are NaN themselves (a NaN of written cells ends the waiting).
FP32 log-odds: Z within 1e-6 of the FP64 oracle, the bits of any grid equal."""
import numpy as np
import pytest

from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


def _scores(L, W, seed):
    rng = np.random.default_rng(seed)
    u = rng.uniform(-30.0, -8.0, L)
    p = u[:, None] + u[None, :] + rng.normal(-2.0, 2.5, (L, L))
    k = np.arange(L)[None, :] - np.arange(L)[:, None]
    p[(k < 1) | (k > W)] = -np.inf
    return u, np.asfortranarray(np.maximum(p, p.T))


def _run(u, p, monkeypatch, ctas, threads=0):
    from messi_gb300 import api
    for name, v in (("MESSI_WAVE_CTAS", ctas), ("MESSI_WAVE_THREADS", threads)):
        if v:
            monkeypatch.setenv(name, str(v))
        else:
            monkeypatch.delenv(name, raising=False)
    ctx = api.Context(0)
    try:
        return api.computeinsideKH99(u, p, ctx=ctx), api.computeinsideKH99(u, p, zonly=False, ctx=ctx)
    finally:
        ctx.close()


@pytest.mark.parametrize("L,W", [(1, 1), (2, 1), (3, 2), (4, 3), (5, 1), (8, 7), (33, 16), (151, 150), (305, 40)])
def test_small_alignments_against_the_oracle(L, W, monkeypatch):
    u, p = _scores(L, W, 100 + L)
    ref = co.inside(u, p)[0, 0, L - 1]
    got = [_run(u, p, monkeypatch, *form) for form in ((0, 0), (3, 256), (0, 512))]
    for z, t in got:
        assert abs(z - ref) <= 1e-6 * abs(ref)
        assert z == got[0][0]
        np.testing.assert_array_equal(t, got[0][1])


@pytest.mark.parametrize("L,ctas", [(64, 1), (65, 1), (130, 2), (511, 1), (513, 1), (514, 1), (1027, 1), (1100, 2), (2440, 0)])
def test_cells_per_cta(L, ctas, monkeypatch):
    u, p = _scores(L, 23, L)
    z0, t0 = _run(u, p, monkeypatch, 0)
    z1, t1 = _run(u, p, monkeypatch, ctas, 0 if ctas else 256)
    assert z0 == z1
    np.testing.assert_array_equal(t0, t1)
    ref = co.inside_banded_Z(u, p, 23)
    assert abs(z0 - ref) <= 1e-6 * abs(ref)


@pytest.mark.parametrize("where", ["pair", "column"])
def test_nan_scores_end_in_nan(where, monkeypatch):
    u, p = _scores(90, 60, 7)
    if where == "pair":
        p[10, 40] = p[40, 10] = np.inf  # (a NaN pair score counts as forbidden)
    else:
        u[31] = np.nan
    z, _ = _run(u, p, monkeypatch, 0)
    assert np.isnan(z)
