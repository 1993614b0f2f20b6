"""The outside pass whose CTAs wait for one another's cells: the smallest
alignments, rows per CTA around the 16, 32 and 256 that are finished at a time,
and every CTA size.  Posteriors within 1e-4 of the FP64 oracle, as FP32 log-odds
cells allow; the bits of any grid equal."""
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
        return api.computeposteriors(u, p, ctx=ctx)
    finally:
        ctx.close()


@pytest.mark.parametrize("L,W", [(2, 1), (3, 2), (4, 3), (5, 1), (8, 7), (33, 16), (151, 150), (305, 40)])
def test_small_alignments_against_the_oracle(L, W, monkeypatch):
    u, p = _scores(L, W, 200 + L)
    ins = co.inside(u, p)
    single, pair = co.basepairprobs(ins, co.outside(ins, u, p), u, p)
    got = [_run(u, p, monkeypatch, *form) for form in ((0, 0), (3, 256), (0, 512), (0, 1024))]
    for z, s, q in got:
        assert abs(z - ins[0, 0, L - 1]) <= 1e-6 * abs(ins[0, 0, L - 1])
        assert np.max(np.abs(s - single)) <= 1e-4
        assert np.max(np.abs(q - pair)) <= 1e-4
        assert z == got[0][0]
        np.testing.assert_array_equal(s, got[0][1])
        np.testing.assert_array_equal(q, got[0][2])


@pytest.mark.parametrize("L,ctas", [(16, 1), (17, 1), (33, 1), (64, 2), (255, 1), (256, 1), (257, 1), (258, 1), (515, 1),
                                    (700, 2), (800, 0)])
def test_rows_per_cta(L, ctas, monkeypatch):
    u, p = _scores(L, 23, L)
    z0, s0, q0 = _run(u, p, monkeypatch, 0)
    z1, s1, q1 = _run(u, p, monkeypatch, ctas, 0 if ctas else 256)
    assert z0 == z1
    np.testing.assert_array_equal(s0, s1)
    np.testing.assert_array_equal(q0, q1)
