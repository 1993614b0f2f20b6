"""The suffix recurrences of bands wider than their shared-memory window (the
pull form, blocks of 32 cells), on small cases with the window made smaller:
whole and ragged blocks, spans below and above a block.  Z within 1e-6 of the
FP64 oracle; posteriors within 2e-4 of the windowed form's (each form within
1e-4 of the exact ones, as FP32 log-odds cells allow); a batch gives the bits of
its single calls."""
import numpy as np
import pytest

from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


def _run(u, p, monkeypatch, window):
    from messi_gb300 import api
    if window is not None:
        monkeypatch.setenv("MESSI_SUFFIX_WINDOW", str(window))
    ctx = api.Context(0)
    try:
        return api.computeposteriors(u, p, ctx=ctx)
    finally:
        ctx.close()


@pytest.mark.parametrize("L,W", [(3, 1), (20, 3), (33, 1), (40, 7), (97, 31), (160, 64), (333, 100)])
def test_pull_form(L, W, monkeypatch):
    rng = np.random.default_rng(L)
    u = rng.uniform(-30.0, -8.0, L)
    p = u[:, None] + u[None, :] + rng.normal(-2.0, 2.5, (L, L))
    k = np.arange(L)[None, :] - np.arange(L)[:, None]
    p[(k < 1) | (k > W)] = -np.inf
    p = np.asfortranarray(np.maximum(p, p.T))
    z0, s0, q0 = _run(u, p, monkeypatch, None)
    z, s, q = _run(u, p, monkeypatch, 0)
    ref = co.inside_banded_Z(u, p, W)
    assert abs(z - ref) <= 1e-6 * abs(ref)
    assert abs(z0 - ref) <= 1e-6 * abs(ref)
    assert np.max(np.abs(s - s0)) <= 2e-4
    assert np.max(np.abs(q - q0)) <= 2e-4


def test_batch_with_both_forms(monkeypatch):
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    monkeypatch.setenv("MESSI_SUFFIX_WINDOW", "100")  # spans up to 36 fit
    made = [synth.make_workload(dict(numseqs=5, numcols=L, W=W, paired=0.3, mean_bl=0.1), seed=L)
            for L, W in ((150, 20), (200, 70), (90, 89))]
    params = [M.getparams(s.params15, s.dataset.branchlengths) for s in made]
    ctx = api.Context(0)
    try:
        one = [api.computestructureintegratedlikelihood(s.dataset, q, s.W, ctx=ctx) for s, q in zip(made, params)]
        got = api.computestructureintegratedlikelihoods([s.dataset for s in made], params, [s.W for s in made], ctx=ctx)
    finally:
        ctx.close()
    np.testing.assert_array_equal(np.asarray(got), np.asarray(one))
    monkeypatch.delenv("MESSI_SUFFIX_WINDOW")
    ctx = api.Context(0)
    try:
        want = [api.computestructureintegratedlikelihood(s.dataset, q, s.W, ctx=ctx) for s, q in zip(made, params)]
    finally:
        ctx.close()
    np.testing.assert_allclose(one, want, rtol=2e-6, atol=0)
