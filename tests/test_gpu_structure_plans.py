"""The likelihood of a given structure: its plan lies in the context's scratch
from call to call, so structures of growing and shrinking size, none at all and
band likelihoods in between must give the bits that a fresh context gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_structures_of_any_size_in_turn_equal_fresh_contexts(c1):
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    ds = c1.dataset
    params = M.getparams(c1.params15, ds.branchlengths)
    L = ds.numcols
    rng = np.random.default_rng(3)
    structures = [np.zeros(L, np.int32)]
    for W, share in ((8, 0.05), (L - 1, 0.5), (20, 0.2), (L - 1, 0.9), (6, 0.02)):
        q = synth.random_structure(rng, L, max(4, min(W, L - 1)), share)
        structures.append(np.where(q >= 0, q + 1, 0).astype(np.int32))
    structures.append(structures[0])

    def value(ctx, s):
        return api.computemodellikelihood(None, ds, params, s, useprior=False, ctx=ctx)

    fresh = []
    for s in structures:
        ctx = api.Context(0)
        try:
            fresh.append(value(ctx, s))
        finally:
            ctx.close()
    ctx = api.Context(0)
    try:
        got, Z = [], []
        for s in structures + structures[::-1]:
            got.append(value(ctx, s))
            Z.append(api.computestructureintegratedlikelihood(ds, params, c1.W, ctx=ctx))
    finally:
        ctx.close()
    assert got == fresh + fresh[::-1]
    assert len(set(Z)) == 1
