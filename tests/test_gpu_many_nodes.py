"""A batch with more tree nodes than eight times 65,535, the most CTAs that a
grid's second dimension takes: every alignment gives its own call's value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_of_many_nodes():
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    s = synth.make_workload(dict(numseqs=250, numcols=3, W=2, paired=0.3, mean_bl=0.05), seed=6)
    params = M.getparams(s.params15, s.dataset.branchlengths, 1)
    count = 8 * 65535 // s.dataset.numnodes + 2
    ctx = api.Context(0)
    try:
        one = api.computestructureintegratedlikelihood(s.dataset, params, s.W, ctx=ctx)
        got = api.computestructureintegratedlikelihoods([s.dataset] * count, [params] * count, [s.W] * count, ctx=ctx)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got, np.full(count, one))
