"""Site-rate conditionals at the sizes where the kernels' splits end: column
counts around a warp's 32 partners, one to four site-rate categories, columns
without any allowed partner, zero posteriors (relative 1e-6 to the FP64
oracle, the bar of tests/test_gpu_conditionals.py)."""
import numpy as np
import pytest

from oracle import model_ref as mr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,W,site", [(2, 1, 3), (5, 1, 1), (33, 32, 4), (65, 31, 2), (70, 69, 3)])
def test_siterate_forms(L, W, site):
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    s = synth.make_workload(dict(numseqs=7, numcols=L, W=W, paired=0.3, mean_bl=0.1), seed=L + site)
    ds = s.dataset
    rng = np.random.default_rng(L)
    pair = rng.random((L, L)) ** 8
    pair[rng.random((L, L)) < 0.3] = 0.0
    pair[0, :] = pair[:, 0] = 0.0
    single = rng.random(L)
    single[-1] = 0.0
    ref = mr.siterate_conditionals(ds.tree_arrays(), ds.masks, mr.getparams(s.params15, ds.branchlengths, site), W, single,
                                   pair)
    got = api.felsensteinposteriorsiterateconditionalscuda(single, pair, ds,
                                                           M.getparams(s.params15, ds.branchlengths, site), None, W)
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(got))
    assert np.abs((got[fin] - ref[fin]) / np.maximum(np.abs(ref[fin]), 1.0)).max() <= 1e-6
