"""The symmetric L x L matrix of pair log-likelihoods at column counts around the
8 x 32 cells that a CTA writes: both triangles and the diagonal against the FP64
oracle (relative 1e-6, the bar of every pair log-likelihood)."""
import numpy as np
import pytest

from oracle import model_ref as mr

pytestmark = pytest.mark.gpu

REL = 1e-6


@pytest.mark.parametrize("ncol,W", [(2, 1), (7, 6), (8, 7), (31, 30), (32, 31), (32, 9), (63, 62), (64, 40), (65, 64)])
def test_dense_matrix_at_tile_edges(ncol, W):
    from messi_gb300 import api
    from messi_gb300 import model as M
    from messi_gb300.dataset import Dataset
    rng = np.random.default_rng(ncol * 100 + W)
    seqs = ["".join(r) for r in rng.choice(list("ACGU-"), p=[0.24, 0.24, 0.24, 0.24, 0.04], size=(4, ncol))]
    ds = Dataset.from_sequences([f"s{k}" for k in range(4)], seqs, "((s0:0.1,s1:0.2):0.05,s2:0.3,s3:0.1);")
    p15 = M.DEFAULT_PARAMS15.copy()
    got, _ = api.felsensteincuda(ds, M.getparams(p15, ds.branchlengths), None, W)
    ref, _ = mr.pair_loglik(ds.tree_arrays(), ds.masks, mr.getparams(p15, ds.branchlengths), W, per_lambda=True)
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(got))
    assert np.all(got[~fin] == -np.inf)
    np.testing.assert_array_equal(got, got.T)
    assert np.abs((got[fin] - ref[fin]) / ref[fin]).max() <= REL
