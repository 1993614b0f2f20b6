"""Tree segments of the pruning: trees whose segments take every shape (one
long path, set-aside messages on a balanced tree, more nodes than a segment
holds, single-node segments from heavy column compression), with pair counts
around the edges of the 32-pair tiles, against the FP64 oracle (relative
1e-6, the bar of every pair log-likelihood)."""
import numpy as np
import pytest

from oracle import model_ref as mr

pytestmark = pytest.mark.gpu

REL = 1e-6


def _newick(shape, names, rng):
    bl = lambda: f":{rng.exponential(0.1) + 1e-3:.6f}"
    if shape == "path":
        s = f"{names[0]}{bl()}"
        for n in names[1:-2]:
            s = f"({s},{n}{bl()}){bl()}"
        return f"({s},{names[-2]}{bl()},{names[-1]}{bl()});"
    nodes = [n + bl() for n in names]
    while len(nodes) > 3:
        if len(nodes) == 4:
            nodes = [f"({nodes[0]},{nodes[1]}){bl()}"] + nodes[2:]
            continue
        nodes = [f"({nodes[i]},{nodes[i + 1]}){bl()}" if i + 1 < len(nodes) else nodes[i]
                 for i in range(0, len(nodes), 2)]
    return f"({','.join(nodes)});"


# (tree, sequences, columns, distinct columns, span)
CASES = [("path", 12, 9, 9, 8),       # 36 pairs: one full tile and four more
         ("path", 60, 40, 40, 39),    # more nodes than one segment holds
         ("balanced", 24, 33, 33, 32),
         ("balanced", 64, 24, 24, 11),  # set-aside messages, a band
         ("balanced", 17, 70, 5, 69),   # few distinct columns: tables everywhere
         ("path", 4, 3, 3, 2)]


@pytest.mark.parametrize("shape,nseq,ncol,distinct,W", CASES)
def test_segments_match_oracle(shape, nseq, ncol, distinct, W):
    from messi_gb300 import api
    from messi_gb300 import model as M
    from messi_gb300.dataset import Dataset
    rng = np.random.default_rng(nseq * 1000 + ncol)
    cols = rng.choice(list("ACGU-"), p=[0.24, 0.24, 0.24, 0.24, 0.04], size=(nseq, distinct))
    seqs = ["".join(r) for r in cols[:, rng.integers(0, distinct, ncol) if distinct < ncol else np.arange(ncol)]]
    names = [f"s{k}" for k in range(nseq)]
    ds = Dataset.from_sequences(names, seqs, _newick(shape, names, rng))
    p15 = M.DEFAULT_PARAMS15.copy()
    rp = mr.getparams(p15, ds.branchlengths)
    got, per = api.felsensteincuda(ds, M.getparams(p15, ds.branchlengths), None, W, True)
    ref, refl = mr.pair_loglik(ds.tree_arrays(), ds.masks, rp, W, per_lambda=True)
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(got))
    assert np.abs((got[fin] - ref[fin]) / ref[fin]).max() <= REL
    for a, b in zip(per, refl):
        assert np.abs((a[fin] - b[fin]) / b[fin]).max() <= REL
    total = api.computestructureintegratedlikelihood(ds, M.getparams(p15, ds.branchlengths), W)
    want, _ = mr.structure_integrated_likelihood(ds.tree_arrays(), ds.masks, ds.gapfrequency, p15, W)
    assert abs(total - want) <= REL * abs(want)
