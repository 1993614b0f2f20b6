"""Pruning at the bottom of FP32's range: two clades of identical sequences that
differ in every column and are joined by branches of length zero, so that a row's
largest state is denormal where they meet.  The two forms of the node update give
the same bits, and each value is within 1e-6 of the FP64 oracle plus what FP32
loses there: 64 roundings (16 states, four products) of half the smallest denormal,
2^-150, relative to the likelihood."""
import numpy as np
import pytest

from oracle import model_ref as mr

pytestmark = pytest.mark.gpu


def _clade(names, bl):
    s = f"{names[0]}:{bl}"
    for n in names[1:]:
        s = f"({s},{n}:{bl}):0.0"
    return s


@pytest.mark.parametrize("k,bl", [(6, 0.005), (7, 0.005), (8, 0.005), (8, 0.01), (9, 0.01)])
def test_denormal_rows(k, bl, monkeypatch):
    from messi_gb300 import api
    from messi_gb300 import model as M
    from messi_gb300.dataset import Dataset
    a, g = [f"a{i}" for i in range(k)], [f"g{i}" for i in range(k)]
    tree = f"(({_clade(a, bl)},{_clade(g, bl)}):0.0,x:0.1,y:0.1);"
    ds = Dataset.from_sequences(a + g + ["x", "y"], ["ACGUACGA"] * k + ["GUACCGAU"] * k + ["-" * 8] * 2, tree)
    p15 = M.DEFAULT_PARAMS15.copy()
    ref, _ = mr.pair_loglik(ds.tree_arrays(), ds.masks, mr.getparams(p15, ds.branchlengths), 7)
    got = []
    for shape in ("0", "3"):
        monkeypatch.setenv("MESSI_PRUNE_SHAPE", shape)
        ctx = api.Context(0)
        try:
            r = api.felsensteincuda(ds, M.getparams(p15, ds.branchlengths), None, 7, ctx=ctx)
            got.append(r[0] if isinstance(r, tuple) else r)
        finally:
            ctx.close()
    fin = np.isfinite(ref)
    assert fin.sum() == 56
    for z in got:
        assert np.array_equal(fin, np.isfinite(z))
        bound = 1e-6 * np.abs(ref[fin]) + 2.0 ** -144 / np.exp(ref[fin])
        assert (np.abs(z[fin] - ref[fin]) <= bound).all(), (z[fin] - ref[fin]) / bound
    np.testing.assert_array_equal(got[0], got[1])
