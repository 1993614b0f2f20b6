"""Site-rate conditionals of posteriors that are no probabilities: a NaN or
negative single posterior, or an infinite pair posterior (which enters every
category of the pair, so that infinities meet), makes its own columns NaN and
leaves every other column's bits alone; a NaN pair posterior counts as none, as
any that is not above zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["single nan", "single negative", "pair inf", "pair nan", "both"])
def test_non_finite_posteriors(where):
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    L, W = 70, 60
    s = synth.make_workload(dict(numseqs=6, numcols=L, W=W, paired=0.3, mean_bl=0.1), seed=4)
    rng = np.random.default_rng(5)
    pair = rng.random((L, L)) ** 8
    pair = np.triu(pair, 1) + np.triu(pair, 1).T
    single = rng.random(L)

    def run(a, b):
        return api.felsensteinposteriorsiterateconditionalscuda(
            a, b, s.dataset, M.getparams(s.params15, s.dataset.branchlengths), None, W)

    clean = run(single, pair)
    assert np.isfinite(clean).all()
    bad = []
    if where in ("single nan", "both"):
        single[11] = np.nan
        bad += [11]
    if where == "single negative":
        single[0] = single[69] = -1e-9
        bad += [0, 69]
    if where in ("pair inf", "both"):
        pair[20, 55] = pair[55, 20] = np.inf
        bad += [20, 55]
    if where == "pair nan":
        clean_pair = pair.copy()
        clean_pair[3, 4] = clean_pair[4, 3] = 0.0
        clean = run(single, clean_pair)
        pair[3, 4] = pair[4, 3] = np.nan
    got = run(single, pair)
    assert got.shape[1] == L
    assert np.isnan(got[:, bad]).all()
    rest = np.setdiff1d(np.arange(L), bad)
    np.testing.assert_array_equal(got[:, rest], clean[:, rest])


@pytest.mark.parametrize("at", [(22, 46), (0, 88), (10, 11), (70, 99)])
def test_infinite_pair_posteriors_far_below_their_columns_largest_term(at):
    """The NaN of one partner meets sums of others that are hundreds of nats above
    it (43 diverse sequences), in every lane of the column's warp."""
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    L, W = 100, 88
    s = synth.make_workload(dict(numseqs=43, numcols=L, W=W, paired=0.1, mean_bl=0.6), seed=9)
    rng = np.random.default_rng(5)
    pair = rng.random((L, L)) ** 8
    pair = np.triu(pair, 1) + np.triu(pair, 1).T
    single = rng.random(L)
    params = M.getparams(s.params15, s.dataset.branchlengths, 3, 1)
    clean = api.felsensteinposteriorsiterateconditionalscuda(single, pair, s.dataset, params, None, W)
    pair[at] = np.inf
    got = api.felsensteinposteriorsiterateconditionalscuda(single, pair, s.dataset, params, None, W)
    assert np.isnan(got[:, list(at)]).all()
    rest = np.setdiff1d(np.arange(L), at)
    np.testing.assert_array_equal(got[:, rest], clean[:, rest])
