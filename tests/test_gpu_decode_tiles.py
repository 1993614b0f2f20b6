"""Posterior decoding at the edges of its 16 x 16 tiles: one cell to several
row blocks per CTA, whole and ragged last tiles, ties between split points,
and scores below the recursion's initial maximum (bit-exact against the FP32
oracle)."""
import numpy as np
import pytest

from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


def _case(L, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "ties":  # few distinct values: many equal splits
        p = rng.integers(0, 3, (L, L)) * 0.25
        s = rng.integers(0, 3, L) * 0.25
    elif kind == "zero":
        p, s = np.zeros((L, L)), np.zeros(L)
    else:
        p, s = rng.random((L, L)) ** 6, rng.random(L) * 0.2
    return s.astype(np.float64), (p + p.T).astype(np.float64)


@pytest.mark.parametrize("L,kind,alpha", [(1, "random", 2.0), (2, "random", 2.0), (15, "random", 2.0),
                                          (16, "ties", 2.0), (17, "random", 2.0), (32, "ties", 1.0),
                                          (33, "random", 2.0), (49, "zero", 2.0), (161, "ties", 2.0),
                                          (200, "random", -1.0), (257, "random", 2.0)])
@pytest.mark.parametrize("ctas", [0, 3])
def test_decode_tiles(L, kind, alpha, ctas, monkeypatch):
    from messi_gb300 import api
    single, pair = _case(L, kind, L)
    if ctas:
        monkeypatch.setenv("MESSI_WAVE_CTAS", str(ctas))
    ctx = api.Context(0)
    try:
        e, s = api.computeposteriordecodingcuda(single, pair, alpha, ctx=ctx)
    finally:
        ctx.close()
    e_ref, s_ref = co.posterior_decoding(single, pair, alpha)
    np.testing.assert_array_equal(e, e_ref.astype(np.float64))
    np.testing.assert_array_equal(s, s_ref)
