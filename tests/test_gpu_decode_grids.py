"""Posterior decoding with several row blocks per CTA dealt so that a row block's
next ones belong to other CTAs (4, 5 and 7 CTAs), and with one row block more
than the GPU has SMs, where the default grid reads its rows from global memory
(bit-exact against the FP32 oracle)."""
import numpy as np
import pytest

from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


def _check(L, seed, ctas, monkeypatch):
    from messi_gb300 import api
    rng = np.random.default_rng(seed)
    p, s = rng.random((L, L)) ** 6, rng.random(L) * 0.2
    p += p.T
    if ctas:
        monkeypatch.setenv("MESSI_WAVE_CTAS", str(ctas))
    ctx = api.Context(0)
    try:
        e, t = api.computeposteriordecodingcuda(s, p, 2.0, ctx=ctx)
    finally:
        ctx.close()
    e_ref, t_ref = co.posterior_decoding(s, p, 2.0)
    np.testing.assert_array_equal(e, e_ref.astype(np.float64))
    np.testing.assert_array_equal(t, t_ref)


@pytest.mark.parametrize("L", [160, 305, 449])
@pytest.mark.parametrize("ctas", [4, 5, 7])
def test_row_blocks_over_other_ctas(L, ctas, monkeypatch):
    _check(L, L, ctas, monkeypatch)


def test_more_row_blocks_than_sms(monkeypatch):
    import torch
    _check(16 * torch.cuda.get_device_properties(0).multi_processor_count + 1, 11, 0, monkeypatch)
