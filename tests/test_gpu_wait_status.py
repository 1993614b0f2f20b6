"""The status of every pass of a call counts, not the last one's alone: the
self-test's failed wait is read back first and a pass without a failure after it,
as an inside pass before an outside pass and a decoding, and the call's end still
reports the time-out; the next call starts clean."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_later_pass_does_not_hide_a_time_out():
    from messi_gb300 import _lib, api
    rng = np.random.default_rng(3)
    L = 60
    u = rng.uniform(-30.0, -8.0, L)
    p = u[:, None] + u[None, :] + rng.normal(-2.0, 2.5, (L, L))
    p = np.asfortranarray(np.maximum(p, p.T))
    ctx = api.Context(0)
    try:
        before = api.consensusstructure(u, p, ctx=ctx)
        for _ in range(3):
            assert ctx.selftest_bounded_wait() == _lib.MESSI_ETIMEOUT
            np.testing.assert_array_equal(api.consensusstructure(u, p, ctx=ctx), before)
    finally:
        ctx.close()
