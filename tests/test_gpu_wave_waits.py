"""A warp's bounded wait on the device: with another CTA's failure visible to one
lane alone all 32 lanes leave at the same look, and a wait that nothing ends gives
up; the self-test reports both as MESSI_ETIMEOUT and leaves the context usable."""
import pytest

pytestmark = pytest.mark.gpu


def test_lanes_leave_together(c1):
    from messi_gb300 import _lib, api
    from messi_gb300 import model as M
    ctx = api.Context(0)
    try:
        assert [ctx.selftest_bounded_wait() for _ in range(3)] == [_lib.MESSI_ETIMEOUT] * 3
        params = M.getparams(c1.params15, c1.dataset.branchlengths)
        api.computestructureintegratedlikelihood(c1.dataset, params, c1.W, ctx=ctx)
    finally:
        ctx.close()
