"""Contexts of several host threads whose calls need different amounts of dynamic
shared memory of the same kernel: the limit belongs to the kernel on the device,
so one thread's smaller call may not take it away from another's.  The calls
take turns, and every one gives what it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_turn(calls, turns):
    """calls[t]() in thread t, one call at a time, in the order of `turns`."""
    go = [threading.Semaphore(0) for _ in calls]
    back = threading.Semaphore(0)
    out = [[] for _ in calls]
    err = []

    def run(t):
        for _ in range(turns.count(t)):
            go[t].acquire()
            try:
                out[t].append(calls[t]())
            except Exception as e:  # handed to the test's thread
                err.append((t, e))
            back.release()

    pool = [threading.Thread(target=run, args=(t,)) for t in range(len(calls))]
    for th in pool:
        th.start()
    for t in turns:
        go[t].release()
        back.acquire()
    for th in pool:
        th.join()
    if err:
        raise AssertionError(f"thread {err[0][0]}") from err[0][1]
    return out


def _tree_call(numseqs, numcols, seed):
    from messi_gb300 import api, synth
    from messi_gb300 import model as M
    s = synth.make_workload(dict(numseqs=numseqs, numcols=numcols, W=numcols - 1, paired=0.3, mean_bl=0.3), seed=seed)
    params = M.getparams(s.params15, s.dataset.branchlengths)
    ctx = api.Context(0)
    return ctx, lambda: api.felsensteincuda(s.dataset, params, None, s.W, True, ctx=ctx)


def _mlp_call(width, batch, seed):
    from messi_gb300 import api
    rng = np.random.default_rng(seed)
    ctx = api.Context(0)
    net = api.MLP(20, width, 3, 5, seed=seed, ctx=ctx)
    x, t = rng.normal(size=(batch, 20)), rng.normal(size=(batch, 5))
    return ctx, lambda: (net.forward(x), net.gradients(x, t)[1])


def _decode_call(L, seed):
    from messi_gb300 import api
    rng = np.random.default_rng(seed)
    p, s = rng.random((L, L)) ** 6, rng.random(L)
    ctx = api.Context(0)
    return ctx, lambda: api.computeposteriordecodingcuda(s, p + p.T, 2.0, ctx=ctx)


def _suffix_call(L, W, seed):
    from messi_gb300 import api
    rng = np.random.default_rng(seed)
    u = rng.uniform(-30.0, -8.0, L)
    p = u[:, None] + u[None, :] + rng.normal(-2.0, 2.5, (L, L))
    k = np.arange(L)[None, :] - np.arange(L)[:, None]
    p[(k < 1) | (k > W)] = -np.inf
    p = np.asfortranarray(np.maximum(p, p.T))
    ctx = api.Context(0)
    return ctx, lambda: api.computeposteriors(u, p, ctx=ctx)


def _flat(r):
    if isinstance(r, (list, tuple)):
        return [a for x in r for a in _flat(x)]
    return [np.asarray(r)]


FORMS = {"tree": (lambda: _tree_call(96, 40, 1), lambda: _tree_call(4, 12, 2)),
         "network": (lambda: _mlp_call(300, 20, 1), lambda: _mlp_call(24, 20, 2)),
         "decoding": (lambda: _decode_call(900, 1), lambda: _decode_call(40, 2)),
         "suffix": (lambda: _suffix_call(900, 700, 1), lambda: _suffix_call(90, 20, 2))}


@pytest.mark.parametrize("form", list(FORMS))
def test_large_and_small_calls_in_turn(form):
    made = [make() for make in FORMS[form]]
    try:
        alone = [call() for _, call in made]
        got = _in_turn([call for _, call in made], [0, 1, 0, 1, 1, 0])
    finally:
        for ctx, _ in made:
            ctx.close()
    for t in range(2):
        for r in got[t]:
            for a, b in zip(_flat(r), _flat(alone[t])):
                np.testing.assert_array_equal(a, b)
