"""Performance cases: the calls that a user of messi_gb300 makes, with the
sizes that the repository's own workloads, tests and benchmark have.

A case names a kind of call and its sizes; inputs come from the seed alone.
Every state owns its context (one alignment or one set of scores is what a
program has on a context), so the plans and captured graphs of two states never
meet.  `exact` computes the same outputs in FP64 with torch, from the
alignment, tree and parameters, without the package's numerical code.
"""
import math

import numpy as np
import torch

from messi_gb300 import api, synth
from messi_gb300 import model as M

DEVICE = "cuda"
F64 = torch.float64
NINF = -math.inf


def listed():
    return [
        # The objective of every optimiser step and MCMC proposal: unpaired
        # columns, pair pruning, gap mask, inside pass.  A small family (the
        # smallest useful alignment: latency and launches), the benchmark
        # alignment, and a genome-scale alignment with a band.
        {"name": "likelihood 16x120", "kind": "likelihood", "seqs": 16, "cols": 120, "span": 119, "bl": 0.10},
        {"name": "likelihood 64x1000", "kind": "likelihood", "seqs": 64, "cols": 1000, "span": 500, "bl": 0.10},
        {"name": "likelihood 30x9000", "kind": "likelihood", "seqs": 30, "cols": 9000, "span": 800, "bl": 0.05},
        # The reference-facing calls with host matrices: unpaired columns and
        # the dense pair matrix of a deep alignment, every pair, odd length.
        {"name": "pairs 100x733", "kind": "pairs", "seqs": 100, "cols": 733, "span": 732, "bl": 0.10},
        # Many alignments of uneven depth and length in one evaluation.
        {"name": "batch of 24", "kind": "batch", "count": 24, "seqs": 64, "cols": 600, "bl": 0.10},
        # The likelihood of one sampled structure, the MCMC's other target.
        {"name": "structure 64x1000", "kind": "structure", "seqs": 64, "cols": 1000, "span": 500, "bl": 0.10},
        # Site-rate conditionals given the structure posteriors (once per
        # sampled structure, the rate-resampling step).
        {"name": "site rates 64x600", "kind": "siterates", "seqs": 64, "cols": 600, "span": 300, "bl": 0.10},
        # The grammar passes on host scores: Z alone with every span allowed
        # (the reference's published timing series), the posterior chain, and
        # the decoding of posteriors into a structure.
        {"name": "inside 2001", "kind": "inside", "cols": 2001, "span": 2000},
        {"name": "posteriors 1000", "kind": "posteriors", "cols": 1000, "span": 500},
        {"name": "decoding 1000", "kind": "decoding", "cols": 1000, "span": 500},
        # The learned proposal: one draw, and the gradients of a training batch.
        {"name": "proposal draw", "kind": "forward", "batch": 1, "width": 256},
        {"name": "proposal gradients", "kind": "gradients", "batch": 256, "width": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["likelihood", "likelihood", "pairs", "batch", "structure", "siterates", "inside", "posteriors",
                       "decoding", "forward", "gradients"])
    bl = rng.choice([0.05, 0.1, 0.2])
    if kind in ("likelihood", "pairs", "structure", "siterates"):
        top = {"likelihood": 3000, "pairs": 733, "structure": 1500, "siterates": 600}[kind]
        cols = _log(rng, 80, top)
        span = cols - 1 if kind == "pairs" or rng.random() < 0.4 else max(10, min(cols - 1, 800, _log(rng, 30, cols)))
        seqs = _log(rng, 6, 128 if cols <= 733 else 64)
        if kind == "siterates":
            seqs, span = min(seqs, 64), min(span, 300)
        return {"kind": kind, "seqs": seqs, "cols": cols, "span": span, "bl": bl}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 24), "seqs": _log(rng, 8, 64), "cols": _log(rng, 100, 600), "bl": bl}
    if kind in ("inside", "posteriors", "decoding"):
        cols = _log(rng, 60, 2001 if kind == "inside" else 1000)
        span = cols - 1 if rng.random() < 0.4 else max(5, _log(rng, 20, cols - 1))
        if kind == "posteriors":
            span = min(span, 500)
        return {"kind": kind, "cols": cols, "span": span}
    return {"kind": kind, "batch": _log(rng, 1, 64) if kind == "forward" else _log(rng, 16, 256),
            "width": rng.choice([64, 128, 256])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
IN_DIM, NCOMP, DIM = 44, 4, 11  # the learned proposal's network (messi_gb300/mcmc.py)


def _alignment(case, seed, cols=None, seqs=None):
    """A seeded alignment on a random tree, and its parameters."""
    cols = cols or case["cols"]
    s = synth.make_workload({"numseqs": seqs or case["seqs"], "numcols": cols, "W": case.get("span", cols - 1),
                             "paired": 0.3, "mean_bl": case["bl"]}, seed=seed)
    return s, M.getparams(s.params15, s.dataset.branchlengths)


def _members(case, seed):
    """The alignments of a batch: uneven lengths and depths up to the case's."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        cols = int(rng.integers(min(80, case["cols"] // 2), case["cols"] + 1))
        seqs = int(rng.integers(min(8, case["seqs"]), case["seqs"] + 1))
        out.append(_alignment(case, int(rng.integers(1, 1 << 31)), cols, max(3, seqs)))
    return out


def _helices(rng, L, W):
    """Columns of a random nested structure (partner or -1)."""
    return synth.random_structure(rng, L, max(4, min(W, L - 1)), 0.3) if L > 8 else np.full(L, -1)


def _scores(case, seed):
    """Unpaired and pair log-likelihoods as the pruning gives them: pairs of
    unrelated columns a little below the product of the two columns, coevolving
    pairs several nats above it, forbidden beyond the span and on gap columns."""
    L, W = case["cols"], case["span"]
    rng = np.random.default_rng(seed)
    u = -rng.gamma(6.0, 9.0, L)
    p = u[:, None] + u[None, :] + rng.normal(-1.5, 1.2, (L, L))
    partner = _helices(rng, L, W)
    x = np.where(partner > np.arange(L))[0]
    p[x, partner[x]] += rng.gamma(4.0, 1.5, len(x)) + 1.5
    gap = rng.random(L) < 0.01
    span = np.arange(L)[None, :] - np.arange(L)[:, None]
    p[(span < 1) | (span > W) | gap[:, None] | gap[None, :]] = NINF
    p = np.maximum(p, p.T)
    return u, np.asfortranarray(p)


def _posteriors(case, seed):
    """Row-normalised posteriors: helices with high probability, a faint
    background of other pairs within the span."""
    L, W = case["cols"], case["span"]
    rng = np.random.default_rng(seed)
    partner = _helices(rng, L, W)
    q = rng.gamma(0.2, 2e-3, (L, L))
    x = np.where(partner > np.arange(L))[0]
    q[x, partner[x]] += rng.gamma(2.0, 2.0, len(x))
    span = np.arange(L)[None, :] - np.arange(L)[:, None]
    q[(span < 1) | (span > W)] = 0.0
    q = q + q.T
    single = rng.gamma(2.0, 0.5, L)
    tot = single + q.sum(axis=1)
    scale = 1.0 / np.sqrt(tot[:, None] * tot[None, :])
    pair = q * scale
    return np.maximum(1.0 - pair.sum(axis=1), 1e-3), np.asfortranarray(pair)


def _network(case, seed):
    rng = np.random.default_rng(seed)
    H, out = case["width"], NCOMP + 2 * NCOMP * DIM
    w = [rng.uniform(-1, 1, (H, IN_DIM)) * math.sqrt(3 / IN_DIM), rng.normal(0, 0.05, H),
         rng.uniform(-1, 1, (H, H)) * math.sqrt(3 / H), rng.normal(0, 0.05, H),
         rng.uniform(-1, 1, (out, H)) * 0.1 * math.sqrt(3 / H), rng.normal(0, 0.05, out)]
    w = [a.astype(np.float32) for a in w]
    x = rng.normal(0, 1, (case["batch"], IN_DIM)).astype(np.float32)
    t = rng.normal(0, 1, (case["batch"], DIM)).astype(np.float32)
    return w, x, t


class _State:
    """What the program holds; gives its device memory back when dropped."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for name in ("batch", "mlp", "ctx"):
            h = getattr(self, name, None)
            if h is not None:
                h.close()


def prepare(case, seed):
    kind = case["kind"]
    st = _State(kind=kind, ctx=api.Context(0))
    if kind in ("likelihood", "pairs", "siterates", "structure"):
        s, st.params = _alignment(case, seed)
        st.dataset, st.span = s.dataset, case["span"]
        if kind == "structure":
            st.paired = np.where(s.paired >= 0, s.paired + 1, 0).astype(np.int32)
            st.ctx.dataset(st.dataset, 1)
        else:
            st.ctx.dataset(st.dataset, st.span)
        if kind == "pairs":
            st.ctx.dataset(st.dataset, 1)
        if kind == "siterates":
            st.single, st.pair = _posteriors(case, seed)
    elif kind == "batch":
        members = _members(case, seed)
        st.params = [p for _, p in members]
        st.batch = api.Batch([s.dataset for s, _ in members], ctx=st.ctx)
    elif kind in ("inside", "posteriors"):
        st.u, st.p = _scores(case, seed)
        st.span = case["span"]
    elif kind == "decoding":
        st.single, st.pair = _posteriors(case, seed)
    else:
        w, st.x, st.t = _network(case, seed)
        st.mlp = api.MLP(IN_DIM, case["width"], NCOMP, DIM, ctx=st.ctx)
        st.mlp.set_params(np.concatenate([a.ravel() for a in w]))
    return st


def run(st):
    kind = st.kind
    if kind == "likelihood":
        total, Z, u = api.computestructureintegratedlikelihood(st.dataset, st.params, st.span, ctx=st.ctx,
                                                               return_unpaired=True)
        return {"total": total, "Z": Z, "unpaired": u}
    if kind == "pairs":
        u = api.computeunpairedlikelihoods(st.dataset, st.params, ctx=st.ctx)
        mat, _ = api.felsensteincuda(st.dataset, st.params, None, st.span, ctx=st.ctx)
        return {"unpaired": u, "paired": mat}
    if kind == "batch":
        return st.batch.likelihood(st.params)
    if kind == "structure":
        return api.computemodellikelihood(None, st.dataset, st.params, st.paired, useprior=False, ctx=st.ctx)
    if kind == "siterates":
        return api.felsensteinposteriorsiterateconditionalscuda(st.single, st.pair, st.dataset, st.params, None, st.span,
                                                                 ctx=st.ctx)
    if kind == "inside":
        return api.computeinsideKH99(st.u, st.p, 1.0, True, True, st.span, ctx=st.ctx)
    if kind == "posteriors":
        Z, single, pair = api.computeposteriors(st.u, st.p, st.span, ctx=st.ctx)
        return {"Z": Z, "single": single, "pair": pair}
    if kind == "decoding":
        e, s = api.computeposteriordecodingcuda(st.single, st.pair, 2.0, ctx=st.ctx)
        return {"e": e, "s": s}
    if kind == "forward":
        return st.mlp.forward(st.x)
    loss, grads = st.mlp.gradients(st.x, st.t)
    return {"loss": loss, "grads": grads}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
# Of the (column pair, tree node) combinations about three tenths have subtree
# patterns of their own on the random trees used here (0.35 at 64 x 1000, 0.33
# at 16 x 120, 0.16 at 30 x 9000); each costs a 16 x 16 product in 36 categories.
DISTINCT = 0.3
CATEGORIES = 36


def _band(L, W):
    W = min(W, L - 1)
    return L * W - W * (W + 1) / 2


def _splits(L, W):
    """Split terms of a banded inside pass: sum over spans of cells x span."""
    W = min(W, L - 1)
    d = np.arange(1, W + 1, dtype=np.float64)
    return float(((L - d) * d).sum()) + max(0, L - 1 - W) * float(W + 1)


def work(case):
    kind = case["kind"]
    if kind in ("forward", "gradients"):
        H, out, B = case["width"], NCOMP + 2 * NCOMP * DIM, case["batch"]
        n = H * IN_DIM + H * H + out * H
        f = 2.0 * n * B * (1 if kind == "forward" else 3)
        return {"bytes": 4.0 * (n + B * (IN_DIM + out)) + (0 if kind == "forward" else 4.0 * n), "flops": f}
    if kind == "batch":
        L, N = 0.5 * (min(80, case["cols"] // 2) + case["cols"]), 0.5 * (min(8, case["seqs"]) + case["seqs"])
        pairs = case["count"] * L * L / 2
        return {"bytes": case["count"] * L * N, "flops": DISTINCT * pairs * N * CATEGORIES * 512}
    L = case["cols"]
    if kind == "decoding":
        return {"bytes": 8.0 * L * L + 16.0 * L * L, "flops": 2.0 * _splits(L, L - 1)}
    W = case["span"]
    dense = 8.0 * L * min(L, 2 * W + 1)
    if kind == "inside":
        return {"bytes": dense / 2, "flops": 4.0 * _splits(L, W)}
    if kind == "posteriors":
        return {"bytes": dense / 2 + 8.0 * L * L, "flops": 20.0 * _splits(L, W)}
    N = case["seqs"]
    per_pair = DISTINCT * (N - 1) * CATEGORIES * 512.0
    if kind == "structure":
        return {"bytes": float(L * N + 4 * L), "flops": per_pair * 0.15 * L + L * N * 3 * 64.0}
    if kind == "siterates":
        return {"bytes": L * N + dense + 24.0 * L, "flops": per_pair * 1.25 * _band(L, W) + 30.0 * 4 * 3 * _band(L, W)}
    flops = per_pair * _band(L, W)
    if kind == "pairs":
        return {"bytes": L * N + 8.0 * L * L, "flops": flops}
    return {"bytes": float(L * N + 8 * L), "flops": flops + 4.0 * _splits(L, W)}


# ---------------------------------------------------------------------------
# the same outputs in FP64
# ---------------------------------------------------------------------------
RULES = [math.log(v) for v in (0.868534, 0.117609877998, 0.013856122002, 0.787640, 0.21236, 0.894603, 0.105397)]


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=DEVICE)


def _reversible(Q, pi, bls):
    """exp(Q t) for every branch length, row = state at the parent."""
    d = np.sqrt(pi)
    S = (d[:, None] * Q) / d[None, :]
    w, U = np.linalg.eigh(0.5 * (S + S.T))
    P = np.einsum("ak,nk,dk->nad", U, np.exp(w[None, :] * np.asarray(bls)[:, None]), U)
    return np.maximum(P * (d[None, None, :] / d[None, :, None]), 0.0)


def _gtr(q, pi):
    S = np.zeros((4, 4))
    for k, (i, j) in enumerate([(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]):
        S[i, j] = S[j, i] = q[k]
    S = S * pi[None, :]
    return S - np.diag(S.sum(axis=1))


def _paired_model(params, k, r1, r2):
    """Rate matrix and frequencies of the 16-state model of coevolution
    category k at site rates r1, r2."""
    lam = np.ones((4, 4))
    for (a, b), v in (((1, 2), params.lambdaratesGC), ((0, 3), params.lambdaratesAT), ((2, 3), params.lambdaratesGT)):
        lam[a, b] = lam[b, a] = v[k] + 1.0
    lam = lam.ravel()
    pi4 = np.asarray(params.freqs)
    pi = np.outer(pi4, pi4).ravel() * lam ** 2
    pi /= pi.sum()
    g = _gtr(params.q, np.ones(4))
    Q = np.zeros((16, 16))
    for h in range(16):
        for v in range(16):
            if h // 4 == v // 4 and h != v:
                Q[h, v] = g[h % 4, v % 4] * r2 * pi4[v % 4] * lam[v] / lam[h]
            elif h % 4 == v % 4 and h != v:
                Q[h, v] = g[h // 4, v // 4] * r1 * pi4[v // 4] * lam[v] / lam[h]
    return Q - np.diag(Q.sum(axis=1)), pi


def _prune(ds, P, pi, leaf_row, n):
    """log sum_a pi_a x_a at the root for n items; leaf_row(seq) gives the
    items' row numbers into the table of indicator rows and that table."""
    children = ds.children
    msg = {}
    for v in range(ds.numnodes - 1, -1, -1):
        if children[v, 0] < 0:
            rows, table = leaf_row(int(ds.seqindex[v]))
            msg[v] = ((table @ P[v].T)[rows], None)
            continue
        (a, la), (b, lb) = msg.pop(int(children[v, 0])), msg.pop(int(children[v, 1]))
        x = a * b
        del a, b
        lg = la if lb is None else (lb if la is None else la + lb)
        if v == 0:
            t = torch.log(x @ pi)
            return t if lg is None else t + lg
        m = x.amax(dim=1).clamp_min(1e-300)
        lg = torch.log(m) if lg is None else lg + torch.log(m)
        msg[v] = ((x / m[:, None]) @ P[v].T, lg)
    raise AssertionError("no root")


def _bits(masks):
    return ((masks[..., None].astype(np.int64) >> np.arange(4)) & 1).astype(np.float64)


def _unpaired(ds, params):
    """Per-site-rate and mixed log-likelihoods of the single columns."""
    codes = torch.as_tensor(ds.masks.astype(np.int64), device=DEVICE)
    table = _t(_bits(np.arange(16)))
    Q = _gtr(np.asarray(params.q), np.asarray(params.freqs))
    per = []
    for r in params.siteRates:
        P = _t(_reversible(Q * r, np.asarray(params.freqs), ds.branchlengths))
        per.append(_prune(ds, P, _t(params.freqs), lambda s: (codes[s], table), ds.numcols))
    per = torch.stack(per)
    return per, torch.logsumexp(per + torch.log(_t(params.siteWeights))[:, None], dim=0)


def _categories(params):
    for a, r1 in enumerate(params.siteRates):
        for b, r2 in enumerate(params.siteRates):
            for k, w in enumerate(params.lambdaweightsGC):
                yield a, b, k, r1, r2, math.log(params.siteWeights[a] * params.siteWeights[b] * w)


def _pair_loglik(ds, params, x, y, each=None):
    """Mixed log-likelihood of the pairs (x, y); `each` sees every category."""
    b4 = _bits(np.arange(16))
    table = _t(np.einsum("ia,jb->ijab", b4, b4).reshape(256, 16))
    codes = torch.as_tensor(ds.masks.astype(np.int64), device=DEVICE)
    step = 1 << 20
    out = torch.full((len(x),), NINF, dtype=F64, device=DEVICE)
    for a, b, k, r1, r2, logw in _categories(params):
        Q, pi = _paired_model(params, k, r1, r2)
        P, pit = _t(_reversible(Q, pi, ds.branchlengths)), _t(pi)
        for i in range(0, len(x), step):
            xs, ys = x[i:i + step], y[i:i + step]
            ll = _prune(ds, P, pit, lambda s: (codes[s][xs] * 16 + codes[s][ys], table), len(xs))
            out[i:i + step] = torch.logaddexp(out[i:i + step], ll + logw)
            if each is not None:
                each(a, b, i, ll + logw)
    return out


def _band_pairs(L, W):
    x = torch.arange(L, device=DEVICE).repeat_interleave(min(W, L - 1))
    y = x + torch.arange(1, min(W, L - 1) + 1, device=DEVICE).repeat(L)
    ok = y < L
    return x[ok], y[ok]


def _pair_band(L, W, x, y, vals):
    """p[i][k] = score of (i, i + k)."""
    p = torch.full((L, W + 1), NINF, dtype=F64, device=DEVICE)
    p[x, y - x] = vals
    return p


def _inside(u, p, L, W):
    """Z and the banded tables X[i][k] = X(i, i + k), column tables by
    Xc[j][k] = X(j - k, j); p as from _pair_band."""
    r = RULES
    S, F, Lt, Sc, Lc = (torch.full((L, W + 1), NINF, dtype=F64, device=DEVICE) for _ in range(5))
    S[:, 0], Lt[:, 0] = u + r[1], u + r[5]
    Sc[:, 0], Lc[:, 0] = S[:, 0], Lt[:, 0]
    for d in range(1, W + 1):
        n = L - d
        tmp = torch.logsumexp(Lt[:n, :d] + Sc[d:, :d].flip(1), dim=1)
        v = p[:n, d] + (F[1:n + 1, d - 2] if d >= 2 else NINF)
        S[:n, d] = torch.logaddexp(tmp + r[0], v + r[2])
        F[:n, d] = torch.logaddexp(tmp + r[4], v + r[3])
        Lt[:n, d] = v + r[6]
        Sc[d:, d], Lc[d:, d] = S[:n, d], Lt[:n, d]
    suf = torch.full((L,), NINF, dtype=F64, device=DEVICE)
    i = torch.arange(max(0, L - 1 - W), L, device=DEVICE)
    suf[i] = S[i, L - 1 - i]
    for i in range(L - 2 - W, -1, -1):
        suf[i] = r[0] + torch.logsumexp(Lt[i] + suf[i + 1:i + W + 2], dim=0)
    return suf, S, F, Lt, Sc, Lc


def _posterior_chain(u, p, L, W):
    """Row-normalised posteriors from dense FP64 inside and outside tables
    (spans beyond the band are forbidden by their scores)."""
    r = RULES
    full = torch.full((L, L), NINF, dtype=F64, device=DEVICE)
    full[:, :W + 1] = p
    p = full
    suf, S, F, Lt, Sc, Lc = _inside(u, p, L, L - 1)
    OS, OF, OL, OSc, OFc = (torch.full((L, L), NINF, dtype=F64, device=DEVICE) for _ in range(5))
    for d in range(L - 1, -1, -1):
        n = L - d
        i = torch.arange(n, device=DEVICE)
        j = i + d
        if d < L - 1:
            m = L - 1 - d  # parents up to span d + m
            oR = torch.logaddexp(OS[:n, d + 1:] + r[0], OF[:n, d + 1:] + r[4])
            sib = torch.full((n, m), NINF, dtype=F64, device=DEVICE)
            sib[:-1] = S[d + 1:, :m]
            OL[:n, d] = torch.logsumexp(oR + sib, dim=1)
            oC = torch.logaddexp(OSc[d:, d + 1:] + r[0], OFc[d:, d + 1:] + r[4])
            left = torch.full((n, m), NINF, dtype=F64, device=DEVICE)
            left[1:] = Lc[:n - 1, :m]
            OS[:n, d] = torch.logsumexp(oC + left, dim=1)
            if d <= L - 3:
                e = d + 2
                k = L - e
                OF[1:k + 1, d] = p[:k, e] + torch.logsumexp(
                    torch.stack([OS[:k, e] + r[2], OF[:k, e] + r[3], OL[:k, e] + r[6]]), dim=0)
        else:
            OS[0, d] = 0.0
        OSc[j, d], OFc[j, d] = OS[i, d], OF[i, d]
    Z = suf[0]
    single = torch.logaddexp(OS[:, 0] + r[1], OL[:, 0] + r[5]) + u - Z
    enclosed = torch.full((L, L), NINF, dtype=F64, device=DEVICE)
    enclosed[:-1, 2:] = F[1:, :-2]
    post = torch.logsumexp(torch.stack([OS + r[2], OF + r[3], OL + r[6]]), dim=0) + enclosed + p - Z
    x = torch.arange(L, device=DEVICE)
    k = x[None, :] - x[:, None]
    pair = torch.where(k >= 1, post.gather(1, k.clamp(0, L - 1)), NINF)
    pair = torch.maximum(pair, pair.T)
    norm = torch.logaddexp(torch.logsumexp(pair, dim=1), single)
    return Z, torch.exp(single - norm), torch.exp(pair - norm[:, None])


def _likelihood(ds, params, W):
    L = ds.numcols
    W = min(W, L - 1)
    _, u = _unpaired(ds, params)
    x, y = _band_pairs(L, W)
    gap = torch.as_tensor(np.asarray(ds.gapfrequency) >= 1.0, device=DEVICE)
    ll = _pair_loglik(ds, params, x, y)
    ll[gap[x] | gap[y]] = NINF
    return _inside(u, _pair_band(L, W, x, y, ll), L, W)[0][0].item(), u


def _mixture(y, t):
    K, D = NCOMP, DIM
    logit, mean, ls = y[:, :K], y[:, K:K + K * D].reshape(-1, K, D), y[:, K + K * D:].reshape(-1, K, D).clamp(-7.0, 5.0)
    z = (t[:, None, :] - mean) * torch.exp(-ls)
    comp = (-0.5 * z * z - ls).sum(dim=2) - 0.5 * math.log(2 * math.pi) * D
    return -torch.logsumexp(torch.log_softmax(logit, dim=1) + comp, dim=1).mean()


def _mlp(w, x):
    h = torch.nn.functional.silu(x @ w[0].T + w[1])
    h = torch.nn.functional.silu(h @ w[2].T + w[3])
    return h @ w[4].T + w[5]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradients"):
        w, x, t = _network(case, seed)
        w, x, t = [_t(a) for a in w], _t(x), _t(t)
        if kind == "forward":
            return _mlp(w, x)
        w = [a.requires_grad_(True) for a in w]
        loss = _mixture(_mlp(w, x), t)
        grads = torch.autograd.grad(loss, w)
        return {"loss": float(loss), "grads": torch.cat([g.reshape(-1) for g in grads])}
    if kind == "batch":
        return np.array([_likelihood(s.dataset, p, s.dataset.numcols - 1)[0] for s, p in _members(case, seed)])
    L = case["cols"]
    if kind == "decoding":
        single, pair = (_t(a) for a in _posteriors(case, seed))
        e = torch.zeros((L, L), dtype=F64, device=DEVICE)   # e[i][k] = e(i, i + k)
        ec = torch.zeros((L, L), dtype=F64, device=DEVICE)  # ec[j][k] = e(j - k, j)
        at = torch.arange(L, device=DEVICE)
        pr = pair.gather(1, (at[:, None] + at[None, :]).clamp_max(L - 1))
        for d in range(1, L):
            n = L - d
            best = torch.maximum(single[:n] + e[1:n + 1, d - 1], 2.0 * pr[:n, d] + (e[1:n + 1, d - 2] if d >= 2 else 0.0))
            if d >= 2:  # column i pairs i + k, 1 <= k < d
                inner = torch.cat([torch.zeros((n, 1), dtype=F64, device=DEVICE), e[1:n + 1, :d - 2]], dim=1)
                rest = ec[d:, :d - 1].flip(1)
                best = torch.maximum(best, (2.0 * pr[:n, 1:d] + inner + rest).amax(dim=1))
            e[:n, d] = best
            ec[d:, d] = best
        k = at[None, :] - at[:, None]
        return {"e": torch.where(k >= 0, e.gather(1, k.clamp_min(0)), torch.zeros((), dtype=F64, device=DEVICE)), "s": None}
    if kind in ("inside", "posteriors"):
        W = min(case["span"], L - 1)
        u, p = (_t(a) for a in _scores(case, seed))
        x, y = _band_pairs(L, W)
        band = _pair_band(L, W, x, y, p[x, y])
        if kind == "inside":
            return _inside(u, band, L, W)[0][0].item()
        Z, single, pair = _posterior_chain(u, band, L, W)
        return {"Z": Z.item(), "single": single, "pair": pair}
    s, params = _alignment(case, seed)
    ds, W = s.dataset, min(case["span"], L - 1)
    if kind == "likelihood":
        Z, u = _likelihood(ds, params, W)
        return {"total": Z + _logprior(params), "Z": Z, "unpaired": u}
    per, u = _unpaired(ds, params)
    if kind == "structure":
        i = np.where(s.paired > np.arange(L))[0]
        x, y = (torch.as_tensor(a, device=DEVICE) for a in (i, s.paired[i]))
        free = torch.as_tensor(s.paired < 0, device=DEVICE)
        return float(u[free].sum() + (_pair_loglik(ds, params, x, y).sum() if len(i) else 0.0))
    x, y = _band_pairs(L, W)
    if kind == "pairs":
        out = torch.full((L, L), NINF, dtype=F64, device=DEVICE)
        out[x, y] = out[y, x] = _pair_loglik(ds, params, x, y)
        return {"unpaired": u, "paired": out}
    single, pair = (_t(a) for a in _posteriors(case, seed))
    terms = [[] for _ in params.siteRates]

    def each(a, b, i, ll):
        n = len(ll)
        v = ll + torch.log(pair[x[i:i + n], y[i:i + n]])
        for cat, col in ((a, x[i:i + n]), (b, y[i:i + n])):
            m = torch.full((L,), NINF, dtype=F64, device=DEVICE).scatter_reduce(0, col, v, "amax")
            base = torch.where(torch.isfinite(m), m, 0.0)
            t = torch.zeros(L, dtype=F64, device=DEVICE).index_add(0, col, torch.exp(v - base[col]))
            terms[cat].append(base + torch.log(t))

    _pair_loglik(ds, params, x, y, each)
    out = torch.empty((len(terms), L), dtype=F64, device=DEVICE)
    for c, w in enumerate(params.siteWeights):
        out[c] = torch.logsumexp(torch.stack(terms[c] + [math.log(w) + torch.log(single) + per[c]]), dim=0)
    return out


def _logprior(params):
    """The prior of the model parameters (branch lengths not sampled)."""
    shapes = (params.lambdaGammaShapeGC, params.lambdaGammaScaleGC, params.lambdaGammaShapeAT,
              params.lambdaGammaScaleAT, params.lambdaGammaShapeGT, params.lambdaGammaScaleGT)
    lam = (params.lambdaGC - 1.0) + (params.lambdaAT - 1.0) + (params.lambdaGT - 1.0)
    w = params.lambdazeroweight
    return (-0.1 * (lam + float(np.sum(params.q)) + sum(shapes) + params.siteGammaShape)
            + math.log(6.0) + math.log(w) + math.log1p(-w))
