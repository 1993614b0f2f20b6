// plan.cpp -- per-dataset pair plan: column-pattern compression, unique pair
// lists per tree node, the tree's segments with their programs and gather
// indices, level schedule and message arena layout.
//
// Semantics follow getindexdict (src/FelsensteinCUDA.jl:77-142) and
// Dataset.subcolumnrefs (src/Dataset.jl:180-196): at node v two root pairs
// share one partial when their columns have the same subtree patterns at v.
// The set of unique pairs at v is derived from the parent's unique list, so
// every node computes each distinct (pattern_v(x), pattern_v(y)) exactly
// once.  Results do not depend on the dedup, only the work does.
#include <algorithm>
#include <cstring>
#include <functional>

#include "internal.h"

namespace messi {

namespace {

// Open-addressing int64 -> int32 map.
struct KeyMap {
    std::vector<int64_t> keys;
    std::vector<int32_t> vals;
    uint64_t mask = 0;
    void reset(size_t expected)
    {
        size_t cap = 16;
        while (cap < 2 * expected + 2) cap <<= 1;
        keys.assign(cap, -1);
        vals.resize(cap);
        mask = cap - 1;
    }
    // Returns the value for key, inserting `next` if absent (then *inserted = true).
    int32_t get_or_insert(int64_t key, int32_t next, bool* inserted)
    {
        uint64_t h = ((uint64_t)key * 0x9E3779B97F4A7C15ull) >> 20;
        uint64_t s = h & mask;
        while (keys[s] >= 0 && keys[s] != key) s = (s + 1) & mask;
        if (keys[s] < 0) {
            keys[s] = key;
            vals[s] = next;
            *inserted = true;
            return next;
        }
        *inserted = false;
        return vals[s];
    }
};

}  // namespace

// ---------------------------------------------------------------------------
// Segments.  A node whose unique pairs are nearly as many as its ancestor's
// gains little from being computed once per unique pair: its rows would be
// written and read back (68 bytes each way) to save few updates.  Such a node
// joins its ancestor's segment and is recomputed in registers for each of the
// segment's pairs.  A child joins when it has at least this share of the pairs
// of the segment's top node (GB300, pruning of 64 x 1,000 / 30 x 9,000 / 100 x
// 733 columns: 0.7: 5.80 / 19.5 / 6.08 ms, 0.6: 5.72 / 18.3 / 5.70, 0.5: 6.19 /
// 19.5 / 6.38, 0.35: 6.80 / 24.3 / 7.15: below it the recomputed updates cost
// more than the rows).
// ---------------------------------------------------------------------------
constexpr double kFuseShare = 0.6;

struct SegBuilder {
    messi_dataset* ds;
    std::vector<char> in;      // node belongs to the segment being built
    std::vector<int> need;     // set-aside messages its evaluation needs

    bool internal(int v) const { return ds->children[2 * v] >= 0; }
    // fused children of v, the one that needs more set-aside messages first
    int fused(int v, int (&c)[2]) const
    {
        int k = 0;
        for (int side = 0; side < 2; side++) {
            const int w = ds->children[2 * v + side];
            if (internal(w) && in[w]) c[k++] = w;
        }
        if (k == 2 && need[c[1]] > need[c[0]]) std::swap(c[0], c[1]);
        return k;
    }
    void drop(int v)  // takes v's subtree out of the segment
    {
        in[v] = 0;
        for (int side = 0; side < 2; side++) {
            const int w = ds->children[2 * v + side];
            if (internal(w) && in[w]) drop(w);
        }
    }
    void emit(Segment& sg, int v, bool push)
    {
        int c[2];
        const int k = fused(v, c);
        const int flag = (v == 0 ? kStepRoot : 0) | (push ? kStepPush : 0);
        if (k == 2) {
            emit(sg, c[0], true);
            emit(sg, c[1], false);
            sg.steps.push_back({-1, v, flag | kStepPop});
        } else {
            int a = ds->children[2 * v], b = ds->children[2 * v + 1];
            if (k == 1) {
                emit(sg, c[0], false);
                if (a == c[0]) a = b;
            } else {
                // the larger table first: its rows are asked for a step ahead
                if (ds->nunique[b] > ds->nunique[a]) std::swap(a, b);
                sg.steps.push_back({a, v, kStepGather | kStepInit | (sg.nb++ << kStepSlotShift)});
                a = b;
            }
            sg.steps.push_back({a, v, flag | kStepGather | (sg.nb++ << kStepSlotShift)});
        }
        if (v != 0) sg.nmat++;
    }

    // Segment with top node r, then (recursively) the segments below it.
    void build(int r0)
    {
        std::vector<int> todo{r0};
        while (!todo.empty()) {
            const int r = todo.back();
            todo.pop_back();
            // nodes, largest first, until the segment is full
            std::vector<int> members{r}, cand;
            in[r] = 1;
            auto offer = [&](int v) {
                for (int side = 0; side < 2; side++) {
                    const int w = ds->children[2 * v + side];
                    if (ds->fuse && internal(w) && (double)ds->nunique[w] >= kFuseShare * (double)ds->nunique[r])
                        cand.push_back(w);
                }
            };
            offer(r);
            while (!cand.empty() && (int)members.size() < kSegMaxNodes) {
                size_t best = 0;
                for (size_t k = 1; k < cand.size(); k++)
                    if (ds->nunique[cand[k]] > ds->nunique[cand[best]]) best = k;
                const int v = cand[best];
                cand.erase(cand.begin() + (long)best);
                in[v] = 1;
                members.push_back(v);
                offer(v);
            }
            // children have larger numbers: descending order is bottom-up
            std::sort(members.begin(), members.end(), std::greater<int>());
            for (int v : members) {
                if (!in[v]) continue;
                int c[2];
                int k = fused(v, c);
                if (k == 2 && std::max(need[c[0]], 1 + need[c[1]]) > kSegMaxDepth) {
                    // too many set-aside messages: the child with fewer pairs becomes a table
                    const int w = ds->nunique[c[0]] < ds->nunique[c[1]] ? c[0] : c[1];
                    drop(w);
                    k = fused(v, c);
                }
                need[v] = (k == 2) ? std::max(need[c[0]], 1 + need[c[1]]) : (k == 1 ? need[c[0]] : 0);
            }
            Segment sg;
            sg.root = r;
            sg.n = ds->nunique[r];
            sg.depth = need[r];
            emit(sg, r, false);
            ds->seg_of[r] = (int)ds->segs.size();
            ds->segs.push_back(std::move(sg));
            for (int v : members) {
                if (!in[v]) continue;
                for (int side = 0; side < 2; side++) {
                    const int w = ds->children[2 * v + side];
                    if (internal(w) && !in[w]) todo.push_back(w);
                }
            }
            for (int v : members) in[v] = 0;
        }
    }
};

void level_add(SegLevel* lv, const Segment& sg)
{
    lv->warps += (sg.n + 31) / 32;
    lv->max_steps = std::max(lv->max_steps, (int)sg.steps.size());
    lv->max_nb = std::max(lv->max_nb, sg.nb);
    lv->max_depth = std::max(lv->max_depth, sg.depth);
    lv->units += (double)sg.n * (sg.nmat + (sg.root == 0 ? 1 : 0));
}

// Four pair groups per CTA, all categories in turn, where the level's pairs alone
// give every SM twelve warps (GB300: 1,824); below that one pair group per CTA,
// whose warps share the categories (launch_prune_level).  With the line at 4,096
// warps a level of 3,803 took 171 us and takes 118, one of 3,344 (a batch) 341 ->
// 251, the 1,872 of a root segment of 100 sequences 2,107 -> 1,517 (warps that
// share the categories do not share their matrices in L1); below the line 1,807
// take 475 us as they are and would take 505, 1,672 399 and 530.
constexpr int64_t kGroupWarpsPerSm = 12;

void level_shape(SegLevel* lv, bool fuse, int num_sms)
{
    lv->pg = (lv->warps >= kGroupWarpsPerSm * num_sms || !fuse) ? 4 : 1;
}

int build_plan(messi_dataset* ds, const messi_alignment* aln, int W, const uint8_t* pairmask, std::string* err,
               const std::vector<int2>* pairs, std::vector<int32_t>* pair_unique)
{
    const int N = aln->numseqs, L = aln->numcols, nn = aln->numnodes;
    if (N < 2 || L < 1 || nn != 2 * N - 1 || !aln->masks || !aln->children || !aln->seqindex) {
        *err = "alignment: need numseqs >= 2, numcols >= 1, numnodes == 2*numseqs-1 and all arrays";
        return MESSI_EINVAL;
    }
    if (W < 1) W = 1;
    if (W > L - 1) W = (L > 1) ? L - 1 : 1;
    ds->N = N;
    ds->L = L;
    ds->numnodes = nn;
    ds->W = W;
    ds->children.assign(aln->children, aln->children + 2 * nn);
    ds->seqindex.assign(aln->seqindex, aln->seqindex + nn);
    ds->masks.assign(aln->masks, aln->masks + (size_t)N * L);
    for (size_t i = 0; i < ds->masks.size() && !pairs; i++)  // (a list's alignment is a dataset's, checked before)
        if (ds->masks[i] == 0 || ds->masks[i] > 15) {
            *err = "alignment: nucleotide masks must be in 1..15";
            return MESSI_EINVAL;
        }
    // ---- validate the tree: binary, pre-order numbering, every node reached once
    ds->parent.assign(nn, -1);
    std::vector<int> seen_seq(N, 0);
    for (int v = 0; v < nn; v++) {
        int c0 = ds->children[2 * v], c1 = ds->children[2 * v + 1];
        if ((c0 < 0) != (c1 < 0)) { *err = "tree: every internal node needs two children"; return MESSI_EINVAL; }
        if (c0 < 0) {
            int s = ds->seqindex[v];
            if (s < 0 || s >= N || seen_seq[s]) { *err = "tree: leaves must map one-to-one to sequences"; return MESSI_EINVAL; }
            seen_seq[s] = 1;
        } else {
            for (int c : {c0, c1}) {
                if (c <= v || c >= nn || ds->parent[c] >= 0) {
                    *err = "tree: children must be later pre-order nodes with a single parent";
                    return MESSI_EINVAL;
                }
                ds->parent[c] = v;
            }
        }
    }
    for (int v = 1; v < nn; v++)
        if (ds->parent[v] < 0) { *err = "tree: node not reachable from the root"; return MESSI_EINVAL; }
    // post-order and levels
    ds->postorder.clear();
    {
        std::vector<int> stack{0};
        std::vector<char> expanded(nn, 0);
        while (!stack.empty()) {
            int v = stack.back();
            if (ds->children[2 * v] < 0 || expanded[v]) {
                ds->postorder.push_back(v);
                stack.pop_back();
            } else {
                expanded[v] = 1;
                stack.push_back(ds->children[2 * v + 1]);
                stack.push_back(ds->children[2 * v]);
            }
        }
    }
    ds->level.assign(nn, 0);
    int maxdepth = 0;
    {
        std::vector<int> depth(nn, 0);
        for (int v = 1; v < nn; v++) depth[v] = depth[ds->parent[v]] + 1;  // parent < v
        for (int v = 0; v < nn; v++) maxdepth = std::max(maxdepth, depth[v]);
    }
    if (maxdepth + 2 > kMaxStack) { *err = "tree: height above the supported limit (510)"; return MESSI_EINVAL; }
    for (int v : ds->postorder)
        if (ds->children[2 * v] >= 0)
            ds->level[v] = 1 + std::max(ds->level[ds->children[2 * v]], ds->level[ds->children[2 * v + 1]]);
    ds->H = ds->level[0];

    // ---- program of the unpaired columns: internal nodes in post-order, the
    // subtree whose evaluation stacks more first
    std::vector<int4> uops;
    {
        std::vector<int> need(nn, 0);  // results stacked while the subtree is evaluated
        for (int v : ds->postorder) {
            const int a = ds->children[2 * v], b = ds->children[2 * v + 1];
            if (a < 0) continue;
            const bool ia = ds->children[2 * a] >= 0, ib = ds->children[2 * b] >= 0;
            if (ia && ib) need[v] = std::max(std::max(need[a], need[b]), 1 + std::min(need[a], need[b]));
            else need[v] = ia ? need[a] : (ib ? need[b] : 0);
        }
        std::vector<std::pair<int, char>> stack{{0, 0}};
        while (!stack.empty()) {
            const auto [v, expanded] = stack.back();
            stack.pop_back();
            int a = ds->children[2 * v], b = ds->children[2 * v + 1];
            if (a < 0) continue;
            const bool ia = ds->children[2 * a] >= 0, ib = ds->children[2 * b] >= 0;
            // a: the child whose result comes last (the top), or the leaf when both are leaves
            if (ia && ib) {
                if (need[a] > need[b]) std::swap(a, b);
            } else if (ib) {
                std::swap(a, b);
            }
            if (expanded) {
                uops.push_back(make_int4(a, b, ds->seqindex[a], ds->children[2 * b] < 0 ? ds->seqindex[b] : -1));
                if (ds->children[2 * a] >= 0) uops.back().z = -1;
            } else {
                stack.push_back({v, 1});
                stack.push_back({a, 0});
                stack.push_back({b, 0});  // evaluated first
            }
        }
        ds->unpaired_depth = need[0];
    }

    // ---- column pattern ids per node (dense, first-occurrence order)
    // (of the pairs' columns alone where a list of pairs is given)
    std::vector<int32_t> cols;
    if (pairs) {
        std::vector<char> in(L, 0);
        for (const int2& p : *pairs)
            if (p.x >= 0 && p.x < p.y && p.y < L) in[p.x] = in[p.y] = 1;
        for (int x = 0; x < L; x++)
            if (in[x]) cols.push_back(x);
    } else {
        cols.resize(L);
        for (int x = 0; x < L; x++) cols[x] = x;
    }
    std::vector<std::vector<int32_t>> pid(nn);
    std::vector<int32_t> npat(nn, 0);
    KeyMap km;
    for (int v : ds->postorder) {
        pid[v].resize(L);
        if (ds->children[2 * v] < 0) {
            int first[16];
            for (int k = 0; k < 16; k++) first[k] = -1;
            const uint8_t* row = &ds->masks[(size_t)ds->seqindex[v] * L];
            int n = 0;
            for (int x : cols) {
                if (first[row[x]] < 0) first[row[x]] = n++;
                pid[v][x] = first[row[x]];
            }
            npat[v] = n;
        } else {
            int c0 = ds->children[2 * v], c1 = ds->children[2 * v + 1];
            km.reset(std::min<size_t>(cols.size(), (size_t)npat[c0] * npat[c1]));
            int n = 0;
            for (int x : cols) {
                bool ins;
                int64_t key = (int64_t)pid[c0][x] * npat[c1] + pid[c1][x];
                pid[v][x] = km.get_or_insert(key, n, &ins);
                if (ins) n++;
            }
            npat[v] = n;
        }
    }

    // ---- unique pairs at the root (band + mask, or an explicit pair list), band index map
    const int W1 = W + 1;
    std::vector<int32_t> bandidx(pairs ? (size_t)1 : (size_t)L * W1, -1);
    std::vector<std::vector<int32_t>> rep(nn);  // representative (x, y) per unique pair, interleaved
    ds->nunique.assign(nn, 0);
    if (pairs) {
        ds->band_pairs = (int64_t)pairs->size();
        km.reset((size_t)std::min<int64_t>(ds->band_pairs, (int64_t)npat[0] * npat[0]));
        pair_unique->assign(pairs->size(), -1);
        int32_t n = 0;
        for (size_t p = 0; p < pairs->size(); p++) {
            const int x = (*pairs)[p].x, y = (*pairs)[p].y;
            if (x < 0 || y >= L || x >= y) {
                *err = "structure: pairs must satisfy 0 <= x < y < numcols";
                return MESSI_EINVAL;
            }
            bool ins;
            const int64_t key = (int64_t)pid[0][x] * npat[0] + pid[0][y];
            const int32_t u = km.get_or_insert(key, n, &ins);
            if (ins) {
                rep[0].push_back(x);
                rep[0].push_back(y);
                n++;
            }
            (*pair_unique)[p] = u;
        }
        ds->nroot = n;
        ds->nunique[0] = n;
    } else {
        int64_t count_band = 0;
        for (int x = 0; x < L; x++) {
            int kmax = std::min(W, L - 1 - x);
            for (int k = 1; k <= kmax; k++)
                if (!pairmask || pairmask[(size_t)x + (size_t)(x + k) * L]) count_band++;
        }
        ds->band_pairs = count_band;
        km.reset((size_t)std::min<int64_t>(count_band, (int64_t)npat[0] * npat[0]));
        int32_t n = 0;
        for (int x = 0; x < L; x++) {
            int kmax = std::min(W, L - 1 - x);
            for (int k = 1; k <= kmax; k++) {
                int y = x + k;
                if (pairmask && !pairmask[(size_t)x + (size_t)y * L]) continue;
                bool ins;
                int64_t key = (int64_t)pid[0][x] * npat[0] + pid[0][y];
                int32_t u = km.get_or_insert(key, n, &ins);
                if (ins) {
                    rep[0].push_back(x);
                    rep[0].push_back(y);
                    n++;
                }
                bandidx[(size_t)x * W1 + k] = u;
            }
        }
        ds->nroot = n;
        ds->nunique[0] = n;
    }

    // ---- unique pairs per node from the parent's list (pre-order: parents first)
    std::vector<std::vector<int32_t>> li(nn), ri(nn);
    for (int v = 0; v < nn; v++) {
        if (ds->children[2 * v] < 0) continue;
        const int64_t nv = ds->nunique[v];
        for (int side = 0; side < 2; side++) {
            int c = ds->children[2 * v + side];
            std::vector<int32_t>& idx = side ? ri[v] : li[v];
            idx.resize(nv);
            km.reset((size_t)std::min<int64_t>(nv, (int64_t)npat[c] * npat[c]));
            int32_t n = 0;
            for (int64_t u = 0; u < nv; u++) {
                int x = rep[v][2 * u], y = rep[v][2 * u + 1];
                bool ins;
                int64_t key = (int64_t)pid[c][x] * npat[c] + pid[c][y];
                int32_t cu = km.get_or_insert(key, n, &ins);
                if (ins) {
                    rep[c].push_back(x);
                    rep[c].push_back(y);
                    n++;
                }
                idx[u] = cu;
            }
            ds->nunique[c] = n;
        }
        if (v != 0) { std::vector<int32_t>().swap(rep[v]); }
    }

    // ---- segments, their levels (a segment's rows are read by one segment
    // above it) and statistics
    ds->segs.clear();
    ds->seg_of.assign(nn, -1);
    {
        SegBuilder sb{ds, std::vector<char>(nn, 0), std::vector<int>(nn, 0)};
        sb.build(0);
    }
    // a segment comes after the one that reads it: levels bottom-up in reverse order
    std::vector<int> reader(ds->segs.size(), -1);
    for (int g = (int)ds->segs.size() - 1; g >= 0; g--) {
        Segment& sg = ds->segs[g];
        for (const PlanStep& st : sg.steps)
            if (st.child >= 0 && ds->seg_of[st.child] >= 0) {
                const int below = ds->seg_of[st.child];
                sg.level = std::max(sg.level, ds->segs[below].level);
                reader[below] = g;
            }
        sg.level++;
    }
    ds->SH = ds->segs[0].level;
    ds->seg_levels.assign(ds->SH + 1, SegLevel{});
    for (const Segment& sg : ds->segs) level_add(&ds->seg_levels[sg.level], sg);
    for (SegLevel& lv : ds->seg_levels) level_shape(&lv, ds->fuse, ds->ctx->num_sms);
    ds->executed = 0;
    for (const SegLevel& lv : ds->seg_levels) ds->executed += (int64_t)lv.units;
    ds->naive = ds->band_pairs * (int64_t)(N - 1);

    // ---- leaf rows: the 16 pair states allowed by the two column masks
    ds->leaf_off.assign(nn, -1);
    int64_t leaf_rows = 0;
    for (int v = 0; v < nn; v++)
        if (ds->children[2 * v] < 0) { ds->leaf_off[v] = leaf_rows; leaf_rows += ds->nunique[v]; }
    ds->leaf_rows = leaf_rows;
    std::vector<int2>& leaf = ds->leaf_host;
    leaf.assign((size_t)std::max<int64_t>(leaf_rows, 1), make_int2(0, 1));
    for (int v = 0; v < nn; v++) {
        if (ds->children[2 * v] >= 0) continue;
        const uint8_t* row = &ds->masks[(size_t)ds->seqindex[v] * L];
        for (int64_t u = 0; u < ds->nunique[v]; u++) {
            const uint8_t mx = row[rep[v][2 * u]], my = row[rep[v][2 * u + 1]];
            int states = 0;
            for (int a = 0; a < 16; a++) states |= (((mx >> (a / 4)) & 1) & ((my >> (a % 4)) & 1)) << a;
            leaf[(size_t)(ds->leaf_off[v] + u)] = make_int2(v, states);
        }
    }

    // ---- arena layout over levels: a segment's rows live from its level to its reader's
    {
        struct Iv { int64_t off, len; int last; };
        std::vector<Iv> live;
        int64_t peak = 0;
        for (int lv = 1; lv < ds->SH; lv++) {
            live.erase(std::remove_if(live.begin(), live.end(), [&](const Iv& iv) { return iv.last < lv; }),
                       live.end());
            for (size_t g = 1; g < ds->segs.size(); g++) {  // the root (0) writes mixtures, not rows
                Segment& sg = ds->segs[g];
                if (sg.level != lv) continue;
                std::sort(live.begin(), live.end(), [](const Iv& x, const Iv& y) { return x.off < y.off; });
                int64_t pos = 0;
                for (const Iv& iv : live) {
                    if (iv.off - pos >= sg.n) break;
                    pos = std::max(pos, iv.off + iv.len);
                }
                live.push_back({pos, sg.n, ds->segs[reader[g]].level});
                sg.row_off = pos;
                peak = std::max(peak, pos + sg.n);
            }
        }
        ds->arena_rows = std::max<int64_t>(peak, 1);
    }

    // ---- gather indices: for every segment the child lists to follow from its
    // top node down (composed on the device), parents before children
    std::vector<IdxOp> idx_ops;
    std::vector<IdxSeg> idx_segs;
    std::vector<int64_t> lr_off(nn, -1);
    int64_t lr_total = 0, idx_total = 0, max_seg_n = 0;
    for (int v = 0; v < nn; v++)
        if (ds->children[2 * v] >= 0) { lr_off[v] = lr_total; lr_total += 2 * ds->nunique[v]; }
    {
        std::vector<int> slot(nn, -1), local(nn, -1), inside;
        ds->nsteps = 0;
        for (Segment& sg : ds->segs) {
            sg.idx_off = idx_total;
            idx_total += ((sg.n + 31) / 32) * 32 * sg.nb;
            max_seg_n = std::max(max_seg_n, sg.n);
            ds->nsteps += (int)sg.steps.size();
            IdxSeg is{sg.idx_off, (int)idx_ops.size(), 0, (int)sg.n, sg.nb};
            inside.assign(1, sg.root);
            for (const PlanStep& st : sg.steps) {
                if (st.child >= 0) slot[st.child] = st.flags >> kStepSlotShift;
                if (!(st.flags & kStepInit) && st.self != sg.root) inside.push_back(st.self);
            }
            std::sort(inside.begin(), inside.end());
            for (size_t k = 0; k < inside.size(); k++) local[inside[k]] = (int)k;
            for (int v : inside)
                for (int side = 0; side < 2; side++) {
                    const int c = ds->children[2 * v + side];
                    idx_ops.push_back({lr_off[v] + side * ds->nunique[v], local[v], local[c] >= 0 ? local[c] : ~slot[c]});
                }
            for (int v : inside) local[v] = -1;
            is.op1 = (int)idx_ops.size();
            idx_segs.push_back(is);
        }
    }

    // ---- upload static device data
    cudaError_t e = cudaSuccess;
    int* d_lr = nullptr;
    IdxOp* d_ops = nullptr;
    IdxSeg* d_isegs = nullptr;
    std::vector<int32_t> lr((size_t)std::max<int64_t>(lr_total, 1));
    for (int v = 0; v < nn; v++)
        if (ds->children[2 * v] >= 0) {
            std::copy(li[v].begin(), li[v].end(), lr.begin() + lr_off[v]);
            std::copy(ri[v].begin(), ri[v].end(), lr.begin() + lr_off[v] + ds->nunique[v]);
        }
    std::vector<int> tree((size_t)nn * 4);
    for (int v = 0; v < nn; v++) {
        tree[4 * v] = ds->children[2 * v];
        tree[4 * v + 1] = ds->children[2 * v + 1];
        tree[4 * v + 2] = ds->seqindex[v];
        tree[4 * v + 3] = 0;
    }
    // tiles per level
    std::vector<int2> tiles;
    for (int lv = 1; lv <= ds->SH; lv++) {
        SegLevel& sl = ds->seg_levels[lv];
        sl.tile_off = (int)tiles.size();
        for (size_t g = 0; g < ds->segs.size(); g++)
            if (ds->segs[g].level == lv)
                for (int64_t b = 0; b < ds->segs[g].n; b += 32 * sl.pg) tiles.push_back(make_int2((int)g, (int)b));
        sl.tile_cnt = (int)tiles.size() - sl.tile_off;
    }
    if (tiles.empty()) tiles.push_back(make_int2(0, 0));

    // device buffers: what is uploaded, then what is only laid out
    struct Buffer {
        void** p;
        const void* src;
        size_t bytes;
        bool temporary;
    };
    const Buffer buffers[] = {
        {(void**)&ds->d_bandidx, bandidx.data(), bandidx.size() * sizeof(int32_t), false},
        {(void**)&d_lr, lr.data(), lr.size() * sizeof(int32_t), true},
        {(void**)&d_ops, idx_ops.data(), idx_ops.size() * sizeof(IdxOp), true},
        {(void**)&d_isegs, idx_segs.data(), idx_segs.size() * sizeof(IdxSeg), true},
        {(void**)&ds->d_leaf, leaf.data(), leaf.size() * sizeof(int2), false},
        {(void**)&ds->d_masks, ds->masks.data(), ds->masks.size(), false},
        {(void**)&ds->d_tree, tree.data(), tree.size() * sizeof(int), false},
        {(void**)&ds->d_uops, uops.data(), uops.size() * sizeof(int4), false},
        {(void**)&ds->d_tiles, tiles.data(), tiles.size() * sizeof(int2), false},
        {(void**)&ds->d_idx, nullptr, (size_t)std::max<int64_t>(idx_total, 1) * sizeof(int), false},
        {(void**)&ds->d_mix, nullptr, sizeof(double) * std::max<int64_t>(ds->nroot, 1), false},
        {(void**)&ds->d_mixlam, nullptr, sizeof(double) * kMaxLambda * std::max<int64_t>(ds->nroot, 1), false},
        {(void**)&ds->d_segs, nullptr, sizeof(SegDev) * ds->segs.size(), false},
        {(void**)&ds->d_steps, nullptr, sizeof(StepDev) * std::max(1, ds->nsteps), false},
    };
    auto room = [](size_t bytes) { return (bytes + 255) & ~size_t(255); };
    size_t total = 0, uploaded = 0;
    for (const Buffer& b : buffers) {
        total += room(b.bytes);
        if (b.src) uploaded += room(b.bytes);
    }
    if (ds->lent && total <= kKeptPlanBytes) {
        // one copy into the context's scratch, in its stream's order (a dozen
        // allocations and their frees took 0.2 ms of a structure's call)
        void* slab = nullptr;
        if (const int rc = ensure(ds->ctx, kSlotPlan, total, &slab)) {
            *err = "dataset upload: " + ds->ctx->last_error;
            return rc;
        }
        ds->lent_plan = true;
        std::vector<char> stage(uploaded);
        size_t at = 0;
        for (const Buffer& b : buffers) {
            *b.p = (char*)slab + at;
            if (b.src && b.bytes) std::memcpy(stage.data() + at, b.src, b.bytes);
            at += room(b.bytes);
        }
        e = cudaMemcpyAsync(slab, stage.data(), uploaded, cudaMemcpyHostToDevice, ds->ctx->stream);
        if (e == cudaSuccess && launch_segment_indices(d_isegs, d_ops, (int)idx_segs.size(), max_seg_n, d_lr, ds->d_idx,
                                                       ds->ctx->stream))
            e = cudaGetLastError();
        if (e == cudaSuccess) return MESSI_OK;
    } else {
        for (const Buffer& b : buffers) {
            if (e == cudaSuccess) e = cudaMalloc(b.p, b.bytes);
            if (e == cudaSuccess && b.src) e = cudaMemcpy(*b.p, b.src, b.bytes, cudaMemcpyHostToDevice);
        }
        if (e == cudaSuccess &&
            launch_segment_indices(d_isegs, d_ops, (int)idx_segs.size(), max_seg_n, d_lr, ds->d_idx, 0))
            e = cudaGetLastError();
        // the index kernel ran on the default stream: done before any context stream reads its output
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        for (const Buffer& b : buffers)
            if (b.temporary) cudaFree(*b.p);
        if (e == cudaSuccess) return MESSI_OK;
    }
    *err = std::string("dataset upload: ") + cudaGetErrorString(e);
    return (e == cudaErrorMemoryAllocation) ? MESSI_ENOMEM : MESSI_ECUDA;
}

void fill_descriptors(const messi_dataset* ds, float* rows, int* exps, int64_t row_base, int64_t cstride,
                      int64_t leaf_base, int64_t leaf_cstride, int node_base, int grp, const StepDev* d_steps,
                      SegDev* segs, StepDev* steps)
{
    size_t at = 0;
    for (size_t g = 0; g < ds->segs.size(); g++) {
        const Segment& sg = ds->segs[g];
        SegDev d{};
        d.steps = d_steps + at;
        d.idx = ds->d_idx + sg.idx_off;
        d.rows = rows;
        d.exps = exps;
        d.n = (int)sg.n;
        d.nsteps = (int)sg.steps.size();
        d.nb = sg.nb;
        d.grp = grp;
        if (sg.root != 0) {
            d.out = (unsigned)(row_base + sg.row_off);
            d.ocs = (unsigned)cstride;
        } else {
            d.mix = ds->d_mix;
            d.mixlam = ds->d_mixlam;
        }
        segs[g] = d;
        for (const PlanStep& st : sg.steps) {
            StepDev& o = steps[at++];
            o = StepDev{};
            o.self = node_base + st.self;
            o.flags = st.flags;
            if (st.child < 0) continue;
            const int below = ds->seg_of[st.child];
            if (below < 0) {
                o.row = (unsigned)(leaf_base + ds->leaf_off[st.child]);
                o.cs = (unsigned)leaf_cstride;
                o.flags |= kStepLeaf;
            } else {
                o.row = (unsigned)(row_base + ds->segs[below].row_off);
                o.cs = (unsigned)cstride;
            }
        }
    }
}

// Allocate the message arena for C categories (as many per pass as fit) and
// fill the segment descriptors.
int allocate_arena(messi_dataset* ds, int C, std::string* err)
{
    size_t freeb = 0, totalb = 0;
    cudaMemGetInfo(&freeb, &totalb);
    const size_t row_bytes = 16 * sizeof(float) + sizeof(int);
    size_t budget = freeb / 2;
    const int64_t leaf_rows = std::max<int64_t>(ds->leaf_rows, 1);
    int chunk = C;
    const int64_t all_rows = ds->arena_rows + leaf_rows;
    while (chunk > 1 && ((size_t)chunk * all_rows * row_bytes > budget || chunk * all_rows > (int64_t)UINT32_MAX))
        chunk = (chunk + 1) / 2;
    if (all_rows > (int64_t)UINT32_MAX) {
        *err = "message arena: more than 2^32 rows";
        return MESSI_ENOMEM;
    }
    if (ds->chunk != chunk) {
        if (ds->d_arena_f && !ds->lent_arena) cudaFree(ds->d_arena_f);
        if (ds->d_arena_e && !ds->lent_arena) cudaFree(ds->d_arena_e);
        ds->d_arena_f = nullptr;
        ds->d_arena_e = nullptr;
        ds->d_leafmsg = nullptr;
        ds->chunk = 0;
        const size_t fbytes = (size_t)chunk * all_rows * 16 * sizeof(float), ebytes = (size_t)chunk * ds->arena_rows * sizeof(int);
        ds->lent_arena = ds->lent && fbytes + ebytes <= kKeptPlanBytes;
        // segment rows, then the leaf messages (which have no exponents)
        cudaError_t e = cudaSuccess;
        if (ds->lent_arena) {
            void* rows = nullptr;
            if (const int rc = ensure(ds->ctx, kSlotPlanRows, fbytes + ebytes, &rows)) {
                *err = "message arena: " + ds->ctx->last_error;
                return rc;
            }
            ds->d_arena_f = (float*)rows;
            ds->d_arena_e = (int*)((char*)rows + fbytes);
        } else {
            e = cudaMalloc((void**)&ds->d_arena_f, fbytes);
            if (e == cudaSuccess) e = cudaMalloc((void**)&ds->d_arena_e, ebytes);
        }
        if (e != cudaSuccess) {
            *err = std::string("message arena: ") + cudaGetErrorString(e);
            return MESSI_ENOMEM;
        }
        ds->d_leafmsg = ds->d_arena_f + (size_t)chunk * ds->arena_rows * 16;
        ds->chunk = chunk;
    }
    ds->arena_gen++;
    ds->segs_host.assign(ds->segs.size(), SegDev{});
    ds->steps_host.assign((size_t)ds->nsteps, StepDev{});
    fill_descriptors(ds, ds->d_arena_f, ds->d_arena_e, 0, ds->arena_rows, (int64_t)ds->chunk * ds->arena_rows,
                     leaf_rows, 0, 0, ds->d_steps, ds->segs_host.data(), ds->steps_host.data());
    // in the stream's order: behind the last reader, before the next
    auto upload = [&](void* dst, const void* src, size_t bytes) {
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ds->ctx->stream);
    };
    cudaError_t e = upload(ds->d_segs, ds->segs_host.data(), sizeof(SegDev) * ds->segs.size());
    if (e == cudaSuccess) e = upload(ds->d_steps, ds->steps_host.data(), sizeof(StepDev) * (size_t)ds->nsteps);
    if (e != cudaSuccess) {
        *err = std::string("segment descriptors: ") + cudaGetErrorString(e);
        return MESSI_ECUDA;
    }
    return MESSI_OK;
}

}  // namespace messi
