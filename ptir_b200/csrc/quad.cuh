// Traversal with four lanes a ray ("quad"): the calls of traverse.cuh, decision for decision, with the
// work of one node visit spread over the lanes instead of looped over.
//
// Lane c of a quad tests child c of the 4-wide node and, when that is a leaf, the leaf's candidate
// test, so the leaf tests of a visit run side by side; the k-buffer is spread over the quad (lane c
// holds entries c K/4 to (c+1) K/4 - 1); the order of the children comes from comparing keys across
// the quad, and up to four stack entries are popped at a time. A visit decides what the one-lane visit
// decides: the leaf tests of a node see the K-th distance as it was before the node, but an entry at or
// past the current K-th distance enters the sorted buffer nowhere, which is the one-lane test's
// rejection; children are visited and stacked in the same order (quad_order). What a small launch can differ in from a
// large one is a grazing candidate: the one-lane kernels seed a first round's cut (wavefront.cu), the four-lane
// ones do not.
//
// Bound: latency. A visit is a chain of a node load, box tests, leaf loads and tests, insertions and
// the descent. With one lane a ray that chain took 0.9 to 1.2 us a visit (leaf tests one after the
// other, an insertion a chain of 16 selects, 32 registers of k-buffer), and the longest of a launch's
// rays (up to 5000 visits on a million Gaussians) set the time of every bounce stage. See k_wf_trace_quad.
#pragma once

#include "leaf.cuh"

namespace ptir {

constexpr int kQuadStackEntries = kStackDepth + 2;  // quads of a warp start in different shared-memory banks

// A trace call of a quad's ray. Everything but the k-buffer part (kt, kid) is the same in its four lanes.
template <int K>
struct QuadTrace {
    static constexpr int L = K / 4;  // k-buffer entries a lane
    float3 inv;
    float tmin, tend;
    float slack, cap, floor;  // as TraceState
    float tk;                 // the K-th distance
    int node, sp;
    float kt[L];
    unsigned kid[L];
};

// What an insertion takes from the lane before: its last distance (-kFarT in the quad's first lane: nothing moves in
// there), and with it the first id of the run of equal distances that ends there. A run may start any number of
// lanes before: a lane that lies wholly in one hands on what it is handed. That takes five equal distances (three with
// K = 8), so a vote skips it for nearly every insertion (1 to 2 % of the stage: 24.8 -> 25.2 ms at 90k rays over 300k
// Gaussians). `first`: the same id for the lane's own last entry.
template <int K>
PTIR_DEV void quad_before(const QuadTrace<K>& t, unsigned c, unsigned mask, float& pt, unsigned& pid, unsigned& first) {
    constexpr int L = QuadTrace<K>::L;
    pt = __shfl_up_sync(mask, t.kt[L - 1], 1, 4);
    if (c == 0) pt = -kFarT;
    first = t.kid[0];
#pragma unroll
    for (int j = 1; j < L; ++j) first = t.kt[j] == t.kt[j - 1] ? first : t.kid[j];
    pid = __shfl_up_sync(mask, first, 1, 4);
    const bool whole = t.kt[L - 1] == pt && t.kt[0] == pt && pt < kFarT;
    if (__any_sync(mask, whole)) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {  // lanes 1, 2 and 3 in turn
            if (whole) first = pid;
            pid = __shfl_up_sync(mask, first, 1, 4);
        }
    }
}

// Insert (ts, id) into the quad's sorted k-buffer, behind equal distances; kFarT goes nowhere. Called by
// every lane of `mask` with its quad's entry. kbuf_insert's chain of swaps moves the first entry of a run of
// equal distances behind the run when something is inserted before it (an entry passes only what is
// strictly farther); so does this: an entry moves on only past a strictly nearer one (`moves`), and what arrives
// behind a run is the run's first (`run`, or `pid` where the run starts in a lane before).
template <int K>
PTIR_DEV void quad_insert(QuadTrace<K>& t, float ts, unsigned id, float pt, unsigned pid) {
    constexpr int L = QuadTrace<K>::L;
    unsigned run[L];
#pragma unroll
    for (int j = 0; j < L; ++j) run[j] = (j > 0 && t.kt[j] == t.kt[j > 0 ? j - 1 : 0]) ? run[j > 0 ? j - 1 : 0] : t.kid[j];
#pragma unroll
    for (int j = L - 1; j >= 0; --j) {
        const float prev = j > 0 ? t.kt[j > 0 ? j - 1 : 0] : pt;
        unsigned prev_id = j > 0 ? run[j > 0 ? j - 1 : 0] : pid;
        if (j > 0 && t.kt[j > 0 ? j - 1 : 0] == t.kt[0] && t.kt[0] == pt) prev_id = pid;
        const float in = fmaxf(prev, ts);
        const bool moves = in < t.kt[j];
        t.kid[j] = moves ? (ts < prev ? prev_id : id) : t.kid[j];
        t.kt[j] = moves ? in : t.kt[j];
    }
}
template <int K>
PTIR_DEV void quad_insert(QuadTrace<K>& t, float ts, unsigned id, unsigned c, unsigned mask) {
    float pt;
    unsigned pid, first;
    quad_before(t, c, mask, pt, pid, first);
    quad_insert(t, ts, id, pt, pid);
}

// number of filled entries of this lane's part
template <int K>
PTIR_DEV unsigned quad_count(const QuadTrace<K>& t) {
    return kbuf_count(t.kt);
}

// trace_start for a quad: true when node visits remain
template <int K>
PTIR_DEV bool quad_start(const AccelView& A, float3 o, float3 d, float tmin, float tend, QuadTrace<K>& t,
                         TraceCounters& ctr, unsigned c, float cap) {
    t.cap = cap;
    t.floor = -kFarT;
    t.tk = kFarT;
    kbuf_clear(t.kt, t.kid);
    if (c == 0) ++ctr.calls;
    if (A.n <= 0) return false;
    t.tmin = tmin;
    t.tend = tend;
    if (A.n == 1) {
        if (c == 0) {
            ++ctr.leaves;
            float ts;
            unsigned id;
            if (leaf_candidate_wide(A, 0, o, d, tmin, tend, kFarT, ts, id, -kFarT)) {
                t.kt[0] = ts;
                t.kid[0] = id;
                ++ctr.candidates;
            }
        }
        return false;
    }
    t.inv = make_float3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    t.slack = A.cull_slack > 0.0f ? A.cull_slack / sqrtf(dot(d, d)) : 0.0f;
    t.node = 0;
    t.sp = 0;
    return true;
}

// trace_continue for a quad
template <int K>
PTIR_DEV void quad_continue(QuadTrace<K>& t, TraceCounters& ctr) {
    ctr.candidates -= quad_count(t);
    t.floor = t.cap;
    t.cap = kFarT;
    t.node = 0;
    t.sp = 0;
}

// descend's order (traverse.cuh) over a node's children, of which lane c holds child c, `inner` when it is an internal
// one to be visited, and its key. The nearest is visited next, the lowest child of equal keys; the others are
// stacked largest key first, the lowest child first of equal keys. Returns the number of stacked children, -1 when
// there is no internal child; `best`: the next child's lane in the quad; `at`: a stacked child's place above the
// stack's top. A key comes from an interval a <= b with a above 0, so it is no NaN and compares as an integer.
// (Of equal keys those of lower children: c ^ 1 is lower where c is odd, c ^ 2 and c ^ 3 where c > 1; and the next
// child, where its key is the lane's own, is not stacked.) Integer keys with the lane in their two lowest bits took
// 4 % less of the stage (23.9 against 24.8 ms at 90k rays over 300k Gaussians), but they order keys that are equal or
// within four units of the last place otherwise than descend.
PTIR_DEV int quad_order(bool inner, float key, unsigned c, unsigned base, unsigned mask, unsigned& best, int& at) {
    const int ik = inner ? __float_as_int(key) : 0x7FFFFFFF;
    const int k1 = __shfl_xor_sync(mask, ik, 1), k2 = __shfl_xor_sync(mask, ik, 2), k3 = __shfl_xor_sync(mask, ik, 3);
    const int least = min(min(ik, k1), min(k2, k3));
    best = __ffs((__ballot_sync(mask, ik == least) >> base) & 15u) - 1;
    const int i1 = ik - (int)(c & 1u), i2 = ik - (int)((c >> 1) & 1u);
    const int np = __popc((__ballot_sync(mask, inner) >> base) & 15u) - 1;
    at = np - 3 + (k1 > i1 ? 1 : 0) + (k2 > i2 ? 1 : 0) + (k3 > i2 ? 1 : 0) - (ik == least ? 1 : 0);
    return np;
}

// One node visit of the quads in `mask` (whole quads, all of them tracing). Returns false when the
// quad's call is complete. `stack` is the quad's, in shared memory.
template <int K, bool kSlack>
PTIR_DEV bool quad_step(const AccelView& A, float3 o, float3 d, QuadTrace<K>& t, StackEntry* stack, unsigned* err,
                        TraceCounters& ctr, unsigned ln, unsigned mask) {
    constexpr int L = QuadTrace<K>::L;
    const unsigned c = ln & 3u, base = ln & 28u;
    const float3 inv = t.inv;
    float4 p, q;  // lo.xyz hi.x | hi.yz child kmax
    ld256(A.quads + 8 * (size_t)t.node + 2 * c, p, q);
    const int child = __float_as_int(q.z);
    const bool px = inv.x >= 0.0f, py = inv.y >= 0.0f, pz = inv.z >= 0.0f;
    // the clipped slab interval of visit_node
    const float3 oi = make_float3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
    const float a = max3f(fmaf(px ? p.x : p.w, inv.x, -oi.x), fmaf(py ? p.y : q.x, inv.y, -oi.y),
                          fmaxf(fmaf(pz ? p.z : q.y, inv.z, -oi.z), t.tmin));
    const float b = min3f(fmaf(px ? p.w : p.x, inv.x, -oi.x), fmaf(py ? q.x : p.y, inv.y, -oi.y),
                          fminf(fmaf(pz ? q.y : p.z, inv.z, -oi.z), t.tend));
    const float sl = (kSlack && t.slack > 0.0f) ? q.w * t.slack : 0.0f;
    const float t0 = kSlack ? a - sl : a;
    const float key = 15.0f * a + b;
    float cut = fminf(t.tk, t.cap);
    const bool hit = child != kNoChild && a <= b && (kSlack ? b + sl : b) >= t.floor && t0 <= cut;
    if (c == 0) ++ctr.nodes;
    float ts = kFarT;
    unsigned id = kNoHit;
    bool cand = false;
    if (hit && child < 0) {
        ++ctr.leaves;
        cand = leaf_candidate_wide(A, ~child, o, d, t.tmin, t.tend, cut, ts, id, t.floor);
    }
    const unsigned cands = __ballot_sync(mask, cand);
    if (cands) {  // uniform over the mask
        unsigned mine = (cands >> base) & 15u;
        do {
            const unsigned src = base + (mine ? __ffs(mine) - 1 : 0u);
            const float tin = __shfl_sync(mask, ts, src);
            const unsigned iin = __shfl_sync(mask, id, src);
            quad_insert(t, mine ? tin : kFarT, iin, c, mask);
            mine &= mine - 1u;
        } while (__any_sync(mask, mine != 0u));
        t.tk = __shfl_sync(mask, t.kt[L - 1], base + 3u);
        cut = fminf(t.tk, t.cap);
    }
    // descent: the internal children still in front of the cut
    const bool inner = hit && child >= 0 && t0 <= cut;
    unsigned best;
    int at;
    const int np = quad_order(inner, key, c, base, mask, best, at);
    const int next = __shfl_sync(mask, child, base + best);
    bool more = true, pop = np < 0;
    if (!pop) {
        if (t.sp + np > kStackDepth) {
            if (c == 0) atomicOr(err, kErrStackOverflow);
            more = false;
        } else {
            if (inner && c != best) stack[t.sp + at] = make_int2(child, __float_as_int(t0));
            t.sp += np;
            t.node = next;
        }
    }
    __syncwarp(mask);
    // pop the next subtree that can still hold a nearer candidate, four entries at a time
    while (__any_sync(mask, pop)) {
        const int i = t.sp - 1 - (int)c;
        StackEntry e = make_int2(0, 0);
        bool ok = false;
        if (pop && i >= 0) {
            e = stack[i];
            ok = __int_as_float(e.y) <= cut;
        }
        const unsigned om = (__ballot_sync(mask, ok) >> base) & 15u;
        const unsigned first = om ? __ffs(om) - 1 : 0u;
        const int popped = __shfl_sync(mask, e.x, base + first);
        if (pop) {
            if (om) {
                t.node = popped;
                t.sp -= 1 + (int)first;
                pop = false;
            } else {
                t.sp -= 4;
                if (t.sp <= 0) {
                    pop = false;
                    more = false;
                }
            }
        }
    }
    // (the entries just read are overwritten only after the next visit's ballots)
    if (!more) ctr.candidates += quad_count(t);
    return more;
}

// ------------------------------------------------------------------------------------
// Resumed calls (traverse.cuh) of a quad: what a call sets aside is appended to the quad's frontier, the entries of
// one step together, in the order in which the one-lane call sets them aside; so the next call comes to
// the same entries in the same order.

// A quad's frontier: two buffers of `cap` (code, lower bound) entries, as Frontier, and where its calls stand in them.
struct QuadFrontier {
    uint2* buf;
    int cap;
    int cur, n, pos, next;
};

constexpr int kQuadPull = (int)0x80000001;  // QuadTrace::node: the call goes on with its frontier

// append the entries of the lanes with `pred`, in lane order
PTIR_DEV void quad_defer(QuadFrontier& F, bool pred, int code, float lower, unsigned c, unsigned base, unsigned mask) {
    const unsigned m = (__ballot_sync(mask, pred) >> base) & 15u;
    if (pred) {
        const int at = F.next + __popc(m & ((1u << c) - 1u));
        if (at < F.cap) F.buf[(1 - F.cur) * F.cap + at] = make_uint2((unsigned)code, __float_as_uint(lower));
    }
    F.next += __popc(m);
}

// quad_insert that gives back the entry pushed out of a full buffer (id kNoHit when none), as kbuf_insert_evict:
// the last entry, or the first of the run of equal distances that ends there
template <int K>
PTIR_DEV void quad_insert_evict(QuadTrace<K>& t, float ts, unsigned id, unsigned c, unsigned base, unsigned mask,
                                float& et, unsigned& eid) {
    constexpr int L = QuadTrace<K>::L;
    float pt;
    unsigned pid, first;
    quad_before(t, c, mask, pt, pid, first);
    et = __shfl_sync(mask, t.kt[L - 1], base + 3u);
    eid = __shfl_sync(mask, first, base + 3u);
    if (!(ts < et)) eid = kNoHit;
    quad_insert(t, ts, id, pt, pid);
}

// trace_start<K, true, true> for a quad: with `resume` the call goes on from what the previous one set aside, unless
// that overflowed the frontier. The caller synchronises the warp between two calls: the lanes read each other's entries.
template <int K>
PTIR_DEV bool quad_start_resume(const AccelView& A, float3 o, float3 d, float tmin, float tend, QuadTrace<K>& t,
                                QuadFrontier& F, bool resume, TraceCounters& ctr, unsigned c) {
    if (!resume) F.cur = F.n = F.pos = F.next = 0;
    if (!quad_start(A, o, d, tmin, tend, t, ctr, c, kFarT)) {
        if (A.n == 1 && t.kid[0] != kNoHit) t.kid[0] = 0u;  // the k-buffer holds leaf record indices
        return false;
    }
    if (resume && F.next <= F.cap) {
        F.cur = 1 - F.cur;
        F.n = F.next;
        F.pos = F.next = 0;
        if (F.n == 0) return false;  // nothing was set aside: no candidate remains
        t.node = kQuadPull;
    } else {
        F.n = F.pos = F.next = 0;
    }
    return true;
}

// One step of a resumable call (trace_step<K, true, true, kSlack>) of the quads in `mask`: a node visit, or up to four
// consecutive leaves of the frontier. The k-buffer holds leaf record indices. False when the call is complete.
template <int K, bool kSlack>
PTIR_DEV bool quad_step_resume(const AccelView& A, float3 o, float3 d, QuadTrace<K>& t, QuadFrontier& F, StackEntry* stack,
                               unsigned* err, TraceCounters& ctr, unsigned ln, unsigned mask) {
    constexpr int L = QuadTrace<K>::L;
    const unsigned c = ln & 3u, base = ln & 28u;
    const bool pulling = t.node == kQuadPull;
    int child = kNoChild;
    float t0 = 0.0f, key = 0.0f;
    bool crossed = false;
    if (pulling) {
        const int at = F.pos + (int)c;
        if (at < F.n) {
            const uint2 e = F.buf[F.cur * F.cap + at];
            child = (int)e.x;
            t0 = __uint_as_float(e.y);
        }
    } else {
        const float3 inv = t.inv;
        float4 p, q;  // lo.xyz hi.x | hi.yz child kmax
        ld256(A.quads + 8 * (size_t)t.node + 2 * c, p, q);
        child = __float_as_int(q.z);
        const bool px = inv.x >= 0.0f, py = inv.y >= 0.0f, pz = inv.z >= 0.0f;
        const float3 oi = make_float3(o.x * inv.x, o.y * inv.y, o.z * inv.z);
        const float a = max3f(fmaf(px ? p.x : p.w, inv.x, -oi.x), fmaf(py ? p.y : q.x, inv.y, -oi.y),
                              fmaxf(fmaf(pz ? p.z : q.y, inv.z, -oi.z), t.tmin));
        const float b = min3f(fmaf(px ? p.w : p.x, inv.x, -oi.x), fmaf(py ? q.x : p.y, inv.y, -oi.y),
                              fminf(fmaf(pz ? q.y : p.z, inv.z, -oi.z), t.tend));
        t0 = (kSlack && t.slack > 0.0f) ? a - q.w * t.slack : a;
        key = 15.0f * a + b;
        crossed = child != kNoChild && a <= b;
        if (c == 0) ++ctr.nodes;
    }
    const bool hit = crossed && t0 <= t.tk;
    quad_defer(F, crossed && !hit, child, t0, c, base, mask);
    // the leading leaves of a pulled group; a node at its head is visited or set aside by itself
    const bool pulled = pulling && child != kNoChild && child < 0;
    const unsigned pm = (__ballot_sync(mask, pulled) >> base) & 15u;
    const unsigned lead = __ffs(~pm) - 1;  // leaves before the first other entry
    const bool leaf = pulling ? c < lead : (hit && child < 0);
    int test = 0;
    float ts = kFarT;
    if (leaf) {
        if (!pulling || t0 <= t.tk) test = leaf_candidate3_wide(A, ~child, o, d, t.tmin, t.tend, t.tk, ts);
        // (an entry past the K-th distance is set aside below: the K-th distance only falls)
    }
    // the leaves in order: set aside, or inserted, what leaves the buffer set aside
    unsigned mine = (__ballot_sync(mask, leaf) >> base) & 15u;
    while (__any_sync(mask, mine != 0u)) {
        const unsigned src = base + (mine ? __ffs(mine) - 1 : 0u);
        const float ti = __shfl_sync(mask, ts, src), lower = __shfl_sync(mask, t0, src);
        const int code = __shfl_sync(mask, child, src), tst = __shfl_sync(mask, test, src);
        const bool live = mine != 0u;
        const bool past = live && pulling && !(lower <= t.tk);
        if (live && !past && c == 0) ++ctr.leaves;
        const bool late = live && !past && tst != 0 && !(ti < t.tk);
        const bool in = live && !past && !late && tst == 3;
        float et;
        unsigned eid;
        quad_insert_evict(t, in ? ti : kFarT, (unsigned)~code, c, base, mask, et, eid);
        const bool out = in && eid != kNoHit;
        quad_defer(F, c == 0 && (past || late || out), out ? ~(int)eid : code, past ? lower : (late ? ti : et), c, base, mask);
        t.tk = __shfl_sync(mask, t.kt[L - 1], base + 3u);
        mine &= mine - 1u;
    }
    if (pulling) F.pos += (int)lead;
    // descent
    const bool child_in = hit && child >= 0;
    const bool inner = child_in && t0 <= t.tk;
    quad_defer(F, child_in && !inner, child, t0, c, base, mask);  // passed over after the leaf tests
    unsigned best;
    int at;
    const int np = quad_order(inner, key, c, base, mask, best, at);
    const int next = __shfl_sync(mask, child, base + best);
    bool more = true, pop = np < 0;
    if (!pop) {
        if (t.sp + np > kStackDepth) {
            if (c == 0) atomicOr(err, kErrStackOverflow);
            more = false;
        } else {
            if (inner && c != best) stack[t.sp + at] = make_int2(child, __float_as_int(t0));
            t.sp += np;
            t.node = next;
        }
    }
    __syncwarp(mask);
    while (__any_sync(mask, pop && t.sp > 0)) {
        const int i = t.sp - 1 - (int)c;
        const bool there = pop && i >= 0;
        StackEntry e = make_int2(0, 0);
        if (there) e = stack[i];
        const bool ok = there && __int_as_float(e.y) <= t.tk;
        const unsigned om = (__ballot_sync(mask, ok) >> base) & 15u;
        const unsigned first = om ? __ffs(om) - 1 : 4u;
        quad_defer(F, there && c < first, e.x, __int_as_float(e.y), c, base, mask);
        const int popped = __shfl_sync(mask, e.x, base + (first & 3u));
        if (pop && t.sp > 0) {
            if (om) {
                t.node = popped;
                t.sp -= 1 + (int)first;
                pop = false;
            } else {
                t.sp = max(t.sp - 4, 0);
            }
        }
    }
    // the stack is empty: the next frontier entries. Leaves are left to the next step; a node is visited, or set
    // aside when it lies past the K-th distance
    while (__any_sync(mask, pop)) {
        const int at = F.pos + (int)c;
        const bool there = pop && at < F.n;
        uint2 e = make_uint2(0u, 0u);
        if (there) e = F.buf[F.cur * F.cap + at];
        const bool is_leaf = there && (int)e.x < 0, visit = there && !is_leaf && __uint_as_float(e.y) <= t.tk;
        const unsigned sm = (__ballot_sync(mask, is_leaf || visit) >> base) & 15u;
        const unsigned vm = (__ballot_sync(mask, visit) >> base) & 15u;
        const unsigned first = sm ? __ffs(sm) - 1 : 4u;
        quad_defer(F, there && c < first, (int)e.x, __uint_as_float(e.y), c, base, mask);
        const int code = (int)__shfl_sync(mask, e.x, base + (first & 3u));
        if (pop) {
            if (sm) {
                const bool v = (vm >> first) & 1u;
                t.node = v ? code : kQuadPull;
                F.pos += (int)first + (v ? 1 : 0);
                pop = false;
            } else {
                F.pos = min(F.pos + 4, F.n);
                if (F.pos >= F.n) {
                    pop = false;
                    more = false;
                }
            }
        }
    }
    if (!more) ctr.candidates += quad_count(t);
    return more;
}

}  // namespace ptir
