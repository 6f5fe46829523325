// One lane a ray with the k-buffer's distances in registers and its ids in a log: the calls of traverse.cuh from
// the root, decision for decision.
//
// While a call runs only the K-th distance is needed. kbuf_insert carries distance and id of 16 entries through a
// chain of compare-and-swap steps, five instructions an entry on the half-rate pipe, and holds 32 registers. Here
// the sorted buffer holds the distances alone (entry j becomes min(kt[j], max(kt[j-1], t)), two independent
// instructions an entry), every inserted (distance, id) is appended to a log in local memory, and the ids
// are put in order once, when the call ends (near_resolve). With 16 registers less the kernel fits 72, seven blocks
// of 128 threads an SM instead of five. Intersection stage of 786k paths over 1M Gaussians, forward and
// adjoint: 147.5 -> 133.0 ms; of 627k over 600k: 72.3 -> 65.6. (With the children sorted by integer keys that hold the
// child in their two lowest bits, in place of descend's whole keys: 135.1 and 67.8, and another order of close keys.)
#pragma once

#include "leaf.cuh"

namespace ptir {

// Log entries a lane, (distance bits, id) in insertion order. A full log drops what is past the K-th
// distance: that leaves at most K - 1 nearer entries and K equal ones.
// A call of 16 inserts about 34 entries. 34 entries of log: 133.9 ms in the stage at 1M Gaussians; 48: 133.0; 64: 132.4.
constexpr int kNearLog = 48;

template <int K>
struct Near {
    static_assert(2 * K - 1 < kNearLog, "a compacted log has room");
    float kt[K];  // sorted distances
    int n;        // log entries
};

template <int K>
PTIR_DEV void near_clear(Near<K>& b) {
#pragma unroll
    for (int j = 0; j < K; ++j) b.kt[j] = kFarT;
    b.n = 0;
}

template <int K>
PTIR_DEV void near_insert(Near<K>& b, uint2* log, float t, unsigned id) {
    log[b.n++] = make_uint2(__float_as_uint(t), id);
#pragma unroll
    for (int j = K - 1; j > 0; --j) b.kt[j] = fminf(b.kt[j], fmaxf(b.kt[j - 1], t));
    b.kt[0] = fminf(b.kt[0], t);
    if (b.n == kNearLog) {
        int m = 0;
#pragma unroll 1
        for (int i = 0; i < kNearLog; ++i) {
            const uint2 e = log[i];
            if (__uint_as_float(e.x) <= b.kt[K - 1]) log[m++] = e;
        }
        b.n = m;
    }
}

// The finished call's candidates in order: entry i at out_t[i * stride], out_id[i * stride], the id kNoHit past
// the last. Where distances are equal (two of the buffer, or one of the buffer and one that left it), the order is
// the one kbuf_insert's chain of swaps leaves, from running that chain over the log: what the log has dropped lay
// past every entry that counts and moved none of them.
template <int K>
PTIR_DEV void near_resolve(const Near<K>& b, const uint2* log, float* out_t, unsigned* out_id, int stride) {
    bool ties = false;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        out_t[j * stride] = b.kt[j];
        out_id[j * stride] = kNoHit;
        if (j > 0) ties = ties || (b.kt[j] == b.kt[j - 1] && b.kt[j] < kFarT);
    }
    int last = 0;  // log entries at the K-th distance
#pragma unroll 1
    for (int i = 0; i < b.n; ++i) {
        const uint2 e = log[i];
        const float t = __uint_as_float(e.x);
        int rank = 0;
#pragma unroll
        for (int j = 0; j < K; ++j) rank += b.kt[j] < t ? 1 : 0;
        if (rank < K) out_id[rank * stride] = e.y;
        last += t == b.kt[K - 1] ? 1 : 0;
    }
    if (!ties && last <= 1) return;
#pragma unroll 1
    for (int j = 0; j < K; ++j) {
        out_t[j * stride] = kFarT;
        out_id[j * stride] = kNoHit;
    }
#pragma unroll 1
    for (int i = 0; i < b.n; ++i) {
        const uint2 e = log[i];
        float t = __uint_as_float(e.x);
        unsigned id = e.y;
#pragma unroll 1
        for (int j = 0; j < K; ++j) {
            const float tt = out_t[j * stride];
            if (t < tt) {
                const unsigned ii = out_id[j * stride];
                out_t[j * stride] = t;
                out_id[j * stride] = id;
                t = tt;
                id = ii;
            }
        }
    }
}

// trace_start: true when node visits remain
template <int K>
PTIR_DEV bool near_start(const AccelView& A, float3 o, float3 d, float tmin, float tend, Near<K>& b, uint2* log,
                         TraceState& t, TraceCounters& ctr, float cap) {
    t.cap = cap;
    t.floor = -kFarT;
    near_clear(b);
    ++ctr.calls;
    if (A.n <= 0) return false;
    t.tmin = tmin;
    t.tend = tend;
    if (A.n == 1) {
        ++ctr.leaves;
        float ts;
        unsigned id;
        if (leaf_candidate_wide(A, 0, o, d, tmin, tend, kFarT, ts, id, -kFarT)) {
            near_insert(b, log, ts, id);
            ++ctr.candidates;
        }
        return false;
    }
    t.inv = make_float3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    t.slack = A.cull_slack > 0.0f ? A.cull_slack / sqrtf(dot(d, d)) : 0.0f;
    t.node = 0;
    t.sp = 0;
    return true;
}

// One 4-wide node visit with its leaf tests (trace_step). Returns false when the call is complete.
template <int K, bool kSlack>
PTIR_DEV bool near_step(const AccelView& A, float3 o, float3 d, TraceState& t, Near<K>& b, uint2* log,
                        StackEntry* stack, unsigned* err, TraceCounters& ctr) {
    NodeVisit v;
    unsigned leaves = visit_node<K, false, kSlack>(A, o, t, b.kt, v, ctr);
    while (leaves) {
        const int k = __ffs(leaves) - 1;
        leaves &= leaves - 1;
        const int c = k == 0 ? v.ch[0] : (k == 1 ? v.ch[1] : (k == 2 ? v.ch[2] : v.ch[3]));
        ++ctr.leaves;
        float ts;
        unsigned id;
        if (leaf_candidate_wide(A, ~c, o, d, t.tmin, t.tend, fminf(b.kt[K - 1], t.cap), ts, id, t.floor))
            near_insert(b, log, ts, id);
    }
    if (descend<K>(t, v, b.kt, stack, err, ctr)) return true;
    ctr.candidates += kbuf_count(b.kt);
    return false;
}

}  // namespace ptir
