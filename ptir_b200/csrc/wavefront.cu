// Wavefront path tracer and adjoint: each path stage is its own kernel over a compacted queue.
//
// Paths are processed in chunks of whole 8x4 pixel tiles (slot q of a chunk = lane q % 32 of
// tile q / 32, so the primary rays of a warp stay coherent). Per chunk, the forward runs
//   camera   : sampler seed and primary ray of every slot              -> intersect queue
//   intersect: primary segment                                        (all slots)
//   primary  : primary outputs, NEE light sample                       -> shadow queue | bounce queue
//   shadow   : stochastic shadow ray of the NEE sample                -> bounce queue
//   bounce d : light gathering, path termination, BRDF sample          -> intersect queue
//   sort     : the intersect queue in (octant, origin cell, direction cell) order, where it holds more than
//              kQuadRays rays
//   intersect: next segment                                            -> bounce queue
// and the backward the same with the adjoint stages, whose re-traversals (the reference's
// rayIntersectBwd) go to a replay queue drained after every bounce stage. Path state lives in
// HBM between stages; queues are appended with one atomic per warp (ballot + popc). The
// intersect, shadow and replay stages take four lanes a ray for queues of up to kQuadRays (quad.cuh) and
// one lane a ray above; the queue's count on the device decides. Lanes and quads are refilled one by one.
// The per-path order of random draws is the megakernel's, so both schedules produce the same paths.

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "radix_sort.cuh"
#include "path.cuh"
#include "near.cuh"
#include "quad_path.cuh"
#include "wavefront.h"

namespace ptir {

namespace {

constexpr int kMaxThreads = 256;  // largest block size; the kernels use warps only, no block barriers

struct WfView {
    Segment* seg;
    PathState* ps;
    unsigned long long* rng;
    unsigned* q[3];          // bounce, intersect, shadow
    unsigned* count;         // [kNumQueueCounts]
    unsigned* cursor;        // [kNumCursors]
    ReplayJob* jobs;
    float* parked;           // intersection: parked accumulators and k-buffer batches, per thread
    uint2* frontier;         // intersection: two frontier buffers of frontier_cap entries per thread
    int frontier_cap;
    unsigned long long tile0;  // first tile of the chunk
    unsigned slots;          // paths in the chunk (32 per tile)
};

enum : int { kQBounce = 0, kQIsect = 1, kQShadow = 2, kQJobs = 3 };

PTIR_DEV unsigned lane() { return threadIdx.x & 31u; }

// the next 32 items of a queue for this warp (uniform across the warp)
PTIR_DEV unsigned fetch32(unsigned* cursor) {
    unsigned base = 0;
    if (lane() == 0) base = atomicAdd(cursor, 32u);
    return __shfl_sync(0xFFFFFFFFu, base, 0);
}

// append `value` for the lanes with `pred` (called by the whole warp)
PTIR_DEV void push(unsigned* items, unsigned* count, unsigned value, bool pred) {
    const unsigned mask = __ballot_sync(0xFFFFFFFFu, pred);
    if (!mask) return;
    const unsigned leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane() == leader) base = atomicAdd(count, __popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (pred) items[base + __popc(mask & ((1u << lane()) - 1u))] = value;
}

PTIR_DEV void push_job(ReplayJob* jobs, unsigned* count, const ReplayJob& j, bool pred) {
    const unsigned mask = __ballot_sync(0xFFFFFFFFu, pred);
    if (!mask) return;
    const unsigned leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane() == leader) base = atomicAdd(count, __popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (pred) jobs[base + __popc(mask & ((1u << lane()) - 1u))] = j;
}

// slot q of the chunk -> view, launch index (x, y, z) and flat launch index li; false for slots
// outside every image
PTIR_DEV bool slot_index(const TraceParams& P, const WfView& W, unsigned q, int& view, unsigned& x, unsigned& y,
                         unsigned& z, size_t& li) {
    return tile_launch(P, (long long)W.tile0 + (q >> 5), q & 31u, view, x, y, z, li);
}

PTIR_DEV void store_rng(const WfView& W, unsigned q, const Pcg32& r) { W.rng[q] = r.state; }
PTIR_DEV Pcg32 load_rng(const WfView& W, unsigned q) {
    Pcg32 r;
    r.state = W.rng[q];
    r.inc = 1ull;
    return r;
}

PTIR_DEV void write_pbr(const FwdOutputs& O, size_t li, const PathState& ps) {
    float* pb = O.pbr + 3 * li;
    pb[0] = ps.acc.x; pb[1] = ps.acc.y; pb[2] = ps.acc.z;
    float* lg = O.light + 3 * li;
    lg[0] = ps.acc_light.x; lg[1] = ps.acc_light.y; lg[2] = ps.acc_light.z;
    float* cp = O.components + 6 * li;
    cp[0] = ps.acc_direct.x; cp[1] = ps.acc_direct.y; cp[2] = ps.acc_direct.z;
    cp[3] = ps.acc_indirect.x; cp[4] = ps.acc_indirect.y; cp[5] = ps.acc_indirect.z;
    if (O.path_sig) O.path_sig[li] = ps.sig;
}

#define PTIR_STAGE_PROLOGUE                         \
    StackEntry stack[kStackDepth];                     \
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0}; \
    CtxT<K> C{P, stack, ctr};

// ---------------------------------------------------------------------------------------
// ray order

// Sort key of a ray: direction octant (3 bits), then the Morton code of its origin's cell (4 bits
// per axis of the scene bounds), then the Morton code of its direction's cell within the octant
// (4 bits per axis of the normalised |d|): 27 bits. Coarse origin cells with fine direction cells keep
// the rays of a warp on similar traversals; against octant + 8-bit origin cells alone this cut
// the intersection stage by 7 % on the 1M-Gaussian scene.
constexpr int kSortKeyBits = 27;

PTIR_DEV unsigned spread3_8(unsigned v) {
    v &= 0xFFu;
    v = (v | (v << 8)) & 0x0000F00Fu;
    v = (v | (v << 4)) & 0x000C30C3u;
    v = (v | (v << 2)) & 0x00249249u;
    return v;
}

// Keys of queue in_q: the intersect queue's segment rays, or the shadow queue's rays toward their
// light samples.
__global__ void __launch_bounds__(kMaxThreads) k_wf_sort_keys(TraceParams P, WfView W, int in_q, unsigned* keys,
                                                              unsigned quad_rays) {
    const unsigned count = W.count[in_q];
    if (count <= quad_rays) return;
    float3 lo = f3(0.0f), scale = f3(0.0f);
    if (P.accel.n > 0) {
        const float4 a = __ldg(P.accel.bounds), b = __ldg(P.accel.bounds + 1);
        lo = make_float3(a.x, a.y, a.z);
        scale = make_float3(255.0f / fmaxf(b.x - a.x, 1e-30f), 255.0f / fmaxf(b.y - a.y, 1e-30f),
                            255.0f / fmaxf(b.z - a.z, 1e-30f));
    }
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const unsigned q = W.q[in_q][i];
        float3 o = W.seg[q].o, d = W.seg[q].d;
        if (in_q == kQShadow) {
            d = W.ps[q].em.dir;
            o = W.seg[q].pos + d * 2e-2f;
        }
        const unsigned oct = (d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u);
        const float3 c = (o - lo) * scale * (1.0f / 16.0f);
        const unsigned cx = (unsigned)fminf(fmaxf(c.x, 0.0f), 15.0f);
        const unsigned cy = (unsigned)fminf(fmaxf(c.y, 0.0f), 15.0f);
        const unsigned cz = (unsigned)fminf(fmaxf(c.z, 0.0f), 15.0f);
        const float dn = rsqrtf(fmaxf(dot(d, d), 1e-30f));
        const unsigned dx = (unsigned)fminf(fabsf(d.x) * dn * 16.0f, 15.0f);
        const unsigned dy = (unsigned)fminf(fabsf(d.y) * dn * 16.0f, 15.0f);
        const unsigned dz = (unsigned)fminf(fabsf(d.z) * dn * 16.0f, 15.0f);
        const unsigned ocell = (spread3_8(cx) << 2) | (spread3_8(cy) << 1) | spread3_8(cz);
        const unsigned dcell = (spread3_8(dx) << 2) | (spread3_8(dy) << 1) | spread3_8(dz);
        keys[i] = (oct << 24) | (ocell << 12) | dcell;
    }
}

// ---------------------------------------------------------------------------------------
// intersection with per-lane refill

PTIR_DEV unsigned lanes_below() { return (1u << lane()) - 1u; }

// The compositing accumulators of a lane's segment, parked in global memory while its warp
// traverses (they are only touched between trace calls, about three times per segment, and stay
// in L2), so that they hold no registers during the traversal and no shared memory: L1 keeps
// all of its capacity for node and leaf records. One float per field and thread, field-major
// with the grid's thread count as stride (coalesced).
constexpr int kParkedFields = 22;

struct Parked {
    float* base;  // this thread's first field
    int stride;   // threads of the grid
    __device__ __forceinline__ float& f(int k) const { return base[k * stride]; }
    __device__ __forceinline__ void save(const Composite& c) const {
        f(0) = c.radiance.x; f(1) = c.radiance.y; f(2) = c.radiance.z;
        f(3) = c.normal.x; f(4) = c.normal.y; f(5) = c.normal.z;
        f(6) = c.albedo.x; f(7) = c.albedo.y; f(8) = c.albedo.z;
        f(9) = c.snrm.x; f(10) = c.snrm.y; f(11) = c.snrm.z;
        f(12) = c.transmittance; f(13) = c.depth; f(14) = c.hit2; f(15) = c.distortion;
        f(16) = c.hits_count; f(17) = c.rough; f(18) = c.metal; f(19) = c.last_hit; f(20) = c.clip_end;
        f(21) = c.hit ? 1.0f : 0.0f;
    }
    __device__ __forceinline__ void load(Composite& c, float3 o, float3 d) const {
        c.o = o;
        c.d = d;
        c.radiance = make_float3(f(0), f(1), f(2));
        c.normal = make_float3(f(3), f(4), f(5));
        c.albedo = make_float3(f(6), f(7), f(8));
        c.snrm = make_float3(f(9), f(10), f(11));
        c.transmittance = f(12); c.depth = f(13); c.hit2 = f(14); c.distortion = f(15);
        c.hits_count = f(16); c.rough = f(17); c.metal = f(18); c.last_hit = f(19); c.clip_end = f(20);
        c.hit = f(21) != 0.0f;
    }
};

// Registers per thread of k_wf_trace (and of k_wf_shadow of the same k-buffer size). The
// kernels use no shared memory, so registers alone set the resident warps. K <= 16: 96, five
// 128-thread blocks per SM, 5 % faster than the compiler's own 127 (four blocks) despite a few
// spills; 80 (six blocks) was 11 % slower (both measured on rounds from the root).
// K = 32: 128, four blocks, 6 % faster for the step than 168 (three blocks); 96 (five blocks) was 23 % slower.
constexpr int trace_regs(int K) { return K > 16 ? 128 : 96; }

// Seed of the k-buffer rounds in the intersection stage: the cut starts at the round's tmin plus
// this multiple of a span, the previous round's (its K-th less its first distance) for a segment's
// later rounds. On 2 views of 512x384x4 (1M Gaussians) 17 % of those rounds were continued past
// the seed at 2, and the step took 150.9 ms, against 163.8 ms unseeded, 154.6 ms at 1.5 and 154.1
// ms at 3. Seeding the first rounds as well (from the lane's last segment) took it to 142.0 ms (5.6 %
// of them continued), against 145.5 ms at 1.5 and 143.2 ms at 3.
constexpr float kSeedSpan = 2.0f;

// Rays up to which an intersection launch takes four lanes a ray. Measured against one lane with ids in registers (the
// stage, ms): 1.92 -> 1.01 at 16k rays over 10k Gaussians, 37.2 -> 25.2 at 90k over 300k. Where the line lies,
// against k_wf_trace_near (lines at 65,536 / 94,720 / 131,072 / 262,144 rays): 24.0 / 25.2 / 25.2 / 25.0 at 90k over
// 300k and 12.5 / 11.5 / 11.5 / 11.6 at 90k over 100k; 7.8 / 7.7 / 7.5 / 7.6 at 278k primary and 80k bounce rays over
// 30k; 65.7 / 66.2 / 65.6 / 73.1 at 627k paths of several views over 600k; 133.0 / 132.9 / 133.0 / 141.9 at 786k
// primary and about 200k bounce rays over 1M.
constexpr unsigned kQuadRays = 1u << 17;

// Intersection stage: each lane carries one segment of queue `in_q` (read from `items`, the
// queue in queue or sorted order) through as many trace calls as it needs (composite_begin /
// trace / composite_hits / composite_end). A lane whose call has finished composites its batch
// and starts the next call, or writes its segment, hands it to queue `out_q` (when >= 0) and
// takes the next one from the queue, so that no lane waits for the slowest segment of its warp.
// The warp leaves its traversal loop once `refill` lanes wait (a finished call, or idle while
// the queue still holds segments). W.parked holds, per thread of the grid, the parked
// accumulators and, while a batch is composited, its k-buffer (kParkedFields + 2K floats).
//
// Three kernels do this: k_wf_trace (two rounds a traversal with K = 32, and resumed rounds), k_wf_trace_near
// (rounds from the root, K <= 16) and k_wf_trace_quad (the same, four lanes a ray, for small launches).
//
// With K = 32 a traversal stands for two of the reference's 16-candidate rounds (the rounds of
// pathTracer.cuh:216-311): its first 16 candidates are the first round, and its last 16 are the
// second when each of them is a candidate of the second round's own call, i.e. lies past the
// first round's last hit and has its instance box crossed within the second round's interval;
// otherwise the second round is traced. The results are those of 16-candidate rounds (a 32-entry
// traversal culls at a farther distance, so it keeps grazing candidates that a 16-entry one can
// cull, as an exact nearest-16 selection would), with about a third fewer node visits per segment.
//
// With kResume (K <= 16) a segment's calls after its first resume from the frontier its previous
// call set aside (traverse.cuh), in a lane's part of W.frontier. kSlack builds the kernel that
// applies the exact-candidate cull slack (only tracers with exact_candidates launch it).
template <int K, bool kMark, bool kSelfOcc, bool kResume, bool kSlack>
__global__ void __maxnreg__(trace_regs(K)) k_wf_trace(TraceParams P, float* vis, WfView W, int in_q,
                                                      const unsigned* items, int out_q, unsigned cursor, int refill,
                                                      unsigned quad_rays) {
    constexpr bool kPair = K == 32;  // traversals gather two 16-candidate rounds (leaf-index k-buffer)
    // the k-buffer holds leaf record indices
    static_assert(kPair != kResume, "rounds from the root with K <= 16 are k_wf_trace_near's and k_wf_trace_quad's");
    static_assert(!(kSlack && kResume), "the exact-candidate slack is applied by the rounds from the root");
    const int nthreads = (int)(gridDim.x * blockDim.x);
    const Frontier F{kResume ? W.frontier + (size_t)(blockIdx.x * blockDim.x + threadIdx.x) * 2 * W.frontier_cap
                             : nullptr,
                     W.frontier_cap};
    float* const base = W.parked + blockIdx.x * blockDim.x + threadIdx.x;
    const Parked pk{base, nthreads};
    float* const batch_t = base + kParkedFields * nthreads;
    unsigned* const batch_id = reinterpret_cast<unsigned*>(batch_t + K * nthreads);
    StackEntry stack[kStackDepth];
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    constexpr unsigned kFull = 0xFFFFFFFFu;
    enum : int { kIdle = 0, kTracing = 1, kReady = 2 };
    const unsigned count = W.count[in_q];
    if (count <= quad_rays) return;  // the quads' launch
    int phase = kIdle;
    unsigned q = 0;
    int rounds = 0;
    bool drained = false;
    float3 ro = f3(0.0f), rd = f3(0.0f);  // the lane's segment ray
    TraceState t;
    float kt[K];  // a call found nothing when kt[0] == kFarT
    unsigned kid[K];
    // next trace call of this lane's segment, or ready with nothing found when it is complete
    auto next_call = [&](const Composite& c) {
        if (!composite_open(P, c)) {
            kt[0] = kFarT;
            phase = kReady;
            return;
        }
        if (++rounds > kMaxRounds + 1) {
            atomicOr(P.error_word, kErrLoopBound);
            kt[0] = kFarT;
            phase = kReady;
            return;
        }
        phase = trace_start<K, true, kResume>(P.accel, ro, rd, composite_tmin(c), composite_tend(c), kt, kid, t, ctr, &F,
                                              rounds > 1)
                    ? kTracing
                    : kReady;
    };
    // the segment is complete: no call remains
    auto no_call = [&]() {
        kt[0] = kFarT;
        phase = kReady;
    };
    while (true) {
        // refill the idle lanes
        const unsigned idle = __ballot_sync(kFull, phase == kIdle);
        if (!drained && idle) {
            const unsigned n_idle = __popc(idle);
            unsigned base = 0;
            if (lane() == 0) base = atomicAdd(W.cursor + cursor, n_idle);
            base = __shfl_sync(kFull, base, 0);
            drained = base + n_idle >= count;
            if (phase == kIdle) {
                const unsigned i = base + __popc(idle & lanes_below());
                if (i < count) {
                    q = items[i];
                    Composite c;
                    composite_begin(P, c, W.seg[q].o, W.seg[q].d);
                    ro = c.o;
                    rd = c.d;
                    ++ctr.segments;
                    rounds = 0;
                    next_call(c);
                    pk.save(c);
                }
            }
        }
        const unsigned busy = __ballot_sync(kFull, phase != kIdle);
        if (!busy) {
            if (drained) break;
            continue;
        }
        // traverse until enough lanes wait
        const unsigned eligible = drained ? busy : kFull;
        while (true) {
            const unsigned tracing = __ballot_sync(kFull, phase == kTracing);
            if (!tracing || __popc(eligible & ~tracing) >= refill) break;
            if (phase == kTracing &&
                !trace_step<K, true, kResume, kSlack>(P.accel, ro, rd, t, kt, kid, stack, P.error_word, ctr, &F))
                phase = kReady;
        }
        // composite the finished calls; hand on the finished segments
        bool done = false;
        if (phase == kReady) {
            Composite c;
            pk.load(c, ro, rd);
            if (kt[0] < kFarT) {
                // the batch goes to the parked buffer, so compositing holds no k-buffer registers
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    batch_t[i * nthreads] = kt[i];
                    batch_id[i * nthreads] = kid[i];
                }
                float* const mark = kMark ? vis : nullptr;
                if constexpr (kPair) {
                    composite_leaf_batch<kSelfOcc>(P, ctr, c, batch_t, batch_id, nthreads, 0, 16, mark);
                    bool call = composite_open(P, c) && batch_id[16 * nthreads] != kNoHit;
                    if (call) {
                        const float tmin2 = composite_tmin(c), tend2 = composite_tend(c);
                        bool second = true;
#pragma unroll 1
                        for (int i = 16; i < 32 && second; ++i) {
                            const unsigned p = batch_id[i * nthreads];
                            if (p == kNoHit) break;
                            second = batch_t[i * nthreads] > tmin2 && leaf_box_hit(P.accel, p, ro, rd, tmin2, tend2);
                        }
                        if (second) {
                            composite_leaf_batch<kSelfOcc>(P, ctr, c, batch_t, batch_id, nthreads, 16, 32, mark);
                            call = composite_open(P, c) && batch_id[31 * nthreads] != kNoHit;
                        }
                    }
                    if (call) next_call(c);
                    else no_call();
                } else {
                    composite_leaf_batch<kSelfOcc>(P, ctr, c, batch_t, batch_id, nthreads, 0, K, mark);
                    // a k-buffer that is not full held every candidate of the call: a later call finds none
                    if (kid[K - 1] != kNoHit) next_call(c);
                    else no_call();
                }
            }
            // nothing found, segment closed, or loop bound: the segment is complete
            if (phase == kReady && kt[0] >= kFarT) {
                Segment s;
                Pcg32 rng = load_rng(W, q);
                composite_end(P, c, W.seg[q].scatter_pdf, W.seg[q].light_pdf, s, rng);
                W.seg[q] = s;
                store_rng(W, q, rng);
                phase = kIdle;
                done = true;
            } else {
                pk.save(c);
            }
        }
        if (out_q >= 0) push(W.q[out_q], W.count + out_q, q, done);
    }
    flush_counters(P, ctr);
}

// k_wf_trace for the rounds from the root (K <= 16), with the k-buffer of near.cuh: the same calls, seeds and
// compositing. 72 registers: on 786k paths over 1M Gaussians (forward and adjoint) the stage took 133.0 ms, against
// 137.5 at 80, 144.6 at 64 and 168.5 at 56.
template <int K, bool kMark, bool kSelfOcc, bool kSlack>
__global__ void __maxnreg__(72) k_wf_trace_near(TraceParams P, float* vis, WfView W, int in_q, const unsigned* items,
                                                int out_q, unsigned cursor, int refill, unsigned quad_rays) {
    const int nthreads = (int)(gridDim.x * blockDim.x);
    float* const base = W.parked + blockIdx.x * blockDim.x + threadIdx.x;
    const Parked pk{base, nthreads};
    float* const batch_t = base + kParkedFields * nthreads;
    unsigned* const batch_id = reinterpret_cast<unsigned*>(batch_t + K * nthreads);
    StackEntry stack[kStackDepth];
    uint2 log[kNearLog];
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    constexpr unsigned kFull = 0xFFFFFFFFu;
    enum : int { kIdle = 0, kTracing = 1, kReady = 2 };
    const unsigned count = W.count[in_q];
    if (count <= quad_rays) return;  // the quads' launch
    int phase = kIdle;
    unsigned q = 0;
    int rounds = 0;
    bool drained = false, seeded = false;
    float3 ro = f3(0.0f), rd = f3(0.0f);
    TraceState t;
    float first_span = 0.0f;
    Near<K> b;
    near_clear(b);
    // next trace call of this lane's segment, or ready with nothing found when it is complete
    auto next_call = [&](const Composite& c) {
        // kt still holds the previous round (a full k-buffer) when there is one
        const float span = rounds > 0 ? b.kt[K - 1] - b.kt[0] : first_span;
        phase = kReady;
        bool call = composite_open(P, c);
        if (call && ++rounds > kMaxRounds + 1) {
            atomicOr(P.error_word, kErrLoopBound);
            call = false;
        }
        if (!call) {
            b.kt[0] = kFarT;
            return;
        }
        float cap = kFarT;
        seeded = false;
        if (K == 16 && span > 0.0f) {
            cap = composite_tmin(c) + kSeedSpan * span;
            seeded = cap < composite_tend(c);
            if (!seeded) cap = kFarT;
        }
        if (near_start<K>(P.accel, ro, rd, composite_tmin(c), composite_tend(c), b, log, t, ctr, cap)) phase = kTracing;
    };
    while (true) {
        // refill the idle lanes
        const unsigned idle = __ballot_sync(kFull, phase == kIdle);
        if (!drained && idle) {
            const unsigned n_idle = __popc(idle);
            unsigned first = 0;
            if (lane() == 0) first = atomicAdd(W.cursor + cursor, n_idle);
            first = __shfl_sync(kFull, first, 0);
            drained = first + n_idle >= count;
            if (phase == kIdle) {
                const unsigned i = first + __popc(idle & lanes_below());
                if (i < count) {
                    q = items[i];
                    Composite c;
                    composite_begin(P, c, W.seg[q].o, W.seg[q].d);
                    ro = c.o;
                    rd = c.d;
                    ++ctr.segments;
                    rounds = 0;
                    next_call(c);
                    pk.save(c);
                }
            }
        }
        const unsigned busy = __ballot_sync(kFull, phase != kIdle);
        if (!busy) {
            if (drained) break;
            continue;
        }
        // traverse until enough lanes wait
        const unsigned eligible = drained ? busy : kFull;
        while (true) {
            const unsigned tracing = __ballot_sync(kFull, phase == kTracing);
            if (!tracing || __popc(eligible & ~tracing) >= refill) break;
            if (phase == kTracing && !near_step<K, kSlack>(P.accel, ro, rd, t, b, log, stack, P.error_word, ctr)) {
                if (seeded && b.kt[K - 1] >= kFarT) {
                    seeded = false;
                    trace_continue(t, b.kt, ctr);
                } else {
                    phase = kReady;
                }
            }
        }
        // composite the finished calls; hand on the finished segments
        bool done = false;
        if (phase == kReady) {
            Composite c;
            pk.load(c, ro, rd);
            if (b.kt[0] < kFarT) {
                near_resolve(b, log, batch_t, batch_id, nthreads);
                composite_hits_strided<kSelfOcc, K>(P, ctr, c, batch_t, batch_id, nthreads, kMark ? vis : nullptr);
                const bool full = b.kt[K - 1] < kFarT;
                if (rounds == 1 && full) first_span = b.kt[K - 1] - t.tmin;
                // a k-buffer that is not full held every candidate of the call: a later call finds none
                if (full) next_call(c);
                else b.kt[0] = kFarT;
            }
            // nothing found, segment closed, or loop bound: the segment is complete
            if (phase == kReady && b.kt[0] >= kFarT) {
                Segment s;
                Pcg32 rng = load_rng(W, q);
                composite_end(P, c, W.seg[q].scatter_pdf, W.seg[q].light_pdf, s, rng);
                W.seg[q] = s;
                store_rng(W, q, rng);
                phase = kIdle;
                done = true;
            } else {
                pk.save(c);
            }
        }
        if (out_q >= 0) push(W.q[out_q], W.count + out_q, q, done);
    }
    flush_counters(P, ctr);
}

// ---------------------------------------------------------------------------------------
// intersection, four lanes a ray

// Shared memory of a quad: its traversal stack (the staging of quad_composite lies over it: no traversal
// is in progress then) and its compositing state.
struct QuadSlot {
    StackEntry stack[kQuadStackEntries];
    QuadComposite comp;
};
static_assert(sizeof(float4) * kQuadStage <= sizeof(StackEntry) * kStackDepth, "the staging fits the stack");
static_assert(sizeof(QuadSlot) % 16 == 0, "float4 members");

constexpr size_t quad_smem(int block) { return sizeof(QuadSlot) * (size_t)(block / 4); }

// Rays a warp carries: all eight quads, or fewer when the queue holds less than the grid's quads, so that
// a small launch spreads over all warps and no ray waits for another's.
PTIR_DEV unsigned quads_in_use(unsigned count) {
    const unsigned warps = gridDim.x * (blockDim.x >> 5);
    return min(8u, max(1u, (count + warps - 1u) / warps));
}

// The rounds from the root (K <= 16) of small launches, a quad of lanes per segment (quad.cuh).
// The decisions, their order and the compositing are k_wf_trace_near's, and no first round is seeded: a quad rarely
// sees more than a few segments. A small launch is bound by the chain of its slowest ray, which one lane walks
// at about 1 us a visit; here the visit's parts run side by side (preview of 2,867 rays over 2k Gaussians:
// 1.41 -> 0.51 ms in the stage). 96 registers hold the visit without spills: 25.2 ms at 90k rays over 300k
// Gaussians, against 26.1 at 72 and 26.9 at 64, where spills cost more than the warps gain, and 27.8 at 128.
template <int K, bool kMark, bool kSelfOcc, bool kSlack>
__global__ void __maxnreg__(96) k_wf_trace_quad(TraceParams P, float* vis, WfView W, int in_q, const unsigned* items,
                                                int out_q, unsigned cursor, int refill, unsigned quad_rays) {
    extern __shared__ float4 quad_mem[];
    constexpr unsigned kFull = 0xFFFFFFFFu;
    enum : int { kIdle = 0, kTracing = 1, kReady = 2 };
    const unsigned ln = lane(), c = ln & 3u, base = ln & 28u;
    QuadSlot& slot = reinterpret_cast<QuadSlot*>(quad_mem)[threadIdx.x >> 2];
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const unsigned count = W.count[in_q];
    if (count > quad_rays) return;
    const bool in_use = (ln >> 2) < quads_in_use(count);
    int phase = kIdle;
    unsigned q = 0;
    int rounds = 0;
    bool drained = false, seeded = false;
    float3 ro = f3(0.0f), rd = f3(0.0f);
    QuadTrace<K> t;
    t.tk = kFarT;
    // next trace call of the quad's segment, or ready with nothing found when it is complete
    auto next_call = [&](float span) {
        t.tk = kFarT;
        const QuadComposite& s = slot.comp;
        bool call = quad_open(P, s);
        if (call && ++rounds > kMaxRounds + 1) {
            if (c == 0) atomicOr(P.error_word, kErrLoopBound);
            call = false;
        }
        phase = kReady;
        if (!call) {
            kbuf_clear(t.kt, t.kid);
            return;
        }
        const float tmin = s.last_hit + 1e-9f, tend = s.clip_end + 1e-9f;
        float cap = kFarT;
        seeded = false;
        if (K == 16 && span > 0.0f) {
            cap = tmin + kSeedSpan * span;
            seeded = cap < tend;
            if (!seeded) cap = kFarT;
        }
        if (quad_start(P.accel, ro, rd, tmin, tend, t, ctr, c, cap)) phase = kTracing;
    };
    while (true) {
        // refill the idle quads
        const unsigned idle = __ballot_sync(kFull, phase == kIdle && in_use && c == 0);
        if (!drained && idle) {
            const unsigned n_idle = __popc(idle);
            unsigned first = 0;
            if (ln == 0) first = atomicAdd(W.cursor + cursor, n_idle);
            first = __shfl_sync(kFull, first, 0);
            drained = first + n_idle >= count;
            const unsigned i = first + __popc(idle & ((1u << base) - 1u));
            const bool take = phase == kIdle && in_use && i < count;
            const unsigned taking = __ballot_sync(kFull, take);
            if (take) {
                q = items[i];
                ro = W.seg[q].o;
                rd = W.seg[q].d;
                rounds = 0;
                quad_composite_begin(P, slot.comp, ro, rd, c, taking);
                if (c == 0) ++ctr.segments;
                next_call(0.0f);
            }
        }
        const unsigned busy = __ballot_sync(kFull, phase != kIdle && c == 0);
        if (!busy) {
            if (drained) break;
            continue;
        }
        // traverse until enough quads wait
        while (true) {
            const unsigned tracing = __ballot_sync(kFull, phase == kTracing);
            if (!tracing || __popc(busy) - (__popc(tracing) >> 2) >= (drained ? 1 : refill)) break;
            if (phase == kTracing && !quad_step<K, kSlack>(P.accel, ro, rd, t, slot.stack, P.error_word, ctr, ln, tracing)) {
                if (seeded && t.tk >= kFarT) {
                    seeded = false;
                    quad_continue(t, ctr);
                } else {
                    phase = kReady;
                }
            }
        }
        // composite the finished calls; hand on the finished segments
        bool done = false;
        const unsigned ready = __ballot_sync(kFull, phase == kReady);
        if (phase == kReady) {
            const float t_first = __shfl_sync(ready, t.kt[0], base);
            const float t_last = __shfl_sync(ready, t.kt[QuadTrace<K>::L - 1], base + 3u);
            bool complete = true;
            const unsigned found = __ballot_sync(ready, t_first < kFarT);
            if (t_first < kFarT) {
                quad_composite<kSelfOcc>(P, ctr, slot.comp, reinterpret_cast<float4*>(slot.stack), t, ro, rd,
                                         kMark ? vis : nullptr, ln, found);
                // a k-buffer that is not full held every candidate of the call: a later call finds none
                if (t_last < kFarT) {
                    next_call(t_last - t_first);
                    complete = phase == kReady;
                }
            }
            if (complete) {
                if (c == 0) {
                    Composite cm;
                    quad_composite_gather(slot.comp, cm, ro, rd);
                    Segment s;
                    Pcg32 rng = load_rng(W, q);
                    composite_end(P, cm, W.seg[q].scatter_pdf, W.seg[q].light_pdf, s, rng);
                    W.seg[q] = s;
                    store_rng(W, q, rng);
                    done = true;
                }
                phase = kIdle;
            }
        }
        __syncwarp();
        if (out_q >= 0) push(W.q[out_q], W.count + out_q, q, done);
    }
    flush_counters(P, ctr);
}

// ---------------------------------------------------------------------------------------
// forward

// Camera segments of the chunk: the sampler seed and the primary ray of every slot inside the
// image, queued for intersection.
__global__ void __launch_bounds__(kMaxThreads) k_wf_camera(TraceParams P, WfView W) {
    while (true) {
        const unsigned base = fetch32(W.cursor + 0);
        if (base >= W.slots) break;
        const unsigned q = base + lane();
        unsigned x = 0, y = 0, z = 0;
        int view = 0;
        size_t li = 0;
        const bool valid = q < W.slots && slot_index(P, W, q, view, x, y, z, li);
        if (valid) {
            Pcg32 rng;
            rng.seed(x, y, z, P.views[view].frame);
            Segment s;
            float3 o, d;
            world_ray(P, view, x, y, z, li, o, d);
            segment_reset(s, o, d, 0.0f);
            W.seg[q] = s;
            store_rng(W, q, rng);
        }
        push(W.q[kQIsect], W.count + kQIsect, q, valid);
    }
}

// primary outputs and the first NEE sample of every camera segment
template <int K>
__global__ void __launch_bounds__(kMaxThreads) k_wf_fwd_primary(TraceParams P, FwdOutputs O, WfView W) {
    PTIR_STAGE_PROLOGUE
    const bool mis = (P.flags & kMis) != 0;
    while (true) {
        const unsigned base = fetch32(W.cursor + 2);
        if (base >= W.slots) break;
        const unsigned q = base + lane();
        unsigned x = 0, y = 0, z = 0;
        int view = 0;
        size_t li = 0;
        const bool valid = q < W.slots && slot_index(P, W, q, view, x, y, z, li);
        bool cont = false, shadow = false;
        if (valid) {
            Pcg32 rng = load_rng(W, q);
            PathState ps;
            path_init(ps, effective_bounces(P));
            Segment s = W.seg[q];
            sig_event(P, ps, sig_segment(s));
            float* r = O.radiance + 3 * li;
            r[0] = s.radiance.x; r[1] = s.radiance.y; r[2] = s.radiance.z;
            O.density[li] = 1.0f - s.transmittance;
            O.hit[2 * li] = s.depth;
            O.hit[2 * li + 1] = s.last_hit;
            O.hit2[li] = s.hit2;
            O.distortion[li] = s.distortion;
            const bool nrm = (P.flags & kNormals) != 0;
            float* n = O.normal + 3 * li;
            n[0] = nrm ? s.normal.x : 0.0f; n[1] = nrm ? s.normal.y : 0.0f; n[2] = nrm ? s.normal.z : 0.0f;
            float* sn = O.snormal + 3 * li;
            sn[0] = nrm ? s.snrm.x : 0.0f; sn[1] = nrm ? s.snrm.y : 0.0f; sn[2] = nrm ? s.snrm.z : 0.0f;
            float* m = O.material + 5 * li;
            m[0] = s.albedo.x; m[1] = s.albedo.y; m[2] = s.albedo.z; m[3] = s.rough; m[4] = s.metal;
            O.hits_count[li] = (P.flags & kHitCounts) ? s.hits_count : 0.0f;
            write_pbr(O, li, ps);  // zeros; rewritten when the path ends
            cont = (P.flags & kVisualizeLights) || s.ivalid;
            if (cont) {
                if (mis) shadow = nee_prepare(C, ps, s, rng);
                W.seg[q] = s;
                W.ps[q] = ps;
                store_rng(W, q, rng);
            }
        }
        push(W.q[kQShadow], W.count + kQShadow, q, cont && shadow);
        push(W.q[kQBounce], W.count + kQBounce, q, cont && !shadow);
    }
    flush_counters(P, ctr);
}

// NEE shadow rays (the stochastic occlusion walk of pathTracer.cuh:161-214, as shadow_occluded in
// path.cuh) with per-lane refill, as in k_wf_trace: a lane whose ray is decided hands its slot
// to the bounce queue and takes the next shadow ray, so that no lane waits for the longest walk
// of its warp. The warp leaves its traversal loop once `refill` lanes wait. The random draws of
// a ray are those of shadow_occluded, in the same order. Against one ray per lane for the whole
// walk this cut the stage by 15 % on the 1M-Gaussian scene, and the register cap of the
// intersection kernel (more resident warps) by 6 % more.
template <int K>
__global__ void __maxnreg__(trace_regs(K)) k_wf_shadow(TraceParams P, WfView W, int refill, const unsigned* items,
                                                          unsigned quad_rays) {
    StackEntry stack[kStackDepth];
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    constexpr unsigned kFull = 0xFFFFFFFFu;
    enum : int { kIdle = 0, kTracing = 1, kReady = 2 };
    const unsigned count = W.count[kQShadow];
    if (count <= quad_rays) return;  // the quads' launch
    int phase = kIdle;
    unsigned q = 0;
    int rounds = 0;
    bool drained = false;
    float3 ro = f3(0.0f), rd = f3(0.0f);
    float start = 0.0f, end = 0.0f;
    Pcg32 rng;
    TraceState t;
    bool seeded = false;      // the lane's call started with a cut estimated from a span, as in k_wf_trace
    float first_span = 0.0f;  // K-th distance less tmin of the first round of the lane's last shadow ray
    float kt[K];
    unsigned kid[K];
    // next trace call of the lane's ray over (start, end), or the ray is decided (unoccluded). Rounds
    // of 16 are seeded as in k_wf_trace: a later round from the previous round's span, a first round
    // from the first-round span of the lane's last shadow ray (a neighbour in the sorted queue).
    auto next_call = [&]() -> bool {
        if (!(start < end)) return false;
        if (++rounds > (1 << 16) + 1) {
            atomicOr(P.error_word, kErrLoopBound);
            return false;
        }
        float cap = kFarT;
        seeded = false;
        if constexpr (K == 16) {
            // kt still holds the previous round (a full k-buffer) when there is one
            const float span = rounds > 1 ? kt[K - 1] - kt[0] : first_span;
            if (span > 0.0f) {
                cap = start + 1e-9f + kSeedSpan * span;
                seeded = cap < end;
                if (!seeded) cap = kFarT;
            }
        }
        phase = trace_start(P.accel, ro, rd, start + 1e-9f, end, kt, kid, t, ctr, nullptr, false, cap) ? kTracing
                                                                                                       : kReady;
        return true;
    };
    while (true) {
        bool done = false, occluded = false;
        const unsigned idle = __ballot_sync(kFull, phase == kIdle);
        if (!drained && idle) {
            const unsigned n_idle = __popc(idle);
            unsigned base = 0;
            if (lane() == 0) base = atomicAdd(W.cursor + 3, n_idle);
            base = __shfl_sync(kFull, base, 0);
            drained = base + n_idle >= count;
            if (phase == kIdle) {
                const unsigned i = base + __popc(idle & lanes_below());
                if (i < count) {
                    q = items[i];
                    const float3 wi = W.ps[q].em.dir;
                    ro = W.seg[q].pos + wi * 2e-2f;
                    rd = wi;
                    rng = load_rng(W, q);
                    ++ctr.segments;
                    rounds = 0;
                    const float2 clip = clip_scene(P, ro, rd);
                    start = fmaxf(0.0f, clip.x - 1e-9f);
                    end = fminf(W.ps[q].em.tmax, clip.y) + 1e-9f;
                    phase = kTracing;
                    if (!next_call()) done = true;  // nothing in front of the light
                }
            }
        }
        const unsigned busy = __ballot_sync(kFull, phase != kIdle && !done);
        if (!busy && !__any_sync(kFull, done)) {
            if (drained) break;
            continue;
        }
        // traverse until enough lanes wait
        const unsigned eligible = drained ? busy : kFull;
        while (true) {
            const unsigned tracing = __ballot_sync(kFull, phase == kTracing && !done);
            if (!tracing || __popc(eligible & ~tracing) >= refill) break;
            if (phase == kTracing && !done &&
                !trace_step(P.accel, ro, rd, t, kt, kid, stack, P.error_word, ctr)) {
                if (seeded && kid[K - 1] == kNoHit) {
                    seeded = false;
                    trace_continue(t, kt, ctr);
                } else {
                    phase = kReady;
                }
            }
        }
        // walk the finished batches: the first hit that occludes decides the ray
        if (phase == kReady && !done) {
            if (rounds == 1 && kid[K - 1] != kNoHit) first_span = kt[K - 1] - t.tmin;
            if (kid[0] == kNoHit) {
                done = true;
            } else {
                float batch_end = start;
                bool stop = false;
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    if (stop || occluded) continue;
                    const unsigned id = kid[i];
                    if (id == kNoHit || kt[i] > end) {
                        stop = true;
                        continue;
                    }
                    batch_end = fmaxf(batch_end, kt[i]);
                    if (self_occluded(P, kt[i], id, rd)) continue;
                    float dns;
                    const Response r = respond(P, id, ro, rd, dns);
                    const float alpha = (r.gres > P.min_response && r.alpha > P.alpha_min) ? r.alpha : 0.0f;
                    if (alpha > 0.0f && rng.uniform() < alpha) occluded = true;
                }
                if (occluded || batch_end <= start || kid[K - 1] == kNoHit) {
                    done = true;  // decided, or no candidate left (the k-buffer was not full)
                } else {
                    start = batch_end;
                    if (!next_call()) done = true;
                }
            }
        }
        if (done) {
            if (occluded) {
                Emitter em = W.ps[q].em;
                emitter_clear(em);
                W.ps[q].em = em;
            }
            if (P.flags & kPathSig) W.ps[q].sig = sig_mix(W.ps[q].sig, kSigShadow | (occluded ? 1u : 0u));
            store_rng(W, q, rng);
            phase = kIdle;
        }
        push(W.q[kQBounce], W.count + kQBounce, q, done);
    }
    flush_counters(P, ctr);
}

// k_wf_shadow for small launches, a quad of lanes a ray (quad.cuh): the same candidates, walked in the same order with
// the same draws; no first round is seeded, as in k_wf_trace_quad. As there a small launch waits for its slowest
// ray: stage of 16k rays over 10k Gaussians 0.57 -> 0.26 ms, of 90k over 300k (forward and adjoint) 6.4 -> 4.2 ms.
// kSlack: with the exact-candidate cull slack.
template <int K, bool kSlack>
__global__ void __maxnreg__(96) k_wf_shadow_quad(TraceParams P, WfView W, int refill, const unsigned* items,
                                                 unsigned quad_rays) {
    extern __shared__ float4 quad_mem[];
    constexpr unsigned kFull = 0xFFFFFFFFu;
    enum : int { kIdle = 0, kTracing = 1, kReady = 2 };
    const unsigned ln = lane(), c = ln & 3u, base = ln & 28u;
    StackEntry* const stack = reinterpret_cast<StackEntry*>(quad_mem) + (threadIdx.x >> 2) * kQuadStackEntries;
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const unsigned count = W.count[kQShadow];
    if (count > quad_rays) return;
    const bool in_use = (ln >> 2) < quads_in_use(count);
    int phase = kIdle;
    unsigned q = 0;
    int rounds = 0;
    bool drained = false, seeded = false;
    float3 ro = f3(0.0f), rd = f3(0.0f);
    float start = 0.0f, end = 0.0f;
    Pcg32 rng;
    QuadTrace<K> t;
    t.tk = kFarT;
    kbuf_clear(t.kt, t.kid);
    // next trace call of the quad's ray over (start, end); false when the ray is decided (unoccluded)
    auto next_call = [&](float span) -> bool {
        if (!(start < end)) return false;
        if (++rounds > (1 << 16) + 1) {
            if (c == 0) atomicOr(P.error_word, kErrLoopBound);
            return false;
        }
        float cap = kFarT;
        seeded = false;
        if (K == 16 && span > 0.0f) {
            cap = start + 1e-9f + kSeedSpan * span;
            seeded = cap < end;
            if (!seeded) cap = kFarT;
        }
        phase = quad_start(P.accel, ro, rd, start + 1e-9f, end, t, ctr, c, cap) ? kTracing : kReady;
        return true;
    };
    while (true) {
        bool done = false, occluded = false;
        const unsigned idle = __ballot_sync(kFull, phase == kIdle && in_use && c == 0);
        if (!drained && idle) {
            const unsigned n_idle = __popc(idle);
            unsigned first = 0;
            if (ln == 0) first = atomicAdd(W.cursor + 3, n_idle);
            first = __shfl_sync(kFull, first, 0);
            drained = first + n_idle >= count;
            const unsigned i = first + __popc(idle & ((1u << base) - 1u));
            if (phase == kIdle && in_use && i < count) {
                q = items[i];
                const float3 wi = W.ps[q].em.dir;
                ro = W.seg[q].pos + wi * 2e-2f;
                rd = wi;
                rng = load_rng(W, q);
                if (c == 0) ++ctr.segments;
                rounds = 0;
                const float2 clip = clip_scene(P, ro, rd);
                start = fmaxf(0.0f, clip.x - 1e-9f);
                end = fminf(W.ps[q].em.tmax, clip.y) + 1e-9f;
                phase = kTracing;
                if (!next_call(0.0f)) done = true;  // nothing in front of the light
            }
        }
        const unsigned busy = __ballot_sync(kFull, phase != kIdle && !done && c == 0);
        if (!busy && !__any_sync(kFull, done)) {
            if (drained) break;
            continue;
        }
        // traverse until enough quads wait
        while (true) {
            const unsigned tracing = __ballot_sync(kFull, phase == kTracing && !done);
            if (!tracing || __popc(busy) - (__popc(tracing) >> 2) >= (drained ? 1 : refill)) break;
            if (phase == kTracing && !done && !quad_step<K, kSlack>(P.accel, ro, rd, t, stack, P.error_word, ctr, ln, tracing)) {
                if (seeded && t.tk >= kFarT) {
                    seeded = false;
                    quad_continue(t, ctr);
                } else {
                    phase = kReady;
                }
            }
        }
        // walk the finished batches: the first hit that occludes decides the ray
        const bool ready = phase == kReady && !done;
        const unsigned ready_m = __ballot_sync(kFull, ready);
        if (ready) {
            const float t_first = __shfl_sync(ready_m, t.kt[0], base);
            const float t_last = __shfl_sync(ready_m, t.kt[QuadTrace<K>::L - 1], base + 3u);
            float batch_end = start;
            occluded = quad_shadow_walk(P, t, ro, rd, end, rng, batch_end, ln, ready_m);
            if (occluded || batch_end <= start || !(t_last < kFarT)) {
                done = true;  // decided, or no candidate left (the k-buffer was not full)
            } else {
                start = batch_end;
                if (!next_call(t_last - t_first)) done = true;
            }
        }
        if (done) {
            if (c == 0) {
                if (occluded) {
                    Emitter em = W.ps[q].em;
                    emitter_clear(em);
                    W.ps[q].em = em;
                }
                if (P.flags & kPathSig) W.ps[q].sig = sig_mix(W.ps[q].sig, kSigShadow | (occluded ? 1u : 0u));
                store_rng(W, q, rng);
            }
            phase = kIdle;
        }
        __syncwarp();
        push(W.q[kQBounce], W.count + kQBounce, q, done && c == 0);
    }
    flush_counters(P, ctr);
}

template <int K>
__global__ void __launch_bounds__(kMaxThreads) k_wf_fwd_bounce(TraceParams P, FwdOutputs O, WfView W, unsigned depth,
                                                            unsigned cursor) {
    PTIR_STAGE_PROLOGUE
    const unsigned count = W.count[kQBounce];
    while (true) {
        const unsigned base = fetch32(W.cursor + cursor);
        if (base >= count) break;
        const unsigned i = base + lane();
        const bool valid = i < count;
        const unsigned q = valid ? W.q[kQBounce][i] : 0u;
        bool cont = false;
        if (valid) {
            Segment s = W.seg[q];
            PathState ps = W.ps[q];
            Pcg32 rng = load_rng(W, q);
            if (depth > 0) sig_event(P, ps, sig_segment(s));
            accumulate_light(C, ps, s);
            ps.active &= (unsigned)((depth + 1u < ps.max_bounces) && s.ivalid);
            if (ps.active) {
                ps.bounces = depth + 1u;
                sample_next(C, ps, s, rng);
                cont = path_continues(ps);
                sig_event(P, ps, kSigCont | (cont ? 1u : 0u));
            }
            if (cont) {
                W.seg[q] = s;
                W.ps[q] = ps;
                store_rng(W, q, rng);
            } else {
                unsigned x, y, z;
                int view;
                size_t li;
                slot_index(P, W, q, view, x, y, z, li);
                write_pbr(O, li, ps);
            }
        }
        push(W.q[kQIsect], W.count + kQIsect, q, cont);
    }
    flush_counters(P, ctr);
}

// ---------------------------------------------------------------------------------------
// backward

// adjoint state and the first NEE sample of every camera segment
template <int K>
__global__ void __launch_bounds__(kMaxThreads) k_wb_primary(TraceParams P, BwdInputs B, WfView W) {
    PTIR_STAGE_PROLOGUE
    const bool mis = (P.flags & kMis) != 0;
    while (true) {
        const unsigned base = fetch32(W.cursor + 2);
        if (base >= W.slots) break;
        const unsigned q = base + lane();
        unsigned x = 0, y = 0, z = 0;
        int view = 0;
        size_t li = 0;
        const bool valid = q < W.slots && slot_index(P, W, q, view, x, y, z, li);
        bool cont = false, shadow = false;
        if (valid) {
            Pcg32 rng = load_rng(W, q);
            PathState ps;
            path_init(ps, effective_bounces(P));
            load_adjoint_inputs(P, B, x, y, z, li, ps);
            Segment s = W.seg[q];
            add_material_output_grad(P, B, x, y, z, li, s);
            cont = (P.flags & kVisualizeLights) || s.ivalid;
            if (cont) {
                if (mis) shadow = nee_prepare(C, ps, s, rng);
                W.seg[q] = s;
                W.ps[q] = ps;
                store_rng(W, q, rng);
            }
        }
        push(W.q[kQShadow], W.count + kQShadow, q, cont && shadow);
        push(W.q[kQBounce], W.count + kQBounce, q, cont && !shadow);
    }
    flush_counters(P, ctr);
}

template <int K>
__global__ void __launch_bounds__(kMaxThreads) k_wb_bounce(TraceParams P, BwdInputs B, WfView W, unsigned depth,
                                                        unsigned cursor) {
    PTIR_STAGE_PROLOGUE
    const unsigned count = W.count[kQBounce];
    while (true) {
        const unsigned base = fetch32(W.cursor + cursor);
        if (base >= count) break;
        const unsigned i = base + lane();
        const bool valid = i < count;
        const unsigned q = valid ? W.q[kQBounce][i] : 0u;
        bool cont = false;
        ReplayJob job[2];
        bool has[2] = {false, false};
        if (valid) {
            Segment s = W.seg[q];
            PathState ps = W.ps[q];
            Pcg32 rng = load_rng(W, q);
            accumulate_light_bwd(C, B, ps, s);
            pending_bwd(ps, s, [&](const ReplayJob& j) {
                job[0] = j;
                has[0] = true;
            });
            ps.active &= (unsigned)((depth + 1u < ps.max_bounces) && s.ivalid);
            if (ps.active) {
                ps.bounces = depth + 1u;
                sample_next_bwd(C, ps, s, rng, [&](const ReplayJob& j) {
                    job[1] = j;
                    has[1] = true;
                });
                cont = ps.active && !(max3(ps.throughput) < 1e-4f);
            }
            if (cont) {
                W.seg[q] = s;
                W.ps[q] = ps;
                store_rng(W, q, rng);
            }
        }
        push_job(W.jobs, W.count + kQJobs, job[0], has[0]);
        push_job(W.jobs, W.count + kQJobs, job[1], has[1]);
        push(W.q[kQIsect], W.count + kQIsect, q, cont);
    }
    flush_counters(P, ctr);
}

template <int K>
__global__ void __launch_bounds__(kMaxThreads) k_wb_replay(TraceParams P, BwdInputs B, WfView W, unsigned cursor,
                                                           bool resume, unsigned quad_jobs) {
    PTIR_STAGE_PROLOGUE
    const unsigned count = W.count[kQJobs];
    if (count <= quad_jobs) return;  // the quads' launch
    // with `resume` a replay's rounds after its first resume from the previous round's frontier
    const Frontier F{resume ? W.frontier + (size_t)(blockIdx.x * blockDim.x + threadIdx.x) * 2 * W.frontier_cap
                            : nullptr,
                     W.frontier_cap};
    while (true) {
        const unsigned base = fetch32(W.cursor + cursor);
        if (base >= count) break;
        const unsigned i = base + lane();
        if (i < count) {
            const ReplayJob j = W.jobs[i];
            replay_material_grad(C, B, j, F.buf ? &F : nullptr);
        }
    }
    flush_counters(P, ctr);
}

// k_wb_replay with resumed rounds (K <= 16) for up to kQuadRays jobs, a quad of lanes a job (quad.cuh): the entries
// that a round sets aside come in the order of the one-lane replay, so the same hits are scattered with the same
// weights. Bound, as there, by the latency of a step, of which a job is a chain. Replay stage, against one lane a job:
// 3.2 -> 2.6 ms (80k paths, 20k Gaussians), 4.9 -> 3.4 (90k, 100k), 7.0 -> 6.1 (90k, 300k); with 786k paths over
// 1M Gaussians it took 41 ms against 18.6 (twice the frontier traffic an issue slot), hence the line. kSlack: with
// the exact-candidate cull slack.
template <int K, bool kSlack>
__global__ void __maxnreg__(128) k_wb_replay_quad(TraceParams P, BwdInputs B, WfView W, unsigned cursor, int refill,
                                                 unsigned quad_jobs) {
    extern __shared__ float4 quad_mem[];
    constexpr unsigned kFull = 0xFFFFFFFFu;
    enum : int { kIdle = 0, kTracing = 1, kReady = 2 };
    const unsigned ln = lane(), c = ln & 3u, base = ln & 28u;
    StackEntry* const stack = reinterpret_cast<StackEntry*>(quad_mem) + (threadIdx.x >> 2) * kQuadStackEntries;
    TraceCounters ctr = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const unsigned count = W.count[kQJobs];
    if (count > quad_jobs) return;
    const bool in_use = (ln >> 2) < quads_in_use(count);
    int phase = kIdle;
    int rounds = 0;
    bool drained = false;
    ReplayState r;
    QuadTrace<K> t;
    t.tk = kFarT;
    kbuf_clear(t.kt, t.kid);
    QuadFrontier F{W.frontier + (size_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 2) * 2 * W.frontier_cap, W.frontier_cap,
                   0, 0, 0, 0};
    // next round of the job, false when it is complete
    auto next_round = [&]() -> bool {
        if (!replay_open(P, r)) return false;
        if (rounds > (1 << 16)) {
            if (c == 0) atomicOr(P.error_word, kErrLoopBound);
            return false;
        }
        const bool resume = rounds++ > 0;
        phase = quad_start_resume(P.accel, r.o, r.d, r.start + 1e-9f, r.end, t, F, resume, ctr, c) ? kTracing : kReady;
        return true;
    };
    while (true) {
        const unsigned idle = __ballot_sync(kFull, phase == kIdle && in_use && c == 0);
        if (!drained && idle) {
            const unsigned n_idle = __popc(idle);
            unsigned first = 0;
            if (ln == 0) first = atomicAdd(W.cursor + cursor, n_idle);
            first = __shfl_sync(kFull, first, 0);
            drained = first + n_idle >= count;
            const unsigned i = first + __popc(idle & ((1u << base) - 1u));
            if (phase == kIdle && in_use && i < count) {
                TraceCounters mine = {0, 0, 0, 0, 0, 0, 0, 0, 0};
                replay_begin(P, W.jobs[i], r, mine);
                if (c == 0) ctr.replay += mine.replay;
                rounds = 0;
                if (!next_round()) phase = kIdle;
            }
        }
        const unsigned busy = __ballot_sync(kFull, phase != kIdle && c == 0);
        if (!busy) {
            if (drained) break;
            continue;
        }
        while (true) {
            const unsigned tracing = __ballot_sync(kFull, phase == kTracing);
            if (!tracing || __popc(busy) - (__popc(tracing) >> 2) >= (drained ? 1 : refill)) break;
            if (phase == kTracing &&
                !quad_step_resume<K, kSlack>(P.accel, r.o, r.d, t, F, stack, P.error_word, ctr, ln, tracing))
                phase = kReady;
        }
        __syncwarp();  // the entries set aside, before the next call reads them
        const unsigned ready = __ballot_sync(kFull, phase == kReady);
        if (phase == kReady) {
            const float t_last = __shfl_sync(ready, t.kt[QuadTrace<K>::L - 1], base + 3u);
            quad_replay_batch(P, B, r, t, ctr, ln, ready);
            // a k-buffer that is not full held every candidate of the round
            if (!(t_last < kFarT && next_round())) phase = kIdle;
        }
        __syncwarp();
    }
    flush_counters(P, ctr);
}

// the four-lane replay, with the exact-candidate cull slack or without
template <int K>
static auto* replay_quad_fn(const WavefrontTuning& tune) {
    return tune.exact_candidates ? k_wb_replay_quad<K, true> : k_wb_replay_quad<K, false>;
}

// persistent grid: resident blocks per SM x SMs (defined below)
int grid_cached(const void* fn, int block, size_t smem);

// The shadow stage with its own k-buffer size. A shadow walk visits the hits in distance order
// until one occludes, whatever the batch size, so its size is free of the intersection's: a
// walk usually ends in its first batch, which a smaller buffer gathers with less traversal.
static void launch_shadow(const WavefrontTuning& tune, const TraceParams& q, const WfView& W, const unsigned* items,
                          cudaStream_t s) {
    const int B = tune.block, R = tune.refill_lanes;
    const bool slack = tune.exact_candidates;
    // up to kQuadRays shadow rays (the queue's count, which only the device knows) go to the quads
    const auto blocks = [&](int grid, unsigned per_block) {
        return (unsigned)std::min<long long>(grid, ((long long)W.slots + per_block - 1) / per_block);
    };
    const size_t stacks = sizeof(StackEntry) * kQuadStackEntries * (size_t)(B / 4);
    const auto lanes = [&](auto* fn, unsigned quad_rays) {
        if (W.slots > quad_rays) fn<<<blocks(grid_cached((const void*)fn, B, 0), B), B, 0, s>>>(q, W, R, items, quad_rays);
    };
    const auto quads = [&](auto* fn) {
        fn<<<blocks(grid_cached((const void*)fn, B, stacks), B / 32), B, stacks, s>>>(q, W, (R + 3) / 4, W.q[kQShadow], kQuadRays);
    };
    switch (tune.shadow_kbuf) {
    case 8: quads(slack ? k_wf_shadow_quad<8, true> : k_wf_shadow_quad<8, false>); lanes(k_wf_shadow<8>, kQuadRays); break;
    case 32: lanes(k_wf_shadow<32>, 0u); break;
    default: quads(slack ? k_wf_shadow_quad<16, true> : k_wf_shadow_quad<16, false>); lanes(k_wf_shadow<16>, kQuadRays); break;
    }
}

// persistent grid: resident blocks per SM x SMs
int grid_for(const void* fn, int block, size_t smem) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, smem) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    return sms * per_sm;
}

// floats of W.parked for every thread the device can hold resident (k-buffer up to 32)
size_t parked_floats() {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
    if (sms <= 0) sms = 148;
    if (per_sm <= 0) per_sm = 2048;
    return (size_t)(kParkedFields + 2 * 32) * (size_t)sms * (size_t)per_sm;
}

// grid of a kernel at a block size, computed once per (kernel, block size)
int grid_cached(const void* fn, int block, size_t smem = 0) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, int> cache;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find({fn, block});
    if (it != cache.end()) return it->second;
    // more than the default 48 KB of dynamic shared memory needs the kernel's opt-in
    if (smem > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int g = grid_for(fn, block, smem);
    cache[{fn, block}] = g;
    return g;
}

}  // namespace

// ---------------------------------------------------------------------------------------
cudaError_t wavefront_reserve(WavefrontBuffers& b, size_t slots, cudaStream_t s) {
    if (slots <= b.slots && b.seg) return cudaSuccess;
    auto rel = [&](void* p) {
        if (p) cudaFreeAsync(p, s);
    };
    rel(b.seg); rel(b.ps); rel(b.rng); rel(b.q[0]); rel(b.q[1]); rel(b.q[2]); rel(b.jobs);
    rel(b.sort_keys[0]); rel(b.sort_keys[1]); rel(b.sorted); rel(b.sort_temp); rel(b.parked);
    void* counters = b.counters;
    void* frontier = b.frontier;
    const size_t frontier_threads = b.frontier_threads;
    b = WavefrontBuffers{};
    b.counters = counters;
    b.frontier = frontier;  // sized by the intersection grid, not by the chunk
    b.frontier_threads = frontier_threads;
    cudaError_t e = cudaSuccess;
    auto get = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMallocAsync(p, bytes, s);
    };
    get(&b.seg, sizeof(Segment) * slots);
    get(&b.ps, sizeof(PathState) * slots);
    get(&b.rng, sizeof(unsigned long long) * slots);
    for (int k = 0; k < 3; ++k) get(&b.q[k], sizeof(unsigned) * slots);
    get(&b.jobs, sizeof(ReplayJob) * 2 * slots);
    if (!b.counters) get(&b.counters, sizeof(unsigned) * (kNumQueueCounts + kNumCursors));
    get(&b.sort_keys[0], sizeof(unsigned) * slots);
    get(&b.sort_keys[1], sizeof(unsigned) * slots);
    get(&b.sorted, sizeof(unsigned) * slots);
    get(&b.parked, sizeof(float) * parked_floats());
    if (e == cudaSuccess) {
        b.sort_temp_bytes = radix_sort_temp_bytes<unsigned>((long long)slots);
        get(&b.sort_temp, b.sort_temp_bytes);
    }
    if (e == cudaSuccess) b.slots = slots;
    return e;
}

size_t wavefront_bytes_per_slot() {
    // path state, RNG, three queues, two replay jobs, two sort keys + the sorted queue, and the
    // radix sort's scratch (a key / value pair per slot and its digit counts, rounded up)
    return sizeof(Segment) + sizeof(PathState) + sizeof(unsigned long long) + 3 * sizeof(unsigned) +
           2 * sizeof(ReplayJob) + 3 * sizeof(unsigned) + 4 * sizeof(unsigned);
}

void wavefront_free(WavefrontBuffers& b) {
    for (void* p : {b.seg, b.ps, b.rng, b.q[0], b.q[1], b.q[2], b.jobs, b.counters, b.sort_keys[0], b.sort_keys[1],
                    b.sorted, b.sort_temp, b.parked, b.frontier})
        if (p) cudaFree(p);
    b = WavefrontBuffers{};
}

// frontier buffers for `threads` threads of the intersection kernel (grown on demand)
cudaError_t frontier_reserve(WavefrontBuffers& b, size_t threads, cudaStream_t s) {
    if (threads <= b.frontier_threads && b.frontier) return cudaSuccess;
    if (b.frontier) cudaFreeAsync(b.frontier, s);
    b.frontier = nullptr;
    b.frontier_threads = 0;
    const cudaError_t e = cudaMallocAsync(&b.frontier, sizeof(uint2) * 2 * (size_t)kFrontierCap * threads, s);
    if (e == cudaSuccess) b.frontier_threads = threads;
    return e;
}

static WfView view_of(const WavefrontBuffers& b, unsigned long long tile0, unsigned slots, bool resume) {
    WfView W;
    W.seg = static_cast<Segment*>(b.seg);
    W.ps = static_cast<PathState*>(b.ps);
    W.rng = static_cast<unsigned long long*>(b.rng);
    for (int k = 0; k < 3; ++k) W.q[k] = static_cast<unsigned*>(b.q[k]);
    W.count = static_cast<unsigned*>(b.counters);
    W.cursor = W.count + kNumQueueCounts;
    W.jobs = static_cast<ReplayJob*>(b.jobs);
    W.parked = static_cast<float*>(b.parked);
    W.frontier = resume ? static_cast<uint2*>(b.frontier) : nullptr;
    W.frontier_cap = resume ? kFrontierCap : 0;
    W.tile0 = tile0;
    W.slots = slots;
    return W;
}

static unsigned long long total_tiles(const TraceParams& p) { return (unsigned long long)p.tiles; }

// Queue in_q in ray order (or as queued when sorting is off): keys, then a key/slot radix sort of what the queue
// holds (the count stays on the device).
static const unsigned* sort_queue(const TraceParams& p, const WavefrontBuffers& b, const WfView& W,
                                  const WavefrontTuning& tune, const StageCtx& sc, cudaStream_t s, bool quads,
                                  int in_q = kQIsect) {
    if (!tune.sort_rays) return W.q[in_q];
    // up to kQuadRays rays are traced by quads, in queue order: each waits for its own ray, and sorting cost more than
    // it gave (16k rays over 10k Gaussians: a trace of 1.29 ms against 1.69, the stage's time the same; 90k
    // over 300k: 36.0 against 36.6). How many rays the queue holds only the device knows.
    const unsigned quad_rays = quads ? kQuadRays : 0u;
    if (W.slots <= quad_rays) return W.q[in_q];
    unsigned* keys_in = static_cast<unsigned*>(b.sort_keys[0]);
    unsigned* keys_out = static_cast<unsigned*>(b.sort_keys[1]);
    unsigned* sorted = static_cast<unsigned*>(b.sorted);
    const int grid = grid_cached((const void*)k_wf_sort_keys, tune.block);
    sc.run(kStageSort, p, s, [&](const TraceParams& q) {
        k_wf_sort_keys<<<grid, tune.block, 0, s>>>(q, W, in_q, keys_in, quad_rays);
        radix_sort_pairs<unsigned>(b.sort_temp, b.sort_temp_bytes, keys_in, keys_out, W.q[in_q], sorted,
                                   (long long)W.slots, 0, kSortKeyBits, s, W.count + in_q, quad_rays);
    });
    return sorted;
}

// Cursor of each stage launch within a chunk: camera 0, primary intersection 1, primary outputs
// 2, shadow 3, then per bounce depth the bounce stage, (the adjoint's replay,) and intersection.
constexpr unsigned kFirstBounceCursor = 4;

// intersection kernels with resumed rounds (K <= 16)
template <int K>
static bool use_resume(const WavefrontTuning& tune) {
    return K <= 16 && tune.resume_isect && !tune.exact_candidates;
}

// An intersection launch: the kernels of its k-buffer size and options, and their persistent grids. Rounds from
// the root with K <= 16 take four lanes a ray (k_wf_trace_quad) in a launch of up to kQuadRays rays and one lane
// a ray (k_wf_trace_near) in a larger one; resumed rounds and K = 32 take one (k_wf_trace).
struct TraceLaunch {
    const void* lane_fn = nullptr;
    const void* quad_fn = nullptr;
    int block, lane_refill, quad_refill, lane_grid = 0, quad_grid = 0;
};

template <int K, bool kMark, bool kSelfOcc>
static TraceLaunch trace_launch(const WavefrontTuning& tune, bool resume) {
    TraceLaunch l;
    l.block = tune.block;
    l.lane_refill = tune.refill_lanes;
    l.quad_refill = (tune.refill_lanes + 3) / 4;
    const bool slack = tune.exact_candidates;
    if constexpr (K <= 16) {
        if (resume) {
            l.lane_fn = (const void*)k_wf_trace<K, kMark, kSelfOcc, true, false>;
        } else {
            l.lane_fn = slack ? (const void*)k_wf_trace_near<K, kMark, kSelfOcc, true>
                              : (const void*)k_wf_trace_near<K, kMark, kSelfOcc, false>;
            l.quad_fn = slack ? (const void*)k_wf_trace_quad<K, kMark, kSelfOcc, true>
                              : (const void*)k_wf_trace_quad<K, kMark, kSelfOcc, false>;
        }
    } else {
        l.lane_fn = slack ? (const void*)k_wf_trace<K, kMark, kSelfOcc, false, true>
                          : (const void*)k_wf_trace<K, kMark, kSelfOcc, false, false>;
    }
    l.lane_grid = grid_cached(l.lane_fn, l.block);
    if (l.quad_fn) l.quad_grid = grid_cached(l.quad_fn, l.block, quad_smem(l.block));
    return l;
}

// The intersection of queue in_q, which holds at most `rays` rays. How many it does hold only the device knows,
// so a queue that might be on either side of kQuadRays gets both launches, and the kernel that it is not for
// returns at once.
static void run_trace(const TraceLaunch& l, long long rays, const TraceParams& q, float* vis, const WfView& W, int in_q,
                      const unsigned* items, int out_q, unsigned cursor, cudaStream_t s) {
    TraceParams p = q;
    WfView w = W;
    const auto blocks = [&](int grid, long long per_block) {
        return dim3((unsigned)std::max<long long>(1, std::min<long long>(grid, (rays + per_block - 1) / per_block)));
    };
    unsigned quad_rays = l.quad_fn ? kQuadRays : 0u;
    int refill;
    void* args[] = {&p, &vis, &w, &in_q, &items, &out_q, &cursor, &refill, &quad_rays};
    if (l.quad_fn) {
        const unsigned* sorted = items;
        items = W.q[in_q];  // as queued (sort_queue)
        refill = l.quad_refill;
        cudaLaunchKernel(l.quad_fn, blocks(l.quad_grid, l.block / 32), dim3((unsigned)l.block), args, quad_smem(l.block), s);
        items = sorted;
    }
    if (rays > (long long)quad_rays) {
        refill = l.lane_refill;
        cudaLaunchKernel(l.lane_fn, blocks(l.lane_grid, l.block), dim3((unsigned)l.block), args, 0, s);
    }
}

template <int K>
static cudaError_t run_fwd(const TraceParams& p, const FwdOutputs& o, WavefrontBuffers& b, const WavefrontTuning& tune,
                           const StageCtx& sc, cudaStream_t s) {
    const unsigned long long tiles = total_tiles(p);
    if (tiles == 0) return cudaSuccess;
    const unsigned chunk_tiles = (unsigned)std::min<unsigned long long>(tune.chunk_tiles, tiles);
    cudaError_t e = wavefront_reserve(b, (size_t)chunk_tiles * 32, s);
    if (e != cudaSuccess) return e;
    const int B = tune.block;
    const int g_camera = grid_cached((const void*)k_wf_camera, B);
    const int g_primary = grid_cached((const void*)k_wf_fwd_primary<K>, B);
    const int g_bounce = grid_cached((const void*)k_wf_fwd_bounce<K>, B);
    const bool resume = use_resume<K>(tune);
    const TraceLaunch trace0 = trace_launch<K, true, false>(tune, resume), trace = trace_launch<K, true, true>(tune, resume);
    if (resume && (e = frontier_reserve(b, (size_t)std::max(trace0.lane_grid, trace.lane_grid) * B, s)) != cudaSuccess) return e;
    const unsigned mb = p.render_opts ? std::min(p.max_bounces, 2u) : p.max_bounces;
    if (kFirstBounceCursor + 2u * mb > (unsigned)kNumCursors) return cudaErrorInvalidValue;
    for (unsigned long long t0 = 0; t0 < tiles; t0 += chunk_tiles) {
        const unsigned nt = (unsigned)std::min<unsigned long long>(chunk_tiles, tiles - t0);
        const WfView W = view_of(b, t0, nt * 32u, resume);
        e = cudaMemsetAsync(b.counters, 0, sizeof(unsigned) * (kNumQueueCounts + kNumCursors), s);
        if (e != cudaSuccess) return e;
        const int cap = (int)std::min<long long>(INT32_MAX, ((long long)nt * 32 + B - 1) / B);
        sc.run(kStageShading, p, s, [&](const TraceParams& q) {
            k_wf_camera<<<std::min(g_camera, cap), B, 0, s>>>(q, W);
        });
        sc.run(kStageIntersect, p, s, [&](const TraceParams& q) {
            run_trace(trace0, (long long)nt * 32, q, o.visibility, W, kQIsect, W.q[kQIsect], -1, 1, s);
        });
        sc.run(kStageShading, p, s, [&](const TraceParams& q) {
            k_wf_fwd_primary<K><<<std::min(g_primary, cap), B, 0, s>>>(q, o, W);
        });
        if (p.flags & kMis) {
            const unsigned* shadow_items = sort_queue(p, b, W, tune, sc, s, tune.shadow_kbuf <= 16, kQShadow);
            sc.run(kStageShadow, p, s,
                   [&](const TraceParams& q) { launch_shadow(tune, q, W, shadow_items, s); });
        }
        unsigned cursor = kFirstBounceCursor;
        for (unsigned depth = 0; depth < mb; ++depth) {
            cudaMemsetAsync(W.count + kQIsect, 0, sizeof(unsigned), s);
            sc.run(kStageShading, p, s, [&](const TraceParams& q) {
                k_wf_fwd_bounce<K><<<g_bounce, B, 0, s>>>(q, o, W, depth, cursor);
            });
            ++cursor;
            if (depth + 1 >= mb) break;
            cudaMemsetAsync(W.count + kQBounce, 0, sizeof(unsigned), s);
            const unsigned* items = sort_queue(p, b, W, tune, sc, s, trace.quad_fn != nullptr);
            sc.run(kStageIntersect, p, s, [&](const TraceParams& q) {
                run_trace(trace, (long long)nt * 32, q, o.visibility, W, kQIsect, items, kQBounce, cursor, s);
            });
            ++cursor;
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <int K>
static cudaError_t run_bwd(const TraceParams& p, const BwdInputs& bi, WavefrontBuffers& b, const WavefrontTuning& tune,
                           const StageCtx& sc, cudaStream_t s) {
    const unsigned long long tiles = total_tiles(p);
    if (tiles == 0) return cudaSuccess;
    const unsigned chunk_tiles = (unsigned)std::min<unsigned long long>(tune.chunk_tiles, tiles);
    cudaError_t e = wavefront_reserve(b, (size_t)chunk_tiles * 32, s);
    if (e != cudaSuccess) return e;
    const int B = tune.block, R = tune.refill_lanes;
    const int g_camera = grid_cached((const void*)k_wf_camera, B);
    const int g_primary = grid_cached((const void*)k_wb_primary<K>, B);
    const int g_bounce = grid_cached((const void*)k_wb_bounce<K>, B);
    const bool resume = use_resume<K>(tune);
    const bool resume_replay = K <= 16 && tune.resume_replay;
    const TraceLaunch trace0 = trace_launch<K, false, false>(tune, resume), trace = trace_launch<K, false, true>(tune, resume);
    // replays with resumed rounds: a quad a job up to kQuadRays jobs (at most two a path), a lane a job above
    const size_t quad_stacks = sizeof(StackEntry) * kQuadStackEntries * (size_t)(B / 4);
    const unsigned quad_jobs = resume_replay ? kQuadRays : 0u;
    const bool lane_jobs = 2ull * 32ull * chunk_tiles > quad_jobs;
    const int g_replay = grid_cached((const void*)k_wb_replay<K>, B);
    int g_replay_quad = 0;
    if constexpr (K <= 16) {
        if (resume_replay) g_replay_quad = grid_cached((const void*)replay_quad_fn<K>(tune), B, quad_stacks);
    }
    // frontiers: one a thread of a resumed kernel, one a quad of the replay
    const size_t fronts = std::max({resume ? (size_t)std::max(trace0.lane_grid, trace.lane_grid) * B : (size_t)0,
                                    resume_replay && lane_jobs ? (size_t)g_replay * B : (size_t)0,
                                    (size_t)g_replay_quad * B / 4});
    if (fronts > 0 && (e = frontier_reserve(b, fronts, s)) != cudaSuccess) return e;
    const unsigned mb = p.render_opts ? std::min(p.max_bounces, 2u) : p.max_bounces;
    if (kFirstBounceCursor + 3u * mb > (unsigned)kNumCursors) return cudaErrorInvalidValue;
    for (unsigned long long t0 = 0; t0 < tiles; t0 += chunk_tiles) {
        const unsigned nt = (unsigned)std::min<unsigned long long>(chunk_tiles, tiles - t0);
        const WfView W = view_of(b, t0, nt * 32u, fronts > 0);
        e = cudaMemsetAsync(b.counters, 0, sizeof(unsigned) * (kNumQueueCounts + kNumCursors), s);
        if (e != cudaSuccess) return e;
        const int cap = (int)std::min<long long>(INT32_MAX, ((long long)nt * 32 + B - 1) / B);
        sc.run(kStageShading, p, s, [&](const TraceParams& q) {
            k_wf_camera<<<std::min(g_camera, cap), B, 0, s>>>(q, W);
        });
        sc.run(kStageIntersect, p, s, [&](const TraceParams& q) {
            run_trace(trace0, (long long)nt * 32, q, nullptr, W, kQIsect, W.q[kQIsect], -1, 1, s);
        });
        sc.run(kStageShading, p, s, [&](const TraceParams& q) {
            k_wb_primary<K><<<std::min(g_primary, cap), B, 0, s>>>(q, bi, W);
        });
        if (p.flags & kMis) {
            const unsigned* shadow_items = sort_queue(p, b, W, tune, sc, s, tune.shadow_kbuf <= 16, kQShadow);
            sc.run(kStageShadow, p, s,
                   [&](const TraceParams& q) { launch_shadow(tune, q, W, shadow_items, s); });
        }
        unsigned cursor = kFirstBounceCursor;
        for (unsigned depth = 0; depth < mb; ++depth) {
            cudaMemsetAsync(W.count + kQIsect, 0, sizeof(unsigned), s);
            cudaMemsetAsync(W.count + kQJobs, 0, sizeof(unsigned), s);
            sc.run(kStageShading, p, s, [&](const TraceParams& q) {
                k_wb_bounce<K><<<g_bounce, B, 0, s>>>(q, bi, W, depth, cursor);
            });
            ++cursor;
            sc.run(kStageReplay, p, s, [&](const TraceParams& q) {
                if constexpr (K <= 16) {
                    if (resume_replay) {
                        const long long need = (2ll * W.slots + B / 32 - 1) / (B / 32);
                        replay_quad_fn<K>(tune)<<<(unsigned)std::min<long long>(g_replay_quad, need), B, quad_stacks, s>>>(
                            q, bi, W, cursor, (R + 7) / 8, quad_jobs);
                    }
                }
                if (lane_jobs) k_wb_replay<K><<<g_replay, B, 0, s>>>(q, bi, W, cursor, resume_replay, quad_jobs);
            });
            ++cursor;
            if (depth + 1 >= mb) break;
            cudaMemsetAsync(W.count + kQBounce, 0, sizeof(unsigned), s);
            const unsigned* items = sort_queue(p, b, W, tune, sc, s, trace.quad_fn != nullptr);
            sc.run(kStageIntersect, p, s, [&](const TraceParams& q) {
                run_trace(trace, (long long)nt * 32, q, nullptr, W, kQIsect, items, kQBounce, cursor, s);
            });
            ++cursor;
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_trace_fwd_wavefront(const TraceParams& p, const FwdOutputs& o, WavefrontBuffers& b,
                                       const WavefrontTuning& tune, const StageCtx& sc, cudaStream_t s) {
    switch (tune.kbuf) {
    case 8: return run_fwd<8>(p, o, b, tune, sc, s);
    case 32: return run_fwd<32>(p, o, b, tune, sc, s);
    default: return run_fwd<16>(p, o, b, tune, sc, s);
    }
}

cudaError_t launch_trace_bwd_wavefront(const TraceParams& p, const BwdInputs& bi, WavefrontBuffers& b,
                                       const WavefrontTuning& tune, const StageCtx& sc, cudaStream_t s) {
    switch (tune.kbuf) {
    case 8: return run_bwd<8>(p, bi, b, tune, sc, s);
    case 32: return run_bwd<32>(p, bi, b, tune, sc, s);
    default: return run_bwd<16>(p, bi, b, tune, sc, s);
    }
}

}  // namespace ptir
