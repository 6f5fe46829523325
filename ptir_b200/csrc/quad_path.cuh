// Compositing and shadow walks of a quad's k-buffer batch (quad.cuh), four hits at a time: lane c
// evaluates hit 4r + c of round r (the particle response and what the hit contributes, none of which
// depends on the hits before it), then the quad goes over the four hits in order. The order-dependent
// part (transmittance, acceptance while it lasts, the sums) is composite_one's, operation for operation,
// so the sums are those of one lane going over the batch, up to how the compiler contracts a term's multiply-adds (with a
// k-buffer of 8 and SH of degree 3 the radiance differs in its last bit, and is the megakernel's).
#pragma once

#include "path.cuh"
#include "quad.cuh"

namespace ptir {

// entry 4r + c of the quad's k-buffer in lane c; `mask`: the lanes calling, whole quads
template <int K>
PTIR_DEV void quad_hit(const QuadTrace<K>& t, int r, unsigned c, unsigned base, unsigned mask, float& ts, unsigned& id) {
    constexpr int L = QuadTrace<K>::L;
    ts = kFarT;
    id = kNoHit;
    const int e = 4 * r + (int)c;
#pragma unroll
    for (int j = 0; j < L; ++j) {
        const float a = __shfl_sync(mask, t.kt[j], base + e / L);
        const unsigned b = __shfl_sync(mask, t.kid[j], base + e / L);
        if (e % L == j) {
            ts = a;
            id = b;
        }
    }
}

// A quad's compositing state in shared memory: the scalars of Composite, then its sums, four to a lane
// (radiance -, albedo roughness, shading normal metallic, normal -).
struct QuadComposite {
    float transmittance, depth, hit2, distortion, hits_count, last_hit, clip_end, hit;
    float4 sums[4];
};

// hits staged for the quad: per hit the four sums' terms and (alpha, hit distance, k-buffer distance, flags)
constexpr int kQuadStage = 4 * 5;  // float4

enum : unsigned { kStageHit = 1u, kStageAccept = 2u };

PTIR_DEV bool quad_open(const TraceParams& P, const QuadComposite& s) {
    return s.last_hit <= s.clip_end && s.transmittance > P.min_transmittance;
}

PTIR_DEV void quad_composite_begin(const TraceParams& P, QuadComposite& s, float3 o, float3 d, unsigned c, unsigned mask) {
    const float2 clip = clip_scene(P, o, d);
    s.sums[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (c == 0) {
        s.transmittance = 1.0f;
        s.depth = s.hit2 = s.distortion = s.hits_count = 0.0f;
        s.last_hit = fmaxf(0.0f, clip.x - 1e-9f);
        s.clip_end = clip.y;
        s.hit = 0.0f;
    }
    __syncwarp(mask);
}

// The batch of the finished call of each quad in `mask` onto its compositing state. `stage` is
// kQuadStage float4 of shared memory of the quad.
template <bool kSelfOcc, int K>
PTIR_DEV void quad_composite(const TraceParams& P, TraceCounters& ctr, QuadComposite& s, float4* stage,
                             const QuadTrace<K>& t, float3 o, float3 d, float* vis, unsigned ln, unsigned mask) {
    const unsigned c = ln & 3u, base = ln & 28u;
    float tr = s.transmittance, depth = s.depth, hit2 = s.hit2, distortion = s.distortion;
    float hits_count = s.hits_count, last_hit = s.last_hit, any = s.hit;
    float4 sum = s.sums[c];
    bool open = tr > P.min_transmittance;
#pragma unroll 1
    for (int r = 0; r < K / 4; ++r) {
        float th;
        unsigned id;
        quad_hit(t, r, c, base, mask, th, id);
        unsigned flags = 0u;
        if (open && id != kNoHit) {
            flags = kStageHit;
            float alpha = 0.0f, hit_t = 0.0f;
            if (!(kSelfOcc && self_occluded(P, th, id, d))) {
                float dns;
                const Response res = respond(P, id, o, d, dns);
                alpha = res.alpha;
                if (res.gres > P.min_response && res.alpha > P.alpha_min) {
                    flags |= kStageAccept;
                    const float3 grds = res.scl * res.grd * dot(res.grd, -res.gro);
                    hit_t = sqrtf(dot(grds, grds));
                    const float3 rad = sh_radiance(P, id, d);
                    float3 alb;
                    float rgh, met;
                    load_material(P.part, id, alb, rgh, met);
                    float3 sn = f3(0.0f), nr = f3(0.0f);
                    if (P.flags & kNormals) {
                        sn = load_snrm(P.part, id);
                        const float3 srot = mul_cols(res.rt, res.scl);
                        nr = normalize_or_keep((res.gro + res.grd * (dot(res.grd, -res.gro) - sqrtf(9.0f - res.d2))) * srot);
                    }
                    float4* v = stage + 5 * c;
                    v[0] = make_float4(rad.x, rad.y, rad.z, 0.0f);
                    v[1] = make_float4(alb.x, alb.y, alb.z, rgh);
                    v[2] = make_float4(sn.x, sn.y, sn.z, met);
                    v[3] = make_float4(nr.x, nr.y, nr.z, 0.0f);
                }
            }
            stage[5 * c + 4] = make_float4(alpha, hit_t, th, 0.0f);
        }
        const unsigned hits = (__ballot_sync(mask, flags != 0u) >> base) & 15u;
        const unsigned acc = (__ballot_sync(mask, (flags & kStageAccept) != 0u) >> base) & 15u;
        __syncwarp(mask);
        for (unsigned i = 0; i < 4; ++i) {
            if (!((hits >> i) & 1u) || !(tr > P.min_transmittance)) continue;
            const float4 h = stage[5 * i + 4];
            if ((acc >> i) & 1u) {
                const float4 v = stage[5 * i + c];
                const float w = h.x * tr;
                sum.x += v.x * w;
                sum.y += v.y * w;
                sum.z += v.z * w;
                sum.w += v.w * w;
                tr *= (1.0f - h.x);
                depth += h.y * w;
                hit2 += h.y * h.y * w;
                any = 1.0f;
                const float op = 1.0f - tr;
                distortion = fmaxf(op * hit2 - depth * depth, 0.0f);
                hits_count += 1.0f;
                if (i == c) {
                    ++ctr.accepted;
                    if (vis) vis[id] = __int_as_float(1);
                }
            }
            last_hit = fmaxf(last_hit, h.z);
        }
        __syncwarp(mask);
        open = tr > P.min_transmittance;
        if (!__any_sync(mask, open && hits == 15u)) break;  // no quad has a further hit to take
    }
    s.sums[c] = sum;
    if (c == 0) {
        s.transmittance = tr;
        s.depth = depth;
        s.hit2 = hit2;
        s.distortion = distortion;
        s.hits_count = hits_count;
        s.last_hit = last_hit;
        s.hit = any;
    }
    __syncwarp(mask);
}

// the one-lane form of a quad's compositing state (for composite_end)
PTIR_DEV void quad_composite_gather(const QuadComposite& s, Composite& c, float3 o, float3 d) {
    c.o = o;
    c.d = d;
    c.radiance = make_float3(s.sums[0].x, s.sums[0].y, s.sums[0].z);
    c.albedo = make_float3(s.sums[1].x, s.sums[1].y, s.sums[1].z);
    c.rough = s.sums[1].w;
    c.snrm = make_float3(s.sums[2].x, s.sums[2].y, s.sums[2].z);
    c.metal = s.sums[2].w;
    c.normal = make_float3(s.sums[3].x, s.sums[3].y, s.sums[3].z);
    c.transmittance = s.transmittance;
    c.depth = s.depth;
    c.hit2 = s.hit2;
    c.distortion = s.distortion;
    c.hits_count = s.hits_count;
    c.last_hit = s.last_hit;
    c.clip_end = s.clip_end;
    c.hit = s.hit != 0.0f;
}

// The shadow walk over the batch of the finished call of each quad in `mask` (shadow_occluded in path.cuh), in
// the batch's order with the ray's own draws, which all four lanes make: whether a hit occludes the ray; else
// `batch_end` is raised to the farthest hit walked.
template <int K>
PTIR_DEV bool quad_shadow_walk(const TraceParams& P, const QuadTrace<K>& t, float3 o, float3 d, float end, Pcg32& rng,
                               float& batch_end, unsigned ln, unsigned mask) {
    const unsigned c = ln & 3u, base = ln & 28u;
    bool occluded = false, stop = false;
#pragma unroll 1
    for (int r = 0; r < K / 4; ++r) {
        float th;
        unsigned id;
        quad_hit(t, r, c, base, mask, th, id);
        const bool hit = !stop && id != kNoHit && !(th > end);
        float alpha = 0.0f;
        if (hit && !self_occluded(P, th, id, d)) {
            float dns;
            const Response res = respond(P, id, o, d, dns);
            alpha = (res.gres > P.min_response && res.alpha > P.alpha_min) ? res.alpha : 0.0f;
        }
        const unsigned hits = (__ballot_sync(mask, hit) >> base) & 15u;
#pragma unroll
        for (unsigned i = 0; i < 4; ++i) {
            const float ai = __shfl_sync(mask, alpha, base + i), ti = __shfl_sync(mask, th, base + i);
            if (stop || occluded) continue;
            if (!((hits >> i) & 1u)) {
                stop = true;
                continue;
            }
            batch_end = fmaxf(batch_end, ti);
            if (ai > 0.0f && rng.uniform() < ai) occluded = true;
        }
        stop = stop || occluded;
        if (!__any_sync(mask, !stop)) break;
    }
    return occluded;
}

// replay_batch (path.cuh) for a quad whose k-buffer holds leaf record indices: each lane evaluates its hits and
// scatters their gradient rows, the transmittance goes through the hits in order.
template <int K>
PTIR_DEV void quad_replay_batch(const TraceParams& P, const BwdInputs& B, ReplayState& r, const QuadTrace<K>& t,
                                TraceCounters& ctr, unsigned ln, unsigned mask) {
    const unsigned c = ln & 3u, base = ln & 28u;
    const bool metallic_on = (P.flags & kMetallic) != 0;
#pragma unroll 1
    for (int k = 0; k < K / 4; ++k) {
        float th;
        unsigned leaf;
        quad_hit(t, k, c, base, mask, th, leaf);
        const bool open = r.tr > P.min_transmittance;
        const bool hit = open && leaf != kNoHit;
        unsigned id = 0u;
        float alpha = 0.0f;
        bool accept = false;
        if (hit) {
            id = leaf_gaussian(P.accel, leaf);
            if (!(r.self_occ && self_occluded(P, th, id, r.d))) {
                float dns;
                const Response res = respond(P, id, r.o, r.d, dns);
                alpha = res.alpha;
                accept = res.gres > P.min_response && res.alpha > P.alpha_min;
            }
        }
        const unsigned hits = (__ballot_sync(mask, hit) >> base) & 15u;
        const unsigned acc = (__ballot_sync(mask, accept) >> base) & 15u;
        float w = 0.0f;
        bool scatter = false;
#pragma unroll
        for (unsigned i = 0; i < 4; ++i) {
            const float ai = __shfl_sync(mask, alpha, base + i), ti = __shfl_sync(mask, th, base + i);
            if (!((hits >> i) & 1u) || !(r.tr > P.min_transmittance)) continue;
            if ((acc >> i) & 1u) {
                if (i == c) {
                    w = ai * r.tr;
                    scatter = true;
                }
                r.tr *= (1.0f - ai);
            }
            r.start = fmaxf(r.start, ti);
        }
        if (scatter) {
            ++ctr.replay_accepted;
            float* g = B.particle_material_grad + 5 * (size_t)id;
            float* cg = B.particle_material_comp ? B.particle_material_comp + 5 * (size_t)id : nullptr;
            float row[5] = {w * r.da.x, w * r.da.y, w * r.da.z, w * r.dr, w * r.dm};
            grad_add_row(P.flags, g, cg, row, metallic_on ? 5 : 4);
        }
        __syncwarp(mask);
        if (!__any_sync(mask, hits == 15u && r.tr > P.min_transmittance)) break;
    }
}

}  // namespace ptir
