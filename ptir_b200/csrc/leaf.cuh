// Candidate test shared by the traversals of more than one lane a ray.
#pragma once

#include "traverse.cuh"

namespace ptir {

// 32 bytes through the read-only path, 32-byte aligned
PTIR_DEV void ld256(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// leaf_candidate (traverse.cuh) on a leaf record fetched with two 32-byte loads
PTIR_DEV bool leaf_candidate_wide(const AccelView& A, int p, float3 o, float3 d, float tmin, float tend, float cut,
                                  float& ts_out, unsigned& id_out, float floor) {
    const float4* rec = A.leaves + 4 * (size_t)p;
    float4 r0, r1, r2, r3;
    ld256(rec, r0, r1);
    ld256(rec + 2, r2, r3);
    const float3 od = make_float3(r0.x * o.x + r0.y * o.y + r0.z * o.z + r0.w,
                                  r1.x * o.x + r1.y * o.y + r1.z * o.z + r1.w,
                                  r2.x * o.x + r2.y * o.y + r2.z * o.z + r2.w);
    const float3 dd = make_float3(r0.x * d.x + r0.y * d.y + r0.z * d.z, r1.x * d.x + r1.y * d.y + r1.z * d.z,
                                  r2.x * d.x + r2.y * d.y + r2.z * d.z);
    const float den = 1.0f / dot(dd, dd);
    const float ts = -dot(od, dd) * den;
    if (!(ts > tmin && ts >= floor && ts < fminf(tend, cut))) return false;
    const float3 inv = make_float3(1.0f / dd.x, 1.0f / dd.y, 1.0f / dd.z);
    float b0, b1;
    slab(f3(-1.0f), f3(1.0f), od, inv, b0, b1);
    if (fmaxf(b0, tmin) > fminf(b1, tend)) return false;
    // The perpendicular distance of a line through the box is at most sqrt(3) instance units, and the rounding of
    // the cross product adds less than 1e-6 |od| to it, with |od| <= ts |dd| + sqrt(3): where den < 1 and ts < 1e5
    // the distance test cannot fail, and it is skipped.
    if (!(den < 1.0f && ts < 1e5f)) {
        const float3 c = cross(normalize_or_keep(dd), od);
        if (!(dot(c, c) * den < 9.0f)) return false;
    }
    ts_out = ts;
    id_out = __float_as_uint(r3.x);
    return true;
}

// leaf_candidate3 (traverse.cuh) of a resumable call, the same way, without its last condition on the cut: 2 when t*
// lies in (tmin, tend), and 1 as well when the leaf is a candidate there (its box test passes; decided only
// for t* before `cut`).
PTIR_DEV int leaf_candidate3_wide(const AccelView& A, int p, float3 o, float3 d, float tmin, float tend, float cut,
                                  float& ts_out) {
    const float4* rec = A.leaves + 4 * (size_t)p;
    float4 r0, r1, r2, r3;
    ld256(rec, r0, r1);
    ld256(rec + 2, r2, r3);
    const float3 od = make_float3(r0.x * o.x + r0.y * o.y + r0.z * o.z + r0.w,
                                  r1.x * o.x + r1.y * o.y + r1.z * o.z + r1.w,
                                  r2.x * o.x + r2.y * o.y + r2.z * o.z + r2.w);
    const float3 dd = make_float3(r0.x * d.x + r0.y * d.y + r0.z * d.z, r1.x * d.x + r1.y * d.y + r1.z * d.z,
                                  r2.x * d.x + r2.y * d.y + r2.z * d.z);
    const float den = 1.0f / dot(dd, dd);
    const float ts = -dot(od, dd) * den;
    if (!(ts > tmin && ts < tend)) return 0;
    ts_out = ts;
    if (!(ts < cut)) return 2;
    const float3 inv = make_float3(1.0f / dd.x, 1.0f / dd.y, 1.0f / dd.z);
    float b0, b1;
    slab(f3(-1.0f), f3(1.0f), od, inv, b0, b1);
    if (fmaxf(b0, tmin) > fminf(b1, tend)) return 2;
    if (!(den < 1.0f && ts < 1e5f)) {  // as in leaf_candidate_wide
        const float3 c = cross(normalize_or_keep(dd), od);
        if (!(dot(c, c) * den < 9.0f)) return 2;
    }
    return 3;
}

}  // namespace ptir
