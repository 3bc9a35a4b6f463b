// The end of a single-pass shadow ray, shared by the transmittance kernels
// over the exact and the quantised nodes.
#pragma once

#include "render_types.hpp"
#include "traversal.cuh"

namespace yrc {
namespace {

// The reference's shadow loop over the kept clear surfaces; returns the RGB
// transmittance, w = 1 when visible, all 0 when occluded, w = -1 when the
// kept surfaces do not decide it.
__device__ __forceinline__ float4 ReplayShadow(const ShadowArgs& A, int64_t ray, const ClearHits& clear) {
    const float4 ra = Ld(A.rays + 2 * ray);
    const float4 rb = Ld(A.rays + 2 * ray + 1);
    float o[3] = {ra.x, ra.y, ra.z};
    const float d[3] = {rb.x, rb.y, rb.z};
    float remaining = rb.w;
    float T[3] = {1.0f, 1.0f, 1.0f}, mc[3] = {1.0f, 1.0f, 1.0f}, md = 1.0f;
    bool medium = false;
    float qmin = ra.w;   // t_min of the current query
    float off = 0.0f;    // distance from the ray origin to the current query's origin
    const float4 occluded = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto black = [&]() { return fmaxf(T[0], fmaxf(T[1], T[2])) <= 1.0e-6f; };
    auto beer = [&](float dist) {
        if (dist <= 0.0f || md <= 0.0f) return;
        const float inv = 1.0f / md;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float c = fminf(fmaxf(mc[k], 1.0e-6f), 1.0f);
            T[k] = T[k] * expf(logf(c) * dist * inv);
        }
    };
    int k = 0;
    for (int query = 0; query < kClearHits; ++query) {
        const bool finite = isfinite(remaining);
        float t = 0.0f;
        int32_t id = 0;
        bool found = false;
        for (; k < clear.n; ++k) {
            t = __fsub_rn(clear.t[k * kTraceBlock], off);
            if (t > qmin && t <= remaining) {
                id = clear.id[k * kTraceBlock];
                found = true;
                ++k;
                break;
            }
        }
        if (!found) {
            // A surface beyond the kept ones would be this query's
            // answer: the exact loop traces this ray instead.
            if (clear.dropped) return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
            if (medium) {
                if (!finite) return occluded;
                beer(remaining);
            }
            return black() ? occluded : make_float4(T[0], T[1], T[2], 1.0f);
        }
        if (medium) {
            beer(t);
            if (black()) return occluded;
        }
        const int32_t material = id >= 0 ? A.prim_material[A.tri_prim[id]] : A.sphere_material[-2 - id];
        if (material < 0 || (A.materials[material].kind != 2 && A.materials[material].kind != 3)) {
            return occluded;
        }
        const DevMaterial& m = A.materials[material];
        float hp[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) hp[c] = __fadd_rn(o[c], __fmul_rn(d[c], t));
        if (m.kind == 3) {
#pragma unroll
            for (int c = 0; c < 3; ++c) T[c] = T[c] * fminf(fmaxf(m.reflectance[c], 0.0f), 1.0f);
            if (black()) return occluded;
        } else if (medium) {
            medium = false;
            mc[0] = mc[1] = mc[2] = 1.0f;
            md = 1.0f;
        } else {
            medium = true;
            mc[0] = m.absorption_color[0];
            mc[1] = m.absorption_color[1];
            mc[2] = m.absorption_color[2];
            md = m.absorption_distance;
        }
        const float bias = fmaxf(1.0e-4f, fmaxf(fabsf(hp[0]), fmaxf(fabsf(hp[1]), fabsf(hp[2]))) * 1.0e-5f);
        if (finite) {
            remaining = __fsub_rn(remaining, __fadd_rn(t, bias));
            if (remaining <= 0.0f) return black() ? occluded : make_float4(T[0], T[1], T[2], 1.0f);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c] = __fadd_rn(hp[c], __fmul_rn(d[c], bias));
        off = __fadd_rn(off, __fadd_rn(t, bias));
        qmin = 1.0e-5f;
    }
    return occluded;  // the reference gives up after 16 queries
}

// Writes the ray's transmittance, or lists it for the exact loop.
__device__ __forceinline__ void FinishShadow(const ShadowArgs& A, int64_t ray, bool hit, bool saw,
                                             const ClearHits& clear) {
    const int32_t slot = A.out_index[ray];
    float4 tr;
    if (hit) {
        tr = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else if (!saw) {
        tr = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    } else {
        tr = ReplayShadow(A, ray, clear);
        if (tr.w < 0.0f) {
            const unsigned long long o = atomicAdd(A.overflow_count, 1ull);
            A.overflow[o] = static_cast<int32_t>(ray);
            return;
        }
    }
    A.transmittance[slot] = tr;
    if (tr.w == 0.0f) CountLanes(A.occluded_count);
}

}  // namespace
}  // namespace yrc
