// The subsurface probe loop of the render path.
#pragma once

#include "traversal.cuh"

namespace yrc {
namespace {

// SampleBssrdfProbe's probe (src/integrators/bssrdf_probe.cpp:51-66) for the
// render path: IntersectAccelerationProbe's loop (closest-hit queries with an
// advancing cursor, target hits kept in t order, at most kProbeMaxHits)
// run twice per probe, first to count the target hits, then to return the
// one the selection sample picks (floor(u * count), clamped), so no per-probe
// hit list is stored.
template <bool kTwo, typename Stack>
__device__ __forceinline__ void ProbeLoop(const RenderProbeArgs& args, int64_t k, Stack& st, int2* col) {
    Traversal s;
    const int4 target = args.targets[k];
    const float t_min = Ld(args.rays + 2 * k).w;
    const float t_max = Ld(args.rays + 2 * k + 1).w;
    // pass == 0 counts; pass == 1 stops at the selected target hit
    int32_t count = 0;
    int32_t selected = -1;
    float4 chosen = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            if (count == 0) break;
            const float u = args.selection[2 * k].w;
            selected = min(max(static_cast<int32_t>(u * static_cast<float>(count)), 0), count - 1);
        }
        int32_t seen = 0;
        float cursor = t_min;
        for (int iter = 0; iter < kProbeMaxIterations; ++iter) {
            bool alive = Begin(args.accel, args.rays, k, cursor, t_max, s);
            while (alive) alive = Step<false, false, kTwo, Stack>(args.accel, args.rays, k, s, st, col, args.error);
            if (!s.best.hit) break;
            const bool inst_ok = !kTwo || target.y < 0 || s.best_inst == target.y;
            const bool is_target = (target.x >= 0 && s.best.id >= 0 && s.best.prim == target.x && inst_ok) ||
                                   (target.z >= 0 && s.best.id == -2 - target.z);
            if (is_target) {
                if (seen >= kProbeMaxHits) break;
                if (pass == 1 && seen == selected) {
                    chosen = make_float4(s.best.t, __int_as_float(s.best.id), s.best.u, s.best.v);
                    break;
                }
                ++seen;
            }
            float next = __fadd_rn(s.best.t, __fmul_rn(1.0e-4f, __fadd_rn(1.0f, fabsf(s.best.t))));
            if (!(next > cursor)) next = __fadd_rn(cursor, 1.0e-4f);
            cursor = next;
            if (cursor >= t_max) break;
        }
        if (pass == 0) count = seen;
    }
    args.hits[k] = count;
    args.hit[k] = chosen;
}

}  // namespace
}  // namespace yrc
