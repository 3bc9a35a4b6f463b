// Closest- and any-hit traversal launches over the quantised nodes
// (quantised.cuh).
#include "probe_loop.cuh"
#include "quantised.cuh"
#include "shadow_replay.cuh"
#include "trace_kernels.hpp"

#include <cuda_runtime.h>

#include <algorithm>

namespace yrc {
namespace {

// The end of a ray: a closest hit was written when it was found, an undecided
// ray is marked and listed for RetraceKernel.
template <bool kAny>
__device__ __forceinline__ void FinishTrace(const TraceArgs& args, int64_t ray, const QTraversal& q) {
    if (kAny) {
        args.occluded[args.out_index ? args.out_index[ray] : ray] = q.id >= 0 ? 1 : 0;
        if (args.occluded_count && q.id >= 0) CountLanes(args.occluded_count);
        return;
    }
    if (q.id < 0) {
        reinterpret_cast<float4*>(args.hits)[ray] =
            make_float4(q.t, __int_as_float(q.id == -1 ? -1 : kUndecidedId), 0.0f, 0.0f);
        if (q.id != -1) {
            // An index that the list cannot hold counts as its overflow.
            const unsigned long long slot = atomicAdd(args.undecided, (ray >> 32) ? kUndecidedMax + 1ull : 1ull);
            if (slot < kUndecidedMax) reinterpret_cast<uint32_t*>(args.undecided + 1)[slot] = static_cast<uint32_t>(ray);
        }
    }
    if (args.instances) {
        args.instances[ray] = q.inst < 0 ? -1 : __float_as_int(Ld(&args.accel.records[q.inst].v0).w);
    }
}

// The exact traversal of the rays the quantised one left undecided, one per
// thread: the listed ones, or, when more than the list holds are, those that
// carry the mark. Nearly always there is none, and the launch costs its 2 us.
template <bool kTwo>
__global__ void __launch_bounds__(kTraceBlock) RetraceKernel(const __grid_constant__ TraceArgs args) {
    __shared__ int2 s_stack[kShortStack * kTraceBlock];
    int2* col = s_stack + threadIdx.x;
    StackStore<kQuantisedExactStack> st;
    Traversal s;
    const unsigned long long listed = *args.undecided;
    if (listed == 0) return;
    const bool scan = listed > kUndecidedMax;
    const unsigned long long n =
        !scan ? listed : args.count_ptr ? *args.count_ptr : static_cast<unsigned long long>(args.count);
    const uint32_t* list = reinterpret_cast<const uint32_t*>(args.undecided + 1);
    for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(kTraceBlock) + threadIdx.x; i < n;
         i += static_cast<unsigned long long>(gridDim.x) * kTraceBlock) {
        const int64_t ray = scan ? static_cast<int64_t>(i) : static_cast<int64_t>(list[i]);
        float4* hit = reinterpret_cast<float4*>(args.hits) + ray;
        if (__float_as_int(hit->y) != kUndecidedId) continue;
        bool alive = Begin(args.accel, args.rays, ray, Ld(args.rays + 2 * ray).w, Ld(args.rays + 2 * ray + 1).w, s);
        while (alive) alive = Step<false, false, kTwo, StackStore<kQuantisedExactStack>>(args.accel, args.rays, ray, s, st, col, args.error);
        *hit = make_float4(s.best.t, __int_as_float(s.best.hit ? s.best.id : -1), s.best.u, s.best.v);
        if (args.instances) args.instances[ray] = s.best.hit ? s.best_inst : -1;
    }
}

// TraceKernel over the quantised nodes (quantised.cuh), no statistics: the
// same persistent lanes, refill and leaf batching.
template <bool kAny, bool kTwo, int kBlock, int kStepsPerRefill, int kMinBlocks, int kLeafBatch>
__global__ void __launch_bounds__(kBlock, kMinBlocks) QTraceKernel(const __grid_constant__ TraceArgs args) {
    __shared__ int2 s_stack[kShortStack * kBlock];
    int2* col = s_stack + threadIdx.x;
    StackStore<kQuantisedStack, kBlock> st;
    QTraversal q;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    int64_t ray = -1;
    bool alive = false;
    bool exhausted = false;
    const unsigned long long count =
        args.count_ptr ? *args.count_ptr : static_cast<unsigned long long>(args.count);

    for (;;) {
        const unsigned need = __ballot_sync(kFull, !alive && !exhausted);
        if (need) {
            unsigned long long base = 0;
            const int leader = __ffs(need) - 1;
            if (static_cast<int>(lane) == leader) {
                base = atomicAdd(args.counter, static_cast<unsigned long long>(__popc(need)));
            }
            base = __shfl_sync(kFull, base, leader);
            if (!alive && !exhausted) {
                const unsigned long long idx = base + __popc(need & lt_mask);
                if (idx >= count) {
                    exhausted = true;
                } else {
                    ray = args.order ? static_cast<int64_t>(__ldg(args.order + idx)) : static_cast<int64_t>(idx);
                    alive = QBegin<kTwo, !kAny>(args.accel, args.rays, ray, q);
                    if (!alive) FinishTrace<kAny>(args, ray, q);
                }
            }
        }
        if (!__any_sync(kFull, alive)) {
            if (__all_sync(kFull, exhausted)) break;
            continue;
        }
#pragma unroll 1
        for (int k = 0; k < kStepsPerRefill; ++k) {
            if (!QVoteStep<kAny ? kQAny : kQClosest, kTwo, kLeafBatch>(
                    args.accel, alive, q, st, col, args.error, nullptr, nullptr, nullptr,
                    [&](float t, int32_t id, float u, float v) {
                        reinterpret_cast<float4*>(args.hits)[ray] = make_float4(t, __int_as_float(id), u, v);
                    },
                    [&] { FinishTrace<kAny>(args, ray, q); })) {
                break;
            }
        }
    }
}

// ShadowTransmittanceKernel over the quantised nodes.
template <bool kTwo, int kMinBlocks, int kLeafBatch>
__global__ void __launch_bounds__(kTraceBlock, kMinBlocks) QShadowKernel(const __grid_constant__ ShadowArgs args) {
    __shared__ int2 s_stack[kShadowShortStack * kTraceBlock];
    __shared__ float s_clear_t[kClearHits * kTraceBlock];
    __shared__ int32_t s_clear_id[kClearHits * kTraceBlock];
    int2* col = s_stack + threadIdx.x;
    StackStore<kQuantisedStack, kTraceBlock, kShadowShortStack> st;
    QTraversal q;
    ClearHits clear{s_clear_t + threadIdx.x, s_clear_id + threadIdx.x, 0, false};
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned long long count = *args.count_ptr;
    int64_t ray = -1;
    bool alive = false;
    bool exhausted = false;
    for (;;) {
        const unsigned need = __ballot_sync(kFull, !alive && !exhausted);
        if (need) {
            unsigned long long base = 0;
            const int leader = __ffs(need) - 1;
            if (static_cast<int>(lane) == leader) {
                base = atomicAdd(args.counter, static_cast<unsigned long long>(__popc(need)));
            }
            base = __shfl_sync(kFull, base, leader);
            if (!alive && !exhausted) {
                const unsigned long long idx = base + __popc(need & lt_mask);
                if (idx >= count) {
                    exhausted = true;
                } else {
                    ray = static_cast<int64_t>(idx);
                    clear.n = 0;
                    clear.dropped = false;
                    alive = QBegin<kTwo, false>(args.accel, args.rays, ray, q);
                    if (!alive) FinishShadow(args, ray, false, false, clear);
                }
            }
        }
        if (!__any_sync(kFull, alive)) {
            if (__all_sync(kFull, exhausted)) break;
            continue;
        }
#pragma unroll 1
        for (int k = 0; k < 8; ++k) {
            if (!QVoteStep<kQFilter, kTwo, kLeafBatch>(
                    args.accel, alive, q, st, col, args.error, args.tri_clear, &clear, nullptr,
                    [](float, int32_t, float, float) {}, [&] { FinishShadow(args, ray, q.id >= 0, q.saw, clear); })) {
                break;
            }
        }
    }
}

// SampleBssrdfProbe's probe over the quantised nodes: one traversal collects
// the segment's surfaces in t order (SurfaceList), and the reference's loop of
// closest-hit queries (ProbeLoop) is replayed over that list, once to count
// the target hits and once to stop at the selected one, instead of being
// traced twice. A probe whose list is open is traced as before. The probe is
// short and few surfaces lie on it, so the traversals were what it cost:
// each query walks the whole tree again.
template <bool kTwo>
__device__ __noinline__ void ProbeExact(const RenderProbeArgs& args, int64_t k) {
    StackStore<kQuantisedExactStack, kTraceBlock, 0> st;
    ProbeLoop<kTwo>(args, k, st, nullptr);
}

template <bool kTwo>
__device__ __forceinline__ void FinishProbe(const RenderProbeArgs& args, int64_t k, const SurfaceList& list) {
    if (list.open) {
        ProbeExact<kTwo>(args, k);
        return;
    }
    const AccelParams& a = args.accel;
    const int4 target = args.targets[k];
    const float4 ra = Ld(args.rays + 2 * k), rb = Ld(args.rays + 2 * k + 1);
    const float t_min = ra.w, t_max = rb.w;
    int32_t count = 0;
    int32_t selected = -1;
    int32_t at = -1;
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            if (count == 0) break;
            const float u = args.selection[2 * k].w;
            selected = min(max(static_cast<int32_t>(u * static_cast<float>(count)), 0), count - 1);
        }
        int32_t seen = 0;
        float cursor = t_min;
        for (int j = 0; j < list.n; ++j) {
            const float t = list.t[j * kTraceBlock];
            if (!(t > cursor)) continue;
            const bool inst_ok = !kTwo || target.y < 0 ||
                                 __float_as_int(Ld(&a.records[list.inst[j * kTraceBlock]].v0).w) == target.y;
            const int32_t prim = __float_as_int(Ld(&a.records[list.rec[j * kTraceBlock]].v2).w);
            if (target.x >= 0 && prim == target.x && inst_ok) {
                if (pass == 1 && seen == selected) {
                    at = j;
                    break;
                }
                ++seen;
            }
            float next = __fadd_rn(t, __fmul_rn(1.0e-4f, __fadd_rn(1.0f, fabsf(t))));
            if (!(next > cursor)) next = __fadd_rn(cursor, 1.0e-4f);
            cursor = next;
            if (cursor >= t_max) break;
        }
        if (pass == 0) count = seen;
    }
    args.hits[k] = count;
    float4 chosen = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (at >= 0) {
        // The chosen surface intersected again for its u, v (the same bits).
        float o[3] = {ra.x, ra.y, ra.z}, d[3] = {rb.x, rb.y, rb.z};
        if (kTwo) ToObject(a, __float_as_int(Ld(&a.records[list.inst[at * kTraceBlock]].v0).w), o, d);
        const Record& r = a.records[list.rec[at * kTraceBlock]];
        const float4 v0 = Ld(&r.v0);
        float t = 0.0f, u = 0.0f, v = 0.0f;
        TriangleIntersect(o, d, v0, Ld(&r.v1), Ld(&r.v2), t_min, t_max, t, u, v);
        chosen = make_float4(t, v0.w, u, v);
    }
    args.hit[k] = chosen;
}

template <bool kTwo>
__global__ void __launch_bounds__(kTraceBlock, 7) QRenderProbeKernel(const __grid_constant__ RenderProbeArgs args) {
    __shared__ int2 s_stack[kShadowShortStack * kTraceBlock];
    __shared__ float s_t[SurfaceList::kMax * kTraceBlock];
    __shared__ int32_t s_rec[SurfaceList::kMax * kTraceBlock];
    __shared__ int32_t s_inst[kTwo ? SurfaceList::kMax * kTraceBlock : 1];
    int2* col = s_stack + threadIdx.x;
    StackStore<kQuantisedStack, kTraceBlock, kShadowShortStack> st;
    QTraversal q;
    q.cur_inst = -1;
    SurfaceList list{s_t + threadIdx.x, s_rec + threadIdx.x, kTwo ? s_inst + threadIdx.x : nullptr, 0, false};
    const unsigned lane = threadIdx.x & 31u;
    const int64_t count = static_cast<int64_t>(*args.count_ptr);
    // Probes are dealt out by grid stride: a warp takes 32 at a time and
    // traces them to the end (they are alike: short segments at a surface).
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t base = blockIdx.x * static_cast<int64_t>(blockDim.x) + (threadIdx.x & ~31u); base < count;
         base += stride) {
        const int64_t k = base + lane;
        list.n = 0;
        list.open = false;
        bool alive = k < count && QBegin<kTwo, false>(args.accel, args.rays, k, q);
        while (QVoteStep<kQCollect, kTwo, 16>(args.accel, alive, q, st, col, args.error, nullptr, nullptr, &list,
                                              [](float, int32_t, float, float) {}, [] {})) {
        }
        if (k < count) FinishProbe<kTwo>(args, k, list);
        __syncwarp();
    }
}

template <bool kAny, bool kTwo, int kStepsPerRefill, int kMinBlocks, int kLeafBatch>
cudaError_t LaunchQOne(const TraceArgs& args, cudaStream_t stream, int sm_count) {
    auto kernel = QTraceKernel<kAny, kTwo, kTraceBlock, kStepsPerRefill, kMinBlocks, kLeafBatch>;
    int64_t blocks = 0;
    const cudaError_t err = PersistentGrid(kernel, kTraceBlock, args.count, sm_count, blocks);
    if (err != cudaSuccess) return err;
    kernel<<<static_cast<unsigned>(blocks), kTraceBlock, 0, stream>>>(args);
    if (!kAny) {
        const int64_t most = std::min<int64_t>(2 * static_cast<int64_t>(sm_count), (args.count + kTraceBlock - 1) / kTraceBlock);
        RetraceKernel<kTwo><<<static_cast<unsigned>(most), kTraceBlock, 0, stream>>>(args);
    }
    return cudaGetLastError();
}

// Blocks of 128 throughout. Flat: 64 registers (8 blocks per SM) and leaf batch
// 8 with a refill every 8 steps, every 4 for any hit, whose rays end sooner
// (2M triangles, 8M incoherent rays: 1.90 ms; 2.04 at 80 registers, 2.02 at 56,
// 2.05 with batch 16; 1.5M shadow rays, 400K triangles: 0.235 ms, 0.248 with a
// refill every 8). Two-level: 72 registers and leaf batch 16, since a leaf there
// may enter an instance (0.68 ms against 0.84 with 64 and 8, which spills; any
// hit 0.56 against 0.68). The launch shapes 9 and 12 ask for leaf batch 16.
template <bool kAny, bool kTwo>
cudaError_t LaunchQShape(const TraceArgs& args, int shape, cudaStream_t stream, int sm_count) {
    if constexpr (kTwo) {
        return LaunchQOne<kAny, true, 8, 7, 16>(args, stream, sm_count);
    } else {
        if (shape == 9 || shape == 12) return LaunchQOne<kAny, false, 8, 8, 16>(args, stream, sm_count);
        return LaunchQOne<kAny, false, kAny ? 4 : 8, 8, kAny ? 8 : 10>(args, stream, sm_count);
    }
}

template <bool kTwo, int kMinBlocks, int kLeafBatch>
cudaError_t LaunchQShadowOne(const ShadowArgs& args, cudaStream_t stream, int sm_count) {
    auto kernel = QShadowKernel<kTwo, kMinBlocks, kLeafBatch>;
    int64_t blocks = 0;
    const cudaError_t err = PersistentGrid(kernel, kTraceBlock, args.capacity, sm_count, blocks);
    if (err != cudaSuccess) return err;
    kernel<<<static_cast<unsigned>(blocks), kTraceBlock, 0, stream>>>(args);
    return cudaGetLastError();
}

template <bool kTwo>
cudaError_t LaunchQRenderProbeOne(const RenderProbeArgs& args, cudaStream_t stream, int sm_count) {
    auto kernel = QRenderProbeKernel<kTwo>;
    int64_t blocks = 0;
    const cudaError_t err = PersistentGrid(kernel, kTraceBlock, args.capacity, sm_count, blocks);
    if (err != cudaSuccess) return err;
    kernel<<<static_cast<unsigned>(blocks), kTraceBlock, 0, stream>>>(args);
    return cudaGetLastError();
}

}  // namespace

cudaError_t LaunchQShadow(const ShadowArgs& args, cudaStream_t stream, int sm_count) {
    return args.accel.two_level ? LaunchQShadowOne<true, 7, 16>(args, stream, sm_count)
                                : LaunchQShadowOne<false, 8, 8>(args, stream, sm_count);
}

cudaError_t LaunchQRenderProbe(const RenderProbeArgs& args, cudaStream_t stream, int sm_count) {
    return args.accel.two_level ? LaunchQRenderProbeOne<true>(args, stream, sm_count)
                                : LaunchQRenderProbeOne<false>(args, stream, sm_count);
}

cudaError_t LaunchQTrace(const TraceArgs& args, bool any_hit, int shape, cudaStream_t stream, int sm_count) {
    const bool two = args.accel.two_level != 0;
    if (any_hit) return two ? LaunchQShape<true, true>(args, shape, stream, sm_count)
                            : LaunchQShape<true, false>(args, shape, stream, sm_count);
    return two ? LaunchQShape<false, true>(args, shape, stream, sm_count)
               : LaunchQShape<false, false>(args, shape, stream, sm_count);
}

}  // namespace yrc
