// Quantised copy of a BVH's node pairs (QNode, device_layout.cuh) and the exact
// boxes of its leaves, for the traversal in quantised.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "quantise.hpp"

namespace yrc {
namespace {

constexpr int kBlock = 256;
constexpr int kMaxCell = 65535;

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ Box ChildBox(const NodePair& p, int side) {
    return side == 0 ? Box{{p.a.x, p.a.y, p.a.z}, {p.a.w, p.b.x, p.b.y}}
                     : Box{{p.b.z, p.b.w, p.c.x}, {p.c.y, p.c.z, p.c.w}};
}

__device__ __forceinline__ double Area(double x, double y, double z) { return x * y + y * z + z * x; }

__global__ void FillBoxesKernel(float4* boxes, int64_t records) {
    const float inf = __int_as_float(0x7f800000);
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < records;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        boxes[2 * i] = make_float4(-inf, -inf, -inf, inf);
        boxes[2 * i + 1] = make_float4(inf, inf, 0.0f, 0.0f);
    }
}

// Cells of box b in the range's grid, one cell outwards; false when it is not
// a box or leaves the grid.
__device__ __forceinline__ bool Cells(const Box& b, const QRange& r, uint32_t w[3], double ext[3], double qext[3]) {
    bool ok = true;
    for (int a = 0; a < 3; ++a) {
        const double l = floor((static_cast<double>(b.lo[a]) - r.lo[a]) / r.cell) - 1.0;
        const double h = ceil((static_cast<double>(b.hi[a]) - r.lo[a]) / r.cell) + 1.0;
        const bool in = b.lo[a] <= b.hi[a] && l >= 0.0 && h <= static_cast<double>(kMaxCell);
        ok = ok && in;
        w[a] = in ? static_cast<uint32_t>(l) | (static_cast<uint32_t>(h) << 16) : 0u;
        ext[a] = static_cast<double>(b.hi[a]) - b.lo[a];
        qext[a] = (h - l) * r.cell;
    }
    return ok;
}

// One thread per pair: the four-wide node that starts there (nodes at the
// depths in between are written too and never referred to: no numbering pass)
// and the exact boxes of the pair's leaf children. Both interior children are
// replaced by theirs; where only one child is interior, so is the larger
// interior one of that child's children. So a step from a node to a child
// that is a node again goes down at least two levels and leaves at most
// three entries on the stack (QuantisedStack). Sets status when a box is
// not a valid one, does not hold the boxes below it (the traversal relies on
// nesting) or leaves the grid; sums the areas before and after. Bound by the
// 64-byte pair reads, mostly in cache after the first; once per scene.
__global__ void __launch_bounds__(kBlock) QuantiseKernel(const NodePair* pairs, int64_t count, const QRange* ranges,
                                                         int32_t range_count, int32_t absent_ref, QNode* out,
                                                         float4* boxes, int* status, double* areas) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    double exact = 0.0, coarse = 0.0;
    if (i < count) {
        int lo = 0, hi = range_count - 1;  // the last range that begins at or before i
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (ranges[m].begin <= i) lo = m;
            else hi = m - 1;
        }
        const QRange r = ranges[lo];
        const double root = Area(static_cast<double>(r.root_hi[0]) - r.root_lo[0],
                                 static_cast<double>(r.root_hi[1]) - r.root_lo[1],
                                 static_cast<double>(r.root_hi[2]) - r.root_lo[2]);
        const NodePair p = pairs[i];
        Box e[4];
        int32_t ref[4];
        int n = 0;
        bool ok = true;
        // Entry k replaced by its children; false when they are not inside.
        auto expand = [&](int k) {
            const NodePair c = pairs[ref[k]];
            const Box b = e[k];
            bool first = true;
            for (int side = 0; side < 2; ++side) {
                const int32_t cref = side == 0 ? c.d.x : c.d.y;
                if (cref == kAbsentRef) continue;
                const int at = first ? k : n++;
                first = false;
                e[at] = ChildBox(c, side);
                ref[at] = cref;
                for (int a = 0; a < 3; ++a) ok = ok && e[at].lo[a] >= b.lo[a] && e[at].hi[a] <= b.hi[a];
            }
            ok = ok && !first;  // a childless interior node: the exact nodes
        };
        for (int side = 0; side < 2; ++side) {
            const int32_t cref = side == 0 ? p.d.x : p.d.y;
            if (cref == kAbsentRef) continue;
            e[n] = ChildBox(p, side);
            ref[n] = cref;
            uint32_t w[3];
            double ext[3], qext[3];
            ok = Cells(e[n], r, w, ext, qext) && ok;
            // As a share of the root box's area, which is what the SAH
            // counts visits by (the ranges have spaces of their own).
            if (root > 0.0) {
                exact += Area(ext[0], ext[1], ext[2]) / root;
                coarse += Area(qext[0], qext[1], qext[2]) / root;
            }
            if (cref < 0) {
                float4* o = boxes + 2 * static_cast<int64_t>(~cref);
                o[0] = make_float4(e[n].lo[0], e[n].lo[1], e[n].lo[2], e[n].hi[0]);
                o[1] = make_float4(e[n].hi[1], e[n].hi[2], 0.0f, 0.0f);
            }
            ++n;
        }
        const int children = n;
        for (int k = 0; k < children; ++k) {
            if (ref[k] >= 0) expand(k);
        }
        if (n == 3) {
            int best = -1;
            double most = -1.0;
            for (int k = 0; k < 3; ++k) {
                const double area = Area(static_cast<double>(e[k].hi[0]) - e[k].lo[0],
                                         static_cast<double>(e[k].hi[1]) - e[k].lo[1],
                                         static_cast<double>(e[k].hi[2]) - e[k].lo[2]);
                if (ref[k] >= 0 && area > most) {
                    most = area;
                    best = k;
                }
            }
            if (best >= 0) expand(best);
        }
        QNode q;
        for (int c = 0; c < 4; ++c) {
            uint32_t* w = q.w + 8 * (c / 2) + 3 * (c & 1);
            uint32_t* wr = q.w + 8 * (c / 2) + 6 + (c & 1);
            w[0] = w[1] = w[2] = static_cast<uint32_t>(kMaxCell);  // lo > hi
            *wr = static_cast<uint32_t>(absent_ref);
            if (c >= n) continue;
            double ext[3], qext[3];
            ok = Cells(e[c], r, w, ext, qext) && ok;
            *wr = static_cast<uint32_t>(ref[c]);
        }
        if (!ok) atomicOr(status, 1);
        out[i] = q;
    }
    for (int o = 16; o > 0; o >>= 1) {
        exact += __shfl_xor_sync(0xffffffffu, exact, o);
        coarse += __shfl_xor_sync(0xffffffffu, coarse, o);
    }
    if ((threadIdx.x & 31) == 0 && coarse > 0.0) {
        atomicAdd(areas, exact);
        atomicAdd(areas + 1, coarse);
    }
}

// The leaf box of a BVH that is a single leaf.
__global__ void RootLeafKernel(const QRange* ranges, int32_t range_count, float4* boxes) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= range_count || ranges[k].root_ref >= 0 || ranges[k].root_ref == kAbsentRef) return;
    const QRange& r = ranges[k];
    float4* o = boxes + 2 * static_cast<int64_t>(~r.root_ref);
    o[0] = make_float4(r.root_lo[0], r.root_lo[1], r.root_lo[2], r.root_hi[0]);
    o[1] = make_float4(r.root_hi[1], r.root_hi[2], 0.0f, 0.0f);
}

}  // namespace

// One cell size for all three axes: a flat box then has cells of its own size
// across, and a ray's origin is never many more cells away on one axis than
// the scene's largest extent explains. Eight cells are left free at the low
// end and about twenty at the high end.
bool MakeQRange(int64_t begin, int32_t root_ref, const float lo[3], const float hi[3], QRange& r) {
    r.begin = begin;
    r.root_ref = root_ref;
    float extent = 0.0f;
    for (int a = 0; a < 3; ++a) {
        if (!(lo[a] <= hi[a]) || !(std::fabs(lo[a]) <= 1.0e18f) || !(std::fabs(hi[a]) <= 1.0e18f)) return false;
        extent = std::max(extent, hi[a] - lo[a]);
        r.root_lo[a] = lo[a];
        r.root_hi[a] = hi[a];
    }
    if (!(extent >= 1.0e-10f)) return false;
    r.cell = extent / 65500.0f;
    for (int a = 0; a < 3; ++a) r.lo[a] = lo[a] - 8.0f * r.cell;
    return true;
}

cudaError_t Quantise(const NodePair* pairs, int64_t pair_count, int64_t record_count, int32_t absent_ref,
                     const std::vector<QRange>& ranges, QNode** qnodes, float4** leaf_boxes, int64_t* bytes,
                     bool* usable) {
    *qnodes = nullptr;
    *leaf_boxes = nullptr;
    *usable = false;
    struct Result {
        double areas[2];
        int status, pad;
    } result{};
    const size_t nodes = static_cast<size_t>(std::max<int64_t>(pair_count, 1)) * sizeof(QNode);
    const size_t boxes = static_cast<size_t>(std::max<int64_t>(record_count, 1)) * 2 * sizeof(float4);
    const size_t table = (ranges.size() * sizeof(QRange) + 255) / 256 * 256;
    // One allocation: nodes, leaf boxes, then what only the build needs.
    char* block = nullptr;
    cudaError_t err = cudaMalloc(reinterpret_cast<void**>(&block), nodes + boxes + table + sizeof(Result));
    QRange* d_ranges = reinterpret_cast<QRange*>(block + nodes + boxes);
    char* d_out = block + nodes + boxes + table;
    *qnodes = reinterpret_cast<QNode*>(block);
    *leaf_boxes = reinterpret_cast<float4*>(block + nodes);
    if (err == cudaSuccess) {
        err = cudaMemcpy(d_ranges, ranges.data(), ranges.size() * sizeof(QRange), cudaMemcpyHostToDevice);
    }
    if (err == cudaSuccess) err = cudaMemset(d_out, 0, sizeof(Result));
    if (err == cudaSuccess) {
        const int32_t n = static_cast<int32_t>(ranges.size());
        FillBoxesKernel<<<static_cast<unsigned>(std::min<int64_t>((record_count + kBlock) / kBlock, 4096)), kBlock>>>(
            *leaf_boxes, record_count);
        if (pair_count > 0) {
            double* areas = reinterpret_cast<double*>(d_out);
            QuantiseKernel<<<static_cast<unsigned>((pair_count + kBlock - 1) / kBlock), kBlock>>>(
                pairs, pair_count, d_ranges, n, absent_ref, *qnodes, *leaf_boxes, reinterpret_cast<int*>(areas + 2),
                areas);
        }
        RootLeafKernel<<<static_cast<unsigned>((n + kBlock - 1) / kBlock), kBlock>>>(d_ranges, n, *leaf_boxes);
        err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaMemcpy(&result, d_out, sizeof(Result), cudaMemcpyDeviceToHost);
    *usable = err == cudaSuccess && result.status == 0 && result.areas[1] <= kQuantisedAreaLimit * result.areas[0];
    if (*usable) {
        *bytes += static_cast<int64_t>(nodes + boxes + table + sizeof(Result));
    } else {
        cudaFree(block);
        *qnodes = nullptr;
        *leaf_boxes = nullptr;
    }
    return err;
}

}  // namespace yrc
