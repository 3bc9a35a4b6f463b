// Quantised node copy (quantise.cu) built when an accelerator is created.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "device_layout.cuh"

namespace yrc {

// One BVH of the pair array (the flat BVH, a BLAS or the TLAS) and its grid.
struct QRange {
    int64_t begin;  // its first pair
    float lo[3];    // grid origin
    float cell;
    int32_t root_ref;
    float root_lo[3], root_hi[3];
};

// Above this ratio of the quantised boxes' summed area to the exact boxes',
// the grid is too coarse for the scene's detail and the exact nodes are kept:
// box tests pass, and leaves are visited, in proportion to the area.
constexpr double kQuantisedAreaLimit = 1.3;
constexpr int64_t kQuantisedMinPairs = 256;

// Deepest stack of the quantised traversal over a hierarchy of `depth` pair
// levels: three entries per step, each at least two levels down.
constexpr int QuantisedStack(int depth) { return 3 * ((depth + 1) / 2) + 1; }

// False when the box has no grid (not finite, empty or a point).
bool MakeQRange(int64_t begin, int32_t root_ref, const float lo[3], const float hi[3], QRange& r);

// Device arrays of the quantised nodes and leaf boxes; `usable` false (and
// null arrays) when the BVH is not one the quantised traversal may take.
// One allocation holds both, freed through `qnodes`.
// Ranges in the order of their pairs; `absent_ref` the leaf an absent child
// stands for.
cudaError_t Quantise(const NodePair* pairs, int64_t pair_count, int64_t record_count, int32_t absent_ref,
                     const std::vector<QRange>& ranges, QNode** qnodes, float4** leaf_boxes, int64_t* bytes,
                     bool* usable);

}  // namespace yrc
