// Traversal of the quantised hierarchy (QNode, device_layout.cuh): the
// closest- and any-hit core of the triangle-only BVHs, with the exact
// traversal's hits (traversal.cuh).
//
// Why the hits are the same bits. The exact traversal visits a leaf when the
// leaf's box and every ancestor's box pass their slab tests and the leaf's
// entry is not beyond the nearest t when it is taken. Boxes are nested
// (checked at creation) and the slab test's rounding is monotone, so the
// ancestors pass whenever the leaf's box passes; the visit is decided by the
// leaf's own box against the nearest t of that moment. Here:
//  * a quantised box test is conservative: its entry is at most, and its exit
//    at least, what the exact slab test computes in floats (the bound stands
//    at SetUp), so no leaf that the exact traversal visits is lost;
//  * a leaf that accepts a triangle has its own exact box tested with the
//    exact slab test and the nearest t from before the leaf, and what it
//    accepted is dropped when that fails, so no other leaf counts.
// The order in which leaves are taken differs (a node holds the boxes one to
// three levels down, nearest entry first). It decides the closest hit only
// where rounding puts a hit's t before its own leaf's entry: a surface between
// the two, visited first, makes the exact traversal skip that leaf. So
// triangles are tested up to the horizon max(t, entry) of the nearest hit and
// boxes a little further (BoxLimit), and a ray that meets a second surface
// there is traced again by the exact traversal. Without one the result is the
// smallest t, an equal t going to the smaller index; between instances, where
// it goes to the one visited first, the exact order is worked out
// (VisitedBefore). From beyond 256 extents away t is so coarse against the
// triangles that this would be common and BoxLimit too tight: such a ray is
// left to the exact traversal at once.
//
// What bounds it: dependent node fetches and the issue slots of divergent
// lanes. Four children per fetch halve the fetches of a ray; a node is 64
// bytes and two loads (the exact pair of two children is 64 bytes and four
// loads, its four-wide form 128 and seven), and a box test is 6 byte permutes
// (which pick the near and far plane by the ray's sign and turn 16 bits into
// a float), 6 fused multiply-adds and 4 min / max.
#pragma once

#include "traversal.cuh"

namespace yrc {
namespace {

struct QTraversal {
    float o[3], d[3];               // current ray (object space inside a BLAS)
    float s[3], bn[3], bf[3];       // plane q -> t: q * s + bn (near), q * s + bf (far)
    uint32_t sel[3];                // byte selector of the near plane
    float tmin;
    float t;                        // nearest hit (its u, v are written out when it is found)
    float h;                        // its horizon: max(t, its leaf's entry)
    int32_t id;                     // flat triangle index, -1 none, -2 - index: Undecided
    int32_t inst;                   // TLAS record of the hit's instance (two-level), -1 none
    int32_t cur, sp;                // node (>= 0) or leaf (~first record); stack pointer
    int32_t level, blas_base, tl_resume;  // two-level, as Traversal
    int32_t cur_inst;               // TLAS record of the instance being traversed
    float wo[3], wd[3];
    bool saw;
};

__device__ __forceinline__ float Max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float Min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The 16 bits of `w` that `sel` picks as the float 2^23 + q.
__device__ __forceinline__ float Plane(uint32_t w, uint32_t sel) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, sel));
}

constexpr uint32_t kSelLow = 0x7610u, kSelHigh = 0x7632u, kSelFlip = kSelLow ^ kSelHigh;

// The ray against a grid (origin glo, cell size). A plane q lies at
// t = (2^23 + q) * s + b with s = cell / d and b = (glo - o) / d - 2^23 s.
// Against the slab test's float value of any plane that q's cell holds, the
// rounding of this form is below 0.52 s + 6 * 2^-24 |(glo - o) / d|: half a
// cell from rounding b at 2^23 cells, the rest relative. The planes are
// stored one cell outwards, and the near / far offsets are moved apart by
// 10 * 2^-24 of the second term, so the test is conservative for any origin.
// A component too small for s (or zero) is taken at |s| = 1e30, where a plane
// more than half a cell away is beyond every t the other components can
// give (|d| >= 1e-10 there); rays outside these ranges get NaN offsets,
// which max / min ignore: the axis does not constrain.
__device__ __forceinline__ void SetUp(QTraversal& q, float gx, float gy, float gz, float cell) {
    const float g[3] = {gx, gy, gz};
    const float dm = fmaxf(fabsf(q.d[0]), fmaxf(fabsf(q.d[1]), fabsf(q.d[2])));
    const bool ray_ok = dm >= 1.0e-10f && dm <= 1.0e10f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float inv = __frcp_rn(q.d[a]);
        const uint32_t sign = __float_as_uint(inv) & 0x80000000u;
        q.sel[a] = sign ? kSelHigh : kSelLow;
        float s = __fmul_rn(cell, inv);
        float b0 = __fmul_rn(__fsub_rn(g[a], q.o[a]), inv);
        if (!(fabsf(s) <= 1.0e30f)) {
            s = __uint_as_float(__float_as_uint(1.0e30f) | sign);
            b0 = __fmul_rn(__fdiv_rn(__fsub_rn(g[a], q.o[a]), cell), s);
        }
        const float e = __fmul_rn(fabsf(b0), 6.0e-7f);
        const bool ok = ray_ok && fabsf(s) >= 1.0e-30f && fabsf(b0) <= 1.0e37f;
        const float nan = __int_as_float(0x7fffffff);
        q.s[a] = ok ? s : 0.0f;
        q.bn[a] = ok ? __fmaf_rn(-8388608.0f, s, __fsub_rn(b0, e)) : nan;
        q.bf[a] = ok ? __fmaf_rn(-8388608.0f, s, __fadd_rn(b0, e)) : nan;
    }
}

__device__ __forceinline__ void RestoreWorldRay(const AccelParams& a, QTraversal& q) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        q.o[k] = q.wo[k];
        q.d[k] = q.wd[k];
    }
    SetUp(q, a.qlo[0], a.qlo[1], a.qlo[2], a.qcell);
}

// As Begin of the exact traversal, with its root box test.
template <bool kTwo, bool kClosest>
__device__ __forceinline__ bool QBeginRay(const AccelParams& a, const float o[3], const float d[3], float tmin,
                                          float tmax, QTraversal& q) {
    RayPre r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.o[k] = q.o[k] = o[k];
        r.d[k] = q.d[k] = d[k];
        if (kTwo) {
            q.wo[k] = o[k];
            q.wd[k] = d[k];
        }
    }
    Precompute(r);
    q.tmin = tmin;
    q.t = q.h = tmax;
    q.id = -1;
    q.inst = -1;
    q.sp = 0;
    q.level = 0;
    q.tl_resume = -1;
    q.saw = false;
    if (a.root_ref == kAbsentRef) return false;
    float entry;
    if (!SlabTest(r, a.root_lo[0], a.root_lo[1], a.root_lo[2], a.root_hi[0], a.root_hi[1], a.root_hi[2], tmin, tmax,
                  entry)) {
        return false;
    }
    SetUp(q, a.qlo[0], a.qlo[1], a.qlo[2], a.qcell);
    q.cur = a.root_ref;
    const float away = entry * fmaxf(fabsf(d[0]), fmaxf(fabsf(d[1]), fabsf(d[2])));
    const bool far = kClosest && away > 256.0f * 65500.0f * a.qcell;
    if (far) q.id = -2;  // Undecided
    return !far;
}

template <bool kTwo, bool kClosest>
__device__ __forceinline__ bool QBegin(const AccelParams& a, const float4* rays, int64_t i, QTraversal& q) {
    const float4 ra = Ld(rays + 2 * i), rb = Ld(rays + 2 * i + 1);
    const float o[3] = {ra.x, ra.y, ra.z}, d[3] = {rb.x, rb.y, rb.z};
    return QBeginRay<kTwo, kClosest>(a, o, d, ra.w, rb.w, q);
}

// Stack and sort key of a child: its entry's bits with the child's number in
// the last two. Signed order is the floats' order for entries >= 0; negative
// ones (a negative t_min) come first. An entry is culled when its key is above
// the nearest t's: never for a smaller entry, nor for a negative one.
__device__ __forceinline__ int32_t EntryKey(float entry, int c) { return (__float_as_int(entry) & ~3) | c; }
__device__ __forceinline__ int32_t CullKey(float t) { return __float_as_int(fmaxf(t, 0.0f)) | 3; }
// Boxes are taken a hundred thousandth beyond the nearest t: a triangle's t lies before
// its box's entry by the rounding of its own intersection, about 2^-23 over the
// cosine of incidence.
__device__ __forceinline__ float BoxLimit(float t) { return __fmaf_rn(fabsf(t), 1.0e-5f, t); }
// A ray whose closest hit the visiting order may decide, until a nearer hit.
__device__ __forceinline__ bool Undecided(const QTraversal& q) { return q.id < -1; }
constexpr int32_t kMissKey = 0x7fffffff;

// Pop of the exact traversal. A hit inside a BLAS is only ever accepted when
// strictly nearer (TriangleAccept), so nothing is merged on leaving it.
template <bool kTwo, typename Stack>
__device__ __forceinline__ bool QPop(const AccelParams& a, QTraversal& q, Stack& st, const int2* col) {
    for (;;) {
        if (kTwo && q.level == 1 && q.sp == q.blas_base) {
            q.level = 0;
            RestoreWorldRay(a, q);
            if (q.tl_resume >= 0) {
                q.cur = ~q.tl_resume;
                return true;
            }
            continue;
        }
        if (q.sp == 0) return false;
        --q.sp;
        const int2 e = st.Get(col, q.sp);
        if (e.y > CullKey(BoxLimit(q.t))) continue;
        q.cur = e.x;
        return true;
    }
}

// A world ray in the space of an instance (TransformPoint / TransformVector by
// world_to_object; the direction is not normalised, so t stays the same).
__device__ __forceinline__ void ToObject(const AccelParams& a, int32_t inst, float o[3], float d[3]) {
    const float4* ip = reinterpret_cast<const float4*>(a.instances + inst);
    const float4 rows[3] = {Ld(ip), Ld(ip + 1), Ld(ip + 2)};
    const float wo[3] = {o[0], o[1], o[2]}, wd[3] = {d[0], d[1], d[2]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 m = rows[k];
        o[k] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m.x, wo[0]), __fmul_rn(m.y, wo[1])), __fmul_rn(m.z, wo[2])),
                         m.w);
        d[k] = __fadd_rn(__fadd_rn(__fmul_rn(m.x, wd[0]), __fmul_rn(m.y, wd[1])), __fmul_rn(m.z, wd[2]));
    }
}

// The exact slab test of a leaf's own box over [tmin, limit].
__device__ __forceinline__ bool LeafBoxPasses(const AccelParams& a, const QTraversal& q, int32_t first, float limit,
                                              float& entry) {
    const float4 x = Ld(a.leaf_boxes + 2 * static_cast<int64_t>(first));
    const float4 y = Ld(a.leaf_boxes + 2 * static_cast<int64_t>(first) + 1);
    RayPre r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.o[k] = q.o[k];
        r.d[k] = q.d[k];
    }
    Precompute(r);
    return SlabTestInterval(r, x.x, x.y, x.z, x.w, y.x, y.y, q.tmin, limit, entry);
}

__device__ __forceinline__ void LoadQNode(const QNode* p, uint32_t w[16]) {
    const unsigned long long pol = NodePolicy();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t* v = w + 8 * h;
        asm volatile("ld.global.nc.L2::cache_hint.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "l"(p->w + 8 * h), "l"(pol));
    }
}

// Whether the exact traversal comes to TLAS record ra before rb on this ray:
// the two part at one pair, whose nearer child it takes first (the left one
// on a tie), and the records of a leaf go in order. Records are numbered
// left subtree first.
__device__ __forceinline__ bool VisitedBefore(const AccelParams& a, const QTraversal& q, int32_t ra, int32_t rb) {
    RayPre r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.o[k] = q.wo[k];
        r.d[k] = q.wd[k];
    }
    Precompute(r);
    int32_t cur = a.root_ref;
    while (cur >= 0) {
        const float4* p = reinterpret_cast<const float4*>(a.pairs + cur);
        const float4 pa = Ld(p), pb = Ld(p + 1), pc = Ld(p + 2);
        const int4 pd = __ldg(reinterpret_cast<const int4*>(p + 3));
        const bool a_right = ra >= pd.z, b_right = rb >= pd.z;
        if (a_right != b_right) {
            const float inf = __int_as_float(0x7f800000);
            float le, re;
            SlabTestInterval(r, pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, q.tmin, inf, le);
            SlabTestInterval(r, pb.z, pb.w, pc.x, pc.y, pc.z, pc.w, q.tmin, inf, re);
            return (le <= re) != a_right;
        }
        cur = a_right ? pd.y : pd.x;
    }
    return ra < rb;
}

enum QMode { kQClosest, kQAny, kQFilter, kQCollect };

// The nearest kMax surfaces on a ray as (t, record, instance), ordered by t and
// then triangle index, in the block's shared memory laid out
// [entry][thread].
struct SurfaceList {
    static constexpr int kMax = 12;
    float* t;       // the lane's column, stride kTraceBlock
    int32_t* rec;
    int32_t* inst;  // two-level only
    int n;
    bool open;      // a farther surface did not fit, or two instances tie

    __device__ __forceinline__ void Add(const AccelParams& a, float tv, int32_t rv, int32_t iv) {
        const int32_t id = __float_as_int(Ld(&a.records[rv].v0).w);
        int j = n;
        while (j > 0) {
            const float tp = t[(j - 1) * kTraceBlock];
            const int32_t rp = rec[(j - 1) * kTraceBlock];
            const int32_t ip = inst ? inst[(j - 1) * kTraceBlock] : 0;
            if (tp < tv) break;
            if (tp == tv) {
                if (inst && ip != iv) open = true;
                if (__float_as_int(Ld(&a.records[rp].v0).w) < id) break;
            }
            if (j < kMax) {
                t[j * kTraceBlock] = tp;
                rec[j * kTraceBlock] = rp;
                if (inst) inst[j * kTraceBlock] = ip;
            } else {
                open = true;
            }
            --j;
        }
        if (j < kMax) {
            t[j * kTraceBlock] = tv;
            rec[j * kTraceBlock] = rv;
            if (inst) inst[j * kTraceBlock] = iv;
        } else {
            open = true;
        }
        if (n < kMax) ++n;
    }
};

// What a lane's ray does next after a step.
enum QNext { kQGoOn, kQPopNext, kQDone };

// A step at an interior node.
template <typename Stack>
__device__ __forceinline__ QNext QNodeStep(const AccelParams& a, QTraversal& q, Stack& st, int2* col, int* error) {
    uint32_t w[16];
    LoadQNode(a.qnodes + q.cur, w);
    const float limit = BoxLimit(q.t);
    const uint32_t fx = q.sel[0] ^ kSelFlip, fy = q.sel[1] ^ kSelFlip, fz = q.sel[2] ^ kSelFlip;
    int32_t k[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t* b = w + 8 * (c / 2) + 3 * (c & 1);
        const float e = Max3(__fmaf_rn(Plane(b[0], q.sel[0]), q.s[0], q.bn[0]),
                             __fmaf_rn(Plane(b[1], q.sel[1]), q.s[1], q.bn[1]),
                             fmaxf(__fmaf_rn(Plane(b[2], q.sel[2]), q.s[2], q.bn[2]), q.tmin));
        const float x = Min3(__fmaf_rn(Plane(b[0], fx), q.s[0], q.bf[0]),
                             __fmaf_rn(Plane(b[1], fy), q.s[1], q.bf[1]),
                             fminf(__fmaf_rn(Plane(b[2], fz), q.s[2], q.bf[2]), limit));
        k[c] = e <= x ? EntryKey(e, c) : kMissKey;
    }
    auto order = [&](int i, int j) {
        const int32_t lo = min(k[i], k[j]);
        k[j] = max(k[i], k[j]);
        k[i] = lo;
    };
    order(0, 1);
    order(2, 3);
    order(0, 2);
    order(1, 3);
    order(1, 2);
    if (k[0] == kMissKey) return kQPopNext;
    auto ref = [&](int32_t key) {
        const uint32_t even = (key & 2) ? w[14] : w[6], odd = (key & 2) ? w[15] : w[7];
        return static_cast<int32_t>((key & 1) ? odd : even);
    };
    if (k[1] != kMissKey) {
        if (q.sp + 3 > Stack::kTotalEntries) {  // unreachable when the host's depth bound holds
            atomicOr(error, kTraceErrorStackOverflow);
            q.id = -1;
            return kQDone;
        }
        if (k[3] != kMissKey) st.Put(col, q.sp++, make_int2(ref(k[3]), k[3]));
        if (k[2] != kMissKey) st.Put(col, q.sp++, make_int2(ref(k[2]), k[2]));
        st.Put(col, q.sp++, make_int2(ref(k[1]), k[1]));
    }
    q.cur = ref(k[0]);
    return kQGoOn;
}

// A step at a TLAS leaf: into the next of its instances whose root box the ray
// hits. The leaf's own box is tested first, since entering an instance costs
// more than the test (records after a leaf's first have an unbounded box: a
// resumed leaf is not tested again).
__device__ __forceinline__ QNext QInstanceStep(const AccelParams& a, QTraversal& q) {
    const int32_t first = ~q.cur;
    int32_t rec = first;
    // TLAS leaf: tested before its instances, since entering one costs
    // more than the test (records after a leaf's first have an unbounded
    // box: a resumed leaf is not tested again).
    const float limit = q.id != -1 ? BoxLimit(q.t) : q.t;
    float entry;
    if (!LeafBoxPasses(a, q, first, limit, entry)) return kQPopNext;
    for (;;) {
        const float4* p = reinterpret_cast<const float4*>(a.records + rec);
        const float4 v0 = Ld(p), v1 = Ld(p + 1);
        const int32_t flags = __float_as_int(v1.w);
        if (((flags >> 1) & 7) == kRecInstance) {
            const int32_t inst = __float_as_int(v0.w);
            const float4* ip = reinterpret_cast<const float4*>(a.instances + inst);
            const float4 ba = Ld(ip + 3), bb = Ld(ip + 4);
            RayPre obj;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                obj.o[k] = q.o[k];
                obj.d[k] = q.d[k];
            }
            ToObject(a, inst, obj.o, obj.d);
            Precompute(obj);
            const int32_t root = __float_as_int(bb.z);
            if (root != kAbsentRef &&
                SlabTestInterval(obj, ba.x, ba.y, ba.z, ba.w, bb.x, bb.y, q.tmin, limit, entry)) {
                const float4 grid = Ld(ip + 5);
                q.level = 1;
                q.blas_base = q.sp;
                q.cur_inst = rec;
                q.tl_resume = (flags & kRecLast) ? -1 : rec + 1;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    q.o[k] = obj.o[k];
                    q.d[k] = obj.d[k];
                }
                SetUp(q, grid.x, grid.y, grid.z, grid.w);
                q.cur = root;
                return kQGoOn;
            }
        }
        if (flags & kRecLast) break;
        ++rec;
    }
    return kQPopNext;
}

// A step at a triangle leaf: the closest or any hit, any hit on a surface that
// does not pass light (the others go to `clear`), or every surface on the
// segment (to `list`). A nearer closest hit is handed to `keep`.
template <QMode kMode, bool kTwo, typename Keep>
__device__ __forceinline__ QNext QLeafStep(const AccelParams& a, QTraversal& q, const uint8_t* tri_clear,
                                           ClearHits* clear, SurfaceList* list, Keep keep) {
    constexpr bool kAny = kMode == kQAny || kMode == kQFilter;
    constexpr bool kFilter = kMode == kQFilter;
    const int32_t first = ~q.cur;
    int32_t rec = first;
    // Triangle leaf: accepted candidates are kept aside until the leaf's
    // exact box has passed.
    float bt = q.t, bu = 0.0f, bv = 0.0f;
    // The leaf's candidate: its index, -1 none, kNear: only a surface within the
    // horizon of the nearest hit (closest).
    constexpr int32_t kNear = -2;
    int32_t bid = -1;
    bool box_ok = false;  // the box was tested already (it passed)
    float entry;
    for (;;) {
        const float4* p = reinterpret_cast<const float4*>(a.records + rec);
        const float4 v0 = Ld(p), v1 = Ld(p + 1), v2 = Ld(p + 2);
        const int32_t flags = __float_as_int(v1.w);
        float t, u, v;
        if (((flags >> 1) & 7) == kRecTriangle &&
            TriangleIntersect(q.o, q.d, v0, v1, v2, q.tmin,
                              kMode == kQClosest && bid < 0 ? q.h : bt, t, u, v)) {
            if (kMode == kQCollect) {
                if (!box_ok && !LeafBoxPasses(a, q, first, q.t, entry)) break;
                box_ok = true;
                list->Add(a, t, rec, q.cur_inst);
            } else {
                const int32_t id = __float_as_int(v0.w);
                // An equal t goes to the smaller index; two-level, that holds
                // inside an instance, whose hit counts only if it is strictly
                // nearer than those of the instances visited before it.
                const int32_t nid = bid >= 0 ? bid : q.id;  // an undecided ray's order no longer matters
                bool take = kTwo ? t < bt : !(t > bt) && !(t == bt && nid >= 0 && id >= nid);
                if (kTwo && !kAny && t == bt && nid >= 0) {
                    take = bid >= 0 || q.inst == q.cur_inst ? id < nid : VisitedBefore(a, q, q.cur_inst, q.inst);
                }
                if (take) {
                    if (kFilter && tri_clear[id]) {
                        if (!box_ok) {
                            if (!LeafBoxPasses(a, q, first, q.t, entry)) break;
                            box_ok = true;
                        }
                        q.saw = true;
                        clear->Add(t, id);
                    } else {
                        bt = t, bu = u, bv = v, bid = id;
                        if (kAny) break;
                    }
                } else if (kMode == kQClosest && bid < 0 && t < q.h) {
                    bid = kNear;
                }
            }
        }
        if (flags & kRecLast) break;
        ++rec;
    }
    if (kMode == kQClosest) {
        const bool had = q.id != -1;
        if (bid != -1 && LeafBoxPasses(a, q, first, had ? __int_as_float(0x7f800000) : q.t, entry)) {
            bool undecided = true;
            if (bid >= 0) {
                undecided = had && q.t < entry;
                q.t = bt;
                q.h = fmaxf(bt, entry);
                q.id = bid;
                if (kTwo) q.inst = q.cur_inst;
                keep(bt, bid, bu, bv);
            }
            if (undecided && q.id >= 0) q.id = -2 - q.id;
        }
    } else if (bid >= 0 && (box_ok || LeafBoxPasses(a, q, first, q.t, entry))) {
        q.id = bid;
        return kQDone;
    }
    return kQPopNext;
}

// One vote and step of the whole warp (every lane calls it; `alive` lanes hold
// a ray). Lanes at interior nodes always step; those at leaves wait, their
// rays' state unchanged, until kBatch lanes are at one or no lane is at a
// node, so that the long branches run for many lanes. Each branch pops for
// itself: popping together after the branches measured 6-18 % slower (2M
// triangles, incoherent 2.01 ms against 1.90, two-level 0.81 against 0.68),
// since the branches' lanes then wait for each other's loads. Returns false
// when no lane holds a ray; `keep` and `done` are called for a new closest hit and is called for a ray that has ended.
template <QMode kMode, bool kTwo, int kBatch, typename Stack, typename Keep, typename Done>
__device__ __forceinline__ bool QVoteStep(const AccelParams& a, bool& alive, QTraversal& q, Stack& st, int2* col,
                                          int* error, const uint8_t* tri_clear, ClearHits* clear, SurfaceList* list,
                                          Keep keep, Done done) {
    const unsigned leaves = __ballot_sync(kFull, alive && q.cur < 0);
    const unsigned nodes = __ballot_sync(kFull, alive && q.cur >= 0);
    if (!(leaves | nodes)) return false;
    const bool run_leaves = nodes == 0u || __popc(leaves) >= kBatch;
    if (alive && (q.cur >= 0 || run_leaves)) {
        if (q.cur >= 0) {
            const QNext next = QNodeStep(a, q, st, col, error);
            if (next != kQGoOn) alive = next == kQPopNext && QPop<kTwo>(a, q, st, col);
        } else if (kTwo && q.level == 0) {
            if (QInstanceStep(a, q) != kQGoOn) alive = QPop<kTwo>(a, q, st, col);
        } else {
            alive = QLeafStep<kMode, kTwo>(a, q, tri_clear, clear, list, keep) == kQPopNext && QPop<kTwo>(a, q, st, col);
        }
        if (!alive) done();
    }
    return true;
}

}  // namespace
}  // namespace yrc
