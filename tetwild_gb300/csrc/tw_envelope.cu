// tw_envelope.cu -- envelope tests against the device LBVH.
//
// Decision (isPointOutEnvelop, LocalOperations.cpp:1034-1044): a point is
// out iff every facet f has sqdist(p, f) > eps2.  The traversal stops at the
// first facet with sqdist <= eps2, as facet_in_envelope_recursive does
// (mesh_AABB.cpp:482-548), and skips a child box only when its squared
// distance exceeds (eps + tau)^2 with tau = 64 * 2^-53 * max|coord|, which
// covers the rounding of both the box distance and the facet distance: no
// facet that tests <= eps2 is ever skipped, so the decision equals the
// brute-force decision over all facets.
//
// Faces (isFaceOutEnvelop_sampling, :1046-1109): first the pieces of a face
// that lie inside as a whole (tw_hull.cuh); where pieces stay open, a warp
// generates sampleTriangle's samples there (Common.cpp:143-228) with the same
// arithmetic as the reference order, tests them, the facet that held the
// previous samples first (the reference's prev_facet hint, :1080-1083), and
// stops at the first sample that is out.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_run_length_encode.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "tw_device.cuh"
#include "tw_internal.h"

namespace tw {

constexpr int kStack = 64;  // > max depth of a 30-bit LBVH with index tie-break (63)
// fine cells a side of a bin of the point test's bin index, and the 32-bit
// words of an entry's fine-cell mask
constexpr int kFine = 8;
constexpr int kFineWords = kFine * kFine * kFine / 32;

__device__ __forceinline__ double prune_threshold(const V3& p, double eps2, double scale) {
    double m = scale;
    m = fmax(m, fabs(p.x));
    m = fmax(m, fabs(p.y));
    m = fmax(m, fabs(p.z));
    double eps = sqrt(eps2);
    double tau = 64.0 * kEps * m + 4.0 * kEps * eps;
    return (eps + tau) * (eps + tau);
}

__device__ __forceinline__ double leaf_sqdist(const double* __restrict__ tri, int32_t leaf,
                                              const V3& p) {
    const double* t = tri + 9 * (int64_t)leaf;
    V3 a{__ldg(t + 0), __ldg(t + 1), __ldg(t + 2)};
    V3 b{__ldg(t + 3), __ldg(t + 4), __ldg(t + 5)};
    V3 c{__ldg(t + 6), __ldg(t + 7), __ldg(t + 8)};
    return point_tri_sqdist(p, a, b, c);
}

constexpr int32_t kTraversalError = -2;

#include "tw_envcert.cuh"

// One atomic per warp for the traversal statistics.
__device__ __forceinline__ void flush_stats(const TravStats& st, unsigned long long* counters,
                                            uint32_t queries) {
    unsigned long long a = st.facets, b = st.fp64, q = queries;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (a) atomicAdd(counters + kCntEnvFacetTests, a);
        if (b) atomicAdd(counters + kCntEnvFp64, b);
        if (q) atomicAdd(counters + kCntEnvQueries, q);
    }
}

// Returns the leaf index of a facet within eps2 of p, -1 if none, or
// kTraversalError if the walk exceeded its bounds (a tree that is not a
// tree); every internal node is visited at most once per query.
__device__ __forceinline__ int32_t find_facet_within(const BvhNode* __restrict__ nodes,
                                                     const double* __restrict__ tri, int32_t nf,
                                                     const V3& p, double eps2, double thr,
                                                     TravStats& st) {
    if (nf == 1) {
        ++st.facets;
        ++st.fp64;
        return leaf_sqdist(tri, 0, p) <= eps2 ? 0 : -1;
    }
    int32_t stack[kStack];
    int sp = 0;
    int32_t cur = 0;
    for (int32_t iter = 0; iter < nf; ++iter) {
        if ((uint32_t)cur >= (uint32_t)(nf - 1)) return kTraversalError;
        const double2* nd = reinterpret_cast<const double2*>(nodes + cur);
        double2 q0 = __ldg(nd + 0), q1 = __ldg(nd + 1), q2 = __ldg(nd + 2);
        double2 q3 = __ldg(nd + 3), q4 = __ldg(nd + 4), q5 = __ldg(nd + 5);
        int2 ch = __ldg(reinterpret_cast<const int2*>(nd + 6));
        double lo0[3] = {q0.x, q0.y, q1.x}, hi0[3] = {q1.y, q2.x, q2.y};
        double lo1[3] = {q3.x, q3.y, q4.x}, hi1[3] = {q4.y, q5.x, q5.y};
        double d0 = point_box_sqdist(p, lo0, hi0);
        double d1 = point_box_sqdist(p, lo1, hi1);
        bool h0 = d0 <= thr, h1 = d1 <= thr;
        if (h0 && ch.x < 0) {
            if ((uint32_t)(~ch.x) >= (uint32_t)nf) return kTraversalError;
            ++st.facets;
            ++st.fp64;
            if (leaf_sqdist(tri, ~ch.x, p) <= eps2) return ~ch.x;
            h0 = false;
        }
        if (h1 && ch.y < 0) {
            if ((uint32_t)(~ch.y) >= (uint32_t)nf) return kTraversalError;
            ++st.facets;
            ++st.fp64;
            if (leaf_sqdist(tri, ~ch.y, p) <= eps2) return ~ch.y;
            h1 = false;
        }
        if (h0 && h1) {
            if (sp >= kStack) return kTraversalError;
            int32_t nearc = (d0 <= d1) ? ch.x : ch.y;
            int32_t farc = (d0 <= d1) ? ch.y : ch.x;
            stack[sp++] = farc;
            cur = nearc;
        } else if (h0) {
            cur = ch.x;
        } else if (h1) {
            cur = ch.y;
        } else {
            if (sp == 0) return -1;
            cur = stack[--sp];
        }
    }
    return kTraversalError;
}

// Query i of the launch is point order[i] (order == nullptr: point i).  With
// the points in Morton order, the lanes of a warp query neighbouring points
// and walk the same nodes: the warp stays converged and the nodes it reads
// are shared in L1.
struct EnvTree {
    const BvhNode* nodes;
    const BvhNode32* nodes32;
    const FacetCull* cull;
    const double* tri;
    int32_t nf;
    double scale;
    float scale_hi;  // scale rounded up to binary32
    const int32_t* facet_id;  // input facet index of each leaf
    // the uniform grid of the certified test (gslot == nullptr: none)
    float glo[3];
    float ginv;
    int32_t gn[3];
    const uint4* gslot;   // (cell, first entry, count, -) per hash slot
    uint32_t gshift, gmask;
    const int32_t* glist;
    // the bin index of the point test (boff == nullptr: none)
    float blo[3];
    float binv;
    int32_t bn[3];
    const uint32_t* boff;   // first entry per bin (Morton index of its coordinates)
    const uint32_t* bmask;  // fine-cell mask word w of entry e at bmask[w * bnt + e]
    const int32_t* bleaf;   // leaf per entry
    int64_t bnt;            // entries
    const int32_t* bid;     // dense id per bin with entries, -1 for an empty bin
    int32_t nocc;           // bins with entries
};

template <bool FP32>
__device__ __forceinline__ int32_t query_point(const EnvTree& T, const V3& p, const EpsParams& E,
                                               TravStats& st) {
    if (FP32)
        return find_facet_within32(T.nodes32, T.cull, T.tri, T.nf, p, cert_query(p, E, T.scale_hi),
                                   E.eps2, st);
    return find_facet_within(T.nodes, T.tri, T.nf, p, E.eps2, prune_threshold(p, E.eps2, T.scale),
                             st);
}

// eps = sqrt(eps2) rounded up and down to binary32, and the scale rounded up.
static EpsParams eps_params(double eps2) {
    EpsParams E;
    E.eps2 = eps2;
    double eps = std::sqrt(eps2);
    float f = (float)eps;
    E.eps_hi = ((double)f < eps) ? std::nextafter(f, INFINITY) : f;
    E.eps_lo = ((double)f > eps) ? std::nextafter(f, 0.0f) : f;
    return E;
}
static float round_up_float(double x) {
    float f = (float)x;
    return ((double)f < x) ? std::nextafter(f, INFINITY) : f;
}
static EnvTree env_tree(const Surface& S);
// The tree with its grid when the grid was built for this eps2.
static EnvTree env_tree_for(const Surface& S, double eps2) {
    EnvTree T = env_tree(S);
    if (S.grid.eps2 != eps2) {
        T.gslot = nullptr;
        T.glist = nullptr;
        T.boff = nullptr;
        T.bmask = nullptr;
        T.bleaf = nullptr;
        T.bid = nullptr;
        T.nocc = 0;
    }
    return T;
}
static EnvTree env_tree(const Surface& S) {
    EnvTree T{S.nodes, S.nodes32, S.cull, S.tri, S.nf, S.scale, round_up_float(S.scale),
              S.facet_id};
    for (int k = 0; k < 3; ++k) {
        T.glo[k] = S.grid.lo[k];
        T.gn[k] = S.grid.n[k];
    }
    T.ginv = S.grid.inv_c;
    T.gslot = S.grid.slot;
    T.gshift = S.grid.shift;
    T.gmask = S.grid.mask;
    T.glist = S.grid.list;
    for (int k = 0; k < 3; ++k) {
        T.blo[k] = S.grid.blo[k];
        T.bn[k] = S.grid.bn[k];
    }
    T.binv = S.grid.binv;
    T.boff = S.grid.boff;
    T.bmask = S.grid.bent;
    T.bleaf = S.grid.bent ? (const int32_t*)(S.grid.bent + kFineWords * S.grid.bnt) : nullptr;
    T.bnt = S.grid.bnt;
    T.bid = S.grid.bid;
    T.nocc = S.grid.nocc;
    return T;
}

template <bool FP32, int MINB = 1>
__global__ void __launch_bounds__(128, MINB) k_env_points(const double* __restrict__ P,
                                                    const int32_t* __restrict__ order, int64_t n,
                                                    EnvTree T, EpsParams E,
                                                    uint8_t* __restrict__ out,
                                                    unsigned long long* __restrict__ counters) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    TravStats st;
    uint32_t nq = 0;
    // every lane runs the same number of iterations so the final warp
    // reduction of the statistics is converged
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t base0 = first - (threadIdx.x & 31);
    for (int64_t b = base0; b < n; b += stride) {
        const int64_t i = b + (threadIdx.x & 31);
        if (i < n) {
            const int64_t j = order ? (int64_t)__ldg(order + i) : i;
            V3 p{__ldg(P + 3 * j), __ldg(P + 3 * j + 1), __ldg(P + 3 * j + 2)};
            int32_t f = query_point<FP32>(T, p, E, st);
            if (f == kTraversalError) atomicOr(counters + kCntError, 1ULL);
            out[j] = (uint8_t)(f == -1);
            ++nq;
        }
    }
    flush_stats(st, counters, nq);
}

// ---------------------------------------------------------------------------
// Warp-shared candidates (certified mode).  With the points in Morton order
// the 32 points of a warp lie close together: the warp walks the tree once
// for the box of its points grown by the largest per-point culling radius
// (sqrt of CertQuery::thr, rounded up), collecting every leaf whose binary32
// box meets it, and each lane then tests its own point against that list.
// Every leaf that the per-point walk could reach (box within sqrt(thr) of the
// point) meets the grown box, and each leaf test is the same certified test,
// so every decision equals the per-point walk's, i.e. FP64's.  A warp whose
// box meets more than 32 leaves falls back to the per-point walk.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool box_meets(const float* lo, const float* hi, const float* qlo,
                                          const float* qhi) {
    return lo[0] <= qhi[0] && hi[0] >= qlo[0] && lo[1] <= qhi[1] && hi[1] >= qlo[1] &&
           lo[2] <= qhi[2] && hi[2] >= qlo[2];
}

// Lane k receives the k-th leaf in cand; returns the count (the same on every
// lane), -1 when above 32, kTraversalError on a malformed tree.  Every lane
// walks the same nodes (uniform control flow, broadcast loads).
__device__ __forceinline__ int warp_candidates32(const EnvTree& T, const float* qlo,
                                                 const float* qhi, int lane, int32_t& cand) {
    const int32_t nf = T.nf;
    if (nf == 1) {
        cand = 0;
        return 1;
    }
    int32_t stack[kStack];
    int sp = 0, cnt = 0;
    int32_t cur = 0;
    for (int32_t iter = 0; iter < nf; ++iter) {
        if ((uint32_t)cur >= (uint32_t)(nf - 1)) return kTraversalError;
        const float4* nd = reinterpret_cast<const float4*>(T.nodes32 + cur);
        float4 q0 = __ldg(nd + 0), q1 = __ldg(nd + 1), q2 = __ldg(nd + 2);
        int4 q3 = __ldg(reinterpret_cast<const int4*>(nd + 3));
        const float lo0[3] = {q0.x, q0.y, q0.z}, hi0[3] = {q0.w, q1.x, q1.y};
        const float lo1[3] = {q1.z, q1.w, q2.x}, hi1[3] = {q2.y, q2.z, q2.w};
        bool h0 = box_meets(lo0, hi0, qlo, qhi), h1 = box_meets(lo1, hi1, qlo, qhi);
        if (h0 && q3.x < 0) {
            if ((uint32_t)(~q3.x) >= (uint32_t)nf) return kTraversalError;
            if (lane == cnt) cand = ~q3.x;
            if (++cnt > 32) return -1;
            h0 = false;
        }
        if (h1 && q3.y < 0) {
            if ((uint32_t)(~q3.y) >= (uint32_t)nf) return kTraversalError;
            if (lane == cnt) cand = ~q3.y;
            if (++cnt > 32) return -1;
            h1 = false;
        }
        if (h0 && h1) {
            if (sp >= kStack) return kTraversalError;
            stack[sp++] = q3.y;
            cur = q3.x;
        } else if (h0) {
            cur = q3.x;
        } else if (h1) {
            cur = q3.y;
        } else {
            if (sp == 0) return cnt;
            cur = stack[--sp];
        }
    }
    return kTraversalError;
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <int MINB>
__global__ void __launch_bounds__(128, MINB) k_env_points_warp(const double* __restrict__ P,
                                                         const int32_t* __restrict__ order,
                                                         int64_t n, EnvTree T, EpsParams E,
                                                         uint8_t* __restrict__ out,
                                                         unsigned long long* __restrict__ counters) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    TravStats st;
    uint32_t nq = 0, fallback = 0;
    const int64_t base0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane;
    for (int64_t b = base0; b < n; b += stride) {
        const int64_t i = b + lane;
        const bool valid = i < n;
        const int64_t j = valid ? (order ? (int64_t)__ldg(order + i) : i) : 0;
        V3 p{0.0, 0.0, 0.0};
        if (valid) p = V3{__ldg(P + 3 * j), __ldg(P + 3 * j + 1), __ldg(P + 3 * j + 2)};
        const CertQuery q = cert_query(p, E, T.scale_hi);
        const float inf = __int_as_float(0x7f800000);
        const float r = valid ? __fsqrt_ru(q.thr) : 0.0f;
        const float R = warp_max(r);
        float qlo[3], qhi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            qlo[k] = __fsub_rd(warp_min(valid ? q.ph[k] : inf), R);
            qhi[k] = __fadd_ru(warp_max(valid ? q.ph[k] : -inf), R);
        }
        int32_t cand = -1;
        const int cnt = warp_candidates32(T, qlo, qhi, lane, cand);
        bool in = false;
        if (cnt >= 0) {
            for (int k = 0; k < cnt; ++k) {
                const int32_t lf = __shfl_sync(0xffffffffu, cand, k);
                if (valid && !in) in = cert_leaf_within(T.cull, T.tri, lf, p, q, E.eps2, st);
                if (__all_sync(0xffffffffu, in || !valid)) break;
            }
        } else {
            if (cnt == kTraversalError && lane == 0) atomicOr(counters + kCntError, 1ULL);
            ++fallback;
            if (valid) {
                int32_t f = query_point<true>(T, p, E, st);
                if (f == kTraversalError) atomicOr(counters + kCntError, 1ULL);
                in = f >= 0;
            }
        }
        if (valid) {
            out[j] = (uint8_t)!in;
            ++nq;
        }
    }
    flush_stats(st, counters, nq);
    if (lane == 0 && fallback) atomicAdd(counters + kCntEnvWarpFallback, (unsigned long long)fallback);
}

// ---------------------------------------------------------------------------
// Test through the uniform grid: the leaves listed in the point's own cell
// (see EnvGrid) are every leaf within its culling radius, so the point is in
// iff one of them tests in.  No tree walk; the lanes of a warp loop over
// their own lists in step.  Both precision modes use it: CERT tests each leaf
// with the certified binary32 bounds (FP64 in the band), !CERT tests each
// leaf in FP64.  A leaf whose FP64 distance tests <= eps2 lies within
// eps (1 + 2^-50) + O(2^-52 M) of the point, well inside the culling radius
// R = eps (1 + 2^-18) + 2^-17 M the cell lists cover, so both decide exactly
// as the FP64 tree walk (some facet with computed d^2 <= eps2).
// ---------------------------------------------------------------------------
template <class Tree>   // EnvTree, or the fields of it used here
__device__ __forceinline__ void grid_cell_range(const Tree& T, const CertQuery& q, uint32_t& b,
                                                uint32_t& e) {
    int ix[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float t = __fmul_rn(__fsub_rn(q.ph[k], T.glo[k]), T.ginv);
        int i;
        if (!(t > 0.0f)) i = 0;
        else if (t >= (float)T.gn[k]) i = T.gn[k] - 1;
        else i = min((int)t, T.gn[k] - 1);
        ix[k] = i;
    }
    const uint32_t cell = ((uint32_t)ix[2] * (uint32_t)T.gn[1] + (uint32_t)ix[1]) *
                              (uint32_t)T.gn[0] + (uint32_t)ix[0];
    uint32_t slot = (cell * 0x9E3779B1u) >> T.gshift;
    b = e = 0;
    for (uint32_t probe = 0; probe <= T.gmask; ++probe) {
        const uint4 r = __ldg(T.gslot + slot);   // key and range in one load
        if (r.x == cell) {
            b = r.y;
            e = r.y + r.z;
            return;
        }
        if (r.x == 0xffffffffu) return;   // an empty cell: no leaf within reach
        slot = (slot + 1) & T.gmask;
    }
}

// TW_PRECISION_FP64: a facet whose certified lower bound exceeds eps is culled
// like one whose cell or box is out of reach; every other one is evaluated in
// binary64 (a distance costs some hundred binary64 instructions, the bound
// none but the query's three differences): 300k points, half of them out, took
// 0.25 ms in the test, 0.16 so.
__device__ __forceinline__ bool fp64_leaf_within(const EnvTree& T, int32_t lf, const V3& p,
                                                 const CertQuery& q, double eps2, TravStats& st) {
    ++st.facets;
    if (facet_classify(T.cull, lf, q) == kFacetOut) return false;
    ++st.fp64;
    return leaf_sqdist(T.tri, lf, p) <= eps2;
}

// in iff a leaf of the point's cell tests in; every lane of the warp calls it
template <bool CERT>
__device__ __forceinline__ bool grid_point_in(const EnvTree& T, const EpsParams& E, bool valid,
                                              const V3& p, const CertQuery& q, TravStats& st) {
    uint32_t b = 0, e = 0;
    if (valid) grid_cell_range(T, q, b, e);
    bool in = false;
    // the next list entry is loaded while the current facet is tested, so
    // each test waits on one load (its record) instead of two
    int32_t lf = b < e ? __ldg(T.glist + b) : 0;
    for (uint32_t k = b; k < e; ++k) {
        const int32_t next = k + 1 < e ? __ldg(T.glist + k + 1) : 0;
        if (CERT ? cert_leaf_within(T.cull, T.tri, lf, p, q, E.eps2, st)
                 : fp64_leaf_within(T, lf, p, q, E.eps2, st)) {
            in = true;
            break;
        }
        lf = next;
    }
    return in;
}

// Block b's warps take 32-point groups b*W .. b*W+W-1 together (W warps per
// block), then stride by the grid: in Morton order the warps of a block test
// neighbouring cells at the same time and share their facet records in L1.
template <int BLOCK, int MINB, bool CERT>
__global__ void __launch_bounds__(BLOCK, MINB) k_env_points_grid(const double* __restrict__ P,
                                                           const int32_t* __restrict__ order,
                                                           int64_t n, EnvTree T, EpsParams E,
                                                           uint8_t* __restrict__ out,
                                                           unsigned long long* __restrict__ counters) {
    TravStats st;
    uint32_t nq = 0;
    const int64_t groups = (n + 31) >> 5;
    const int64_t warps = (int64_t)gridDim.x * (BLOCK / 32);
    for (int64_t g = (int64_t)blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5); g < groups;
         g += warps) {
        const int64_t i = (g << 5) + (threadIdx.x & 31);
        if (i < n) {
            // the points, the order and the answers stream through once
            // (evict-first), so the facet records and cell lists stay in L2
            const int64_t j = order ? (int64_t)__ldcs(order + i) : i;
            const V3 p{__ldcs(P + 3 * j), __ldcs(P + 3 * j + 1), __ldcs(P + 3 * j + 2)};
            const CertQuery q = cert_query(p, E, T.scale_hi);
            __stcs(out + j, (uint8_t)!grid_point_in<CERT>(T, E, true, p, q, st));
            ++nq;
        }
    }
    flush_stats(st, counters, nq);
}

// ---------------------------------------------------------------------------
// Test through the bin index: the point's bin and fine cell come from its
// binary32 coordinates, t = (ph - blo) * binv per axis (round to nearest):
// bin i = floor(t) and fine cell floor(8 (t - i)) (t - i is exact: t and i
// are within a factor 2, and x8 is exact), clamped to the grid, so the
// computed fine index is floor(8 t).  t is within 2^-24 |p| binv (the
// rounding of p) + 2^-23 |t| (the subtraction and the product) of its exact
// value (p - blo) binv; inside the grown box |t| / binv is at most its extent
// (below 2 M + 2 R), so that is a distance of at most 2^-24 |p| + 2^-22 (M +
// R) <= 2^-21 M per axis, well inside the 2^-17 M of the culling radius R the
// masks are built for.  A clamped coordinate (outside the grown box) maps to the
// outer cell, whose cube holds the point's projection onto the box face, no
// farther from any facet than the point.  So every leaf within the certified
// culling radius of the point is in its bin's list with its fine-cell bit set,
// and the point is in iff one of those leaves tests in (in CERT, the
// certified binary32 bounds with FP64 in the band; else FP64).
// ---------------------------------------------------------------------------
// The point's bin (Morton index) and fine cell (fz + 8 fx + 64 fy).
__device__ __forceinline__ void bin_cell_of(const EnvTree& T, const CertQuery& q, uint32_t& bin,
                                            int& fine) {
    uint32_t m = 0;
    fine = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float t = __fmul_rn(__fsub_rn(q.ph[k], T.blo[k]), T.binv);
        int i, f;
        if (!(t > 0.0f)) {   // below the grid, or NaN
            i = 0;
            f = 0;
        } else if (t >= (float)T.bn[k]) {
            i = T.bn[k] - 1;
            f = kFine - 1;
        } else {
            i = min((int)t, T.bn[k] - 1);
            f = min((int)(__fsub_rn(t, (float)i) * (float)kFine), kFine - 1);
        }
        m |= morton_expand10((uint32_t)i) << (2 - k);
        fine += f * (k == 2 ? 1 : (k == 0 ? kFine : kFine * kFine));
    }
    bin = m;
}

// The mask words of the bin's entries (the word that holds the point's fine
// cell) are read first, 32 at a time, as independent loads: the hits form a
// bit set and only the hit leaves are tested, in entry order.  DEFER (CERT
// only): a leaf in the certified band is not evaluated here; the point is in
// when another leaf tests in, and otherwise undecided (2), for the FP64 pass.
template <bool CERT, bool DEFER = false>
__device__ __forceinline__ int bins_point_test(const EnvTree& T, const EpsParams& E, const V3& p,
                                               const CertQuery& q, TravStats& st) {
    uint32_t bin;
    int fine;
    bin_cell_of(T, q, bin, fine);
    const uint32_t a = __ldg(T.boff + bin), b = __ldg(T.boff + bin + 1);
    const uint32_t* mw = T.bmask + (int64_t)(fine >> 5) * T.bnt;
    const uint32_t sh = (uint32_t)fine & 31u;
    bool band = false;
    for (uint32_t base = a; base < b; base += 32) {
        const uint32_t cnt = min(b - base, 32u);
        uint32_t hits = 0;
#pragma unroll 16
        for (uint32_t k = 0; k < cnt; ++k) hits |= ((__ldg(mw + base + k) >> sh) & 1u) << k;
        while (hits) {
            const uint32_t k = (uint32_t)(__ffs(hits) - 1);
            hits &= hits - 1u;
            const int32_t lf = __ldg(T.bleaf + base + k);
            if (DEFER) {
                ++st.facets;
                const int cls = facet_classify(T.cull, lf, q);
                if (cls == kFacetIn) return 1;
                band |= cls == kFacetBand;
            } else if (CERT ? cert_leaf_within(T.cull, T.tri, lf, p, q, E.eps2, st)
                            : fp64_leaf_within(T, lf, p, q, E.eps2, st)) {
                return 1;
            }
        }
    }
    return band ? 2 : 0;
}

template <bool CERT>
__device__ __forceinline__ bool bins_point_in(const EnvTree& T, const EpsParams& E, const V3& p,
                                              const CertQuery& q, TravStats& st) {
    return bins_point_test<CERT>(T, E, p, q, st) == 1;
}

// recheck: (count, point indices) of the points the certified test left
// undecided (a leaf in the band and none in), for k_env_points_bins_recheck;
// nullptr: the band is evaluated in FP64 on the spot.
// A lane's point through the surface's index: the bins when built, else the
// grid's hashed cells (the same decisions).  No warp collectives: lanes
// without a point (valid false) take no part.  For point queries, of which
// about half lie outside and test every leaf in reach; face samples and
// collapse checks, mostly inside and decided by their first leaf, keep the
// grid's short cell lists (the bins' mask scan measured slower there: 38.1
// against 34.4 ms for the 200k-star smoothing pass).
template <bool CERT>
__device__ __forceinline__ bool index_point_in(const EnvTree& T, const EpsParams& E, bool valid,
                                               const V3& p, const CertQuery& q, TravStats& st) {
    if (T.boff) return valid && bins_point_in<CERT>(T, E, p, q, st);
    return grid_point_in<CERT>(T, E, valid, p, q, st);
}

// A sorted point as the certified test reads it: its coordinates split in
// binary32 (p = ph + pl, the split of cert_query) and its index.  One 32-byte
// sector, written whole by the placing pass and read in order, where a gather
// of the point's 24 bytes fetches two 64-byte lines of DRAM every other time.
// 10M points: the test 485 -> 390 us (DRAM reads 840 -> 303 MB for 6M), the
// placing pass 91 -> 145.
struct __align__(32) PointRec {
    float4 a;   // ph0 ph1 ph2 pl0
    float4 b;   // pl1 pl2 - index
};

// n_dev (sorted on the dense bin ids): the number of sorted queries, read on
// the device (the others were decided by the binning pass); else n.
// rec (DEFER only): the sorted points' records, read in order in place of
// order and P; nullptr: the point is gathered through order.
template <int BLOCK, int MINB, bool CERT, bool DEFER>
__global__ void __launch_bounds__(BLOCK, MINB) k_env_points_bins(const double* __restrict__ P,
                                                           const int32_t* __restrict__ order,
                                                           int64_t n, EnvTree T, EpsParams E,
                                                           uint8_t* __restrict__ out,
                                                           unsigned long long* __restrict__ counters,
                                                           uint32_t* __restrict__ recheck,
                                                           const uint32_t* __restrict__ n_dev,
                                                           const PointRec* __restrict__ rec) {
    TravStats st;
    uint32_t nq = 0;
    if (n_dev) n = min(n, (int64_t)__ldg(n_dev));
    const int64_t groups = (n + 31) >> 5;
    const int64_t warps = (int64_t)gridDim.x * (BLOCK / 32);
    for (int64_t g = (int64_t)blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5); g < groups;
         g += warps) {
        const int64_t i = (g << 5) + (threadIdx.x & 31);
        if (i < n) {
            // the points, the order and the answers stream through once
            // (evict-first), so the bins, entries and facet records stay in L2
            int64_t j;
            V3 p;
            CertQuery q;
            if (DEFER && rec) {
                const float4 a = __ldcs(&rec[i].a), b = __ldcs(&rec[i].b);
                j = (int64_t)__float_as_int(b.w);
                q = cert_query_split(a.x, a.y, a.z, a.w, b.x, b.y, E, T.scale_hi);
            } else {
                j = order ? (int64_t)__ldcs(order + i) : i;
                p = V3{__ldcs(P + 3 * j), __ldcs(P + 3 * j + 1), __ldcs(P + 3 * j + 2)};
                q = cert_query(p, E, T.scale_hi);
            }
            const int r = bins_point_test<CERT, DEFER>(T, E, p, q, st);
            if (DEFER && r == 2) {
                const uint32_t at = atomicAdd(recheck, 1u);
                recheck[1 + at] = (uint32_t)j;   // at < n: one entry per point
            } else {
                __stcs(out + j, (uint8_t)(r != 1));
            }
            ++nq;
        }
    }
    flush_stats(st, counters, nq);
}

// The undecided points of a deferred certified test (the decision of
// TW_PRECISION_FP64 for them).  One point per warp (lane 0): the points'
// leaves take different paths through the FP64 distance, which in one warp
// would run one after another on the slow FP64 pipe; spread over warps (and
// SMs) they run side by side.
__global__ void k_env_points_bins_recheck(const double* __restrict__ P,
                                          const uint32_t* __restrict__ recheck, EnvTree T,
                                          EpsParams E, uint8_t* __restrict__ out,
                                          unsigned long long* __restrict__ counters) {
    if ((threadIdx.x & 31) != 0) return;
    TravStats st;
    const uint32_t cnt = *recheck;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < cnt; k += warps) {
        const int64_t j = recheck[1 + k];
        const V3 p{P[3 * j], P[3 * j + 1], P[3 * j + 2]};
        const CertQuery q = cert_query(p, E, T.scale_hi);
        // the certified test again, now evaluating the band in FP64 on the
        // spot: only the leaves in the band cost a binary64 distance
        out[j] = (uint8_t)!bins_point_in<true>(T, E, p, q, st);
    }
    // no flush_stats: the counters count each point's certified tests once;
    // the FP64 evaluations are added per thread
    if (st.fp64) atomicAdd(counters + kCntEnvFp64, (unsigned long long)st.fp64);
}

// ---- grid build ----------------------------------------------------------------------
// A regular grid for the separating-axis test: cells of side cs from lo, n a
// side.  hf: half-size of the tested cube; ext[k]: largest |coordinate| of the
// grid on axis k.
struct SatGrid {
    double lo[3];
    double inv_c, Rm;
    int32_t n[3];
    float csf, hf, ext[3];
};
static SatGrid sat_grid(const float* lo, const int64_t* n, double inv_c, double Rm, double slack) {
    SatGrid g;
    const double cs = 1.0 / inv_c;
    for (int k = 0; k < 3; ++k) {
        g.lo[k] = lo[k];
        g.n[k] = (int32_t)n[k];
        g.ext[k] = round_up_float(std::max(std::fabs((double)lo[k]),
                                           std::fabs((double)lo[k] + (double)n[k] * cs)));
    }
    g.inv_c = inv_c;
    g.Rm = Rm;
    g.csf = (float)cs;
    g.hf = (float)(0.5 * cs + Rm + slack) * 1.000001f;
    return g;
}

// Binary32 separating-axis test of one leaf against the cells of a grid: a
// cell is within reach when no axis (the triangle's normal, the nine edge x
// box-axis products and the three box axes) separates the triangle from the
// cube of half-size cs/2 + Rm + slack around the cell's centre, which holds
// the ball of radius Rm around every point of the cell (slack = 2^-30 M
// covers the cell's placement), so a leaf it excludes is farther than Rm from
// the whole cell.  Along axis a the cells not separated are those whose centre
// w has lo <= a.w <= hi, two numbers a leaf and axis (SatSlab); the warp's
// lanes compute the 13 slabs of a leaf, one each.
// Rigorous in binary32: any direction is a valid separating axis, so the
// binary32 axes themselves are used as exact vectors and only the
// projections carry rounding.  The vertices relative to t0 (rounded once) and
// the cell centre relative to t0 (from base = lo - t0 and (x + 1/2) cs) are
// within 2^-20 L of the exact values (L = 2 (M + the grid's extent) bounds
// every coordinate and offset), and the projections of both round by at most
// 8 2^-24 |a|_1 L, so each is within |a|_1 2^-19 L (1 + 2^-1); an axis
// separates only by more than |a|_1 2^-18 L.  Cells no axis separates by that
// margin are kept (a longer list, never a missing leaf).
struct __align__(32) SatSlab {
    float a[3];
    float lo, hi, pad[3];
};
constexpr int kSlabs = 13;

// A slab in units of cells along z: the cell with centre (wx, wy, wz + cs i)
// is within it when l - q <= i <= h - q, q = ax wx + ay wy + az wz.  dq: q's
// step to the column four cells on in y.
struct __align__(32) ColumnSlab {
    float ax, ay, az, l;
    float h, dq, pad[2];
};

// One lane's leaf: vertices relative to t0, the grid's origin relative to t0,
// the error scale and the index box of the leaf grown by Rm.
struct SatLeaf {
    float v1[3], v2[3], base[3], mL;
    int32_t i0[3], nb[3];
};
// A block's first warp prepares 32 leaves, one a lane (their binary64 work
// would cost a warp per leaf 32 times as much), and then the warps take them in
// turn.  With 32 leaves a warp, 3k warps in all, the leaves with the most cells
// held the launch: a quarter of the warps resident on the average (100k
// facets: counts 0.22 ms, grid cells 0.14, bin cells 0.091; now 0.155, 0.097,
// 0.071).
constexpr int kSatBlock = 128;
constexpr int kSatWarps = kSatBlock / 32;
struct SatShared {
    SatLeaf leaf[32];
    SatSlab slab[kSatWarps][kSlabs + 3];
    ColumnSlab column[kSatWarps][kSlabs];
};

// false when the box spans more than limit cells
__device__ __forceinline__ bool sat_prepare(const double* __restrict__ tri, int64_t f,
                                            const SatGrid& g, int64_t limit, SatLeaf& l) {
    double t[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) t[k] = __ldg(tri + 9 * f + k);
    float L = 0.0f;
    int64_t box = 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double a = fmin(t[k], fmin(t[3 + k], t[6 + k])) - g.Rm;
        const double b = fmax(t[k], fmax(t[3 + k], t[6 + k])) + g.Rm;
        double u = floor((a - g.lo[k]) * g.inv_c), v = floor((b - g.lo[k]) * g.inv_c);
        u = fmin(fmax(u, 0.0), (double)(g.n[k] - 1));
        v = fmin(fmax(v, 0.0), (double)(g.n[k] - 1));
        l.i0[k] = (int)u;
        l.nb[k] = (int)v - (int)u + 1;
        box *= l.nb[k];
        l.v1[k] = (float)(t[3 + k] - t[k]);
        l.v2[k] = (float)(t[6 + k] - t[k]);
        l.base[k] = (float)(g.lo[k] - t[k]);
        L = fmaxf(L, g.ext[k] + fabsf((float)t[k]) * 1.0000003f);
    }
    L = 2.0f * L;
    // 2^-40 <= L < 2^40 and |a|_1 >= 2^-40 keep every product far from
    // binary32 overflow, and underflow far below the margin (else every cell of
    // the box is kept: mL < 0)
    l.mL = L >= 0x1p-40f && L < 0x1p40f ? L * (0x1p-18f * 1.0001f) : -1.0f;
    return box <= limit;
}

// The leaf's slabs (the whole warp); half: the tested cube's half-size.
__device__ __forceinline__ void sat_slabs(const SatLeaf& l, float half, SatSlab* slab) {
    const int j = threadIdx.x & 31;
    __syncwarp();
    if (j < kSlabs) {
        float a[3] = {0.0f, 0.0f, 0.0f};
        const float e[3][3] = {{l.v1[0], l.v1[1], l.v1[2]},
                               {l.v2[0] - l.v1[0], l.v2[1] - l.v1[1], l.v2[2] - l.v1[2]},
                               {-l.v2[0], -l.v2[1], -l.v2[2]}};
        if (j == 0) {
            a[0] = e[0][1] * e[1][2] - e[0][2] * e[1][1];
            a[1] = e[0][2] * e[1][0] - e[0][0] * e[1][2];
            a[2] = e[0][0] * e[1][1] - e[0][1] * e[1][0];
        } else if (j < 10) {   // unit_k x e_i
            const int i = (j - 1) / 3, k = (j - 1) % 3;
            const float ex = i == 0 ? e[0][0] : i == 1 ? e[1][0] : e[2][0];
            const float ey = i == 0 ? e[0][1] : i == 1 ? e[1][1] : e[2][1];
            const float ez = i == 0 ? e[0][2] : i == 1 ? e[1][2] : e[2][2];
            if (k == 0) {
                a[1] = -ez;
                a[2] = ey;
            } else if (k == 1) {
                a[2] = -ex;
                a[0] = ez;
            } else {
                a[0] = -ey;
                a[1] = ex;
            }
        } else {
            a[0] = j == 10 ? 1.0f : 0.0f;
            a[1] = j == 11 ? 1.0f : 0.0f;
            a[2] = j == 12 ? 1.0f : 0.0f;
        }
        const float a1 = fabsf(a[0]) + fabsf(a[1]) + fabsf(a[2]);
        const float p1 = a[0] * l.v1[0] + a[1] * l.v1[1] + a[2] * l.v1[2];
        const float p2 = a[0] * l.v2[0] + a[1] * l.v2[1] + a[2] * l.v2[2];
        const float r = half * a1 + a1 * l.mL;
        const float inf = __int_as_float(0x7f800000);
        const bool use = a1 >= 0x1p-40f && l.mL > 0.0f;
        SatSlab& s = slab[j];
        s.a[0] = a[0];
        s.a[1] = a[1];
        s.a[2] = a[2];
        s.lo = use ? fminf(0.0f, fminf(p1, p2)) - r : -inf;
        s.hi = use ? fmaxf(0.0f, fmaxf(p1, p2)) + r : inf;
    }
    __syncwarp();
}

// Cell centre (wx, wy, wz) (relative to t0) within reach of the leaf?
__device__ __forceinline__ bool sat_within(const SatSlab* slab, float wx, float wy, float wz) {
    bool in = true;
#pragma unroll
    for (int j = 0; j < kSlabs; ++j) {
        const float p = fmaf(slab[j].a[0], wx, fmaf(slab[j].a[1], wy, slab[j].a[2] * wz));
        in = in && !(p < slab[j].lo) && !(p > slab[j].hi);
    }
    return in;
}
// Cell q (x fastest) of the leaf's box: its indices and whether it is within reach.
__device__ __forceinline__ bool sat_cell(const SatLeaf& l, const SatSlab* slab, float cs, int q,
                                         int& x, int& y, int& z) {
    x = l.i0[0] + q % l.nb[0];
    y = l.i0[1] + (q / l.nb[0]) % l.nb[1];
    z = l.i0[2] + q / (l.nb[0] * l.nb[1]);
    return sat_within(slab, l.base[0] + ((float)x + 0.5f) * cs, l.base[1] + ((float)y + 0.5f) * cs,
                      l.base[2] + ((float)z + 0.5f) * cs);
}

// The cells within reach of every leaf.  Counting (fcnt != nullptr): the
// leaf's count and the total; a leaf whose box spans more than limit cells
// marks the grid unsuitable (*too_big), and the counts, which nothing then
// reads, are left there (uploading 3k facets of all sizes: 1.62 ms without that,
// 0.50 so; 1.25 with a warp a leaf).  Filling: each leaf's cells from
// foff[leaf] on, in box order (fill(at, leaf, x, y, z), one lane each).
template <class Fill>
__device__ __forceinline__ void sat_cells(const double* __restrict__ tri, int32_t nf,
                                          const SatGrid& g, int64_t limit,
                                          unsigned long long* __restrict__ total,
                                          uint32_t* __restrict__ fcnt,
                                          const uint32_t* __restrict__ foff,
                                          int* __restrict__ too_big, Fill fill) {
    __shared__ SatShared sh;
    __shared__ unsigned usable;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t f0 = (int64_t)blockIdx.x * 32;
    if (warp == 0) {
        bool ok = false;
        if (f0 + lane < nf) {
            ok = sat_prepare(tri, f0 + lane, g, limit, sh.leaf[lane]);
            if (!ok && too_big) atomicExch(too_big, 1);
            if (!ok && fcnt) fcnt[f0 + lane] = 0;
        }
        const unsigned b = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) usable = b;
    }
    __syncthreads();
    unsigned long long sum = 0;
    for (int k = warp; k < 32; k += kSatWarps) {
        if (!((usable >> k) & 1u)) continue;
        const SatLeaf& l = sh.leaf[k];
        sat_slabs(l, g.hf, sh.slab[warp]);
        const int nbox = l.nb[0] * l.nb[1] * l.nb[2];
        uint32_t at = fcnt ? 0u : __ldg(foff + f0 + k);
        const uint32_t end = fcnt ? 0xffffffffu : __ldg(foff + f0 + k + 1);
        for (int q0 = 0; q0 < nbox; q0 += 32) {
            if (too_big && q0 && (q0 & 1023) == 0 &&   // long boxes only: a load each
                __shfl_sync(0xffffffffu, *(volatile const int*)too_big, 0))
                return;
            int x = 0, y = 0, z = 0;
            const bool in = q0 + lane < nbox && sat_cell(l, sh.slab[warp], g.csf, q0 + lane, x, y, z);
            const unsigned bal = __ballot_sync(0xffffffffu, in);
            const uint32_t w = at + __popc(bal & ((1u << lane) - 1u));
            if (!fcnt && in && w < end) fill(w, (int32_t)(f0 + k), x, y, z);
            at += __popc(bal);
        }
        if (fcnt && lane == 0) fcnt[f0 + k] = at;
        sum += at;
    }
    if (fcnt && lane == 0 && sum) atomicAdd(total, sum);
}
constexpr int64_t kMaxLeafCells = 65536, kMaxLeafBins = 4096;

__global__ void __launch_bounds__(kSatBlock) k_cells_count(const double* __restrict__ tri, int32_t nf,
                                                           SatGrid g, int64_t limit,
                                                           unsigned long long* __restrict__ total,
                                                           uint32_t* __restrict__ fcnt,
                                                           int* __restrict__ too_big) {
    sat_cells(tri, nf, g, limit, total, fcnt, nullptr, too_big,
              [](uint32_t, int32_t, int, int, int) {});
}

// The grid's (cell << 32 | leaf) pairs.
__global__ void __launch_bounds__(kSatBlock) k_grid_cells(const double* __restrict__ tri, int32_t nf,
                                                          SatGrid g, const uint32_t* __restrict__ foff,
                                                          unsigned long long* __restrict__ pairs) {
    sat_cells(tri, nf, g, kMaxLeafCells, nullptr, nullptr, foff, nullptr,
              [=](uint32_t at, int32_t f, int x, int y, int z) {
                  const uint32_t cell = ((uint32_t)z * (uint32_t)g.n[1] + (uint32_t)y) *
                                            (uint32_t)g.n[0] + (uint32_t)x;
                  pairs[at] = ((unsigned long long)cell << 32) | (uint32_t)f;
              });
}

// The bin index's entries: the bins within reach of every leaf (the Morton
// index of their coordinates in keys, the entry's index in vals, the leaf in
// leaves), before their masks.
__global__ void __launch_bounds__(kSatBlock) k_bin_cells(const double* __restrict__ tri, int32_t nf,
                                                         SatGrid g, const uint32_t* __restrict__ foff,
                                                         uint32_t* __restrict__ keys,
                                                         uint32_t* __restrict__ vals,
                                                         uint32_t* __restrict__ leaves) {
    sat_cells(tri, nf, g, kMaxLeafBins, nullptr, nullptr, foff, nullptr,
              [=](uint32_t at, int32_t f, int x, int y, int z) {
                  keys[at] = (morton_expand10((uint32_t)x) << 2) |
                             (morton_expand10((uint32_t)y) << 1) | morton_expand10((uint32_t)z);
                  vals[at] = at;
                  leaves[at] = (uint32_t)f;
              });
}

__device__ __forceinline__ uint32_t morton_compact10(uint32_t v) {
    v &= 0x49249249u;
    v = (v | (v >> 2)) & 0xC30C30C3u;
    v = (v | (v >> 4)) & 0x0F00F00Fu;
    v = (v | (v >> 8)) & 0xFF0000FFu;
    v = (v | (v >> 16)) & 0x000003FFu;
    return v;
}

// The slabs in units of cells along z (the whole warp).  An axis with |a_z| <
// 2^-20 |a|_1 takes 2^-20 |a|_1 for a_z in the unit: its projection moves by
// at most 7 of those units over a column, so its interval, 8 wider below and
// 16 above, holds all of a column that a cell of it is within.  An axis whose
// numbers could leave binary32 is not used.
__device__ __forceinline__ void column_slabs(const SatLeaf& l, const SatSlab* slab, float cs,
                                             ColumnSlab* column) {
    const int j = threadIdx.x & 31;
    if (j < kSlabs) {
        const float a0 = slab[j].a[0], a1 = slab[j].a[1], a2 = slab[j].a[2];
        const float n1 = fabsf(a0) + fabsf(a1) + fabsf(a2);
        const bool flat = !(fabsf(a2) >= n1 * 0x1p-20f);
        const float inv = flat ? 0x1p20f / (n1 * cs) : 1.0f / (a2 * cs);
        const bool use = n1 >= 0x1p-40f && fabsf(inv) * n1 * l.mL < 0x1p80f;   // false for NaN
        const float inf = __int_as_float(0x7f800000);
        const float u = slab[j].lo * inv, v = slab[j].hi * inv;
        ColumnSlab c;
        c.ax = use ? a0 * inv : 0.0f;
        c.ay = use ? a1 * inv : 0.0f;
        c.az = use ? a2 * inv : 0.0f;
        c.l = use ? fminf(u, v) - (flat ? 8.0f : 0.0f) : -inf;
        c.h = use ? fmaxf(u, v) + (flat ? 16.0f : 0.0f) : inf;
        c.dq = c.ay * (4.0f * cs);
        column[j] = c;
    }
    __syncwarp();
}

// The fine-cell mask of every entry, 16 words an entry: bit fz + 8 fx + 64 fy
// set when the bin's fine cell (a grid of 8n cells a side: g) is within reach
// of the leaf.  A lane takes two columns of eight cells along z (fx, fy =
// lane % 8, lane / 8 and lane / 8 + 4); each slab leaves an interval of a
// column, which is a byte of the mask, and four lanes make two words.  Bound
// by its instructions, so a column costs its 13 slabs once instead of a
// 13-axis test per cell (100k facets: 13.1 ms in two passes, counting and
// filling; 1.28 ms, the count taking whole bins), the slabs are scaled once a leaf
// (four differences and bounds a slab and two columns where a quotient took
// twice that) and the mask's bits lie along the columns (ballots of the cells
// across them took 80 instructions more): 0.62 ms, and
// 0.46 with a block's warps sharing its 32 leaves.  The scaled numbers are off by
// 10 2^-24 |a|_1 L in the projection, inside the margin.
__global__ void __launch_bounds__(kSatBlock) k_bin_masks(const double* __restrict__ tri, int32_t nf,
                                                         SatGrid g, const uint32_t* __restrict__ foff,
                                                         const uint32_t* __restrict__ keys,
                                                         uint32_t* __restrict__ masks) {
    __shared__ SatShared sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t f0 = (int64_t)blockIdx.x * 32;
    if (warp == 0 && f0 + lane < nf) sat_prepare(tri, f0 + lane, g, INT64_MAX, sh.leaf[lane]);
    __syncthreads();
    const int leaves = (int)(nf - f0 < 32 ? nf - f0 : 32);
    const ColumnSlab* column = sh.column[warp];
    for (int k = warp; k < leaves; k += kSatWarps) {
        const SatLeaf& l = sh.leaf[k];
        sat_slabs(l, g.hf, sh.slab[warp]);
        column_slabs(l, sh.slab[warp], g.csf, sh.column[warp]);
        const uint32_t end = __ldg(foff + f0 + k + 1);
        for (uint32_t at = __ldg(foff + f0 + k); at < end; ++at) {
            const uint32_t key = __ldg(keys + at);
            const float x = (float)(kFine * morton_compact10(key >> 2) + (lane & 7));
            const float y = (float)(kFine * morton_compact10(key >> 1) + (lane >> 3));
            const float z = (float)(kFine * morton_compact10(key));
            const float wx = l.base[0] + (x + 0.5f) * g.csf, wy = l.base[1] + (y + 0.5f) * g.csf,
                        wz = l.base[2] + (z + 0.5f) * g.csf;
            float l0 = 0.0f, h0 = 7.0f, l1 = 0.0f, h1 = 7.0f;
#pragma unroll
            for (int j = 0; j < kSlabs; ++j) {
                const ColumnSlab& c = column[j];
                const float q0 = fmaf(c.ax, wx, fmaf(c.ay, wy, c.az * wz)), q1 = q0 + c.dq;
                l0 = fmaxf(l0, c.l - q0);
                h0 = fminf(h0, c.h - q0);
                l1 = fmaxf(l1, c.l - q1);
                h1 = fminf(h1, c.h - q1);
            }
            // the cells ceil(l) .. floor(h) of each column, none for l > 7 or h < 0
            const int i0 = (int)ceilf(fminf(l0, 8.0f)), i1 = (int)ceilf(fminf(l1, 8.0f));
            const int e0 = (int)floorf(fmaxf(h0, -1.0f)), e1 = (int)floorf(fmaxf(h1, -1.0f));
            const uint32_t m0 = (0xffu >> (7 - e0)) & (0xffu << i0);
            const uint32_t m1 = (0xffu >> (7 - e1)) & (0xffu << i1);
            const int sh8 = 8 * (lane & 3);
            uint32_t w0 = (m0 & 0xffu) << sh8, w1 = (m1 & 0xffu) << sh8;
            w0 |= __shfl_xor_sync(0xffffffffu, w0, 1);
            w1 |= __shfl_xor_sync(0xffffffffu, w1, 1);
            w0 |= __shfl_xor_sync(0xffffffffu, w0, 2);
            w1 |= __shfl_xor_sync(0xffffffffu, w1, 2);
            if ((lane & 3) < 2)
                masks[(int64_t)at * kFineWords + (lane >> 2) + 8 * (lane & 3)] = lane & 1 ? w1 : w0;
        }
    }
}

// Sorted bins with the indices of their unsorted entries -> the entries
// (kFineWords mask-word arrays of n, then the leaves), and the entry count of
// each bin (zeroed before).
__global__ void k_bin_split(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ src,
                            const uint32_t* __restrict__ masks, const uint32_t* __restrict__ leaves,
                            int64_t n, uint32_t* __restrict__ ent, uint32_t* __restrict__ cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t from = src[i];
    const uint4* m = reinterpret_cast<const uint4*>(masks + from * kFineWords);
#pragma unroll
    for (int w = 0; w < kFineWords / 4; ++w) {
        const uint4 v = __ldg(m + w);
        ent[(4 * w) * n + i] = v.x;
        ent[(4 * w + 1) * n + i] = v.y;
        ent[(4 * w + 2) * n + i] = v.z;
        ent[(4 * w + 3) * n + i] = v.w;
    }
    ent[kFineWords * n + i] = leaves[from];
    atomicAdd(cnt + keys[i], 1u);
}

// 1 for a bin with entries, else 0 (boff: nb + 1 exclusive sums).
__global__ void k_bin_flags(const uint32_t* __restrict__ boff, int64_t nb,
                            int32_t* __restrict__ flag) {
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m < nb) flag[m] = boff[m + 1] > boff[m] ? 1 : 0;
}

// Exclusive sums of the flags -> the dense id of each bin with entries, -1
// for the others; *nocc: how many have entries.
__global__ void k_bin_ids(const uint32_t* __restrict__ boff, int64_t nb, int32_t* __restrict__ bid,
                          int32_t* __restrict__ nocc) {
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nb) return;
    const bool has = boff[m + 1] > boff[m];
    const int32_t v = bid[m];
    if (m == nb - 1) *nocc = v + (has ? 1 : 0);
    bid[m] = has ? v : -1;
}

// Sorted pairs -> the cell of each entry and the leaf list.
__global__ void k_grid_split(const unsigned long long* __restrict__ pairs, int64_t n,
                             uint32_t* __restrict__ cells, int32_t* __restrict__ list) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long v = pairs[i];
    cells[i] = (uint32_t)(v >> 32);
    list[i] = (int32_t)(v & 0xffffffffu);
}

// Inserts the distinct cells into the hash table (bounded linear probing).
__global__ void k_grid_insert(const uint32_t* __restrict__ uniq, const uint32_t* __restrict__ cnt,
                              const uint32_t* __restrict__ start, const int* __restrict__ nuniq,
                              uint4* __restrict__ slots, uint32_t shift, uint32_t mask,
                              int* __restrict__ failed) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nuniq) return;
    const uint32_t c = uniq[i];
    uint32_t slot = (c * 0x9E3779B1u) >> shift;
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const uint32_t prev = atomicCAS(&slots[slot].x, 0xffffffffu, c);
        if (prev == 0xffffffffu || prev == c) {
            slots[slot].y = start[i];
            slots[slot].z = cnt[i];
            slots[slot].w = 0u;
            return;
        }
        slot = (slot + 1) & mask;
    }
    atomicExch(failed, 1);
}

// Point order for the traversal: a counting sort of the query points into the
// 2^(3b) Morton cells of the surface box (b bits a side).  The order only
// changes how much work the traversal does, never its results, so the bin
// is computed in binary32 (integer-rounded inputs) and the order of points
// within a bin is whatever the atomic increments give.
__global__ void k_point_bins(const double* __restrict__ P, int64_t n, float lx, float ly,
                             float lz, float sx, float sy, float sz, float side,
                             uint2* __restrict__ bin_rank, uint32_t* __restrict__ count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float c[3] = {(d2f_rn(__ldcs(P + 3 * i)) - lx) * sx,
                        (d2f_rn(__ldcs(P + 3 * i + 1)) - ly) * sy,
                        (d2f_rn(__ldcs(P + 3 * i + 2)) - lz) * sz};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float v = fminf(fmaxf(c[k] * side, 0.0f), side - 1.0f);   // NaN -> 0
        q[k] = (uint32_t)v;
    }
    const uint32_t bin =
        (morton_expand10(q[0]) << 2) | (morton_expand10(q[1]) << 1) | morton_expand10(q[2]);
    bin_rank[i] = make_uint2(bin, atomicAdd(count + bin, 1u));
}

// The same sort on the bin index's own bins (Morton order of the bin
// coordinates shifted right by sh): consecutive queries then share a bin and
// its entries.  The bin coordinates are computed as in bins_point_in.
__global__ void k_point_bins_idx(const double* __restrict__ P, int64_t n, float lx, float ly,
                                 float lz, float inv, int32_t n0, int32_t n1, int32_t n2, int sh,
                                 uint2* __restrict__ bin_rank, uint32_t* __restrict__ count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float c[3] = {__fmul_rn(__fsub_rn(d2f_rn(__ldcs(P + 3 * i)), lx), inv),
                        __fmul_rn(__fsub_rn(d2f_rn(__ldcs(P + 3 * i + 1)), ly), inv),
                        __fmul_rn(__fsub_rn(d2f_rn(__ldcs(P + 3 * i + 2)), lz), inv)};
    const int32_t nb[3] = {n0, n1, n2};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int v = !(c[k] > 0.0f) ? 0 : (c[k] >= (float)nb[k] ? nb[k] - 1 : min((int)c[k], nb[k] - 1));
        q[k] = (uint32_t)v >> sh;
    }
    const uint32_t bin =
        (morton_expand10(q[0]) << 2) | (morton_expand10(q[1]) << 1) | morton_expand10(q[2]);
    bin_rank[i] = make_uint2(bin, atomicAdd(count + bin, 1u));
}

// The same on the dense ids of the bins with entries (bid): a point whose bin
// has no entry has no leaf within its culling radius, so it is out, decided
// here (marked 0xffffffff for the placing pass, counted as a query).
__global__ void k_point_bins_cid(const double* __restrict__ P, int64_t n, float lx, float ly,
                                 float lz, float inv, int32_t n0, int32_t n1, int32_t n2,
                                 const int32_t* __restrict__ bid, uint2* __restrict__ bin_rank,
                                 uint32_t* __restrict__ count, uint8_t* __restrict__ out,
                                 unsigned long long* __restrict__ counters) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float c[3] = {__fmul_rn(__fsub_rn(d2f_rn(__ldcs(P + 3 * i)), lx), inv),
                        __fmul_rn(__fsub_rn(d2f_rn(__ldcs(P + 3 * i + 1)), ly), inv),
                        __fmul_rn(__fsub_rn(d2f_rn(__ldcs(P + 3 * i + 2)), lz), inv)};
    const int32_t nb[3] = {n0, n1, n2};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int v = !(c[k] > 0.0f) ? 0 : (c[k] >= (float)nb[k] ? nb[k] - 1 : min((int)c[k], nb[k] - 1));
        q[k] = (uint32_t)v;
    }
    const uint32_t m =
        (morton_expand10(q[0]) << 2) | (morton_expand10(q[1]) << 1) | morton_expand10(q[2]);
    const int32_t id = __ldg(bid + m);
    const bool empty = id < 0;
    if (empty) {
        out[i] = 1;
        bin_rank[i] = make_uint2(0xffffffffu, 0u);
    } else {
        bin_rank[i] = make_uint2((uint32_t)id, atomicAdd(count + id, 1u));
    }
    const unsigned act = __activemask();
    const unsigned dec = __ballot_sync(act, empty);
    if (dec && (threadIdx.x & 31) == (unsigned)(__ffs(act) - 1))
        atomicAdd(counters + kCntEnvQueries, (unsigned long long)__popc(dec));
}

// idx[first of bin + rank] = i, with count holding each bin's first position
__global__ void k_point_place(const uint2* __restrict__ bin_rank, int64_t n,
                              const uint32_t* __restrict__ first, int32_t* __restrict__ idx) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 br = __ldcs(bin_rank + i);
    if (br.x == 0xffffffffu) return;   // decided by the binning pass
    idx[__ldg(first + br.x) + br.y] = (int32_t)i;
}

// The same with the points' records in place of their indices.
__global__ void k_point_place_rec(const double* __restrict__ P,
                                  const uint2* __restrict__ bin_rank, int64_t n,
                                  const uint32_t* __restrict__ first, PointRec* __restrict__ rec) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 br = __ldcs(bin_rank + i);
    const V3 p{__ldcs(P + 3 * i), __ldcs(P + 3 * i + 1), __ldcs(P + 3 * i + 2)};
    if (br.x == 0xffffffffu) return;   // decided by the binning pass
    float ph[3], pl[3];
    cert_split(p, ph, pl);
    PointRec* r = rec + __ldg(first + br.x) + br.y;
    r->a = make_float4(ph[0], ph[1], ph[2], pl[0]);
    r->b = make_float4(pl[1], pl[2], 0.0f, __int_as_float((int32_t)i));
}

// bits a side of the sort grid: the knob (2..8), or the smallest b with
// 2^(3b) >= n, between 3 and 8 (8: cells of 1/256 of the box, about one
// envelope-grid cell on a 100k-facet surface)
static int sort_bits(int64_t n, int knob) {
    if (knob >= 2) return std::min(knob, 8);
    int b = 3;
    while (b < 8 && (int64_t(1) << (3 * b)) < n) ++b;
    return b;
}

struct SortLayout {
    uint2* bin_rank;
    int32_t* idx;    // sorted point indices, or
    PointRec* rec;   // records in the same place (nullptr: no room was asked for)
    uint32_t* count;
    int64_t nbins;
    uint32_t* recheck;   // count, then up to n point indices
    void* temp;
    size_t temp_bytes;
};

static size_t cub_scan_bytes(int64_t nbins) {
    size_t b = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, b, (uint32_t*)nullptr, (int)nbins);
    return b;
}

static SortLayout sort_layout(void* base, int64_t n, int knob, bool records) {
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    char* q = static_cast<char*>(base);
    SortLayout L;
    L.nbins = int64_t(1) << (3 * sort_bits(n, knob));
    L.bin_rank = (uint2*)q; q += al(8 * (size_t)n);
    L.idx = (int32_t*)q;
    L.rec = records ? (PointRec*)q : nullptr;
    q += al((records ? sizeof(PointRec) : 4) * (size_t)n);
    L.count = (uint32_t*)q; q += al(4 * (size_t)L.nbins);
    L.recheck = (uint32_t*)q; q += al(4 * (size_t)n + 4);
    L.temp = q;
    L.temp_bytes = cub_scan_bytes(L.nbins);
    return L;
}

size_t env_sort_scratch_bytes(int64_t n, int knob, bool records) {
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const int64_t nbins = int64_t(1) << (3 * sort_bits(n, knob));
    return al(8 * (size_t)n) + al((records ? sizeof(PointRec) : 4) * (size_t)n) + al(4 * (size_t)nbins) +
           al(4 * (size_t)n + 4) + al(cub_scan_bytes(nbins)) + 256;
}

size_t env_record_bytes(int64_t n) { return sizeof(PointRec) * (size_t)n; }

// Batches below this size are traversed in input order (sorting would cost
// more than it saves).
constexpr int64_t kSortMin = 4096;

// The certified bulk test through the bins needs no more of a point than its
// record; the other tests gather the binary64 coordinates.
bool env_points_use_records(const Surface& S, int64_t n, double eps2, int precision, int knob) {
    return precision == TW_PRECISION_FP32_CERTIFIED && knob != 0 && n >= kSortMin &&
           n <= INT32_MAX && S.grid.boff && S.grid.eps2 == eps2;
}

void launch_env_points(const Surface& S, const double* P, int64_t n, double eps2, uint8_t* out,
                       int precision, unsigned long long* counters, void* sort_scratch,
                       int sort_knob, void* records, int point_block, cudaStream_t s,
                       cudaEvent_t ev_begin, cudaEvent_t ev_end) {
    if (n <= 0) return;
    const int block = 128;
    const int32_t* order = nullptr;
    uint32_t* recheck = nullptr;
    PointRec* rec = nullptr;
    const uint32_t* n_dev = nullptr;   // sorted queries, when the binning pass decides some
    const EnvTree T = env_tree_for(S, eps2);
    const EpsParams E = eps_params(eps2);
    if (sort_scratch && n >= kSortMin && n <= INT32_MAX) {
        SortLayout L = sort_layout(sort_scratch, n, sort_knob, records == sort_scratch);
        const unsigned nb = (unsigned)((n + 255) / 256);
        const int bits = sort_bits(n, sort_knob);
        if (T.boff && T.bid && sort_knob == 1 && (int64_t)T.nocc + 1 <= L.nbins) {
            // on the dense ids of the bins with entries (a 4-byte count each)
            cudaMemsetAsync(L.count, 0, 4 * ((size_t)T.nocc + 1), s);
            k_point_bins_cid<<<nb, 256, 0, s>>>(P, n, T.blo[0], T.blo[1], T.blo[2], T.binv,
                                                T.bn[0], T.bn[1], T.bn[2], T.bid, L.bin_rank,
                                                L.count, out, counters);
            size_t tb = L.temp_bytes;
            cub::DeviceScan::ExclusiveSum(L.temp, tb, L.count, T.nocc + 1, s);
            n_dev = L.count + T.nocc;
        } else if (T.boff) {
            // on the bin index's own bins (or a coarser Morton prefix of them)
            const int b = std::min(bits, S.grid.bbits);
            cudaMemsetAsync(L.count, 0, 4 * ((size_t)1 << (3 * b)), s);
            k_point_bins_idx<<<nb, 256, 0, s>>>(P, n, T.blo[0], T.blo[1], T.blo[2], T.binv,
                                                T.bn[0], T.bn[1], T.bn[2], S.grid.bbits - b,
                                                L.bin_rank, L.count);
            size_t tb = L.temp_bytes;
            cub::DeviceScan::ExclusiveSum(L.temp, tb, L.count, 1 << (3 * b), s);
        } else {
            double sc[3];
            for (int k = 0; k < 3; ++k) {
                double ext = S.hi[k] - S.lo[k];
                sc[k] = ext > 0.0 ? 1.0 / ext : 0.0;
            }
            cudaMemsetAsync(L.count, 0, 4 * (size_t)L.nbins, s);
            k_point_bins<<<nb, 256, 0, s>>>(P, n, (float)S.lo[0], (float)S.lo[1], (float)S.lo[2],
                                            (float)sc[0], (float)sc[1], (float)sc[2],
                                            std::ldexp(1.0f, bits), L.bin_rank, L.count);
            size_t tb = L.temp_bytes;
            cub::DeviceScan::ExclusiveSum(L.temp, tb, L.count, (int)L.nbins, s);
        }
        if (records && env_points_use_records(S, n, eps2, precision, sort_knob)) {
            rec = L.rec ? L.rec : static_cast<PointRec*>(records);
            k_point_place_rec<<<nb, 256, 0, s>>>(P, L.bin_rank, n, L.count, rec);
        } else {
            k_point_place<<<nb, 256, 0, s>>>(L.bin_rank, n, L.count, L.idx);
            order = L.idx;
        }
        recheck = L.recheck;
    }
    // the tree-walk kernels: at least 6 blocks of 128 threads per SM (85
    // registers), measured best of 1, 6 and 8 on the 10M-point workload (8
    // spills)
    if (ev_begin) cudaEventRecord(ev_begin, s);
    if (T.boff && precision == TW_PRECISION_FP32_CERTIFIED && recheck) {
        // no FP64 code in the bulk kernel (64 registers): 4 blocks of 256 per SM
        // (10M points, gathered: 0.564 ms against 0.592 for 8 of 128, 0.646 for 2
        // of 512, 0.665 for 1 of 1024; from records: 0.39 against 0.49, 0.56 and
        // 0.72 for 5, 6 and 8 blocks of 256)
        cudaMemsetAsync(recheck, 0, 4, s);
        k_env_points_bins<256, 4, true, true><<<grid_for(n, 256, 16), 256, 0, s>>>(
            P, order, n, T, E, out, counters, recheck, n_dev, rec);
        k_env_points_bins_recheck<<<grid_for(INT32_MAX, 128, 4), 128, 0, s>>>(P, recheck, T, E,
                                                                             out, counters);
    } else if (T.boff && precision == TW_PRECISION_FP32_CERTIFIED) {
        k_env_points_bins<384, 2, true, false><<<grid_for(n, 384, 6), 384, 0, s>>>(
            P, order, n, T, E, out, counters, nullptr, n_dev, nullptr);
    } else if (T.boff) {
        k_env_points_bins<384, 2, false, false><<<grid_for(n, 384, 6), 384, 0, s>>>(
            P, order, n, T, E, out, counters, nullptr, n_dev, nullptr);
    } else if (T.gslot && precision == TW_PRECISION_FP32_CERTIFIED) {
        // 768 resident threads per SM (85 registers) in every block shape
        switch (point_block) {
        case 256:
            k_env_points_grid<256, 3, true><<<grid_for(n, 256, 8), 256, 0, s>>>(P, order, n, T,
                                                                               E, out, counters);
            break;
        case 128:
            k_env_points_grid<128, 6, true><<<grid_for(n, 128, 16), 128, 0, s>>>(P, order, n, T,
                                                                                E, out, counters);
            break;
        case 768:
            k_env_points_grid<768, 1, true><<<grid_for(n, 768, 3), 768, 0, s>>>(P, order, n, T,
                                                                               E, out, counters);
            break;
        default:   // 384: measured best of the four on 10M points (1.11 vs 1.15 ms at 128)
            k_env_points_grid<384, 2, true><<<grid_for(n, 384, 6), 384, 0, s>>>(P, order, n, T,
                                                                               E, out, counters);
        }
    } else if (T.gslot) {
        // FP64 through the same sort and grid
        k_env_points_grid<384, 2, false><<<grid_for(n, 384, 6), 384, 0, s>>>(P, order, n, T, E,
                                                                            out, counters);
    }
    else if (precision == TW_PRECISION_FP32_CERTIFIED && order)
        k_env_points_warp<6><<<grid_for(n, block, 16), block, 0, s>>>(P, order, n, T, E, out,
                                                                      counters);
    else if (precision == TW_PRECISION_FP32_CERTIFIED)
        k_env_points<true, 6><<<grid_for(n, block, 16), block, 0, s>>>(P, order, n, T, E, out,
                                                                       counters);
    else
        k_env_points<false><<<grid_for(n, block, 16), block, 0, s>>>(P, order, n, T, E, out,
                                                                     counters);
    if (ev_end) cudaEventRecord(ev_end, s);
}

// ---------------------------------------------------------------------------
// sampleTriangle arithmetic (geogram vec3 semantics, as in the oracle).
// ---------------------------------------------------------------------------
__device__ __forceinline__ V3 vsub(const V3& a, const V3& b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 vadd(const V3& a, const V3& b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 vmul(const V3& a, double s) { return V3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 smul(double s, const V3& a) { return V3{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ V3 vdiv(const V3& a, double s) { return V3{a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ double vlen2(const V3& a) { return (a.x * a.x + a.y * a.y) + a.z * a.z; }
__device__ __forceinline__ double vlen(const V3& a) { return sqrt(vlen2(a)); }
__device__ __forceinline__ double vdist(const V3& a, const V3& b) { return vlen(vsub(a, b)); }
__device__ __forceinline__ V3 vnormalize(const V3& a) {
    double s = vlen(a);
    if (s > 1e-30) s = 1.0 / s;
    return smul(s, a);
}
__device__ __forceinline__ int trunc_int(double x) {
    if (!(x == x)) return 0;
    if (x >= 2147483647.0) return 2147483647;
    if (x <= -2147483648.0) return -2147483647 - 1;
    return (int)x;
}

// The per-face constants of sampleTriangle.  The face's vertices from the
// longest edge on (v0, v1 its ends) are kept apart (FaceVerts): the kernels
// read them from the face itself.  The edge directions are n01, n12 (v1->v2)
// and -n02 (v2->v0).
struct FaceVerts {
    V3 v0, v1, v2;
};
struct SampleHeader {
    V3 n01, n02, n12;
    double N;           // base-row bound after the N == int(N) adjustment
    double sin_v0, tan_v0, sin_v1;
    double NE, NF;      // edge bounds after the N == int(N) adjustment
    int max_i;          // v0 is the face's vertex max_i
    int trivial;        // N <= 1: the three vertices only
    int M;              // number of candidate rows (M < 1: base row, v1, v2 only)
    int8_t hasE, hasF;  // the reference samples an edge only when its raw N > 1
    // sample spacing along v0->v1, v1->v2, v2->v0 and row spacing, each in
    // units of the edge (the row's: of v0->v2)
    float r01, r12, r20, rrow;
};

__device__ __forceinline__ FaceVerts face_verts(const double* t, int max_i) {
    const V3 a{t[0], t[1], t[2]}, b{t[3], t[4], t[5]}, c{t[6], t[7], t[8]};
    return max_i == 0 ? FaceVerts{a, b, c} : max_i == 1 ? FaceVerts{b, c, a} : FaceVerts{c, a, b};
}

__device__ __forceinline__ void sample_header(const double* t, double sd, SampleHeader& h,
                                              FaceVerts& v) {
    const double sqrt3_2 = sqrt(3.0) / 2.0;
    const V3 a{t[0], t[1], t[2]}, b{t[3], t[4], t[5]}, c{t[6], t[7], t[8]};
    const double lab = vlen2(vsub(a, b)), lbc = vlen2(vsub(b, c)), lca = vlen2(vsub(c, a));
    int max_i = 0;
    double l01 = lab, l12 = lbc, l20 = lca;
    if (!(lbc < l01)) {
        max_i = 1;
        l01 = lbc; l12 = lca; l20 = lab;
    }
    if (!(lca < l01)) {
        max_i = 2;
        l01 = lca; l12 = lab; l20 = lbc;
    }
    h.max_i = max_i;
    v = face_verts(t, max_i);
    double N = sqrt(l01) / sd;
    h.trivial = (N <= 1) ? 1 : 0;
    h.M = 0;
    h.r01 = h.r12 = h.r20 = h.rrow = 0.0f;
    if (h.trivial) return;
    h.r01 = 1.0f / d2f_rn(N);
    if (N == (double)trunc_int(N)) N -= 1;
    h.N = N;
    h.n01 = vnormalize(vsub(v.v1, v.v0));
    double hh = vdist(vadd(vdiv(smul(dot3(vsub(v.v2, v.v0), vsub(v.v1, v.v0)), vsub(v.v1, v.v0)),
                               l01),
                          v.v0),
                     v.v2);
    h.M = trunc_int(hh / (sqrt3_2 * sd));
    if (h.M < 1) return;
    h.n02 = vnormalize(vsub(v.v2, v.v0));
    h.n12 = vnormalize(vsub(v.v2, v.v1));
    double cr0 = vlen(cross3(vsub(v.v2, v.v0), vsub(v.v1, v.v0)));
    double cr1 = vlen(cross3(vsub(v.v2, v.v1), vsub(v.v0, v.v1)));
    const double d02 = vdist(v.v0, v.v2), d01 = vdist(v.v0, v.v1);
    h.sin_v0 = cr0 / (d02 * d01);
    h.tan_v0 = cr0 / dot3(vsub(v.v2, v.v0), vsub(v.v1, v.v0));
    h.sin_v1 = cr1 / (vdist(v.v1, v.v2) * d01);
    h.rrow = d2f_rn(sqrt3_2 * sd) / (d2f_rn(h.sin_v0) * d2f_rn(d02));
    double NE = sqrt(l12) / sd;
    h.hasE = NE > 1;
    h.r12 = 1.0f / d2f_rn(NE);
    if (h.hasE && NE == (double)trunc_int(NE)) NE -= 1;
    h.NE = NE;
    double NF = sqrt(l20) / sd;
    h.hasF = NF > 1;
    h.r20 = 1.0f / d2f_rn(NF);
    if (h.hasF && NF == (double)trunc_int(NF)) NF -= 1;
    h.NF = NF;
}

// Row m (1 <= m <= M): start point v, its distance delta_d from the edge
// v0->v2 and last index N1; returns false when the row triggers the
// reference's break (distance(v0_m, v1_m) <= sd).
__device__ __forceinline__ bool sample_row(const SampleHeader& h, const FaceVerts& f, double sd,
                                           int m, V3& v, int& N1, double& delta_d) {
    const double sqrt3_2 = sqrt(3.0) / 2.0;
    int n = trunc_int(sqrt3_2 / h.tan_v0 * m + 0.5);
    int n1 = trunc_int(sqrt3_2 / h.tan_v0 * m);
    if (m % 2 == 0 && n == n1) n += 1;
    V3 v0_m = vadd(f.v0, smul((double)m * sqrt3_2 * sd / h.sin_v0, h.n02));
    V3 v1_m = vadd(f.v1, smul((double)m * sqrt3_2 * sd / h.sin_v1, h.n12));
    if (vdist(v0_m, v1_m) <= sd) return false;
    delta_d = (((double)n + (m % 2) / 2.0) - (double)m * sqrt3_2 / h.tan_v0) * sd;
    v = vadd(v0_m, smul(delta_d, h.n01));
    N1 = trunc_int(vdist(v, v1_m) / sd);
    return true;
}
__device__ __forceinline__ V3 row_point(const SampleHeader& h, const V3& v, double sd, int i) {
    return vadd(v, vmul(smul((double)i, h.n01), sd));
}
__device__ __forceinline__ V3 base_point(const SampleHeader& h, const FaceVerts& f, double sd,
                                         int n) {
    return vadd(f.v0, vmul(vmul(h.n01, sd), (double)n));
}
__device__ __forceinline__ V3 edge_point(const V3& o, const V3& dir, double sd, int n) {
    return vadd(o, vmul(vmul(dir, sd), (double)n));
}
__device__ __forceinline__ V3 vneg(const V3& a) { return V3{-a.x, -a.y, -a.z}; }
// number of integers n with lo <= n <= N (N a double), lo >= 0
__device__ __forceinline__ int count_upto(double N, int lo) {
    if (!(N >= (double)lo)) return 0;
    double f = floor(N);
    if (f > 2147483000.0) f = 2147483000.0;
    return (int)f - lo + 1;
}

// Exact collinearity (Triangle_3f::is_degenerate): the three 2x2 minors of
// [a - c, b - c] vanish.
__device__ __forceinline__ bool minor2_zero(double px, double py, double qx, double qy, double rx,
                                            double ry) {
    double a[2], b[2], c[2], d[2], m[16];
    int na = exp_diff(px, rx, a), nb = exp_diff(qy, ry, b);
    int nc = exp_diff(py, ry, c), nd = exp_diff(qx, rx, d);
    int k = exp_minor(a, na, b, nb, c, nc, d, nd, m);
    return m[k - 1] == 0.0;
}
__device__ __noinline__ bool tri_collinear(const double* t) {
    if (!minor2_zero(t[0], t[1], t[3], t[4], t[6], t[7])) return false;
    if (!minor2_zero(t[0], t[2], t[3], t[5], t[6], t[8])) return false;
    return minor2_zero(t[1], t[2], t[4], t[5], t[7], t[8]);
}

struct FaceCtx {
    EnvTree T;
    EpsParams E;
    unsigned long long* counters;
};

// Largest per-face sample grid the kernel accepts (about 4e6 samples per edge
// row); a larger face would keep one warp busy for seconds, so it is flagged
// as an error instead.
constexpr double kMaxSamplesPerRow = 4.0e6;

__device__ __forceinline__ bool header_too_large(const SampleHeader& h) {
    if (h.trivial) return false;
    if (!(h.N <= kMaxSamplesPerRow)) return true;
    if (h.M > (int)kMaxSamplesPerRow) return true;
    if (h.M >= 1 && h.hasE && !(h.NE <= kMaxSamplesPerRow)) return true;
    if (h.M >= 1 && h.hasF && !(h.NF <= kMaxSamplesPerRow)) return true;
    return false;
}

// Per-lane sample test with the facet hint.
template <bool FP32>
__device__ __forceinline__ bool sample_out(const FaceCtx& F, const V3& p, int32_t& hint,
                                           TravStats& st) {
    if (hint >= 0) {
        ++st.facets;
        if (FP32) {
            int cls = facet_classify(F.T.cull, hint, cert_query(p, F.E, F.T.scale_hi));
            if (cls == kFacetIn) return false;
            if (cls == kFacetBand) {
                ++st.fp64;
                if (leaf_sqdist(F.T.tri, hint, p) <= F.E.eps2) return false;
            }
        } else {
            ++st.fp64;
            if (leaf_sqdist(F.T.tri, hint, p) <= F.E.eps2) return false;
        }
    }
    int32_t f = query_point<FP32>(F.T, p, F.E, st);
    if (f == kTraversalError) {
        atomicOr(F.counters + kCntError, 1ULL);
        return false;
    }
    if (f < 0) return true;
    hint = f;
    return false;
}

// Binary32 box of the face's vertices grown by the largest culling radius of
// any sample (CertQuery::thr with M = the surface's and the face's largest
// coordinate) plus 2^-20 M for the rounding of the sample construction, all
// rounded outward: every sample's binary32 point and everything within its
// culling radius lie inside.
__device__ __forceinline__ void face_query_box(const double* t, const FaceCtx& F, float* qlo,
                                               float* qhi) {
    double m = 0.0;
    for (int k = 0; k < 9; ++k) m = fmax(m, fabs(t[k]));
    const CertQuery q = cert_query(V3{m, m, m}, F.E, F.T.scale_hi);
    const float mu = fmaxf(q.ph[0], F.T.scale_hi);
    const float R = __fadd_ru(__fsqrt_ru(q.thr), __fmul_ru(9.5367431640625e-07f, mu));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double lo = fmin(t[k], fmin(t[3 + k], t[6 + k]));
        const double hi = fmax(t[k], fmax(t[3 + k], t[6 + k]));
        float flo = d2f_rn(lo), fhi = d2f_rn(hi);
        if (f2d_exact(flo) > lo) flo = nextafterf(flo, -__int_as_float(0x7f800000));
        if (f2d_exact(fhi) < hi) fhi = nextafterf(fhi, __int_as_float(0x7f800000));
        qlo[k] = __fsub_rd(flo, R);
        qhi[k] = __fadd_ru(fhi, R);
    }
}

#include "tw_hull.cuh"

constexpr int kProbe = 1 << 20;   // 32 kProbe: more than the samples of a face's rim
// The samples of one face with its header already computed, the whole warp:
// 1 if some sample is out, 0 otherwise.  Samples in a cut known to be inside
// (hull) are passed over; the others collect in the warp's queue (64 words of
// shared memory, as rows_held) and are built and tested 32 at a time, so that the binary64
// construction and the facet tests run on full warps.  slice / slices: the
// warp takes every slices-th step of 32 samples; stop (shared, may be null):
// set by another warp of the face that found a sample out.  With slices = kProbe
// the first 32 samples only.  Out of line: the sampling kernel calls it from two
// places.
// !CUT: no part of the face is known to be inside (no hull, no queue): each step
// of 32 samples is tested as it comes.
template <bool FP32, bool CUT>
__device__ __noinline__ uint8_t env_face_samples(const SampleHeader& h,
                                                    const double* __restrict__ tri,
                                                    const FaceCuts& hull, int k2, uint32_t* queue,
                                                    int32_t* rows_held,
                                                    const FaceCtx& Fr, double sd, int slice,
                                                    int slices, const volatile int* stop,
                                                    TravStats& st, uint32_t& nq) {
    // a copy keeps the tree's pointers in registers for the walk; the cut faces'
    // tests through the grid are as fast without (and the registers short)
    typename std::conditional<CUT, const FaceCtx&, const FaceCtx>::type F = Fr;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    double tv[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) tv[k] = __ldg(tri + k);
    const FaceVerts fv = face_verts(tv, h.max_i);
    int32_t hint = -1;
    // certified mode without a grid: the leaves within reach of the face, shared
    // by the warp (see k_env_points_warp); -1 when above 32 (per-sample walks)
    int32_t cand = -1;
    int cnt = -1, kh = 0;
    if (FP32 && !F.T.gslot) {
        float qlo[3], qhi[3];
        face_query_box(tv, F, qlo, qhi);
        cnt = warp_candidates32(F.T, qlo, qhi, lane, cand);
        if (cnt == kTraversalError) {
            if (lane == 0) atomicOr(F.counters + kCntError, 1ULL);
            cnt = -1;
        }
    }
    // out iff the lane's sample (have) is out; called by the whole warp
    auto lane_out = [&](bool have, const V3& p) -> bool {
        if (F.T.gslot) {
            CertQuery q;
            if (have) q = cert_query(p, F.E, F.T.scale_hi);
            return have && !grid_point_in<FP32>(F.T, F.E, have, p, q, st);
        }
        if (cnt < 0) {
            bool o = false;
            if (have) o = sample_out<FP32>(F, p, hint, st);
            return o;
        }
        bool in = !have;
        CertQuery q;
        if (have) q = cert_query(p, F.E, F.T.scale_hi);
        for (int k = 0; k < cnt; ++k) {
            const int kk = (k + kh) % cnt;
            const int32_t lf = __shfl_sync(0xffffffffu, cand, kk);
            if (!in && cert_leaf_within(F.T.cull, F.T.tri, lf, p, q, F.E.eps2, st)) {
                in = true;
                kh = kk;
            }
            if (__all_sync(0xffffffffu, in)) break;
        }
        return !in;
    };
    // passed over: the sample at v0 + s (v1 - v0) + t (v2 - v0)
    auto inside = [&](float s, float t) -> bool {
        const float r = (1.0f - s) - t;
        return h.max_i == 0   ? hull_inside(hull, k2, s, t)
               : h.max_i == 1 ? hull_inside(hull, k2, r, s)
                              : hull_inside(hull, k2, t, r);
    };
    int qn = 0;
    // tests queued samples in full warps (all: to the last); true when one is out
    auto drain = [&](bool all, auto&& point) -> bool {
        while (qn >= 32 || (all && qn > 0)) {
            const int m = min(qn, 32);
            qn -= m;
            const bool have = lane < m;
            const uint32_t e = have ? queue[qn + lane] : 0u;
            const V3 p = point(have, e);
            const bool o = lane_out(have, p);
            if (have) ++nq;
            if (__any_sync(0xffffffffu, o || (stop && *stop))) return true;
        }
        return false;
    };
    auto push = [&](bool want, uint32_t e) {
        const unsigned bal = __ballot_sync(0xffffffffu, want);
        if (want) queue[qn + __popc(bal & lt)] = e;
        qn += __popc(bal);
        __syncwarp();
    };
    if (h.trivial) {
        const bool have = lane < 3;
        const bool o = lane_out(have, lane == 1 ? fv.v1 : lane == 2 ? fv.v2 : fv.v0);
        if (have) ++nq;
        return __any_sync(0xffffffffu, o) ? 1 : 0;
    }
    // The samples as flat index ranges that the 32 lanes walk in step (the
    // order of the tests changes only the work: the face is out iff some
    // sample is).  First the base row, v1, v2 and the two other edges...
    const int NA = count_upto(h.N, 0);
    const int NE = (h.M >= 1 && h.hasE) ? count_upto(h.NE, 1) : 0;
    const int NF = (h.M >= 1 && h.hasF) ? count_upto(h.NF, 1) : 0;
    const int NX = NA + 2 + NE + NF;
    // !CUT: the lane's sample at once; true when one of the warp's is out
    auto test = [&](bool have, const V3& p) -> bool {
        const bool o = lane_out(have, p);
        if (have) ++nq;
        return __any_sync(0xffffffffu, o || (stop && *stop));
    };
    auto rim = [&](bool have, uint32_t e) -> V3 {
        const int s = (int)e;
        if (!have) return fv.v0;
        if (s < NA) return base_point(h, fv, sd, s);
        if (s == NA) return fv.v1;
        if (s == NA + 1) return fv.v2;
        if (s < NA + 2 + NE) return edge_point(fv.v1, h.n12, sd, s - NA - 1);
        return edge_point(fv.v2, vneg(h.n02), sd, s - NA - 1 - NE);
    };
    for (int s0 = 32 * slice; s0 < NX; s0 += 32 * slices) {
        const int s = s0 + lane;
        if (!CUT) {
            if (test(s < NX, rim(s < NX, (uint32_t)s))) return 1;
            continue;
        }
        float x, y;   // the sample along v0->v1 and v0->v2
        if (s < NA) {
            x = (float)s * h.r01;
            y = 0.0f;
        } else if (s < NA + 2) {
            y = (float)(s - NA);
            x = 1.0f - y;
        } else if (s < NA + 2 + NE) {
            y = (float)(s - NA - 1) * h.r12;
            x = 1.0f - y;
        } else {
            x = 0.0f;
            y = 1.0f - (float)(s - NA - 1 - NE) * h.r20;
        }
        push(s < NX && !inside(x, y), (uint32_t)s);
        if (drain(false, rim)) return 1;
    }
    if (CUT && drain(true, rim)) return 1;
    if (slices == kProbe) return 0;
    // ...then the rows 1..M: those that meet an open cut are listed, and 32 at a
    // time each lane sets up one (start point and last index), the reference's
    // break (a row with distance(v0_m, v1_m) <= sd ends the rows) applies, and
    // the lanes walk their samples by flat index.  Rows shorten by at least sd
    // each (v0 v1 is the longest edge), so only the last two can break, which are
    // always listed: passing over rows never passes over a break.
    int held = 0;
    for (int base = 1; base <= h.M || held > 0; base += 32) {
        if (CUT && base <= h.M) {
            const int m = base + lane;
            const bool want = m <= h.M && (m + 1 >= h.M || hull_row_open(hull, k2, h.max_i,
                                                                         (float)m * h.rrow));
            const unsigned bal = __ballot_sync(0xffffffffu, want);
            if (want) rows_held[held + __popc(bal & lt)] = m;
            held += __popc(bal);
            __syncwarp();
            if (held < 32 && base + 32 <= h.M) continue;
        }
        const int batch = CUT ? min(held, 32) : min(h.M - base + 1, 32);
        int m = base + lane;
        if (CUT) {
            m = lane < batch ? rows_held[lane] : 0;
            // what is left moves to the front (at most 31 entries)
            held -= batch;
            const int rest = lane < held ? rows_held[32 + lane] : 0;
            __syncwarp();
            if (lane < held) rows_held[lane] = rest;
            __syncwarp();
        }
        V3 v{0.0, 0.0, 0.0};
        int N1 = -1;
        double dd = 0.0;
        const bool valid = lane < batch;
        const bool brk = valid && !sample_row(h, fv, sd, m, v, N1, dd);
        const unsigned bal = __ballot_sync(0xffffffffu, brk);
        const int first_brk = bal ? __ffs(bal) - 1 : 32;
        int rows = 0;
        if (valid && lane < first_brk) {
            if (N1 > (int)kMaxSamplesPerRow) {
                atomicOr(F.counters + kCntError, 2ULL);
            } else {
                rows = N1 + 1;
            }
        }
        // the row's first sample along v0->v1 (delta_d in units of the edge), and its
        // place along v0->v2
        const float sx = d2f_rn(dd) / d2f_rn(sd) * h.r01, sy = (float)m * h.rrow;
        int incl = rows;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int excl = incl - rows;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        auto in_row = [&](bool, uint32_t e) -> V3 {   // e: lane of the row << 26 | index (below 2^23)
            const int r = (int)(e >> 26);
            const V3 w{__shfl_sync(0xffffffffu, v.x, r), __shfl_sync(0xffffffffu, v.y, r),
                       __shfl_sync(0xffffffffu, v.z, r)};
            return row_point(h, w, sd, (int)(e & 0x3ffffffu));
        };
        for (int s0 = 32 * slice; s0 < total; s0 += 32 * slices) {
            const int s = s0 + lane;
            // the row holding flat index s: the last lane whose first index is
            // <= s (first indices never decrease; empty rows share the next one's)
            int r = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int c = r + step;
                const int ex = __shfl_sync(0xffffffffu, excl, c & 31);
                if (c < 32 && ex <= s) r = c;
            }
            const int i = s - __shfl_sync(0xffffffffu, excl, r);
            if (!CUT) {
                if (test(s < total, in_row(s < total, ((uint32_t)r << 26) | (uint32_t)max(i, 0))))
                    return 1;
                continue;
            }
            const float x = fmaf((float)i, h.r01, __shfl_sync(0xffffffffu, sx, r));
            const float y = __shfl_sync(0xffffffffu, sy, r);
            push(s < total && !inside(x, y), ((uint32_t)r << 26) | (uint32_t)i);
            if (drain(false, in_row)) return 1;
        }
        if (CUT && drain(true, in_row)) return 1;
        if (bal) break;
    }
    return 0;
}

// Header stage of one face (one thread): 0 = degenerate (not out), 1 = beyond
// the per-row sample bound (error bit 2, counted out), 2 = sample it.  shaped:
// known not to be degenerate (hull_prepare).
__device__ __forceinline__ int face_prepare(const double* t, double sd, bool shaped,
                                            SampleHeader& h, unsigned long long* counters) {
    if (!shaped && tri_collinear(t)) return 0;
    FaceVerts v;
    sample_header(t, sd, h, v);
    if (header_too_large(h)) {
        atomicOr(counters + kCntError, 2ULL);
        return 1;
    }
    return 2;
}

// Faces run in two launches.  The first cuts every face, a warp a face, in
// binary32 only, and answers those that are inside as a whole (0) or have a
// vertex certainly out (1); the others it marks open (kFaceOpen in out).  The
// second samples the open faces: their binary64 headers, one a thread, then a
// face by a warp, which cuts it again, now keeping its open pieces, and tests
// the samples there.  (In one kernel the cut was held to the 16 warps per SM
// of the sampling's 128 registers, and half of its stalls were barriers.)
// Sampling every face in full, as before: 12.4 ms for 300k faces (edges 4e-3
// to 3e-2, eps 1e-3, spacing eps / 2, 100k-facet sphere, certified) and 2.7 ms
// for 20k (edges 0.02 to 0.17, spacing 2.4 eps, binary64); now 2.0 and 0.25.
// Ctx(f, F, sd) gives face f's tree, eps and sampling distance.
constexpr int kFaceBlock = 128;
constexpr int kFaceWarps = kFaceBlock / 32;
constexpr int kCutBlocks = 8, kSampleBlocks = 4;   // blocks per SM
constexpr uint8_t kFaceOpen = 2;
// pieces of the second cut that a sample is worth, at most (300k certified faces:
// 4.1-4.3 ms with 0.3, 2.05 with 0.6, 2.00 with 1.2; 20k binary64 faces: 0.345 ms
// with 0.5, 0.262 with 1.0, 0.27-0.28 with 2.0)
constexpr float kSampleCost32 = 0.6f, kSampleCost64 = 1.0f;

// The warps take tiles of faces from a counter (faces over many small facets
// cost tens of times the others), an eighth of a warp's share each (4 to 32
// faces), so that small batches spread over all SMs and large ones balance; up
// to a face a warp, one each (the call of 8 certified faces of 0.1 eps, 1.5 eps
// out: 59 us with tiles of four, 46 so).
template <bool FP32, class Ctx>
__device__ __forceinline__ void faces_cut(const double* __restrict__ tris, int64_t n,
                                          unsigned long long* counters, Ctx ctx,
                                          uint8_t* __restrict__ out) {
    __shared__ CutTables tab;
    __shared__ FaceFrame frame[kFaceWarps][32];
    fill_cut_tables(tab);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    TravStats st;
    uint32_t nq = 0, nopen = 0;
    const int64_t warps = (int64_t)gridDim.x * kFaceWarps, share = n / (warps * 8);
    const int tile = n <= warps ? 1 : (int)(share < 4 ? 4 : share > 32 ? 32 : share);
    for (;;) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(counters + kCntFaceCut, (unsigned long long)tile);
        const int64_t base = (int64_t)__shfl_sync(0xffffffffu, at, 0);
        if (base >= n) break;
        const int faces = (int)(n - base < tile ? n - base : tile);
        if (lane < faces) {
            FaceCtx F;
            double sd, t[9];
            ctx(base + lane, F, sd);
#pragma unroll
            for (int k = 0; k < 9; ++k) t[k] = __ldg(tris + 9 * (base + lane) + k);
            hull_prepare(t, F.T, F.E, sd, FP32 ? kSampleCost32 : kSampleCost64,
                         frame[warp][lane]);
        }
        __syncwarp();
        int o = kFaceOpen;
        for (int k = 0; k < faces; ++k) {
            const FaceFrame& h = frame[warp][k];
            if (h.k2 < 0) continue;
            FaceCtx F;
            double sd;
            ctx(base + k, F, sd);
            const int r = hull_cut<false>(F.T, F.E, h, tris + 9 * (base + k), tab, nullptr, 0, 1,
                                          st, nq);
            if (lane == k) o = r;
        }
        if (lane < faces) {
            out[base + lane] = (uint8_t)o;
            nopen += o == kFaceOpen;
        }
        __syncwarp();
    }
    nopen = __reduce_add_sync(0xffffffffu, nopen);
    if (lane == 0 && nopen) atomicAdd(counters + kCntFaceOpen, (unsigned long long)nopen);
    flush_stats(st, counters, nq);
}

// Samples of a face from which on the block's warps share it (200k-star pass:
// 10.3-10.8 ms with 128, 9.9 with 384, 9.9-10.1 with 1152; 20k binary64 faces:
// 0.313, 0.262, 0.22).
constexpr int kSharedFace = 384;

// The open faces are sparse and their work differs by orders of magnitude
// (the ideal length against refined edges, samples near a vertex of many
// facets).  Blocks take ranges of faces from a counter, each long enough to
// hold about a quarter of a block's share of the open ones (at most one a
// thread); every thread prepares one of them, the warps take the small ones in
// turn, and then the four warps share the samples and second cuts of each
// large one (a launch otherwise lasts as long as its largest face).  A large
// face that was not cut (its vertices not tested) is probed by one warp first:
// one that is out ends there, where the four would have tested four times the
// samples (8 binary64 faces of 40 sample spacings, 1.5 eps out, no grid: 0.90 ms,
// with that and a block a face 0.32).  !CUT: every face is open (no cutting launch
// ran), and none is shared where each warp has one to itself, since each would walk
// the tree for its candidate leaves; with the cut's queue and hull tests in its
// place 54k such faces took 4.3 ms, 2.6 so (2.7 a face a warp in fixed blocks).
template <bool FP32, bool CUT, class Ctx>
__device__ __forceinline__ void faces_sample(const double* __restrict__ tris, int64_t n,
                                             unsigned long long* counters, Ctx ctx,
                                             uint8_t* __restrict__ out) {
    constexpr bool all = !CUT;
    __shared__ CutTables tab;
    __shared__ FaceFrame frame[kFaceBlock];
    __shared__ SampleHeader head[kFaceBlock];
    __shared__ FaceCuts cuts[kFaceWarps];
    __shared__ uint32_t queue[kFaceWarps][64];
    __shared__ int32_t rows_held[kFaceWarps][64];
    __shared__ uint16_t list[kFaceBlock];
    __shared__ uint8_t small[kFaceBlock], large[kFaceBlock], probe[kFaceBlock];
    __shared__ int held, nsmall, nlarge, next, found;
    __shared__ unsigned long long at;
    const unsigned long long nopen = all ? (unsigned long long)n : counters[kCntFaceOpen];
    if (nopen == 0) return;
    if (!all) fill_cut_tables(tab);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    TravStats st;
    uint32_t nq = 0;
    const int rot = (int)(blockIdx.x / ((gridDim.x + 3) / 4)) % kFaceWarps;
    const bool few = nopen <= gridDim.x, share = !all || nopen <= (unsigned long long)kFaceWarps * gridDim.x;
    const double want = fmin(fmax((double)nopen / (4.0 * gridDim.x), few ? 1.0 : 2.0), (double)kFaceBlock);
    const int range = (int)fmin(want * ((double)n / (double)nopen), 4096.0) + (few ? 0 : 1);
    // a face a block: no counter (which the launch then leaves as it is)
    const bool single = all && n <= (int64_t)gridDim.x;
    for (bool first = true;; first = false) {
        if (threadIdx.x == 0)
            at = !single ? atomicAdd(counters + kCntFaceNext, (unsigned long long)range)
                 : first ? (unsigned long long)blockIdx.x
                         : (unsigned long long)n;
        __syncthreads();
        const int64_t base = (int64_t)at;
        if (base >= n) break;
        const int faces = (int)(n - base < range ? n - base : range);
        int r0 = 0;
        while (r0 < faces) {
            // the next open faces of the range, at most one a thread
            if (threadIdx.x == 0) held = nsmall = nlarge = next = found = 0;
            __syncthreads();
            int before = 0;   // held before this step, the same on every thread
            while (r0 < faces && before <= kFaceBlock - kFaceBlock / 4) {
                // a quarter block of flags a step by each warp in turn would idle
                // the others: all threads read, and stop before the list can overflow
                const int step = min(kFaceBlock - before, faces - r0);
                const int f = r0 + threadIdx.x;
                if ((int)threadIdx.x < step && (all || out[base + f] == kFaceOpen))
                    list[atomicAdd(&held, 1)] = (uint16_t)f;
                r0 += step;
                __syncthreads();
                before = held;
                __syncthreads();
            }
            const int batch = before;
            // one thread a face, from warp `rot` on: the blocks of an SM (a quarter of
            // the grid apart) then put a small batch's binary64 work on different
            // quarters of the SM
            const int mine = (int)((threadIdx.x + kFaceBlock - 32 * rot) % kFaceBlock);
            if (mine < batch) {
                const int64_t f = base + list[mine];
                FaceCtx F;
                double sd, t[9];
                ctx(f, F, sd);
#pragma unroll
                for (int k = 0; k < 9; ++k) t[k] = __ldg(tris + 9 * f + k);
                hull_prepare(t, F.T, F.E, sd, FP32 ? kSampleCost32 : kSampleCost64, frame[mine]);
                SampleHeader& h = head[mine];
                const int state = face_prepare(t, sd, frame[mine].k2 >= 0, h, counters);
                if (state != 2) {
                    out[f] = (uint8_t)state;
                } else {
                    const bool big = share && !h.trivial &&
                                     h.N * (3.0 + 0.5 * (double)h.M) > (double)kSharedFace;
                    probe[mine] = big;
                    if (big) large[atomicAdd(&nlarge, 1)] = (uint8_t)mine;
                    if (!big || frame[mine].k2 < 0) small[atomicAdd(&nsmall, 1)] = (uint8_t)mine;
                }
            }
            __syncthreads();
            for (;;) {
                int j = 0;
                if (lane == 0) j = atomicAdd(&next, 1);
                j = __shfl_sync(0xffffffffu, j, 0);
                if (j >= nsmall) break;
                const int k = small[j];
                const int64_t f = base + list[k];
                const bool big = probe[k];
                FaceCtx F;
                double sd;
                ctx(f, F, sd);
                if (CUT && frame[k].k2 >= 0)
                    hull_cut<true>(F.T, F.E, frame[k], tris + 9 * f, tab, &cuts[warp], 0, 1, st, nq);
                const uint8_t o =
                    env_face_samples<FP32, CUT>(head[k], tris + 9 * f, cuts[warp], frame[k].k2,
                                           queue[warp], rows_held[warp], F, sd, 0,
                                           big ? kProbe : 1, nullptr, st, nq);
                __syncwarp();
                if (lane == 0) {
                    out[f] = o;
                    probe[k] = big && o;   // decided
                }
                __syncwarp();
            }
            for (int j = 0; j < nlarge; ++j) {
                const int k = large[j];
                const int64_t f = base + list[k];
                __syncthreads();   // cuts[0] is free, found is 0, the probes are done
                if (frame[k].k2 < 0 && probe[k]) continue;
                FaceCtx F;
                double sd;
                ctx(f, F, sd);
                if (CUT && frame[k].k2 >= 0)
                    hull_cut<true>(F.T, F.E, frame[k], tris + 9 * f, tab, &cuts[0], warp,
                                   kFaceWarps, st, nq);
                __syncthreads();
                if (env_face_samples<FP32, CUT>(head[k], tris + 9 * f, cuts[0], frame[k].k2,
                                           queue[warp], rows_held[warp], F, sd, warp, kFaceWarps,
                                           &found, st, nq))
                    found = 1;
                __syncthreads();
                if (threadIdx.x == 0) {
                    out[f] = (uint8_t)found;
                    found = 0;
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
    flush_stats(st, counters, nq);
}

// All faces with one tree; n_dev (may be null): the count, known only on the
// device (at most n, for which the grids are sized; warps beyond it exit at once).
struct OneFaceCtx {
    FaceCtx F;
    double sd;
    __device__ __forceinline__ void operator()(int64_t, FaceCtx& Fo, double& sdo) const {
        Fo = F;
        sdo = sd;
    }
};
__device__ __forceinline__ int64_t faces_count(int64_t n, const unsigned long long* n_dev) {
    return n_dev ? (int64_t)min((unsigned long long)n, *n_dev) : n;
}
template <bool FP32>
__global__ void __launch_bounds__(kFaceBlock, kCutBlocks)
    k_env_faces_cut(const double* __restrict__ tris, int64_t n,
                    const unsigned long long* __restrict__ n_dev, OneFaceCtx C,
                    uint8_t* __restrict__ out) {
    faces_cut<FP32>(tris, faces_count(n, n_dev), C.F.counters, C, out);
}
template <bool FP32, bool CUT>
__global__ void __launch_bounds__(kFaceBlock, kSampleBlocks)
    k_env_faces(const double* __restrict__ tris, int64_t n,
                const unsigned long long* __restrict__ n_dev, OneFaceCtx C,
                uint8_t* __restrict__ out) {
    faces_sample<FP32, CUT>(tris, faces_count(n, n_dev), C.F.counters, C, out);
}

// n_dev: nullptr, or the device count of the faces (at most n)
void launch_env_faces_dev(const Surface& S, const double* tris, const unsigned long long* n_dev,
                          int64_t n, double eps2, double sd, uint8_t* out, int precision,
                          unsigned long long* counters, cudaStream_t s) {
    if (n <= 0) return;
    // a surface without a grid cuts no face: the sampling launch takes them all
    const int block = kFaceBlock;
    const int gc = grid_for(n, kFaceWarps, kCutBlocks), gs = grid_for(n, 1, kSampleBlocks);
    const OneFaceCtx C{FaceCtx{env_tree_for(S, eps2), eps_params(eps2), counters}, sd};
    const bool cut = C.F.T.gslot != nullptr;
    if (cut || n_dev || n > gs)
        cudaMemsetAsync(counters + kCntFaceOpen, 0, 3 * sizeof(unsigned long long), s);
    const bool cert = precision == TW_PRECISION_FP32_CERTIFIED;
    if (!cut) {
        auto kernel = cert ? k_env_faces<true, false> : k_env_faces<false, false>;
        kernel<<<gs, block, 0, s>>>(tris, n, n_dev, C, out);
    } else if (cert) {
        k_env_faces_cut<true><<<gc, block, 0, s>>>(tris, n, n_dev, C, out);
        k_env_faces<true, true><<<gs, block, 0, s>>>(tris, n, n_dev, C, out);
    } else {
        k_env_faces_cut<false><<<gc, block, 0, s>>>(tris, n, n_dev, C, out);
        k_env_faces<false, true><<<gs, block, 0, s>>>(tris, n, n_dev, C, out);
    }
}

void launch_env_faces(const Surface& S, const double* tris, int64_t n, double eps2, double sd,
                      uint8_t* out, int precision, unsigned long long* counters, cudaStream_t s) {
    launch_env_faces_dev(S, tris, nullptr, n, eps2, sd, out, precision, counters, s);
}

// ---------------------------------------------------------------------------
// Several jobs in one launch (the serving loop): query i belongs to the last
// segment whose begin is <= i; each segment names its job's tree and eps.
// ---------------------------------------------------------------------------
struct EnvSeg {
    int64_t begin;
    EnvTree T;
    EpsParams E;
    double sd;
};

size_t env_seg_bytes() { return sizeof(EnvSeg); }

void fill_env_seg(void* dst, const Surface& S, int64_t begin, double eps2, double sd) {
    EnvSeg g;
    g.begin = begin;
    g.T = env_tree_for(S, eps2);
    g.E = eps_params(eps2);
    g.sd = sd;
    std::memcpy(dst, &g, sizeof g);
}

__device__ __forceinline__ int find_seg(const EnvSeg* __restrict__ segs, int nsegs, int64_t i) {
    int lo = 0, hi = nsegs - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(&segs[mid].begin) <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <bool FP32>
__global__ void __launch_bounds__(128) k_env_points_segs(const double* __restrict__ P, int64_t n,
                                                         const EnvSeg* __restrict__ segs, int nsegs,
                                                         uint8_t* __restrict__ out,
                                                         unsigned long long* __restrict__ counters) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    TravStats st;
    uint32_t nq = 0;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t base0 = first - (threadIdx.x & 31);
    for (int64_t b = base0; b < n; b += stride) {
        const int64_t i = b + (threadIdx.x & 31);
        if (i < n) {
            const EnvSeg& g = segs[find_seg(segs, nsegs, i)];
            const EnvTree T = g.T;
            const EpsParams E = g.E;
            V3 p{__ldg(P + 3 * i), __ldg(P + 3 * i + 1), __ldg(P + 3 * i + 2)};
            if (T.gslot) {
                const CertQuery q = cert_query(p, E, T.scale_hi);
                out[i] = (uint8_t)!index_point_in<FP32>(T, E, true, p, q, st);
            } else {
                int32_t f = query_point<FP32>(T, p, E, st);
                if (f == kTraversalError) atomicOr(counters + kCntError, 1ULL);
                out[i] = (uint8_t)(f == -1);
            }
            ++nq;
        }
    }
    flush_stats(st, counters, nq);
}

struct SegFaceCtx {
    const EnvSeg* segs;
    int nsegs;
    unsigned long long* counters;
    __device__ __forceinline__ void operator()(int64_t f, FaceCtx& Fo, double& sdo) const {
        const EnvSeg& g = segs[find_seg(segs, nsegs, f)];
        Fo = FaceCtx{g.T, g.E, counters};
        sdo = g.sd;
    }
};
template <bool FP32>
__global__ void __launch_bounds__(kFaceBlock, kCutBlocks)
    k_env_faces_segs_cut(const double* __restrict__ tris, int64_t n, SegFaceCtx C,
                         uint8_t* __restrict__ out) {
    faces_cut<FP32>(tris, n, C.counters, C, out);
}
template <bool FP32>
__global__ void __launch_bounds__(kFaceBlock, kSampleBlocks)
    k_env_faces_segs(const double* __restrict__ tris, int64_t n, SegFaceCtx C,
                     uint8_t* __restrict__ out) {
    faces_sample<FP32, true>(tris, n, C.counters, C, out);
}

void launch_env_points_segs(const double* P, int64_t n, const void* segs, int nsegs, uint8_t* out,
                            int precision, unsigned long long* counters, cudaStream_t s) {
    if (n <= 0 || nsegs <= 0) return;
    const int block = 128;
    const int grid = grid_for(n, block, 6);
    const EnvSeg* g = static_cast<const EnvSeg*>(segs);
    if (precision == TW_PRECISION_FP32_CERTIFIED)
        k_env_points_segs<true><<<grid, block, 0, s>>>(P, n, g, nsegs, out, counters);
    else
        k_env_points_segs<false><<<grid, block, 0, s>>>(P, n, g, nsegs, out, counters);
}

void launch_env_faces_segs(const double* tris, int64_t n, const void* segs, int nsegs, uint8_t* out,
                           int precision, unsigned long long* counters, cudaStream_t s) {
    if (n <= 0 || nsegs <= 0) return;
    const int block = kFaceBlock;
    const int gc = grid_for(n, kFaceWarps, kCutBlocks), gs = grid_for(n, 1, kSampleBlocks);
    cudaMemsetAsync(counters + kCntFaceOpen, 0, 3 * sizeof(unsigned long long), s);
    const SegFaceCtx C{static_cast<const EnvSeg*>(segs), nsegs, counters};
    if (precision == TW_PRECISION_FP32_CERTIFIED) {
        k_env_faces_segs_cut<true><<<gc, block, 0, s>>>(tris, n, C, out);
        k_env_faces_segs<true><<<gs, block, 0, s>>>(tris, n, C, out);
    } else {
        k_env_faces_segs_cut<false><<<gc, block, 0, s>>>(tris, n, C, out);
        k_env_faces_segs<false><<<gs, block, 0, s>>>(tris, n, C, out);
    }
}

// ---------------------------------------------------------------------------
// Nearest facet (MeshFacetsAABBWithEps::nearest_facet, mesh_AABB.h:130-141,
// mesh_AABB.cpp:381-480): the facet with the smallest computed squared
// distance and its closest point; equal distances go to the smallest input
// facet index.  A child box is skipped only when its squared distance exceeds
// (b + tau)^2, b = sqrt(best so far), tau = 64 * 2^-53 * max|coord| +
// 16 * 2^-53 * b, so no facet that could tie or beat the best is skipped and
// the result is the exact minimum over all facets, independent of the tree.
// Returns the input facet index, or kTraversalError.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double nearest_threshold(double best, double m) {
    if (!(best < INFINITY)) return INFINITY;
    double b = sqrt(best);
    double tau = 64.0 * kEps * m + 16.0 * kEps * b;
    return (b + tau) * (b + tau);
}

__device__ __forceinline__ void nearest_leaf(const EnvTree& T, int32_t leaf, const V3& p,
                                             double& best, int32_t& best_id, V3& best_q) {
    const double* t = T.tri + 9 * (int64_t)leaf;
    V3 a{__ldg(t + 0), __ldg(t + 1), __ldg(t + 2)};
    V3 b{__ldg(t + 3), __ldg(t + 4), __ldg(t + 5)};
    V3 c{__ldg(t + 6), __ldg(t + 7), __ldg(t + 8)};
    V3 q;
    double d = point_tri_nearest(p, a, b, c, q);
    int32_t id = __ldg(T.facet_id + leaf);
    if (d < best || (d == best && id < best_id)) {
        best = d;
        best_id = id;
        best_q = q;
    }
}

__device__ int32_t nearest_facet(const EnvTree& T, const V3& p, V3& q, double& sqd) {
    double m = T.scale;
    m = fmax(m, fabs(p.x));
    m = fmax(m, fabs(p.y));
    m = fmax(m, fabs(p.z));
    double best = INFINITY;
    int32_t best_id = 0x7fffffff;
    V3 best_q{0.0, 0.0, 0.0};
    const int32_t nf = T.nf;
    if (nf == 1) {
        nearest_leaf(T, 0, p, best, best_id, best_q);
        q = best_q;
        sqd = best;
        return best_id;
    }
    int32_t stack[kStack];
    double sdist[kStack];
    int sp = 0;
    int32_t cur = 0;
    for (int32_t iter = 0; iter < 2 * nf; ++iter) {
        if ((uint32_t)cur >= (uint32_t)(nf - 1)) return kTraversalError;
        const double2* nd = reinterpret_cast<const double2*>(T.nodes + cur);
        double2 q0 = __ldg(nd + 0), q1 = __ldg(nd + 1), q2 = __ldg(nd + 2);
        double2 q3 = __ldg(nd + 3), q4 = __ldg(nd + 4), q5 = __ldg(nd + 5);
        int2 ch = __ldg(reinterpret_cast<const int2*>(nd + 6));
        double lo0[3] = {q0.x, q0.y, q1.x}, hi0[3] = {q1.y, q2.x, q2.y};
        double lo1[3] = {q3.x, q3.y, q4.x}, hi1[3] = {q4.y, q5.x, q5.y};
        double d0 = point_box_sqdist(p, lo0, hi0);
        double d1 = point_box_sqdist(p, lo1, hi1);
        // nearer child first
        int32_t cn = ch.x, cf = ch.y;
        double dn = d0, df = d1;
        if (d1 < d0) {
            cn = ch.y; cf = ch.x;
            dn = d1; df = d0;
        }
        bool hn = dn <= nearest_threshold(best, m);
        if (hn && cn < 0) {
            if ((uint32_t)(~cn) >= (uint32_t)nf) return kTraversalError;
            nearest_leaf(T, ~cn, p, best, best_id, best_q);
            hn = false;
        }
        bool hf = df <= nearest_threshold(best, m);
        if (hf && cf < 0) {
            if ((uint32_t)(~cf) >= (uint32_t)nf) return kTraversalError;
            nearest_leaf(T, ~cf, p, best, best_id, best_q);
            hf = false;
        }
        if (hn && hf) {
            if (sp >= kStack) return kTraversalError;
            stack[sp] = cf;
            sdist[sp] = df;
            ++sp;
            cur = cn;
        } else if (hn) {
            cur = cn;
        } else if (hf) {
            cur = cf;
        } else {
            // pop the next subtree still within reach of the best distance
            cur = -1;
            while (sp > 0) {
                --sp;
                if (sdist[sp] <= nearest_threshold(best, m)) {
                    cur = stack[sp];
                    break;
                }
            }
            if (cur < 0) {
                q = best_q;
                sqd = best;
                return best_id;
            }
        }
    }
    return kTraversalError;
}

// The nearest facet through the envelope grid: the minimum over the leaves of
// the point's cell.  When that minimum is <= eps2 it is the minimum over all
// facets (every facet within eps of the point is in the cell's list, see
// EnvGrid), ties included; otherwise it returns false and the tree decides.
// Only leaves that may attain the minimum take the binary64 distance: with
// the certified bounds L, U of the exact distances, and 16 u64 M the most a
// computed distance is off, a leaf whose L exceeds the least U by 32 u64 M
// cannot (2^-18 covers the binary32 sums, as in facet_classify).  Of the two to
// three leaves of a cell one is left, mostly: 100k projections 1.36 -> 0.49 ms.
__device__ __forceinline__ bool nearest_facet_grid(const EnvTree& T, double eps2, const V3& p,
                                                   V3& q, double& sqd, int32_t& fid) {
    if (!T.gslot) return false;
    const CertQuery cq = cert_query(p, EpsParams{0.0, 0.0f, 0.0f}, T.scale_hi);
    uint32_t b, e;
    grid_cell_range(T, cq, b, e);
    float umin = __int_as_float(0x7f800000), L2, U2;
    if (e - b > 1) {
        for (uint32_t k = b; k < e; ++k) {
            facet_bounds(T.cull, __ldg(T.glist + k), cq, L2, U2);
            umin = fminf(umin, U2);
        }
    }
    // slack = 16 u64 M = Mu2 / 32 (Mu2 = 16 u^2 M, u64 = u^2 / 32); from 1e-35 on
    // what a bound's squares lose to underflow, below 2^-147, is far inside the 2^-18
    const float t = __fmul_ru(__fadd_ru(__fsqrt_ru(umin), cq.Mu2), 1.00000381f);
    const float lim = fmaxf(__fmul_ru(t, t), 1e-35f);
    double best = INFINITY;
    int32_t best_id = 0x7fffffff;
    V3 best_q{0.0, 0.0, 0.0};
    for (uint32_t k = b; k < e; ++k) {
        const int32_t lf = __ldg(T.glist + k);
        if (e - b > 1) {
            facet_bounds(T.cull, lf, cq, L2, U2);
            if (L2 > lim) continue;
        }
        nearest_leaf(T, lf, p, best, best_id, best_q);
    }
    if (!(best <= eps2)) return false;
    q = best_q;
    sqd = best;
    fid = best_id;
    return true;
}

__global__ void k_nearest_points(EnvTree T, double eps2, const double* __restrict__ P, int64_t n,
                                 double* __restrict__ Q, double* __restrict__ D,
                                 int32_t* __restrict__ Fo, unsigned long long* __restrict__ counters) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        V3 p{__ldg(P + 3 * i), __ldg(P + 3 * i + 1), __ldg(P + 3 * i + 2)};
        V3 q;
        double d;
        int32_t f;
        if (!nearest_facet_grid(T, eps2, p, q, d, f)) f = nearest_facet(T, p, q, d);
        if (f == kTraversalError) {
            atomicOr(counters + kCntError, 1ULL);
            q = p;
            d = 0.0;
            f = -1;
        }
        if (Q) {
            Q[3 * i] = q.x;
            Q[3 * i + 1] = q.y;
            Q[3 * i + 2] = q.z;
        }
        if (D) D[i] = d;
        if (Fo) Fo[i] = f;
    }
}

void free_env_grid(tw_ctx* c, EnvGrid& G) {
    if (G.slot) dev_free(c, G.slot, G.slot_bytes);
    if (G.list) dev_free(c, G.list, G.list_bytes);
    if (G.boff) dev_free(c, G.boff, G.boff_bytes);
    if (G.bent) dev_free(c, G.bent, G.bent_bytes);
    if (G.bid) dev_free(c, G.bid, G.bid_bytes);
    G = EnvGrid{};
}

namespace {
// Device blocks of a build, released on every exit path unless kept.
struct BuildScratch {
    tw_ctx* c;
    std::vector<std::pair<void*, size_t>> blocks;
    void* get(size_t bytes, int& st) {
        void* p = nullptr;
        st = dev_alloc(c, bytes, &p);
        if (st == TW_OK) blocks.emplace_back(p, bytes);
        return p;
    }
    void keep() { blocks.clear(); }
    void release() {
        for (auto& b : blocks) dev_free(c, b.first, b.second);
        blocks.clear();
    }
    ~BuildScratch() { release(); }
};
// Offsets of the parts of one allocation.
struct Parts {
    size_t at = 0;
    size_t add(size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) & ~size_t(255);
        return o;
    }
};

// The grid of cells cs over the box grown by Rm: origin rounded down to
// binary32 and cells a side; false when it cannot be had below the limit (cs
// grows by `step` until good(n)).
template <class Good>
bool fit_grid(const Surface& S, double Rm, double cs, double step, Good good, float* lo, int64_t* n,
              float& inv) {
    for (int iter = 0; iter < 64; ++iter) {
        inv = (float)(1.0 / cs);
        for (int k = 0; k < 3; ++k) {
            const double a = S.box_lo[k] - Rm;
            float f = (float)a;
            if ((double)f > a) f = std::nextafter(f, -INFINITY);
            lo[k] = f;
            n[k] = (int64_t)std::floor((S.box_hi[k] + Rm - (double)f) * (double)inv) + 2;
        }
        if (good(n)) break;
        cs *= step;
    }
    return good(n);
}
}  // namespace

// The envelope grid (EnvGrid) of a surface for eps2, and its bin index
// (EnvGrid::boff, bent): bins of side c->bin_cell x the mean facet extent, but
// at least 1/250 of the grown box's largest side (at most 256 bins a side).
// Each is left absent when unsuitable: a leaf over too many cells or bins,
// more than 2^27 entries.  Both are counted together, filled and sorted on
// the cell or bin alone (the leaves are emitted in order and the radix sorts
// are stable, so a cell's leaves stay ascending); the host waits three times
// (the entry counts, the distinct cells, the end), and the temporaries are
// two allocations: opening a 100k-facet surface took 19.4 ms, now 3.5.
int build_env_grid(tw_ctx* c, Surface& S, double eps2, double cell_factor, cudaStream_t s) {
    if (S.nf <= 0 || !(eps2 >= 0.0)) return TW_OK;
    if (S.grid.slot && S.grid.eps2 == eps2 && S.grid.cell_factor == cell_factor &&
        S.grid.bin_factor == c->bin_cell)
        return TW_OK;
    free_env_grid(c, S.grid);
    const int32_t nf = S.nf;
    // culling radius of any point of the grown box, plus the cell-index margin
    const double eps = std::sqrt(eps2);
    double M = S.scale, ext = 0.0;
    for (int k = 0; k < 3; ++k)
        M = std::max(M, std::max(std::fabs(S.box_lo[k]), std::fabs(S.box_hi[k])));
    M = M + 2.0 * eps + 1e-300;
    const double Rm = eps * (1.0 + std::ldexp(1.0, -18)) + std::ldexp(M, -17);
    const double slack = std::ldexp(M, -30);
    for (int k = 0; k < 3; ++k) ext = std::max(ext, S.box_hi[k] - S.box_lo[k] + 2.0 * Rm);
    float lo[3], blo[3], inv = 0.0f, binv = 0.0f;
    int64_t n[3], bn[3];
    if (!fit_grid(S, Rm, std::max(cell_factor * S.mean_extent, 2.0 * Rm), 1.25,
                  [](const int64_t* m) { return m[0] * m[1] * m[2] < (int64_t(1) << 31); }, lo, n,
                  inv))
        return TW_OK;   // the tree walk serves
    const double bcs = std::max(c->bin_cell * S.mean_extent, ext / 250.0);
    bool bins = c->bin_cell > 0.0 && bcs > 0.0 && std::isfinite(bcs) &&
                fit_grid(S, Rm, bcs, 1.01,
                         [](const int64_t* m) { return std::max(m[0], std::max(m[1], m[2])) <= 256; },
                         blo, bn, binv);
    const SatGrid G = sat_grid(lo, n, (double)inv, Rm, slack);
    SatGrid GB{}, GF{};
    int bits = 0;
    if (bins) {
        GB = sat_grid(blo, bn, (double)binv, Rm, slack);
        const int64_t fine[3] = {kFine * bn[0], kFine * bn[1], kFine * bn[2]};
        GF = sat_grid(blo, fine, (double)kFine * (double)binv, Rm, slack);
        while ((int64_t(1) << bits) < std::max(bn[0], std::max(bn[1], bn[2]))) ++bits;
    }
    const int64_t nmorton = int64_t(1) << (3 * bits);

    // counts per leaf (nf + 1 entries, the last 0) and their exclusive sums
    BuildScratch B{c, {}};
    int st = TW_OK;
    size_t tb_scan = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb_scan, (uint32_t*)nullptr, (uint32_t*)nullptr, nf + 1,
                                  s);
    Parts P;
    const size_t nfb = 4 * ((size_t)nf + 1);
    // acc: [0] grid entries, [1] unsuitable, [2] bin entries, [3] unsuitable,
    // [4] distinct cells, [5] insert failure, [6] bins with entries
    const size_t o_acc = P.add(64), o_cnt = P.add(nfb), o_off = P.add(nfb), o_bcnt = P.add(nfb),
                 o_boff = P.add(nfb), o_tmp = P.add(tb_scan + 16);
    char* q = (char*)B.get(P.at, st);
    if (st != TW_OK) return st;
    unsigned long long* acc = (unsigned long long*)(q + o_acc);
    uint32_t *fcnt = (uint32_t*)(q + o_cnt), *foff = (uint32_t*)(q + o_off);
    uint32_t *bfcnt = (uint32_t*)(q + o_bcnt), *bfoff = (uint32_t*)(q + o_boff);
    const unsigned leaf_grid = (unsigned)(((int64_t)nf + 31) / 32);   // 32 leaves a block
    cudaMemsetAsync(acc, 0, 64, s);
    cudaMemsetAsync(fcnt + nf, 0, 4, s);
    cudaMemsetAsync(bfcnt + nf, 0, 4, s);
    k_cells_count<<<leaf_grid, kSatBlock, 0, s>>>(S.tri, nf, G, kMaxLeafCells, acc, fcnt,
                                                  (int*)(acc + 1));
    if (bins)
        k_cells_count<<<leaf_grid, kSatBlock, 0, s>>>(S.tri, nf, GB, kMaxLeafBins, acc + 2, bfcnt,
                                                      (int*)(acc + 3));
    unsigned long long hacc[8] = {0};
    cudaMemcpyAsync(hacc, acc, 64, cudaMemcpyDeviceToHost, s);
    cub::DeviceScan::ExclusiveSum(q + o_tmp, tb_scan, fcnt, foff, nf + 1, s);
    if (bins) cub::DeviceScan::ExclusiveSum(q + o_tmp, tb_scan, bfcnt, bfoff, nf + 1, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(c, e, "grid build");
    auto suitable = [](unsigned long long total, unsigned long long flag) {
        return (flag & 0xffffffffULL) == 0 && total > 0 && total <= (1ULL << 27);
    };
    if (!suitable(hacc[0], hacc[1])) return TW_OK;   // the tree walk serves
    bins = bins && suitable(hacc[2], hacc[3]);
    const int64_t nt = (int64_t)hacc[0], bt = bins ? (int64_t)hacc[2] : 0;

    // what stays; the bin index apart, which gives way to the grid where memory
    // does not suffice for both (the call then ends with that error, the grid
    // built and the bins left out)
    BuildScratch K{c, {}}, KB{c, {}};
    int st_bins = TW_OK;
    auto drop_bins = [&]() {
        st_bins = st;
        st = TW_OK;
        bins = false;
        KB.release();
    };
    const size_t list_bytes = 4 * (size_t)nt + 16, off_bytes = 4 * ((size_t)nmorton + 1),
                 ent_bytes = 4 * (size_t)(kFineWords + 1) * (size_t)bt, bid_bytes = 4 * (size_t)nmorton;
    int32_t* list = (int32_t*)K.get(list_bytes, st);
    if (st != TW_OK) return st;
    uint32_t *boff = nullptr, *bent = nullptr;
    int32_t* bid = nullptr;
    if (bins) {
        boff = (uint32_t*)KB.get(off_bytes, st);
        if (st == TW_OK) bent = (uint32_t*)KB.get(ent_bytes, st);
        if (st == TW_OK) bid = (int32_t*)KB.get(bid_bytes, st);
        if (st != TW_OK) drop_bins();
    }
    // the temporaries: the grid's (pairs twice, start) and the bins' (keys,
    // vals twice, leaves, masks, counts) follow one another in time
    int cell_bits = 0;
    while (cell_bits < 32 && (int64_t(1) << cell_bits) < n[0] * n[1] * n[2]) ++cell_bits;
    size_t tb = 0, tb_bins = 0, tbk = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, tbk, (unsigned long long*)nullptr,
                                   (unsigned long long*)nullptr, (int)nt, 32, 32 + cell_bits, s);
    tb = std::max(tb, tbk);
    cub::DeviceRunLengthEncode::Encode(nullptr, tbk, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                       (uint32_t*)nullptr, (int*)nullptr, (int)nt, s);
    tb = std::max(tb, tbk);
    cub::DeviceScan::ExclusiveSum(nullptr, tbk, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)nt, s);
    tb = std::max(tb, tbk);
    if (bins) {
        cub::DeviceRadixSort::SortPairs(nullptr, tbk, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                        (uint32_t*)nullptr, (uint32_t*)nullptr, (int)bt, 0,
                                        std::max(1, 3 * bits), s);
        tb_bins = std::max(tb_bins, tbk);
        cub::DeviceScan::ExclusiveSum(nullptr, tbk, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                      (int)(nmorton + 1), s);
        tb_bins = std::max(tb_bins, tbk);
        cub::DeviceScan::ExclusiveSum(nullptr, tbk, (int32_t*)nullptr, (int32_t*)nullptr,
                                      (int)nmorton, s);
        tb_bins = std::max(tb_bins, tbk);
    }
    Parts T;
    const size_t o_temp = T.add(tb + 16);
    const size_t o_pairs = T.add(8 * (size_t)nt), o_pairs2 = T.add(8 * (size_t)nt),
                 o_start = T.add(4 * (size_t)nt + 16);
    Parts TB;
    TB.add(tb_bins + 16);   // at o_temp too
    const size_t bb = 4 * (size_t)bt, o_k = TB.add(bb), o_k2 = TB.add(bb), o_v = TB.add(bb),
                 o_v2 = TB.add(bb), o_lf = TB.add(bb), o_m = TB.add(kFineWords * bb),
                 o_bc = TB.add(off_bytes);
    char* w = (char*)B.get(std::max(T.at, bins ? TB.at : 0), st);
    if (st != TW_OK && bins) {
        drop_bins();
        w = (char*)B.get(T.at, st);
    }
    if (st != TW_OK) return st;
    void* temp = w + o_temp;

    unsigned long long *pairs = (unsigned long long*)(w + o_pairs),
                       *pairs2 = (unsigned long long*)(w + o_pairs2);
    k_grid_cells<<<leaf_grid, kSatBlock, 0, s>>>(S.tri, nf, G, foff, pairs);
    size_t t1 = tb;
    cub::DeviceRadixSort::SortKeys(temp, t1, pairs, pairs2, (int)nt, 32, 32 + cell_bits, s);
    // the entry cells (into the unsorted buffer) and the final leaf list; the
    // distinct cells, their counts and first entries (in the sorted one, read by then)
    uint32_t *ecell = (uint32_t*)pairs, *uniq = (uint32_t*)pairs2, *cnt = uniq + nt,
             *start = (uint32_t*)(w + o_start);
    int* d_nuniq = (int*)(acc + 4);
    int* d_failed = (int*)(acc + 5);
    k_grid_split<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(pairs2, nt, ecell, list);
    t1 = tb;
    cub::DeviceRunLengthEncode::Encode(temp, t1, ecell, uniq, cnt, d_nuniq, (int)nt, s);
    int nuniq = 0;
    cudaMemcpyAsync(&nuniq, d_nuniq, 4, cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(c, e, "grid build");
    if (nuniq <= 0) return TW_OK;
    t1 = tb;
    cub::DeviceScan::ExclusiveSum(temp, t1, cnt, start, nuniq, s);
    // the hash table: a power of two at least twice the distinct cells
    uint32_t hbits = 1;
    while ((1ULL << hbits) < 2ULL * (unsigned long long)nuniq) ++hbits;
    const size_t H = size_t(1) << hbits;
    uint4* slots = (uint4*)K.get(16 * H, st);
    if (st != TW_OK && bins) {
        drop_bins();
        slots = (uint4*)K.get(16 * H, st);
    }
    if (st != TW_OK) return st;
    cudaMemsetAsync(slots, 0xff, 16 * H, s);
    k_grid_insert<<<(unsigned)((nuniq + 255) / 256), 256, 0, s>>>(
        uniq, cnt, start, d_nuniq, slots, 32 - hbits, (uint32_t)(H - 1), d_failed);

    if (bins) {
        uint32_t *keys = (uint32_t*)(w + o_k), *keys2 = (uint32_t*)(w + o_k2),
                 *vals = (uint32_t*)(w + o_v), *vals2 = (uint32_t*)(w + o_v2),
                 *leaves = (uint32_t*)(w + o_lf), *masks = (uint32_t*)(w + o_m),
                 *bcnt = (uint32_t*)(w + o_bc);
        k_bin_cells<<<leaf_grid, kSatBlock, 0, s>>>(S.tri, nf, GB, bfoff, keys, vals, leaves);
        k_bin_masks<<<leaf_grid, kSatBlock, 0, s>>>(S.tri, nf, GF, bfoff, keys, masks);
        t1 = tb_bins;
        cub::DeviceRadixSort::SortPairs(temp, t1, keys, keys2, vals, vals2, (int)bt, 0,
                                        std::max(1, 3 * bits), s);
        cudaMemsetAsync(bcnt, 0, off_bytes, s);
        k_bin_split<<<(unsigned)((bt + 255) / 256), 256, 0, s>>>(keys2, vals2, masks, leaves, bt,
                                                                 bent, bcnt);
        t1 = tb_bins;
        cub::DeviceScan::ExclusiveSum(temp, t1, bcnt, boff, (int)(nmorton + 1), s);
        // the dense ids of the bins with entries, for the point sort
        const unsigned gm = (unsigned)((nmorton + 255) / 256);
        k_bin_flags<<<gm, 256, 0, s>>>(boff, nmorton, bid);
        t1 = tb_bins;
        cub::DeviceScan::ExclusiveSum(temp, t1, bid, bid, (int)nmorton, s);
        k_bin_ids<<<gm, 256, 0, s>>>(boff, nmorton, bid, (int32_t*)(acc + 6));
    }
    cudaMemcpyAsync(hacc, acc, 64, cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);   // the temporaries are released on return
    if (e != cudaSuccess) return cuda_fail(c, e, "grid build");
    if ((hacc[5] & 0xffffffffULL) != 0) return TW_OK;
    K.keep();
    KB.keep();
    EnvGrid& g = S.grid;
    for (int k = 0; k < 3; ++k) {
        g.lo[k] = lo[k];
        g.n[k] = (int32_t)n[k];
    }
    g.inv_c = inv;
    g.slot = slots;
    g.shift = 32 - hbits;
    g.mask = (uint32_t)(H - 1);
    g.list = list;
    g.eps2 = eps2;
    g.cell_factor = cell_factor;
    g.slot_bytes = 16 * H;
    g.list_bytes = list_bytes;
    g.bin_factor = c->bin_cell;   // built for it, or found unsuitable
    if (!bins) return st_bins;
    for (int k = 0; k < 3; ++k) {
        g.blo[k] = blo[k];
        g.bn[k] = (int32_t)bn[k];
    }
    g.binv = binv;
    g.bbits = bits;
    g.boff = boff;
    g.bent = bent;
    g.bnt = bt;
    g.bid = bid;
    g.nocc = (int32_t)(hacc[6] & 0xffffffffULL);
    g.boff_bytes = off_bytes;
    g.bent_bytes = ent_bytes;
    g.bid_bytes = bid_bytes;
    return TW_OK;
}

// Point checks of candidate collapses (EdgeCollapser.cpp:286-329): the
// degenerate-edge flag, then v2 against the boundary envelope when v1 is on
// the boundary and v2 is not, and against the envelope when v1 is on the
// surface and v2 is not.  ENVELOP (3) or kCollapsePending.
template <bool FP32>
__global__ void k_collapse_points(EnvTree Tin, EnvTree Tb, EpsParams E,
                                  const double* __restrict__ vx, const double* __restrict__ vy,
                                  const double* __restrict__ vz, const int32_t* __restrict__ v12,
                                  const uint8_t* __restrict__ flags, int32_t n,
                                  uint8_t* __restrict__ status, uint8_t* __restrict__ degenerate,
                                  unsigned long long* __restrict__ counters) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    TravStats st;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int32_t v1 = v12[2 * i], v2 = v12[2 * i + 1];
        const double dx = vx[v1] - vx[v2], dy = vy[v1] - vy[v2], dz = vz[v1] - vz[v2];
        const bool deg = sqrt((dx * dx + dy * dy) + dz * dz) == 0.0;
        degenerate[i] = deg;
        const uint8_t fl = flags[i];
        const V3 p{vx[v2], vy[v2], vz[v2]};
        uint8_t res = kCollapsePending;
        for (int pass = 0; pass < 2 && res == kCollapsePending; ++pass) {
            const bool bnd = pass == 0;
            const uint8_t need = bnd ? TW_CV_V1_BOUNDARY : TW_CV_V1_SURFACE;
            const uint8_t has = bnd ? TW_CV_V2_BOUNDARY : TW_CV_V2_SURFACE;
            if (!(fl & need) || (fl & has) || deg) continue;
            const EnvTree& T = bnd ? Tb : Tin;
            if (T.nf <= 0) {
                atomicOr(counters + kCntError, 4ULL);
                res = 3;
                break;
            }
            int32_t f;
            if (T.gslot) {
                const CertQuery q = cert_query(p, E, T.scale_hi);
                f = grid_point_in<FP32>(T, E, true, p, q, st) ? 0 : -1;
            } else {
                f = query_point<FP32>(T, p, E, st);
            }
            if (f == kTraversalError) atomicOr(counters + kCntError, 1ULL);
            if (f == -1) res = 3;
        }
        status[i] = res;
    }
}

void launch_collapse_points(const Surface& Sin, const Surface& Sb, double eps2, int precision,
                            const double* vx, const double* vy, const double* vz,
                            const int32_t* v12, const uint8_t* flags, int32_t n, uint8_t* status,
                            uint8_t* degenerate, unsigned long long* counters, cudaStream_t s) {
    if (n <= 0) return;
    const int block = 128;
    const EnvTree Ti = env_tree_for(Sin, eps2), Tb = env_tree_for(Sb, eps2);
    const EpsParams E = eps_params(eps2);
    if (precision == TW_PRECISION_FP32_CERTIFIED)
        k_collapse_points<true><<<grid_for(n, block, 8), block, 0, s>>>(
            Ti, Tb, E, vx, vy, vz, v12, flags, n, status, degenerate, counters);
    else
        k_collapse_points<false><<<grid_for(n, block, 8), block, 0, s>>>(
            Ti, Tb, E, vx, vy, vz, v12, flags, n, status, degenerate, counters);
}

void launch_nearest_points(const Surface& S, double eps2, const double* P, int64_t n, double* Q,
                           double* D, int32_t* F, unsigned long long* counters, cudaStream_t s) {
    if (n <= 0 || S.nf <= 0) return;
    const int block = 128;
    k_nearest_points<<<grid_for(n, block, 8), block, 0, s>>>(env_tree_for(S, eps2), eps2, P, n, Q,
                                                             D, F, counters);
}

// Projection step of surface smoothing (VertexSmoother.cpp:353-363): every
// star whose status is kSmoothPendingProject moves its Newton position to the
// closest point of the nearest facet of the input surface (kind 1) or of the
// boundary surface (kind 2).  A boundary star without a boundary surface is
// an argument error (error bit 4) and is left invalid.
__global__ void k_smooth_project(EnvTree Tin, EnvTree Tb, double eps2,
                                 const uint8_t* __restrict__ kinds,
                                 int32_t nstars, uint8_t* __restrict__ status,
                                 double* __restrict__ pnew,
                                 unsigned long long* __restrict__ counters) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nstars; i += stride) {
        if (status[i] != kSmoothPendingProject) continue;
        const bool bnd = kinds[i] == TW_STAR_BOUNDARY;
        const EnvTree& T = bnd ? Tb : Tin;
        if (T.nf <= 0) {
            atomicOr(counters + kCntError, 4ULL);
            status[i] = TW_SMOOTH_INVALID;
            continue;
        }
        V3 p{pnew[3 * i], pnew[3 * i + 1], pnew[3 * i + 2]};
        V3 q;
        double d;
        int32_t f;
        if (!nearest_facet_grid(T, eps2, p, q, d, f) && nearest_facet(T, p, q, d) == kTraversalError) {
            atomicOr(counters + kCntError, 1ULL);
            status[i] = TW_SMOOTH_INVALID;
            continue;
        }
        pnew[3 * i] = q.x;
        pnew[3 * i + 1] = q.y;
        pnew[3 * i + 2] = q.z;
    }
}

void launch_smooth_project(const Surface& Sin, const Surface& Sb, double eps2,
                           const uint8_t* kinds, int32_t nstars, uint8_t* status, double* pnew,
                           unsigned long long* counters, cudaStream_t s) {
    if (nstars <= 0) return;
    const int block = 128;
    k_smooth_project<<<grid_for(nstars, block, 8), block, 0, s>>>(
        env_tree_for(Sin, eps2), env_tree_for(Sb, eps2), eps2, kinds, nstars, status, pnew,
        counters);
}

// One thread generates the full sample list in the reference order with the
// same helpers (for checking the device sampling arithmetic).  *count = -1
// when the face exceeds the per-row sample bound.
__global__ void k_sample_triangle(const double* __restrict__ t, double sd, double* out,
                                  int64_t cap, int64_t* count) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double tv[9];
    for (int k = 0; k < 9; ++k) tv[k] = t[k];
    SampleHeader h;
    FaceVerts f;
    sample_header(tv, sd, h, f);
    if (header_too_large(h)) {
        *count = -1;
        return;
    }
    int64_t cnt = 0;
    auto emit = [&](const V3& p) {
        if (cnt < cap) {
            out[3 * cnt] = p.x;
            out[3 * cnt + 1] = p.y;
            out[3 * cnt + 2] = p.z;
        }
        ++cnt;
    };
    if (h.trivial) {
        for (int i = 0; i < 3; ++i) emit(V3{tv[3 * i], tv[3 * i + 1], tv[3 * i + 2]});
        *count = cnt;
        return;
    }
    for (int n = 0; n <= h.N; ++n) emit(base_point(h, f, sd, n));
    emit(f.v1);
    if (h.M < 1) {
        emit(f.v2);
        *count = cnt;
        return;
    }
    for (int m = 1; m <= h.M; ++m) {
        V3 v;
        int N1;
        double dd;
        if (!sample_row(h, f, sd, m, v, N1, dd)) break;
        if (N1 > (int)kMaxSamplesPerRow) {
            *count = -1;
            return;
        }
        for (int i = 0; i <= N1; ++i) emit(row_point(h, v, sd, i));
    }
    emit(f.v2);
    if (h.hasE)
        for (int n = 1; n <= h.NE; ++n) emit(edge_point(f.v1, h.n12, sd, n));
    if (h.hasF)
        for (int n = 1; n <= h.NF; ++n) emit(edge_point(f.v2, vneg(h.n02), sd, n));
    *count = cnt;
}

void launch_sample_triangle(const double* tri, double sd, double* out, int64_t cap,
                            int64_t* count, cudaStream_t s) {
    k_sample_triangle<<<1, 32, 0, s>>>(tri, sd, out, cap, count);
}

}  // namespace tw
