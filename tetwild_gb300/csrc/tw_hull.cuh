// tw_hull.cuh -- regions of a face that lie inside the envelope as a whole
// (included by tw_envelope.cu inside namespace tw, after the envelope grid).
//
// The distance to one facet is a convex function, so a triangle whose three
// corners are within r of the same facet lies within r of it, and every
// sample in it is in: the face's samples (some hundreds at eps / 2 spacing)
// need not be built or tested there.  Across a crease two facets do together
// (crease_inside).  A face is cut into 5 x 5 similar triangles, one per lane
// (25 of 32; a 6 x 6 cut would take two steps), and those that fail are cut
// again into k2 x k2 when that leaves pieces larger than the sample spacing.
// What no cut decides is sampled as the reference does.
//
// Notation as in tw_envcert.cuh (u = 2^-24, M the largest |coordinate| of the
// face and the surface; an edge is at most 2 sqrt3 M).  Corners are formed in
// binary32 as p0 + a d1 + b d2 (p0, d1, d2 rounded once from binary64):
// 14u M a component, 24u M in all.  The cut that a sample falls into comes
// from its binary32 barycentric coordinates, 8u off at most (the third one
// 16u): 83u M, and 14u M in cut_of.  The sample's own binary64 construction
// stays within 2^-22 M = 4u M of the exact triangle when the face's height is
// at least 2^-10 of its longest edge (the header's sines are then accurate to
// 2^-40).  A point of the crease test is within 4u M of its side.  So a sample
// lies within 129u M of the hulls of its piece's corners, and a piece is inside
// when the certified upper bounds of those distances are below eps - 135u M
// (with the margin of the certified test for the binary64 rounding): the
// binary64 distance of each of its samples to a facet is then <= eps.
#pragma once

constexpr int kCut = 5;
constexpr int kCuts = kCut * kCut;

struct FaceFrame {
    float p0[3], d1[3], d2[3];
    float Mu2, e2in;   // CertQuery's error term; inside when U^2 < e2in
    int32_t k2;        // the second cut: k2 x k2; 0: none, -1: the face is not cut
};
struct FaceCuts {
    uint32_t open;           // cuts not known to be inside
    uint32_t open2[kCuts];   // of each open cut: the pieces of its second cut not inside
};

// Thread-level preparation of one face (t: its nine coordinates).
// sample_cost: pieces that one sample's test is worth.
__device__ __forceinline__ void hull_prepare(const double* t, const EnvTree& T, const EpsParams& E,
                                             double sd, float sample_cost, FaceFrame& h) {
    float d1[3], d2[3], m = T.scale_hi;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float p = d2f_rn(t[k]);
        d1[k] = d2f_rn(t[3 + k] - t[k]);
        d2[k] = d2f_rn(t[6 + k] - t[k]);
        m = fmaxf(m, fmaxf(fabsf(p), fmaxf(fabsf(d2f_rn(t[3 + k])), fabsf(d2f_rn(t[6 + k])))));
        h.p0[k] = p;
        h.d1[k] = d1[k];
        h.d2[k] = d2[k];
    }
    float a2 = 0.0f, b2 = 0.0f, e2 = 0.0f, c2 = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int i = (k + 1) % 3, j = (k + 2) % 3;
        const float e = d2[k] - d1[k], c = d1[i] * d2[j] - d1[j] * d2[i];
        a2 = fmaf(d1[k], d1[k], a2);
        b2 = fmaf(d2[k], d2[k], b2);
        e2 = fmaf(e, e, e2);
        c2 = fmaf(c, c, c2);
    }
    const float l2 = fmaxf(a2, fmaxf(b2, e2));
    const float mu = __fmul_ru(m, 1.00000012f);
    const float slack = __fmul_ru(mu, 8.1e-06f);   // 135u M and 16 u64 M
    const float el = __fsub_rd(E.eps_lo, slack);
    h.e2in = el > 0.0f ? __fmul_rd(__fmul_rd(el, el), 0.999996185f) : 0.0f;
    h.Mu2 = __fmul_ru(5.684341886080802e-14f, mu);
    const float edge = sqrtf(l2), sdf = d2f_rn(sd);
    // well shaped (height at least 2^-10 of the longest edge), far from the bound
    // on a row's samples (an error that the header reports), binary32-safe
    const bool ok = T.gslot && el > 0.0f && l2 > 1e-16f && l2 < 1e16f &&
                    c2 > l2 * l2 * 9.6e-07f && edge < 1e6f * sdf;
    // pieces of about eps (one that meets a crease is then mostly within eps of
    // one of the two facets), and no more of them than the cut's samples are
    // worth (h1^2 / (2 sd^2) of them)
    const float h1 = edge * (1.0f / kCut);
    const int k2 = (int)fminf(fminf(ceilf(h1 / E.eps_lo), sample_cost * h1 / sdf), (float)kCut);
    h.k2 = !ok ? -1 : k2 >= 2 ? k2 : 0;
}

// Cut q of a k x k cut: rows from the bottom, in each the lower
// (ia, ib), (ia+1, ib), (ia, ib+1) and the upper (ia+1, ib+1), (ia, ib+1),
// (ia+1, ib) in turn (in units of 1/k of the edges).
// The cut of a k x k cut that holds the point (a, b) (in units of 1/k), and
// the point from the cut's first corner along the cut's own edges.
__device__ __forceinline__ int cut_of(int k, float a, float b, float& fa, float& fb) {
    const int ib = min((int)fmaxf(b, 0.0f), k - 1);
    const int ia = min((int)fmaxf(a, 0.0f), k - 1 - ib);
    fa = a - (float)ia;
    fb = b - (float)ib;
    int q = 2 * k * ib - ib * ib + 2 * ia;
    if (fa + fb > 1.0f && ia + ib < k - 1) {
        fa = 1.0f - fa;
        fb = 1.0f - fb;
        ++q;
    }
    return q;
}

// Is the sample at (a, b) (in units of the face's edges d1, d2) in a cut known
// to be inside?
__device__ __forceinline__ bool hull_inside(const FaceCuts& h, int k2, float a, float b) {
    if (k2 < 0) return false;
    float fa, fb;
    const int q = cut_of(kCut, a * (float)kCut, b * (float)kCut, fa, fb);
    if (!((h.open >> q) & 1u)) return true;
    if (k2 == 0) return false;
    float ga, gb;
    const int q2 = cut_of(k2, fa * (float)k2, fb * (float)k2, ga, gb);
    return !((h.open2[q] >> q2) & 1u);
}

// May the sample row at t along v0->v2 (v0 the face's vertex max_i) meet an
// open cut?  The cuts of strip i = floor(kCut t) (and of its neighbour within
// the rounding of t) toward v2, which is the face's vertex (max_i + 2) % 3.
__device__ __forceinline__ bool hull_row_open(const FaceCuts& h, int k2, int max_i, float t) {
    if (k2 < 0) return true;
    const float u = t * (float)kCut;
    const int i0 = max(0, min((int)(u - 1e-4f), kCut - 1)), i1 = max(0, min((int)(u + 1e-4f), kCut - 1));
    // strips toward vertex 2 are rows ib; toward vertex 1 columns ia; toward
    // vertex 0 the diagonals (lower cuts with ia + ib, upper with ia + ib + 1,
    // counted from the opposite edge)
    uint32_t m = 0;
#pragma unroll 1
    for (int q = 0, ib = 0, w = 2 * kCut - 1, r = 0; q < kCuts; ++q) {
        const int ia = r >> 1, up = r & 1;
        const int strip = max_i == 0 ? ib : max_i == 2 ? ia : kCut - 1 - ia - ib - up;
        if (strip >= i0 && strip <= i1) m |= 1u << q;
        if (++r == w) {
            r = 0;
            w -= 2;
            ++ib;
        }
    }
    return (h.open & m) != 0;
}

// Vertex (ia, ib) of a k x k cut's lattice: row by row from the bottom, the
// k + 1 - ib vertices of row ib ((k + 1)(k + 2) / 2 in all).
__device__ __forceinline__ int lattice_id(int k, int ia, int ib) {
    return ib * (2 * k + 3 - ib) / 2 + ia;
}
__device__ __forceinline__ void lattice_vertex(int k, int v, float& a, float& b) {
    int ib = 0;
    for (int w = k + 1; v >= w; --w) {
        v -= w;
        ++ib;
    }
    a = (float)v;
    b = (float)ib;
}
// The three lattice vertices of cut q as a bit set.
__device__ __forceinline__ uint32_t cut_vertices(int k, int q) {
    int ib = 0;
    for (int w = 2 * k - 1; q >= w; w -= 2) {
        q -= w;
        ++ib;
    }
    const int ia = q >> 1;
    const uint32_t b1 = (1u << lattice_id(k, ia + 1, ib)) | (1u << lattice_id(k, ia, ib + 1));
    return b1 | (1u << ((q & 1) ? lattice_id(k, ia + 1, ib + 1) : lattice_id(k, ia, ib)));
}

// The certified upper bound U^2 of the distance from x to facet f when it is
// below lim, else some number not below lim.  facet_classify_rec's U alone,
// with pl = 0.
__device__ __forceinline__ float facet_upper(const FacetCull* __restrict__ f, const float* x,
                                             float Mu2, float lim) {
    const float4* w = reinterpret_cast<const float4*>(f);
    const float4 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3),
                 w4 = __ldg(w + 4), w5 = __ldg(w + 5), w6 = __ldg(w + 6);
    const float inf = __int_as_float(0x7f800000);
    const float rx = (x[0] - w0.x) - w0.w, ry = (x[1] - w0.y) - w1.x, rz = (x[2] - w0.z) - w1.y;
    const float R1 = fabsf(rx) + fabsf(ry) + fabsf(rz);
    const float n0 = w1.z, n1 = w1.w, n2 = w2.x;
    const float hhi = fabsf(fmaf(n2, rz, fmaf(n1, ry, n0 * rx))) + fmaf(8.0f * kUf, R1, Mu2);
    const float h2 = hhi * hhi;
    if (__float_as_uint(w6.w) == 0u || !(h2 < lim)) return inf;
    const float ne[3][3] = {{w2.y, w2.z, w2.w}, {w3.x, w3.y, w3.z}, {w3.w, w4.x, w4.y}};
    const float c[3] = {w4.z, w4.w, w5.x}, o[3] = {w5.y, w5.z, w5.w}, len[3] = {w6.x, w6.y, w6.z};
    float s[3], ds[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        s[e] = fmaf(ne[e][2], rz, fmaf(ne[e][1], ry, ne[e][0] * rx)) - c[e];
        ds[e] = fmaf(10.0f * kUf, R1 + fabsf(c[e]), Mu2);
    }
    if (s[0] + ds[0] < 0.0f && s[1] + ds[1] < 0.0f && s[2] + ds[2] < 0.0f) return h2;
    float u = inf;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const float shi = fabsf(s[e]) + ds[e];
        // an edge whose line may be crossed: the nearest of those segments bounds it
        if (!(s[e] + ds[e] >= 0.0f) || !(fmaf(shi, shi, h2) < lim)) continue;
        const float t0 = fmaf(n1, ne[e][2], -n2 * ne[e][1]);
        const float t1 = fmaf(n2, ne[e][0], -n0 * ne[e][2]);
        const float t2 = fmaf(n0, ne[e][1], -n1 * ne[e][0]);
        const float tau = fmaf(t2, rz, fmaf(t1, ry, t0 * rx)) - o[e];
        const float dtau = fmaf(12.0f * kUf, R1 + fabsf(o[e]), Mu2);
        const float xhi = fmaxf(fmaxf(-tau, tau - len[e]), 0.0f) +
                          fmaf(2.0f * kUf, fabsf(tau) + len[e], dtau);
        u = fminf(u, fmaf(hhi, hhi, fmaf(shi, shi, xhi * xhi)));
    }
    return u;
}
__device__ __forceinline__ bool facet_upper_in(const FacetCull* __restrict__ f, const float* x,
                                               float Mu2, float e2in) {
    return facet_upper(f, x, Mu2, e2in) < e2in;
}

// A piece over a crease: o within reach of facet f, p and q of facet g.  Where
// the sides o-p and o-q leave f (its most exceeded edge line), take points m1,
// m2; when both are within reach of f and of g, the triangle o m1 m2 is within
// reach of f and the quadrilateral m1 p q m2 of g, so the piece is inside
// however far it extends to either side; by one facet alone a piece may reach
// past a crease by eps only, so faces over many facets stayed open (39% of the
// 20k faces with edges 12 to 120 eps on a 5k-facet sphere, 0.76 ms; 0.27 so).
// (m1, m2 are formed within 4u M of the sides.)
__device__ __forceinline__ bool crease_inside(const FacetCull* __restrict__ f,
                                              const FacetCull* __restrict__ g, const float* o,
                                              const float* p, const float* q, float Mu2,
                                              float e2in) {
    float m1[3], m2[3];
    {
        const float4* w = reinterpret_cast<const float4*>(f);
        const float4 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3),
                     w4 = __ldg(w + 4), w5 = __ldg(w + 5);
        const float ne[3][3] = {{w2.y, w2.z, w2.w}, {w3.x, w3.y, w3.z}, {w3.w, w4.x, w4.y}};
        const float c[3] = {w4.z, w4.w, w5.x};
        float so[3], sp[3], sq[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            so[e] = ne[e][0] * (o[0] - w0.x) + ne[e][1] * (o[1] - w0.y) + ne[e][2] * (o[2] - w0.z) - c[e];
            sp[e] = ne[e][0] * (p[0] - w0.x) + ne[e][1] * (p[1] - w0.y) + ne[e][2] * (p[2] - w0.z) - c[e];
            sq[e] = ne[e][0] * (q[0] - w0.x) + ne[e][1] * (q[1] - w0.y) + ne[e][2] * (q[2] - w0.z) - c[e];
        }
        float ap = sp[0], bp = so[0], aq = sq[0], bq = so[0];
#pragma unroll
        for (int e = 1; e < 3; ++e) {
            if (sp[e] > ap) {
                ap = sp[e];
                bp = so[e];
            }
            if (sq[e] > aq) {
                aq = sq[e];
                bq = so[e];
            }
        }
        // 0 <= t <= 1 also for the degenerate quotients (NaN -> 0)
        const float tp = fminf(fmaxf(__fdividef(-bp, ap - bp), 0.0f), 1.0f);
        const float tq = fminf(fmaxf(__fdividef(-bq, aq - bq), 0.0f), 1.0f);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            m1[k] = fmaf(tp, p[k] - o[k], o[k]);
            m2[k] = fmaf(tq, q[k] - o[k], o[k]);
        }
    }
    bool in = true;
#pragma unroll 1
    for (int i = 0; i < 4 && in; ++i)
        in = facet_upper_in(i < 2 ? f : g, (i & 1) ? m2 : m1, Mu2, e2in);
    return in;
}

// A leaf near two vertices (two near leaves each, kNone where there is none).
constexpr uint32_t kNone = 0xffffffffu;
__device__ __forceinline__ uint32_t common_leaf(uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1) {
    return (a0 == b0 || a0 == b1) ? a0 : (a1 == b0 || a1 == b1) ? a1 : kNone;
}

// The pieces where a cell lists more than kDenseCell leaves (facets not larger
// than eps, or a vertex of many): merging the lists would take a step per
// leaf, and most leaves reach only part of a piece.  Each piece takes the leaf
// nearest to its centroid, among up to kDenseTries of the centroid's cell
// spread over the list, and its three vertices are tested against that one.
// Out of line, its values passed singly: the common path keeps its registers.
// The call of 300k faces on the lat-long sphere (up to 500 facets a cell at its
// poles; two runs, ms): kDenseCell 10 2.10-2.12, 28 2.03-2.06, 40 2.07-2.11, no
// dense path 2.40-2.47; kDenseTries 8 2.08-2.16, 12 1.92-2.00, 24 2.03-2.06, 48
// 2.18-2.32 (fewer tries leave more faces open, and the 200k-star pass at 9.9
// either way).
constexpr int kDenseCell = 28, kDenseTries = 24;
struct GridView {   // EnvTree's grid, passed by value
    float glo[3], ginv;
    int32_t gn[3];
    uint32_t gshift, gmask;
    const uint4* gslot;
    const int32_t* glist;
    const FacetCull* cull;
};
__device__ __noinline__ bool dense_pieces_inside(GridView T, float Mu2, float e2in, float x0,
                                                 float x1, float x2, uint32_t need) {
    const uint32_t r1 = need & (need - 1u), r2 = r1 & (r1 - 1u);
    const int va = need ? __ffs(need) - 1 : 0, vb = r1 ? __ffs(r1) - 1 : 0, vc = r2 ? __ffs(r2) - 1 : 0;
    const float a[3] = {__shfl_sync(0xffffffffu, x0, va), __shfl_sync(0xffffffffu, x1, va),
                        __shfl_sync(0xffffffffu, x2, va)};
    const float b[3] = {__shfl_sync(0xffffffffu, x0, vb), __shfl_sync(0xffffffffu, x1, vb),
                        __shfl_sync(0xffffffffu, x2, vb)};
    const float c[3] = {__shfl_sync(0xffffffffu, x0, vc), __shfl_sync(0xffffffffu, x1, vc),
                        __shfl_sync(0xffffffffu, x2, vc)};
    if (!need) return false;
    float y[3];
    CertQuery q;
#pragma unroll
    for (int k = 0; k < 3; ++k) q.ph[k] = y[k] = (a[k] + b[k] + c[k]) * 0.333333343f;
    uint32_t i, e;
    grid_cell_range(T, q, i, e);
    const uint32_t stride = (e - i + kDenseTries - 1) / kDenseTries;
    float best = e2in;
    int32_t leaf = -1;
    for (; i < e; i += stride) {
        const int32_t lf = __ldg(T.glist + i);
        const float u = facet_upper(T.cull + lf, y, Mu2, best);
        if (u < best) {
            best = u;
            leaf = lf;
        }
    }
    bool in = leaf >= 0;
#pragma unroll 1
    for (int v = 0; v < 3 && in; ++v) {
#pragma unroll
        for (int k = 0; k < 3; ++k) y[k] = v == 0 ? a[k] : v == 1 ? b[k] : c[k];
        in = facet_upper_in(T.cull + leaf, y, Mu2, e2in);
    }
    return in;
}

// The whole warp tests the pieces of one or more cuts: lanes with vert hold a
// lattice vertex at x, lanes with need a piece (its vertices' lanes as a bit
// set); true for a lane whose piece lies within reach of one facet, or of two
// across a crease.  A facet within eps of a vertex is listed in its grid cell,
// so the lanes merge their cells' ascending lists: each step takes the
// smallest leaf left, and tests it, one record for the whole warp, when it is
// listed for a vertex of a piece still open.  At most kCutLeaves leaves are
// taken (a face over many small facets: its pieces stay open; 300k faces: 2.70
// ms with 16, 2.05 with 32, 2.00-2.10 with 64).
constexpr int kCutLeaves = 32;
__device__ __forceinline__ bool pieces_inside(const EnvTree& T, const FaceFrame& h, bool vert,
                                              const float* x, uint32_t need) {
    uint32_t i = 0, e = 0;
    if (vert) {
        CertQuery q;
#pragma unroll
        for (int k = 0; k < 3; ++k) q.ph[k] = x[k];
        grid_cell_range(T, q, i, e);
    }
    if (__reduce_max_sync(0xffffffffu, e - i) > (uint32_t)kDenseCell) {
        const GridView g{{T.glo[0], T.glo[1], T.glo[2]}, T.ginv, {T.gn[0], T.gn[1], T.gn[2]},
                         T.gshift, T.gmask, T.gslot, T.glist, T.cull};
        return dense_pieces_inside(g, h.Mu2, h.e2in, x[0], x[1], x[2], need);
    }
    // the list is read one entry ahead of the leaf at hand
    uint32_t cur = i < e ? (uint32_t)__ldg(T.glist + i) : kNone;
    uint32_t nxt = i + 1 < e ? (uint32_t)__ldg(T.glist + i + 1) : kNone;
    uint32_t near0 = kNone, near1 = kNone;   // leaves within reach of the vertex
    const float Mu2 = h.Mu2, e2in = h.e2in;
    bool inside = false;
    for (int step = 0; step < kCutLeaves; ++step) {
        const uint32_t lf = __reduce_min_sync(0xffffffffu, cur);
        if (lf == kNone) break;
        const bool has = cur == lf;
        if (has) {
            cur = nxt;
            ++i;
            nxt = i + 1 < e ? (uint32_t)__ldg(T.glist + i + 1) : kNone;
        }
        const uint32_t listed = __ballot_sync(0xffffffffu, has);
        if (!__any_sync(0xffffffffu, !inside && (listed & need) != 0u)) continue;
        bool in = false;
        if (has) {
            in = facet_upper_in(T.cull + lf, x, Mu2, e2in);
            if (in) {
                near1 = near0 == kNone ? near1 : near1 == kNone ? lf : near1;
                near0 = near0 == kNone ? lf : near0;
            }
        }
        const uint32_t near = __ballot_sync(0xffffffffu, in);
        inside = inside || (need && (near & need) == need);
        if (__all_sync(0xffffffffu, inside || !need)) return inside;
    }
    // pieces across a crease
    const bool open = need && !inside;
    const uint32_t r1 = need & (need - 1u), r2 = r1 & (r1 - 1u);
    const int va = need ? __ffs(need) - 1 : 0, vb = r1 ? __ffs(r1) - 1 : 0, vc = r2 ? __ffs(r2) - 1 : 0;
    const uint32_t a0 = __shfl_sync(0xffffffffu, near0, va), a1 = __shfl_sync(0xffffffffu, near1, va);
    const uint32_t b0 = __shfl_sync(0xffffffffu, near0, vb), b1 = __shfl_sync(0xffffffffu, near1, vb);
    const uint32_t c0 = __shfl_sync(0xffffffffu, near0, vc), c1 = __shfl_sync(0xffffffffu, near1, vc);
    uint32_t f = kNone, g = kNone;
    int vo = va, vp = vb, vq = vc;   // the vertex apart, and the other two
    if (a0 != kNone && b0 != kNone && c0 != kNone) {
        g = common_leaf(b0, b1, c0, c1);
        f = a0;
        if (g == kNone) {
            g = common_leaf(a0, a1, c0, c1);
            f = b0;
            vo = vb;
            vp = va;
        }
        if (g == kNone) {
            g = common_leaf(a0, a1, b0, b1);
            f = c0;
            vo = vc;
            vp = va;
            vq = vb;
        }
    }
    const bool test = open && g != kNone;
    if (!__any_sync(0xffffffffu, test)) return inside;
    float o[3], p[3], q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o[k] = __shfl_sync(0xffffffffu, x[k], vo);
        p[k] = __shfl_sync(0xffffffffu, x[k], vp);
        q[k] = __shfl_sync(0xffffffffu, x[k], vq);
    }
    if (test) inside = crease_inside(T.cull + f, T.cull + g, o, p, q, Mu2, e2in);
    return inside;
}

// Per lane and cut size k = 2..5: the lattice vertex (a, b) and the piece's
// vertices, filled once per block (k * 32 + lane).
struct CutTables {
    float a[4 * 32], b[4 * 32];
    uint32_t need[4 * 32];
};
__device__ __forceinline__ void fill_cut_tables(CutTables& t) {
    for (int i = threadIdx.x; i < 4 * 32; i += blockDim.x) {
        const int k = 2 + (i >> 5), l = i & 31;
        const int verts = (k + 1) * (k + 2) / 2, per = k * k;
        const int cuts = 32 / max(verts, per);   // cuts of a second step
        lattice_vertex(k, l % verts, t.a[i], t.b[i]);
        t.need[i] = l / per < cuts ? cut_vertices(k, l % per) << (l / per * verts) : 0u;
    }
    __syncthreads();
}

// The whole warp tests whether a vertex of the face (t) whose cut is open is
// certainly out: every facet listed in its grid cell has a certified lower
// bound above eps.  The vertices of a face that is not degenerate are samples
// of it, so the face is out.
__device__ __forceinline__ bool vertex_out(const EnvTree& T, const EpsParams& E,
                                           const double* __restrict__ t, uint32_t open,
                                           TravStats& st, uint32_t& nq) {
    const int lane = threadIdx.x & 31;
    const int cut = lane == 0 ? 0 : lane == 1 ? 2 * kCut - 2 : kCuts - 1;   // at vertex `lane`
    bool out = false;
    if (lane < 3 && ((open >> cut) & 1u)) {
        const V3 p{__ldg(t + 3 * lane), __ldg(t + 3 * lane + 1), __ldg(t + 3 * lane + 2)};
        const CertQuery q = cert_query(p, E, T.scale_hi);
        uint32_t i, e;
        grid_cell_range(T, q, i, e);
        out = true;
        for (; out && i < e; ++i) {
            out = facet_classify(T.cull, __ldg(T.glist + i), q) == kFacetOut;
            ++st.facets;
        }
        ++nq;
    }
    return __any_sync(0xffffffffu, out);
}

// The whole warp cuts the face t: 0 when all of it is inside.  KEEP: the open
// cuts and pieces are written to c (shared memory); otherwise it stops at the
// first open piece, and answers 1 when a vertex is certainly out.  2: open.
// With KEEP the warps slice = 0 .. slices - 1 of a block may share the second
// cuts, each writing its own cuts' pieces (the caller synchronises; open then
// keeps cuts whose pieces are all inside, with open2 = 0).  st and nq count
// the vertices tested, not the pieces (which are no samples).
template <bool KEEP>
__device__ __forceinline__ int hull_cut(const EnvTree& T, const EpsParams& E, const FaceFrame& h,
                                        const double* __restrict__ t, const CutTables& tab,
                                        FaceCuts* c, int slice, int slices, TravStats& st,
                                        uint32_t& nq) {
    const int lane = threadIdx.x & 31;
    constexpr int kVerts = (kCut + 1) * (kCut + 2) / 2;
    const int k2 = h.k2;
    // second cuts: as many cuts as fit a step (vertices and pieces each on lanes
    // of their own); vs, ps: the lane's vertex' and piece's cut
    int per = 1, cuts = 0, vs = 0, ps = 0;
    float va = 0.0f, vb = 0.0f;
    uint32_t need2 = 0, open = 0, left = 0, still = 0;
    // One loop for the first cut (turn -1) and the second cuts, so that
    // pieces_inside is in the code once: with two copies a quarter of the cut's
    // stalls were instruction fetches (300k faces: 1.55 ms, 1.36 so).
#pragma unroll 1
    for (int turn = -1; turn < 0 || left; ++turn) {
        int qv = -1, qp = -1;
        bool vert;
        uint32_t need;
        float ra, rb;
        if (turn < 0) {
            const int row = (kCut - 2) * 32 + lane;
            ra = tab.a[row] * (1.0f / kCut);
            rb = tab.b[row] * (1.0f / kCut);
            vert = lane < kVerts;
            need = tab.need[row];
        } else {
            for (int s = 0; s < cuts && left; ++s, left &= left - 1) {
                const int q = __ffs(left) - 1;
                if (s == vs) qv = q;
                if (s == ps) qp = q;
            }
            if (KEEP && slices > 1 && turn % slices != slice) continue;
            // along the cut's own edges from its first corner (an upper cut's
            // point backwards)
            int q = max(qv, 0), ib = 0;
            for (int w = 2 * kCut - 1; q >= w; w -= 2) {
                q -= w;
                ++ib;
            }
            const int up = q & 1;
            const float dir = up ? -1.0f : 1.0f;
            ra = fmaf(dir, va, (float)((q >> 1) + up)) * (1.0f / kCut);
            rb = fmaf(dir, vb, (float)(ib + up)) * (1.0f / kCut);
            vert = qv >= 0;
            need = qp >= 0 ? need2 : 0u;
        }
        float x[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) x[k] = fmaf(ra, h.d1[k], fmaf(rb, h.d2[k], h.p0[k]));
        const bool ok = pieces_inside(T, h, vert, x, need);
        const uint32_t bal = __ballot_sync(0xffffffffu, need && !ok);
        if (turn < 0) {
            open = bal;
            if (!open) break;
            if (!KEEP && vertex_out(T, E, t, open, st, nq)) return 1;
            if (k2 <= 0) break;
            left = open;
            const int verts = (k2 + 1) * (k2 + 2) / 2;
            per = k2 * k2;
            cuts = 32 / max(verts, per);
            vs = lane / verts;
            ps = lane / per;
            const int row = (k2 - 2) * 32 + lane;
            const float inv = 1.0f / (float)k2;
            va = tab.a[row] * inv;
            vb = tab.b[row] * inv;
            need2 = tab.need[row];
        } else if (KEEP) {
            const uint32_t mine = qp >= 0 ? (bal >> (ps * per)) & ((1u << per) - 1u) : 0u;
            if (qp >= 0 && lane == ps * per) c->open2[qp] = mine;
            still |= __reduce_or_sync(0xffffffffu, mine ? 1u << qp : 0u);
        } else if (bal) {
            return 2;
        }
    }
    if (k2 > 0 && (!KEEP || slices == 1)) open = still;
    if (KEEP) {
        if (lane == 0 && slice == 0) c->open = open;
        __syncwarp();
    }
    return open ? 2 : 0;
}
