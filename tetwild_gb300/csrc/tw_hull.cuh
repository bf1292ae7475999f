// tw_hull.cuh -- regions of a face that lie inside the envelope as a whole
// (included by tw_envelope.cu inside namespace tw, after the envelope grid).
//
// The distance to one facet is a convex function, so a triangle whose three
// corners are within r of the same facet lies within r of it, and every
// sample in it is in: the face's samples (some hundreds at eps / 2 spacing)
// need not be built or tested there.  A face is cut into 5 x 5 similar
// triangles, one per lane (25 of 32; a 6 x 6 cut would take two steps), and
// those that fail are cut again into k2 x k2 when that leaves pieces larger
// than the sample spacing.  What no cut decides is sampled as the reference
// does.
//
// Notation as in tw_envcert.cuh (u = 2^-24, M the largest |coordinate| of the
// face and the surface; an edge is at most 2 sqrt3 M).  Corners are formed in
// binary32 as p0 + a d1 + b d2 (p0, d1, d2 rounded once from binary64):
// 14u M a component, 24u M in all.  The cut that a sample falls into comes
// from its binary32 barycentric coordinates, 8u off at most (the third one
// 16u): 83u M, and 14u M in cut_of.  The sample's own binary64 construction
// stays within 2^-22 M = 4u M of the exact triangle when the face's height is
// at least 2^-10 of its longest edge (the header's sines are then accurate to
// 2^-40).  So a sample lies within 125u M < 128u M = 2^-17 M of the convex hull
// of its cut's corners, and a cut is inside when the certified upper bounds of its
// corners' distances to one facet are below eps - 2^-17 M (with the margin of
// the certified test for the binary64 rounding): the binary64 distance of
// each of its samples to that facet is then <= eps.
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
    const float slack = __fmul_ru(mu, 7.6293999e-06f);   // 2^-17 M + 16 u64 M
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

// Is the certified upper bound of the distance from x to facet f below the
// limit (U^2 < e2in)?  facet_classify_rec's U alone, with pl = 0.
__device__ __forceinline__ bool facet_upper_in(const FacetCull* __restrict__ f, const float* x,
                                               float Mu2, float e2in) {
    const float4* w = reinterpret_cast<const float4*>(f);
    const float4 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3),
                 w4 = __ldg(w + 4), w5 = __ldg(w + 5), w6 = __ldg(w + 6);
    const float rx = (x[0] - w0.x) - w0.w, ry = (x[1] - w0.y) - w1.x, rz = (x[2] - w0.z) - w1.y;
    const float R1 = fabsf(rx) + fabsf(ry) + fabsf(rz);
    const float n0 = w1.z, n1 = w1.w, n2 = w2.x;
    const float hhi = fabsf(fmaf(n2, rz, fmaf(n1, ry, n0 * rx))) + fmaf(8.0f * kUf, R1, Mu2);
    const float h2 = hhi * hhi;
    if (__float_as_uint(w6.w) == 0u || !(h2 < e2in)) return false;
    const float ne[3][3] = {{w2.y, w2.z, w2.w}, {w3.x, w3.y, w3.z}, {w3.w, w4.x, w4.y}};
    const float c[3] = {w4.z, w4.w, w5.x}, o[3] = {w5.y, w5.z, w5.w}, len[3] = {w6.x, w6.y, w6.z};
    float s[3], ds[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        s[e] = fmaf(ne[e][2], rz, fmaf(ne[e][1], ry, ne[e][0] * rx)) - c[e];
        ds[e] = fmaf(10.0f * kUf, R1 + fabsf(c[e]), Mu2);
    }
    if (s[0] + ds[0] < 0.0f && s[1] + ds[1] < 0.0f && s[2] + ds[2] < 0.0f) return true;
    bool in = false;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const float shi = fabsf(s[e]) + ds[e];
        // an edge whose line may be crossed: the nearest of those segments bounds it
        if (!(s[e] + ds[e] >= 0.0f) || !(fmaf(shi, shi, h2) < e2in)) continue;
        const float t0 = fmaf(n1, ne[e][2], -n2 * ne[e][1]);
        const float t1 = fmaf(n2, ne[e][0], -n0 * ne[e][2]);
        const float t2 = fmaf(n0, ne[e][1], -n1 * ne[e][0]);
        const float tau = fmaf(t2, rz, fmaf(t1, ry, t0 * rx)) - o[e];
        const float dtau = fmaf(12.0f * kUf, R1 + fabsf(o[e]), Mu2);
        const float xhi = fmaxf(fmaxf(-tau, tau - len[e]), 0.0f) +
                          fmaf(2.0f * kUf, fabsf(tau) + len[e], dtau);
        in = in || fmaf(hhi, hhi, fmaf(shi, shi, xhi * xhi)) < e2in;
    }
    return in;
}

// The whole warp tests the pieces of one or more cuts: lanes with vert hold a
// lattice vertex at x, lanes with need a piece (its vertices' lanes as a bit
// set); true for a lane whose piece lies within reach of one facet.  A facet
// within eps of a piece's vertices is listed in the grid cell of each, so
// the lanes merge their cells' ascending lists: each step takes the smallest
// leaf left, and tests it, one record for the whole warp, when it is listed
// for all vertices of a piece still open.  At most kCutLeaves leaves are
// taken (a face over many small facets: its pieces stay open).
constexpr int kCutLeaves = 32;
__device__ __forceinline__ bool pieces_inside(const EnvTree& T, const FaceFrame& h, bool vert,
                                              const float* x, uint32_t need, TravStats& st) {
    uint32_t i = 0, e = 0;
    if (vert) {
        CertQuery q;
#pragma unroll
        for (int k = 0; k < 3; ++k) q.ph[k] = x[k];
        grid_cell_range(T, q, i, e);
    }
    uint32_t cur = i < e ? (uint32_t)__ldg(T.glist + i) : 0xffffffffu;
    const float Mu2 = h.Mu2, e2in = h.e2in;
    bool inside = false;
    for (int step = 0; step < kCutLeaves; ++step) {
        const uint32_t lf = __reduce_min_sync(0xffffffffu, cur);
        if (lf == 0xffffffffu) break;
        const bool has = cur == lf;
        if (has) {
            ++i;
            cur = i < e ? (uint32_t)__ldg(T.glist + i) : 0xffffffffu;
        }
        const uint32_t listed = __ballot_sync(0xffffffffu, has);
        if (!__any_sync(0xffffffffu, need && !inside && (listed & need) == need)) continue;
        bool in = false;
        if (has) {
            in = facet_upper_in(T.cull + lf, x, Mu2, e2in);
            ++st.facets;
        }
        const uint32_t near = __ballot_sync(0xffffffffu, in);
        inside = inside || (need && (near & need) == need);
        if (__all_sync(0xffffffffu, inside || !need)) break;
    }
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
// keeps cuts whose pieces are all inside, with open2 = 0).  nq counts the
// pieces and vertices tested.
template <bool KEEP>
__device__ __forceinline__ int hull_cut(const EnvTree& T, const EpsParams& E, const FaceFrame& h,
                                        const double* __restrict__ t, const CutTables& tab,
                                        FaceCuts* c, int slice, int slices, TravStats& st,
                                        uint32_t& nq) {
    const int lane = threadIdx.x & 31;
    constexpr int kVerts = (kCut + 1) * (kCut + 2) / 2;
    const int row1 = (kCut - 2) * 32 + lane;
    const float a = tab.a[row1] * (1.0f / kCut), b = tab.b[row1] * (1.0f / kCut);
    float x[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = fmaf(a, h.d1[k], fmaf(b, h.d2[k], h.p0[k]));
    const uint32_t need1 = tab.need[row1];
    const bool in = pieces_inside(T, h, lane < kVerts, x, need1, st);
    if (need1) ++nq;
    uint32_t open = __ballot_sync(0xffffffffu, need1 && !in);
    if (!KEEP && open && vertex_out(T, E, t, open, st, nq)) return 1;
    const int k2 = h.k2;
    if (open && k2 > 0) {
        // the open cuts' pieces: as many cuts as fit a step (vertices and pieces
        // each on lanes of their own)
        const int verts = (k2 + 1) * (k2 + 2) / 2, per = k2 * k2;
        const int cuts = 32 / max(verts, per);
        const int vs = lane / verts, ps = lane / per;   // the lane's vertex' and piece's cut
        const int row2 = (k2 - 2) * 32 + lane;
        const uint32_t need2 = tab.need[row2];
        const float inv = 1.0f / (float)k2, va = tab.a[row2] * inv, vb = tab.b[row2] * inv;
        uint32_t still = 0;
        int turn = 0;
        for (uint32_t left = open; left; ++turn) {
            int qv = -1, qp = -1;
            for (int s = 0; s < cuts && left; ++s, left &= left - 1) {
                const int q = __ffs(left) - 1;
                if (s == vs) qv = q;
                if (s == ps) qp = q;
            }
            if (KEEP && slices > 1 && turn % slices != slice) continue;
            if (qv >= 0) {
                // along the cut's own edges from its first corner (an upper cut's
                // point backwards)
                int q = qv, ib = 0;
                for (int w = 2 * kCut - 1; q >= w; w -= 2) {
                    q -= w;
                    ++ib;
                }
                const int up = q & 1;
                const float dir = up ? -1.0f : 1.0f;
                const float ra = fmaf(dir, va, (float)((q >> 1) + up)) * (1.0f / kCut);
                const float rb = fmaf(dir, vb, (float)(ib + up)) * (1.0f / kCut);
#pragma unroll
                for (int k = 0; k < 3; ++k) x[k] = fmaf(ra, h.d1[k], fmaf(rb, h.d2[k], h.p0[k]));
            }
            const bool ok = pieces_inside(T, h, qv >= 0, x, qp >= 0 ? need2 : 0u, st);
            const uint32_t bal = __ballot_sync(0xffffffffu, qp >= 0 && !ok);
            if (qp >= 0) ++nq;
            if (KEEP) {
                const uint32_t mine = qp >= 0 ? (bal >> (ps * per)) & ((1u << per) - 1u) : 0u;
                if (qp >= 0 && lane == ps * per) c->open2[qp] = mine;
                still |= __reduce_or_sync(0xffffffffu, mine ? 1u << qp : 0u);
            } else if (bal) {
                return 2;
            }
        }
        if (!KEEP || slices == 1) open = still;
    }
    if (KEEP) {
        if (lane == 0 && slice == 0) c->open = open;
        __syncwarp();
    }
    return open ? 2 : 0;
}
