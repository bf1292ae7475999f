// tw_star.cuh -- device routines of one-ring stars used by the Newton,
// smoothing and collapse kernels (tw_newton.cu):
// the 3x3 solve, the star view and gathers, the inversion and quality checks
// and the one-ring surface faces.
#pragma once

#include "tw_device.cuh"
#include "tw_internal.h"

namespace tw {

__device__ __forceinline__ void qr_solve3(const double* Hm, const double* bvec, double* x) {
    double R[3][3], c[3];
    int perm[3] = {0, 1, 2};
    for (int i = 0; i < 3; ++i) {
        c[i] = bvec[i];
        for (int j = 0; j < 3; ++j) R[i][j] = Hm[3 * i + j];
    }
    for (int k = 0; k < 3; ++k) {
        int p = k;
        double best = -1.0;
        for (int j = k; j < 3; ++j) {
            double nrm = 0.0;
            for (int i = k; i < 3; ++i) nrm = nrm + R[i][j] * R[i][j];
            if (nrm > best) {
                best = nrm;
                p = j;
            }
        }
        if (p != k) {
            for (int i = 0; i < 3; ++i) {
                double t = R[i][k];
                R[i][k] = R[i][p];
                R[i][p] = t;
            }
            int t = perm[k];
            perm[k] = perm[p];
            perm[p] = t;
        }
        if (k == 2) break;
        double xn = 0.0;
        for (int i = k; i < 3; ++i) xn = xn + R[i][k] * R[i][k];
        xn = sqrt(xn);
        if (xn == 0.0) continue;
        double alpha = (R[k][k] > 0.0) ? -xn : xn;
        double v[3] = {0.0, 0.0, 0.0};
        for (int i = k; i < 3; ++i) v[i] = R[i][k];
        v[k] = v[k] - alpha;
        double vv = 0.0;
        for (int i = k; i < 3; ++i) vv = vv + v[i] * v[i];
        if (vv == 0.0) continue;
        double beta = 2.0 / vv;
        for (int j = k + 1; j < 3; ++j) {
            double s = 0.0;
            for (int i = k; i < 3; ++i) s = s + v[i] * R[i][j];
            s = s * beta;
            for (int i = k; i < 3; ++i) R[i][j] = R[i][j] - s * v[i];
        }
        {
            double s = 0.0;
            for (int i = k; i < 3; ++i) s = s + v[i] * c[i];
            s = s * beta;
            for (int i = k; i < 3; ++i) c[i] = c[i] - s * v[i];
        }
        R[k][k] = alpha;
        for (int i = k + 1; i < 3; ++i) R[i][k] = 0.0;
    }
    double thr = 3.0 * 2.220446049250313e-16 * fabs(R[0][0]);
    int rank = 0;
    for (int k = 0; k < 3; ++k) {
        if (fabs(R[k][k]) > thr)
            rank = k + 1;
        else
            break;
    }
    double y[3] = {0.0, 0.0, 0.0};
    for (int k = rank - 1; k >= 0; --k) {
        double s = c[k];
        for (int j = k + 1; j < rank; ++j) s = s - R[k][j] * y[j];
        y[k] = s / R[k][k];
    }
    for (int k = 0; k < 3; ++k) x[perm[k]] = y[k];
}

struct StarView {
    const double* vx;
    const double* vy;
    const double* vz;
    const int4* tets;
    int32_t nt;
    int32_t v;
    int form;   // TW_ENERGY_FORM_* of the binary64 AMIPS evaluations
};

__device__ __forceinline__ void gather_tet(const StarView& S, int4 tv, int start, const double* pos,
                                           double* T) {
    int id[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int32_t k = id[(start + j) & 3];
        if (k == S.v) {
            T[3 * j] = pos[0];
            T[3 * j + 1] = pos[1];
            T[3 * j + 2] = pos[2];
        } else {
            T[3 * j] = __ldg(S.vx + k);
            T[3 * j + 1] = __ldg(S.vy + k);
            T[3 * j + 2] = __ldg(S.vz + k);
        }
    }
}

// Position of vertex v in the tet (0 when it is none of the four).
__device__ __forceinline__ int centre_index(int4 tv, int32_t v) {
    return (tv.x == v) ? 0 : (tv.y == v) ? 1 : (tv.z == v) ? 2 : (tv.w == v) ? 3 : 0;
}

template <int G>
__device__ __forceinline__ unsigned group_mask(int lane) {
    return (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
}

// ---------------------------------------------------------------------------
// Smoothing pass (VertexSmoother.cpp:114-210 and :244-450), G lanes per star.
// ---------------------------------------------------------------------------
// True when every tet of the star is POSITIVE with the centre at pos.
template <int G>
__device__ __forceinline__ bool star_positive(const StarView& S, const double* pos, int gl,
                                              unsigned gm) {
    bool bad = false;
    for (int c0 = gl; c0 < S.nt; c0 += G) {
        double T[12];
        gather_tet(S, __ldg(S.tets + c0), 0, pos, T);
        bad = bad || (orient3d(T, T + 3, T + 6, T + 9) != 1);
    }
    return !__any_sync(gm, bad);
}

__device__ __forceinline__ int4 tet_at(const StarView& S, int32_t i) { return __ldg(S.tets + i); }
__device__ __forceinline__ int tet_vertex(int4 tv, int j) {
    return j == 0 ? tv.x : j == 1 ? tv.y : j == 2 ? tv.z : tv.w;
}

// The surface face of tet tv opposite its j-th vertex, as a sorted triple.
__device__ __forceinline__ void face_key(int4 tv, int j, int32_t* k) {
    int32_t id[4] = {tv.x, tv.y, tv.z, tv.w};
    int32_t a = id[(j + 1) & 3], b = id[(j + 2) & 3], c = id[(j + 3) & 3];
    int32_t lo = min(a, min(b, c)), hi = max(a, max(b, c));
    k[0] = lo;
    k[1] = (int32_t)((int64_t)a + b + c - lo - hi);
    k[2] = hi;
}

// calTetQuality_AMIPS for a tet already known to be POSITIVE.
__device__ __forceinline__ double positive_tet_quality(const double* T, int form) {
    return quality_from(1, amips_energy_f(T, form));
}

// True when face j of the star's tet c0 is a surface face through the
// centre whose sorted triple does not occur at an earlier (tet, face) of the
// star; writes the triple.
__device__ __forceinline__ bool first_surface_face(const StarView& S, const uint8_t* ff,
                                                   int32_t c0, int4 tv, uint8_t fl, int j,
                                                   int32_t* key) {
    if (tet_vertex(tv, j) == S.v || !((fl >> j) & 1)) return false;
    face_key(tv, j, key);
    for (int32_t i2 = 0; i2 <= c0; ++i2) {
        int4 t2 = tet_at(S, i2);
        uint8_t f2 = __ldg(ff + i2);
        for (int j2 = 0; j2 < 4; ++j2) {
            if (i2 == c0 && j2 >= j) return true;
            if (tet_vertex(t2, j2) == S.v || !((f2 >> j2) & 1)) continue;
            int32_t k2[3];
            face_key(t2, j2, k2);
            if (k2[0] == key[0] && k2[1] == key[1] && k2[2] == key[2]) return false;
        }
    }
    return true;
}

// Differences of the tet's vertices from the first, and a power of two above
// every coordinate's magnitude.
__device__ __forceinline__ float tet_diffs32(const double* T, float* d1, float* d2, float* d3) {
    int m = 0;
#pragma unroll
    for (int k = 0; k < 12; ++k) m = max(m, __double2hiint(T[k]) & 0x7fffffff);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        d1[k] = d2f_rn(T[3 + k] - T[k]);
        d2[k] = d2f_rn(T[6 + k] - T[k]);
        d3[k] = d2f_rn(T[9 + k] - T[k]);
    }
    const int e = (m >> 20) - 1023 + 128;   // of 2^(exponent + 1)
    return e <= 0 ? 1.17549435e-38f : e >= 255 ? __int_as_float(0x7f800000) : __int_as_float(e << 23);
}

// Bounds of the largest quality over the tets a lane of a group has seen
// (certified binary32 energies); sure: every tet had one.
struct MaxBounds {
    float lo = 0.0f, hi = 0.0f;
    bool sure = true;
    __device__ __forceinline__ void add_positive(const float* d1, const float* d2,
                                                 const float* d3, float M) {
        const Energy32 r = amips_energy32(d1, d2, d3, M);
        sure = sure && r.ok && r.E < 1e30f;
        lo = fmaxf(lo, __fmul_rd(r.E, 1.0f - r.rel));
        hi = fmaxf(hi, __fmul_ru(r.E, 1.0f + r.rel));
    }
    __device__ __forceinline__ void add_sentinel() {   // kMaxEnergy, above every energy here
        lo = hi = 3e38f;
    }
    template <int G>
    __device__ __forceinline__ void join(unsigned gm) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            lo = fmaxf(lo, __shfl_xor_sync(gm, lo, o, G));
            hi = fmaxf(hi, __shfl_xor_sync(gm, hi, o, G));
        }
        sure = __all_sync(gm, sure);
    }
};

}  // namespace tw
