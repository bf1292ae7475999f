// tw_newton.cu -- damped Newton smoothing of independent one-ring stars.
//
// Restates VertexSmoother::NewtonsMethod (VertexSmoother.cpp:465-542),
// NewtonsUpdate (:627-702) and getNewEnergy (:544-625) of the default scalar
// build: per step, E/J/H summed over the star's tets in caller order (each
// tet rotated so the centre vertex comes first), X = QR(H)^-1 (H X0 - a J)
// with up to max_it halvings of a, each trial rejected if X is not finite,
// if a tet flips (exact orientation) or if the star energy (tets in stored
// order) does not strictly decrease; stop when |dE| < 1e-5.
// The 3x3 solve is Householder QR with column pivoting (Golub & Van Loan,
// Alg. 5.4.1), the same operations as the oracle's, standing in for Eigen's
// ColPivHouseholderQR (:492).
#include <algorithm>

#include "tw_device.cuh"
#include "tw_internal.h"
#include "tw_star.cuh"

namespace tw {

#include "tw_wave.cuh"

// CERT: signs and the largest qualities are compared as certified binary32
// intervals first, in binary64 where those overlap (the same decisions).
template <int G, bool CERT>
__global__ void __launch_bounds__(256) k_smooth_stage2(
    const double* __restrict__ vx, const double* __restrict__ vy, const double* __restrict__ vz,
    const int32_t* __restrict__ star_off, const int4* __restrict__ tets,
    const uint8_t* __restrict__ face_flags, const int32_t* __restrict__ centers, int32_t nstars,
    const double* __restrict__ pnew, uint8_t* __restrict__ status, double* __restrict__ faces,
    unsigned long long* __restrict__ face_count, int64_t face_cap,
    int32_t* __restrict__ face_base, int32_t* __restrict__ face_cnt,
    unsigned long long* __restrict__ counters, int form) {
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const unsigned gm = group_mask<G>(lane);
    const int64_t gid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / G;
    for (int64_t sid = gid; sid < nstars; sid += ngroups) {
        if (status[sid] != kSmoothPendingProject) continue;  // uniform within the group
        const int32_t b = star_off[sid], nt = star_off[sid + 1] - b;
        StarView S{vx, vy, vz, tets + b, nt, centers[sid], form};
        const double p0[3] = {vx[S.v], vy[S.v], vz[S.v]};
        const double p[3] = {pnew[3 * sid], pnew[3 * sid + 1], pnew[3 * sid + 2]};
        // isFlip at the projected position (:374-378)
        if (!star_positive<G>(S, p, gl, gm)) {
            if (gl == 0) status[sid] = TW_SMOOTH_REJECT_FLIP;
            continue;
        }
        // max calTetQuality before and after (:379-386); max is exact in any order
        int better = -1;   // not known yet
        if (CERT) {
            MaxBounds o, m;
            for (int c0 = gl; c0 < nt; c0 += G) {
                const int4 tv = tet_at(S, c0);
                double T[12];
                float d1[3], d2[3], d3[3];
                gather_tet(S, tv, 0, p0, T);
                float M = tet_diffs32(T, d1, d2, d3);
                o.add_positive(d1, d2, d3, M);
                gather_tet(S, tv, 0, p, T);
                M = tet_diffs32(T, d1, d2, d3);
                m.add_positive(d1, d2, d3, M);
            }
            o.join<G>(gm);
            m.join<G>(gm);
            if (o.sure && m.sure) better = m.hi < o.lo ? 1 : m.lo > o.hi ? 0 : -1;
        }
        if (better < 0) {
            double old_max = 0.0, new_max = 0.0;
            for (int c0 = gl; c0 < nt; c0 += G) {
                double T[12];
                int4 tv = tet_at(S, c0);
                gather_tet(S, tv, 0, p0, T);
                old_max = fmax(old_max, positive_tet_quality(T, S.form));
                gather_tet(S, tv, 0, p, T);
                new_max = fmax(new_max, positive_tet_quality(T, S.form));
            }
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
                old_max = fmax(old_max, __shfl_xor_sync(gm, old_max, o, G));
                new_max = fmax(new_max, __shfl_xor_sync(gm, new_max, o, G));
            }
            better = new_max < old_max;
        }
        if (!better) {
            if (gl == 0) status[sid] = TW_SMOOTH_REJECT_QUALITY;
            continue;
        }
        // one-ring surface faces (:314-326): the first occurrence of each
        // sorted triple; counted, then written at one reservation per star
        const uint8_t* ff = face_flags + b;
        int nmine = 0;
        for (int c0 = gl; c0 < nt; c0 += G) {
            int4 tv = tet_at(S, c0);
            uint8_t fl = __ldg(ff + c0);
            int32_t key[3];
            for (int j = 0; j < 4; ++j) nmine += first_surface_face(S, ff, c0, tv, fl, j, key);
        }
        int incl = nmine;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            int v = __shfl_up_sync(gm, incl, o, G);
            if (gl >= o) incl += v;
        }
        const int total = __shfl_sync(gm, incl, G - 1, G);
        unsigned long long base = 0;
        if (gl == 0 && total > 0) base = atomicAdd(face_count, (unsigned long long)total);
        base = __shfl_sync(gm, base, 0, G);
        if (total > 0 && base + (unsigned long long)total > (unsigned long long)face_cap) {
            if (gl == 0) {
                atomicOr(counters + kCntError, 8ULL);
                status[sid] = TW_SMOOTH_INVALID;
            }
            continue;
        }
        int64_t w = (int64_t)base + (incl - nmine);
        for (int c0 = gl; c0 < nt; c0 += G) {
            int4 tv = tet_at(S, c0);
            uint8_t fl = __ldg(ff + c0);
            for (int j = 0; j < 4; ++j) {
                int32_t key[3];
                if (!first_surface_face(S, ff, c0, tv, fl, j, key)) continue;
                // the face from the centre onward in the cyclic order of its
                // sorted triple (:427-432)
                const int kv = (key[0] == S.v) ? 0 : (key[1] == S.v) ? 1 : 2;
                const int32_t v1 = key[(kv + 1) % 3], v2 = key[(kv + 2) % 3];
                double* f = faces + 9 * w;
                f[0] = p[0];
                f[1] = p[1];
                f[2] = p[2];
                f[3] = __ldg(vx + v1);
                f[4] = __ldg(vy + v1);
                f[5] = __ldg(vz + v1);
                f[6] = __ldg(vx + v2);
                f[7] = __ldg(vy + v2);
                f[8] = __ldg(vz + v2);
                ++w;
            }
        }
        if (gl == 0) {
            face_base[sid] = (int32_t)base;
            face_cnt[sid] = total;
            status[sid] = kSmoothPendingEnvelope;
        }
    }
}

// ---------------------------------------------------------------------------
// Checks of candidate edge collapses v1 -> v2 (EdgeCollapser.cpp:284-446),
// G lanes per edge; the point-envelope checks ran before
// (launch_collapse_points) and left kCollapsePending where they passed.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool tet_has(int4 tv, int32_t v) {
    return tv.x == v || tv.y == v || tv.z == v || tv.w == v;
}

template <int G, bool CERT>
__global__ void __launch_bounds__(256) k_collapse_stage(
    const double* __restrict__ vx, const double* __restrict__ vy, const double* __restrict__ vz,
    const int32_t* __restrict__ off, const int4* __restrict__ tets,
    const uint8_t* __restrict__ face_flags, const int32_t* __restrict__ v12,
    const uint8_t* __restrict__ flags, const uint8_t* __restrict__ degenerate, int32_t n,
    int check_quality, double soft_energy, uint8_t* __restrict__ status,
    double* __restrict__ faces, unsigned long long* __restrict__ face_count, int64_t face_cap,
    int32_t* __restrict__ face_base, int32_t* __restrict__ face_cnt,
    unsigned long long* __restrict__ counters, int form) {
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const unsigned gm = group_mask<G>(lane);
    const int64_t gid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / G;
    for (int64_t e = gid; e < n; e += ngroups) {
        if (status[e] != kCollapsePending) continue;  // uniform within the group
        const int32_t b = off[e], nt = off[e + 1] - b;
        const int32_t v1 = v12[2 * e], v2 = v12[2 * e + 1];
        StarView S{vx, vy, vz, tets + b, nt, v1, form};
        const double p1[3] = {vx[v1], vy[v1], vz[v1]};
        const double p2[3] = {vx[v2], vy[v2], vz[v2]};
        const uint8_t fl = flags[e];
        const bool deg = degenerate[e] != 0;
        // isFlip of the new tets: those without v2, v1 moved onto v2 (:336-384)
        bool bad = false;
        for (int c0 = gl; c0 < nt; c0 += G) {
            const int4 tv = tet_at(S, c0);
            if (tet_has(tv, v2)) continue;
            double T[12];
            gather_tet(S, tv, 0, p2, T);
            bad = bad || (orient3d(T, T + 3, T + 6, T + 9) != 1);
        }
        if (__any_sync(gm, bad)) {
            if (gl == 0) status[e] = 1;  // FLIP
            continue;
        }
        // quality (:390-415): max over the old tets (stored quality, or the soft
        // bound) and the new; an unrounded v1 or a degenerate edge passes
        if (check_quality && !deg && !(fl & TW_CV_V1_UNROUNDED)) {
            const bool soft = soft_energy >= 0.0;
            int worse = -1;   // not known yet
            if (CERT) {
                MaxBounds o, m;
                for (int c0 = gl; c0 < nt; c0 += G) {
                    const int4 tv = tet_at(S, c0);
                    double T[12];
                    float d1[3], d2[3], d3[3];
                    if (!soft) {
                        gather_tet(S, tv, 0, p1, T);
                        const float M = tet_diffs32(T, d1, d2, d3);
                        int ori = orient32_filter(d1, d2, d3);
                        if (ori == 2) ori = orient3d(T, T + 3, T + 6, T + 9);
                        if (ori == 1) o.add_positive(d1, d2, d3, M);
                        else o.add_sentinel();
                    }
                    if (tet_has(tv, v2)) continue;
                    gather_tet(S, tv, 0, p2, T);
                    const float M = tet_diffs32(T, d1, d2, d3);
                    m.add_positive(d1, d2, d3, M);
                }
                o.join<G>(gm);
                m.join<G>(gm);
                if (soft) {
                    o.lo = __double2float_rd(soft_energy);
                    o.hi = __double2float_ru(soft_energy);
                }
                if (o.sure && m.sure) worse = m.hi < o.lo ? 0 : m.lo > o.hi ? 1 : -1;
            }
            if (worse < 0) {
                double old_max = 0.0, new_max = 0.0;
                for (int c0 = gl; c0 < nt; c0 += G) {
                    const int4 tv = tet_at(S, c0);
                    double T[12];
                    if (!soft) {
                        gather_tet(S, tv, 0, p1, T);
                        old_max = fmax(old_max, quality_from(orient3d(T, T + 3, T + 6, T + 9),
                                                             amips_energy_f(T, S.form)));
                    }
                    if (tet_has(tv, v2)) continue;
                    gather_tet(S, tv, 0, p2, T);
                    new_max = fmax(new_max, positive_tet_quality(T, S.form));
                }
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) {
                    old_max = fmax(old_max, __shfl_xor_sync(gm, old_max, o, G));
                    new_max = fmax(new_max, __shfl_xor_sync(gm, new_max, o, G));
                }
                if (soft) old_max = soft_energy;
                worse = !(new_max <= old_max);
            }
            if (worse) {
                if (gl == 0) status[e] = 2;  // QUALITY
                continue;
            }
        }
        if (!(fl & TW_CV_V1_SURFACE) || deg) {
            if (gl == 0) status[e] = 0;  // SUCCESS
            continue;
        }
        // isCollapsable_epsilon (:727-775): the surface faces through v1 as
        // sorted triples without repeats, those through v2 dropped, v1
        // replaced by v2 in place
        const uint8_t* ff = face_flags + b;
        int nmine = 0;
        for (int c0 = gl; c0 < nt; c0 += G) {
            const int4 tv = tet_at(S, c0);
            const uint8_t f8 = __ldg(ff + c0);
            for (int j = 0; j < 4; ++j) {
                int32_t key[3];
                if (!first_surface_face(S, ff, c0, tv, f8, j, key)) continue;
                nmine += (key[0] != v2 && key[1] != v2 && key[2] != v2);
            }
        }
        int incl = nmine;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            int v = __shfl_up_sync(gm, incl, o, G);
            if (gl >= o) incl += v;
        }
        const int total = __shfl_sync(gm, incl, G - 1, G);
        if (total == 0) {
            if (gl == 0) status[e] = 0;
            continue;
        }
        unsigned long long base = 0;
        if (gl == 0) base = atomicAdd(face_count, (unsigned long long)total);
        base = __shfl_sync(gm, base, 0, G);
        if (base + (unsigned long long)total > (unsigned long long)face_cap) {
            if (gl == 0) {
                atomicOr(counters + kCntError, 8ULL);
                status[e] = 3;
            }
            continue;
        }
        int64_t w = (int64_t)base + (incl - nmine);
        for (int c0 = gl; c0 < nt; c0 += G) {
            const int4 tv = tet_at(S, c0);
            const uint8_t f8 = __ldg(ff + c0);
            for (int j = 0; j < 4; ++j) {
                int32_t key[3];
                if (!first_surface_face(S, ff, c0, tv, f8, j, key)) continue;
                if (key[0] == v2 || key[1] == v2 || key[2] == v2) continue;
                double* f = faces + 9 * w;
                for (int k = 0; k < 3; ++k) {
                    if (key[k] == v1) {
                        f[3 * k] = p2[0];
                        f[3 * k + 1] = p2[1];
                        f[3 * k + 2] = p2[2];
                    } else {
                        f[3 * k] = __ldg(vx + key[k]);
                        f[3 * k + 1] = __ldg(vy + key[k]);
                        f[3 * k + 2] = __ldg(vz + key[k]);
                    }
                }
                ++w;
            }
        }
        if (gl == 0) {
            face_base[e] = (int32_t)base;
            face_cnt[e] = total;
            status[e] = kCollapsePendingEnvelope;
        }
    }
}

__global__ void k_collapse_finalize(int32_t n, const int32_t* __restrict__ face_base,
                                    const int32_t* __restrict__ face_cnt,
                                    const uint8_t* __restrict__ face_out,
                                    uint8_t* __restrict__ status) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (status[i] != kCollapsePendingEnvelope) continue;
        bool outside = false;
        const int32_t b = face_base[i], m = face_cnt[i];
        for (int32_t k = 0; k < m && !outside; ++k) outside = face_out[b + k] != 0;
        status[i] = outside ? 3 : 0;
    }
}

__global__ void k_smooth_finalize(int32_t nstars, const int32_t* __restrict__ face_base,
                                  const int32_t* __restrict__ face_cnt,
                                  const uint8_t* __restrict__ face_out,
                                  const double* __restrict__ pnew, double* __restrict__ out,
                                  uint8_t* __restrict__ status) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nstars; i += stride) {
        if (status[i] != kSmoothPendingEnvelope) continue;
        bool outside = false;
        const int32_t b = face_base[i], n = face_cnt[i];
        for (int32_t k = 0; k < n && !outside; ++k) outside = face_out[b + k] != 0;
        if (outside) {
            status[i] = TW_SMOOTH_REJECT_ENVELOPE;
        } else {
            out[3 * i] = pnew[3 * i];
            out[3 * i + 1] = pnew[3 * i + 1];
            out[3 * i + 2] = pnew[3 * i + 2];
            status[i] = TW_SMOOTH_MOVED;
        }
    }
}

// Launch shapes: threads per block of the Newton kernel (64, 128, 256) and
// lanes per star (8, 16, 32) of the smoothing and collapse stages; the Newton
// kernel keeps 4 block / lanes stars a block in flight, at most 32 (shape 0,
// once a thread per star, equals shape 2).
struct NewtonShape {
    int group;
    int block;
};
static const NewtonShape kNewtonShapes[] = {{8, 128},  {8, 64},   {8, 128},  {8, 256},
                                            {16, 64},  {16, 128}, {16, 256}, {32, 64},
                                            {32, 128}, {32, 256}};
int newton_num_shapes() { return (int)(sizeof(kNewtonShapes) / sizeof(kNewtonShapes[0])); }

static int smooth_group(int shape, int* block) {
    if (shape < 0 || shape >= newton_num_shapes()) shape = 5;
    *block = kNewtonShapes[shape].block;
    return kNewtonShapes[shape].group;
}

static int wave_slots(int block, int group) { return std::min(kWaveSlots, 4 * block / group); }
int newton_shape_group(int shape) {
    int block;
    return smooth_group(shape, &block);
}
// Of the ten shapes the Newton kernel has six configurations, 128 and 256
// threads with 32 stars in flight three times each.
bool newton_shapes_alike(int a, int b, bool stages) {
    int ba, bb;
    const int ga = smooth_group(a, &ba), gb = smooth_group(b, &bb);
    return ba == bb && (stages ? ga == gb : wave_slots(ba, ga) == wave_slots(bb, gb));
}

template <bool SMOOTH, bool CERT>
static void launch_wave(int shape, WaveArgs A, cudaStream_t s) {
    int block;
    const int group = smooth_group(shape, &block);
    A.slots = wave_slots(block, group);
    // one star a block before two: the grid fills the SMs first
    const int grid = grid_for(A.nstars, 1, 512 / block);
    if (block == 64) k_newton_wave<SMOOTH, CERT, 64><<<grid, 64, 0, s>>>(A);
    else if (block == 128) k_newton_wave<SMOOTH, CERT, 128><<<grid, 128, 0, s>>>(A);
    else k_newton_wave<SMOOTH, CERT, 256><<<grid, 256, 0, s>>>(A);
}

void launch_newton_stars_shape(int shape, int precision, const double* vx, const double* vy,
                               const double* vz, const int32_t* star_off, const int32_t* tets,
                               const int32_t* centers, int32_t nstars, int max_step, int max_it,
                               double* out, uint8_t* moved, cudaStream_t s, int form) {
    if (nstars <= 0) return;
    const WaveArgs A{vx, vy, vz, star_off, reinterpret_cast<const int4*>(tets), centers, nullptr,
                     nstars, max_step, max_it, 0, form, out, nullptr, moved};
    if (precision == TW_PRECISION_FP32_CERTIFIED) launch_wave<false, true>(shape, A, s);
    else launch_wave<false, false>(shape, A, s);
}

void launch_smooth_stage1(int shape, int precision, const double* vx, const double* vy,
                          const double* vz, const int32_t* star_off, const int32_t* tets,
                          const int32_t* centers, const uint8_t* kinds, int32_t nstars,
                          int max_step, int max_it, double* out, double* pnew, uint8_t* status,
                          cudaStream_t s, int form) {
    if (nstars <= 0) return;
    const WaveArgs A{vx, vy, vz, star_off, reinterpret_cast<const int4*>(tets), centers, kinds,
                     nstars, max_step, max_it, 0, form, out, pnew, status};
    if (precision == TW_PRECISION_FP32_CERTIFIED) launch_wave<true, true>(shape, A, s);
    else launch_wave<true, false>(shape, A, s);
}

void launch_smooth_stage2(int shape, int precision, const double* vx, const double* vy,
                          const double* vz, const int32_t* star_off, const int32_t* tets,
                          const uint8_t* face_flags, const int32_t* centers, int32_t nstars,
                          const double* pnew, uint8_t* status, double* faces,
                          unsigned long long* face_count, int64_t face_cap, int32_t* face_base,
                          int32_t* face_cnt, unsigned long long* counters, cudaStream_t s,
                          int form) {
    if (nstars <= 0) return;
    int block;
    const int G = smooth_group(shape, &block);
    const int grid = grid_for((int64_t)nstars * G, block, 2048 / block);
    const int4* t4 = reinterpret_cast<const int4*>(tets);
    const bool cert = precision == TW_PRECISION_FP32_CERTIFIED;
    auto go = [&](auto kernel) {
        kernel<<<grid, block, 0, s>>>(vx, vy, vz, star_off, t4, face_flags, centers, nstars, pnew,
                                      status, faces, face_count, face_cap, face_base, face_cnt,
                                      counters, form);
    };
    if (G == 8) cert ? go(k_smooth_stage2<8, true>) : go(k_smooth_stage2<8, false>);
    else if (G == 16) cert ? go(k_smooth_stage2<16, true>) : go(k_smooth_stage2<16, false>);
    else cert ? go(k_smooth_stage2<32, true>) : go(k_smooth_stage2<32, false>);
}

void launch_smooth_finalize(int32_t nstars, const int32_t* face_base, const int32_t* face_cnt,
                            const uint8_t* face_out, const double* pnew, double* out,
                            uint8_t* status, cudaStream_t s) {
    if (nstars <= 0) return;
    const int block = 256;
    k_smooth_finalize<<<grid_for(nstars, block, 8), block, 0, s>>>(nstars, face_base, face_cnt,
                                                                   face_out, pnew, out, status);
}

void launch_collapse_stage(int shape, int precision, const double* vx, const double* vy,
                           const double* vz, const int32_t* off, const int32_t* tets,
                           const uint8_t* face_flags, const int32_t* v12, const uint8_t* flags,
                           const uint8_t* degenerate, int32_t n, int check_quality,
                           double soft_energy, uint8_t* status, double* faces,
                           unsigned long long* face_count, int64_t face_cap, int32_t* face_base,
                           int32_t* face_cnt, unsigned long long* counters, cudaStream_t s,
                           int form) {
    if (n <= 0) return;
    int block;
    const int G = smooth_group(shape, &block);
    const int grid = grid_for((int64_t)n * G, block, 2048 / block);
    const int4* t4 = reinterpret_cast<const int4*>(tets);
    const bool cert = precision == TW_PRECISION_FP32_CERTIFIED;
    auto go = [&](auto kernel) {
        kernel<<<grid, block, 0, s>>>(vx, vy, vz, off, t4, face_flags, v12, flags, degenerate, n,
                                      check_quality, soft_energy, status, faces, face_count,
                                      face_cap, face_base, face_cnt, counters, form);
    };
    if (G == 8) cert ? go(k_collapse_stage<8, true>) : go(k_collapse_stage<8, false>);
    else if (G == 16) cert ? go(k_collapse_stage<16, true>) : go(k_collapse_stage<16, false>);
    else cert ? go(k_collapse_stage<32, true>) : go(k_collapse_stage<32, false>);
}

void launch_collapse_finalize(int32_t n, const int32_t* face_base, const int32_t* face_cnt,
                              const uint8_t* face_out, uint8_t* status, cudaStream_t s) {
    if (n <= 0) return;
    k_collapse_finalize<<<grid_for(n, 256, 8), 256, 0, s>>>(n, face_base, face_cnt, face_out,
                                                            status);
}

}  // namespace tw
