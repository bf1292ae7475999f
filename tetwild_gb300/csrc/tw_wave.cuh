// tw_wave.cuh -- NewtonsMethod over many stars at once, a block to a set of
// stars (included by tw_newton.cu inside namespace tw).
//
// The work is binary64 evaluation of tets (the GPU issues one binary64 warp
// instruction per 17 cycles and SM), so what counts is that every lane of
// each binary64 instruction holds a tet of its own.  A block keeps up to 32
// stars in shared memory, each in a state of its own (see WaveState), and
// goes round the states: the tets of all stars in one state are laid out as
// one list that the block's threads evaluate, a tet a thread, whatever the
// stars' sizes; the per-tet terms are summed in tet order by one thread per
// star and component (so the sums round exactly as the sequential loops of
// VertexSmoother.cpp:654-672 and :606-614), and one thread per star solves
// the 3x3 system and takes the step's decisions.  A finished star's slot
// takes the next star.  A fixed group of lanes per star, as before, left a
// third of the lanes idle on the last tets of each star, summed all 13
// components on every lane and solved on every lane: 2 x the binary64
// instructions (20k stars to convergence: 5.5 ms, here 3.2, 2.9 with the
// shorter evaluations of tw_exact.cuh).
//
// CERT (TW_PRECISION_FP32_CERTIFIED): inversion signs come from the certified
// binary32 filter first, and the star energies, which only decide whether a
// trial is taken, as certified binary32 intervals; where an interval cannot
// decide, the star's energies are evaluated in binary64 (kEnergyOld /
// kEnergyNew).  J, H and every position stay binary64, so the results are the
// same bit for bit.  The first stage of the 200k-star pass (one step): 14.6 ms
// with a group of lanes per star, 5.9 here.
#pragma once

enum WaveState : int {
    kIdle,        // no star left for the slot
    kPositive,    // smoothing: all tets positive at the start?
    kUpdate,      // E, J, H at pos (NewtonsUpdate)
    kSolve,       // the step for the current a
    kTrial,       // the tets' signs and the star's energy at the trial position
    kEnergyOld,   // CERT: the energy at old in binary64
    kEnergyNew,   // CERT: the energy at the trial position in binary64
    kFinished,
};

constexpr int kWaveSlots = 32;

template <int BLOCK>
struct WaveShared {
    static constexpr int kItems = BLOCK >= 256 ? 256 : 2 * BLOCK;   // tets per round
    double val[13][kItems + 1];   // per tet: J, H, E (CERT: E and its bound as two floats)
    double pos[3][kWaveSlots], old[3][kWaveSlots], a[kWaveSlots], e_old[kWaveSlots];
    double sum[13][kWaveSlots];
    float lo[2][kWaveSlots], hi[2][kWaveSlots];   // energy interval at old [0], at pos [1]
    int sid[kWaveSlots], off[kWaveSlots], nt[kWaveSlots], v[kWaveSlots], state[kWaveSlots];
    int step[kWaveSlots], it[kWaveSlots];
    int flag[kWaveSlots];         // bit 0: a tet not positive, bit 1: no binary32 energy
    uint8_t kind[kWaveSlots], moved[kWaveSlots], exact[kWaveSlots], pending[kWaveSlots];
    uint8_t status[kWaveSlots];
    int act[kWaveSlots], start[kWaveSlots + 1];
    int nact, fetched, live;
};

struct WaveArgs {
    const double* vx;
    const double* vy;
    const double* vz;
    const int32_t* star_off;
    const int4* tets;
    const int32_t* centers;
    const uint8_t* kinds;      // smoothing (may be null)
    int32_t nstars;
    int max_step, max_it, slots, form;
    double* out;
    double* pnew;              // smoothing
    uint8_t* status;           // smoothing: the state; else moved
};

template <bool SMOOTH, bool CERT, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 512 / BLOCK) k_newton_wave(WaveArgs A) {
    __shared__ WaveShared<BLOCK> W;
    constexpr int kItems = WaveShared<BLOCK>::kItems;
    const int tid = threadIdx.x;

    // ---- one thread per slot ----
    auto enter_update = [&](int s) {
#pragma unroll
        for (int k = 0; k < 3; ++k) W.old[k][s] = W.pos[k][s];
        W.exact[s] = 0;
        W.state[s] = kUpdate;
    };
    auto fetch = [&](int s) {
        const int64_t sid = (int64_t)blockIdx.x + (int64_t)gridDim.x * atomicAdd(&W.fetched, 1);
        if (sid >= A.nstars) {
            W.state[s] = kIdle;
            return;
        }
        const int32_t b = A.star_off[sid], v = A.centers[sid];
        W.sid[s] = (int)sid;
        W.off[s] = b;
        W.nt[s] = A.star_off[sid + 1] - b;
        W.v[s] = v;
        W.pos[0][s] = A.vx[v];
        W.pos[1][s] = A.vy[v];
        W.pos[2][s] = A.vz[v];
        W.kind[s] = SMOOTH && A.kinds ? A.kinds[sid] : (uint8_t)TW_STAR_INTERIOR;
        W.step[s] = 0;
        W.moved[s] = 0;
        if (SMOOTH) {
            W.status[s] = TW_SMOOTH_NOT_MOVED;
            W.state[s] = kPositive;
        } else if (A.max_step > 0) {
            enter_update(s);
        } else {
            W.state[s] = kFinished;
        }
    };
    auto finish = [&](int s) {
        const int64_t sid = W.sid[s];
        const double p[3] = {W.pos[0][s], W.pos[1][s], W.pos[2][s]};
        if (SMOOTH) {
            const bool surface = W.kind[s] == TW_STAR_SURFACE || W.kind[s] == TW_STAR_BOUNDARY;
            uint8_t st = W.status[s];
            if (W.moved[s]) st = surface ? kSmoothPendingProject : (uint8_t)TW_SMOOTH_MOVED;
            const bool moved = st == TW_SMOOTH_MOVED;
            const int32_t v = W.v[s];
            A.out[3 * sid] = moved ? p[0] : A.vx[v];
            A.out[3 * sid + 1] = moved ? p[1] : A.vy[v];
            A.out[3 * sid + 2] = moved ? p[2] : A.vz[v];
#pragma unroll
            for (int k = 0; k < 3; ++k) A.pnew[3 * sid + k] = p[k];
            A.status[sid] = st;
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) A.out[3 * sid + k] = p[k];
            A.status[sid] = W.moved[s];
        }
    };
    auto step_not_taken = [&](int s) {
        W.moved[s] = W.step[s] != 0;
        W.state[s] = kFinished;
    };
    auto reject = [&](int s) {
#pragma unroll
        for (int k = 0; k < 3; ++k) W.pos[k][s] = W.old[k][s];
        W.a[s] = W.a[s] / 2.0;
        if (++W.it[s] >= A.max_it) step_not_taken(s);
        else W.state[s] = kSolve;
    };
    // the trial is taken; small: the energies differ by less than 1e-5
    auto accept = [&](int s, bool small) {
        if (small) {
            step_not_taken(s);
            return;
        }
        W.moved[s] = 1;
        if (++W.step[s] >= A.max_step) W.state[s] = kFinished;
        else enter_update(s);
    };
    auto decide = [&](int s, double sum) {
        if (isinf(sum) || isnan(sum) || sum <= 0.0 || sum > kMaxEnergy) sum = kMaxEnergy;
        const double old_energy = W.e_old[s];
        if (sum >= old_energy) reject(s);
        else accept(s, fabs(sum - old_energy) < 1e-5);
    };
    // after E, J, H (energy: e_old is the binary64 sum): the step's first trial
    auto after_update = [&](int s, bool energy) {
        bool ok = true;
        if (energy) {
            const double e = W.e_old[s];
            ok = !isnan(e) && !(e <= 0.0);
        }
#pragma unroll
        for (int k = 0; k < 12; ++k) ok = ok && isfinite(W.sum[k][s]);
        if (!ok) {
            W.state[s] = kFinished;
            return;
        }
        W.a[s] = 1.0;
        W.it[s] = 0;
        if (A.max_it <= 0) step_not_taken(s);
        else W.state[s] = kSolve;
    };

    // ---- the whole block ----
    // lists the slots in one of the states (a bit set) and their tets
    auto collect = [&](unsigned states) -> int {
        __syncthreads();
        if (tid < 32) {
            const bool in = (states >> W.state[tid]) & 1u;
            const unsigned bal = __ballot_sync(0xffffffffu, in);
            int incl = in ? W.nt[tid] : 0;
            const int own = incl;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += t;
            }
            if (in) {
                const int r = __popc(bal & ((1u << tid) - 1u));
                W.act[r] = tid;
                W.start[r] = incl - own;
                W.flag[tid] = 0;
                const int side = states == (1u << kUpdate) ? 0 : 1;
                W.lo[side][tid] = W.hi[side][tid] = 0.0f;
#pragma unroll
                for (int k = 0; k < 13; ++k)
                    if (k == 12 || states == (1u << kUpdate)) W.sum[k][tid] = 0.0;
            }
            if (tid == 31) {
                W.nact = __popc(bal);
                W.start[__popc(bal)] = incl;
            }
        }
        __syncthreads();
        return W.nact;
    };
    // evaluates eval(slot, tet index, item) for the listed tets, and adds the
    // terms of each round (add(listed star, component, first, end))
    auto sweep = [&](int nact, int ncomp, auto&& eval, auto&& add) {
        const int total = W.start[nact];
        for (int c0 = 0; c0 < total; c0 += kItems) {
            const int cend = min(c0 + kItems, total);
            for (int i = c0 + tid; i < cend; i += BLOCK) {
                int k = 0;
#pragma unroll
                for (int o = kWaveSlots / 2; o > 0; o >>= 1)
                    if (k + o < nact && W.start[k + o] <= i) k += o;
                eval(W.act[k], i - W.start[k], i - c0);
            }
            __syncthreads();
            for (int j = tid; j < nact * ncomp; j += BLOCK) {
                const int k = j / ncomp;
                const int b = max(W.start[k], c0), e = min(W.start[k + 1], cend);
                if (b < e) add(W.act[k], j - k * ncomp, b - c0, e - c0);
            }
            __syncthreads();
        }
    };
    auto view = [&](int s) {
        return StarView{A.vx, A.vy, A.vz, A.tets + W.off[s], W.nt[s], W.v[s], A.form};
    };
    auto add_interval = [&](int s, int side, int b, int e) {
        float lo = W.lo[side][s], hi = W.hi[side][s];
        for (int i = b; i < e; ++i) {
            const float2 er = *reinterpret_cast<const float2*>(&W.val[12][i]);
            lo = __fadd_rd(lo, __fmul_rd(er.x, 1.0f - er.y));
            hi = __fadd_ru(hi, __fmul_ru(er.x, 1.0f + er.y));
        }
        W.lo[side][s] = lo;
        W.hi[side][s] = hi;
    };
    auto add_sum = [&](int s, int c, int b, int e) {
        double x = W.sum[c][s];
        for (int i = b; i < e; ++i) x += W.val[c][i];
        W.sum[c][s] = x;
    };
    auto put_interval = [&](int s, const float* d1, const float* d2, const float* d3, float M,
                            int item) {
        const Energy32 r = amips_energy32(d1, d2, d3, M);
        if (!r.ok) atomicOr(&W.flag[s], 2);
        *reinterpret_cast<float2*>(&W.val[12][item]) = make_float2(r.E, r.rel);
    };

    if (tid == 0) W.fetched = 0;
    if (tid < kWaveSlots) W.state[tid] = kIdle;
    __syncthreads();
    if (tid < A.slots) fetch(tid);
    for (;;) {
        // signs (and energies) at pos
        int nact = collect((1u << kPositive) | (1u << kTrial));
        if (nact) {
            sweep(
                nact, 1,
                [&](int s, int t, int item) {
                    const double p[3] = {W.pos[0][s], W.pos[1][s], W.pos[2][s]};
                    double T[12];
                    const StarView S = view(s);
                    gather_tet(S, __ldg(S.tets + t), 0, p, T);
                    float d1[3], d2[3], d3[3];
                    const float M = tet_diffs32(T, d1, d2, d3);
                    int ori = orient32_filter(d1, d2, d3);
                    if (ori == 2) ori = orient3d(T, T + 3, T + 6, T + 9);
                    if (ori != 1) atomicOr(&W.flag[s], 1);
                    if (W.state[s] == kTrial) {
                        if (CERT) put_interval(s, d1, d2, d3, M, item);
                        else W.val[12][item] = amips_energy_f(T, A.form);
                    }
                },
                [&](int s, int, int b, int e) {
                    if (W.state[s] != kTrial) return;
                    if (CERT) add_interval(s, 1, b, e);
                    else add_sum(s, 12, b, e);
                });
            if (tid < kWaveSlots) {
                const int s = tid;
                if (W.state[s] == kPositive) {
                    if (W.flag[s] & 1) {
                        W.status[s] = TW_SMOOTH_INVALID;
                        W.state[s] = kFinished;
                    } else if (A.max_step > 0) {
                        enter_update(s);
                    } else {
                        W.state[s] = kFinished;
                    }
                } else if (W.state[s] == kTrial) {
                    if (W.flag[s] & 1) {
                        reject(s);
                    } else if (!CERT) {
                        decide(s, W.sum[12][s]);
                    } else {
                        const float olo = W.lo[0][s], ohi = W.hi[0][s];
                        const float nlo = W.lo[1][s], nhi = W.hi[1][s];
                        const bool sure = !(W.flag[s] & 2);
                        if (sure && __fadd_ru(nhi, 1.1e-5f) < olo) accept(s, false);
                        else if (sure && nlo > ohi) reject(s);
                        else if (W.exact[s]) W.state[s] = kEnergyNew;
                        else {
                            W.pending[s] = 1;
                            W.state[s] = kEnergyOld;
                        }
                    }
                }
            }
        }
        if (CERT) {
            // energies in binary64 where the intervals left them open
            nact = collect((1u << kEnergyOld) | (1u << kEnergyNew));
            if (nact) {
                sweep(
                    nact, 1,
                    [&](int s, int t, int item) {
                        const bool o = W.state[s] == kEnergyOld;
                        const double p[3] = {o ? W.old[0][s] : W.pos[0][s],
                                             o ? W.old[1][s] : W.pos[1][s],
                                             o ? W.old[2][s] : W.pos[2][s]};
                        double T[12];
                        const StarView S = view(s);
                        const int4 tv = __ldg(S.tets + t);
                        // the energies of an update are those of the rotated tets
                        gather_tet(S, tv, o ? centre_index(tv, S.v) : 0, p, T);
                        W.val[12][item] = amips_energy_f(T, A.form);
                    },
                    [&](int s, int, int b, int e) { add_sum(s, 12, b, e); });
                if (tid < kWaveSlots) {
                    const int s = tid;
                    if (W.state[s] == kEnergyOld) {
                        double e = W.sum[12][s];
                        if (isinf(e)) e = kMaxEnergy;
                        W.e_old[s] = e;
                        W.exact[s] = 1;
                        W.lo[0][s] = __double2float_rd(e);
                        W.hi[0][s] = __double2float_ru(e);
                        if (W.pending[s]) W.state[s] = kEnergyNew;
                        else after_update(s, true);
                    } else if (W.state[s] == kEnergyNew) {
                        decide(s, W.sum[12][s]);
                    }
                }
            }
        }
        // E, J, H
        nact = collect(1u << kUpdate);
        if (nact) {
            sweep(
                nact, 13,
                [&](int s, int t, int item) {
                    const double p[3] = {W.pos[0][s], W.pos[1][s], W.pos[2][s]};
                    double T[12], J[3], H[9];
                    const StarView S = view(s);
                    const int4 tv = __ldg(S.tets + t);
                    gather_tet(S, tv, centre_index(tv, S.v), p, T);
                    if (CERT) {
                        float d1[3], d2[3], d3[3];
                        const float M = tet_diffs32(T, d1, d2, d3);
                        put_interval(s, d1, d2, d3, M, item);
                        amips_jh_f(T, J, H, A.form);
                    } else {
                        W.val[12][item] = amips_egh_f(T, J, H, A.form);
                    }
#pragma unroll
                    for (int k = 0; k < 3; ++k) W.val[k][item] = J[k];
#pragma unroll
                    for (int k = 0; k < 9; ++k) W.val[3 + k][item] = H[k];
                },
                [&](int s, int c, int b, int e) {
                    if (CERT && c == 12) add_interval(s, 0, b, e);
                    else add_sum(s, c, b, e);
                });
            if (tid < kWaveSlots && W.state[tid] == kUpdate) {
                const int s = tid;
                if (CERT) {
                    if ((W.flag[s] & 2) || W.nt[s] == 0 || !(W.lo[0][s] > 0.0f)) {
                        W.pending[s] = 0;
                        W.state[s] = kEnergyOld;
                    } else {
                        after_update(s, false);
                    }
                } else {
                    double e = W.sum[12][s];
                    if (isinf(e)) e = kMaxEnergy;
                    W.e_old[s] = e;
                    after_update(s, true);
                }
            }
        }
        // the step for the current a; finished stars make room
        __syncthreads();
        if (tid < 32) {
            const int s = tid;
            while (W.state[s] == kSolve) {
                double H[9], rhs[3], X[3];
#pragma unroll
                for (int k = 0; k < 9; ++k) H[k] = W.sum[3 + k][s];
                const double x0 = W.old[0][s], x1 = W.old[1][s], x2 = W.old[2][s], a = W.a[s];
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    rhs[i] = ((H[3 * i] * x0 + H[3 * i + 1] * x1) + H[3 * i + 2] * x2) -
                             a * W.sum[i][s];
                qr_solve3(H, rhs, X);
                if (!isfinite(X[0]) || !isfinite(X[1]) || !isfinite(X[2])) {
                    reject(s);
                    continue;
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) W.pos[k][s] = X[k];
                W.state[s] = kTrial;
            }
            if (W.state[s] == kFinished) {
                finish(s);
                fetch(s);
            }
            const bool any = __any_sync(0xffffffffu, W.state[s] != kIdle);
            if (s == 0) W.live = any;
        }
        __syncthreads();
        if (!W.live) return;
    }
}
