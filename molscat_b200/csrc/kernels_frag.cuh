// LDMD / LDJ / LDMG kernels on DMMA fragments: one warp per matrix (N <= 64).
// Included by propagator.cu after SysDev, JobDev, ref_solutions.
//
// Fragment layout (see warp_dmma.cuh): for every lower 8x8 tile t and lane l,
// the two doubles of positions (l>>2, 2(l&3) + s) of the tile, channels
// 8I + chan_of(l>>2) and 8J + chan_of(2(l&3) + s), are stored at [t][l][s], so
// one warp reads or writes a tile as 512 contiguous bytes.
// VL is stored [term][t][l][s]; the 2HQ(C) table [step][t][l][s].
//
// Padding channels (N .. 8 NT - 1) are uncoupled; every kernel gives those that
// share a pivot block with a real channel a positive diagonal before an
// inversion, so the sweep needs no test for them.  A half tile that is all
// padding is not swept (warp_sweep_invert), so its diagonal is arbitrary:
// LDPROP's drifts by -4.125 a step, LDMG's by 2/(a_k h) a stage.
#pragma once
#include "warp_dmma.cuh"

namespace mgpu {
namespace wf {

constexpr int kWPB = 4;  // warps (matrices) per CTA

// Doubles of shared memory per warp: the sweep's buffers, five channel vectors
// (y14, y14', y23 by position; EINT, CENT by channel) and one tiled matrix
// (LDMD: 2HQ(C_k); LDJ: the parked Z).
template <int NT>
struct WarpSmem {
    static constexpr int PAN = G<NT>::WSM;
    static constexpr int VEC = G<NT>::NPAD;
    static constexpr int QD = G<NT>::NTL * 64;
    static constexpr int DOUBLES = PAN + 5 * VEC + QD;
    static constexpr size_t BYTES = (size_t)DOUBLES * 8;
};

// f(t, I, J, sum0, sum1) for every tile with the coupling sum
// sum_l VL_l P_l(R_ir) (SUMLAM, sumlam.f:29-36,74-86) of this lane's two
// elements: the part of W(R) that does not depend on the energy or on
// EINT/CENT.  Up to CH tiles' sums are formed together, so that their loads
// overlap, and only those are held in registers.
template <int NT, class F>
__device__ __forceinline__ void w_sum_each(const SysDev &S, int lane, int ir, F &&f)
{
    constexpr int NTL = G<NT>::NTL;
    constexpr int CH = NTL <= 15 ? NTL : 9;
    const double *P = S.ptab + (size_t)ir * S.nham;
    const double *V = S.vlt + lane * 2;
    const int *IVT = S.ivt + lane * 2;
#pragma unroll
    for (int t0 = 0; t0 < NTL; t0 += CH) {
        double w[CH][2];
#pragma unroll
        for (int u = 0; u < CH; ++u) w[u][0] = w[u][1] = 0.0;
        for (int l = 0; l < S.nham; ++l) {
            const double *v = V + ((size_t)l * NTL + t0) * 64;
            if (S.ivlfl <= 0) {
                const double pl = __ldg(P + l);
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    if (t0 + u < NTL) {
                        const double2 x = __ldg(reinterpret_cast<const double2 *>(v + u * 64));
                        w[u][0] = fma(x.x, pl, w[u][0]);
                        w[u][1] = fma(x.y, pl, w[u][1]);
                    }
            } else {
                const int *iv = IVT + ((size_t)l * NTL + t0) * 64;
#pragma unroll
                for (int u = 0; u < CH; ++u)
                    if (t0 + u < NTL) {
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const double x = __ldg(v + u * 64 + s);
                            if (x != 0.0) w[u][s] = fma(x, __ldg(P + __ldg(iv + u * 64 + s)), w[u][s]);
                        }
                    }
            }
        }
#pragma unroll
        for (int I = 0; I < NT; ++I)
#pragma unroll
            for (int J = 0; J <= I; ++J)
                if (tix(I, J) >= t0 && tix(I, J) < t0 + CH) f(tix(I, J), I, J, w[tix(I, J) - t0][0], w[tix(I, J) - t0][1]);
    }
}

// The diagonal terms of W(R_ir) (HAMMAT, hammat.f:85-113): CENT/R^2 (the
// 1e16 clamp), EINT, the confinement term, then -ERED.  x is the coupling
// sum of channel i's diagonal element.
__device__ __forceinline__ double w_diag_terms(const SysDev &S, const double *eint, const double *cent, int i, double x,
                                               double rsq, double conf, double ered)
{
    if (S.nrsq == 0) x += rsq * cent[i];
    if (S.nconst == 0) x += eint[i];
    if (S.conlen > 0.0) x += conf;
    return x - ered;
}

__device__ __forceinline__ void w_radial(const SysDev &S, int ir, double &rsq, double &conf)
{
    const double R = __ldg(S.rtab + ir);
    rsq = fmin(1.0 / (R * R), 1.0e16);
    conf = 0.0;
    if (S.conlen > 0.0) {
        const double c2 = S.conlen * S.conlen;
        conf = R * R / (c2 * c2);
    }
}

// Add the diagonal terms to this lane's elements (w0, w1) of diagonal tile I.
__device__ __forceinline__ void w_diag_add(const SysDev &S, const double *eint, const double *cent, int lane, int I,
                                           double rsq, double conf, double ered, double &w0, double &w1)
{
    const int i = frow(I, lane);
    if ((lane & 3) == (lane >> 3) && i < S.n) {
        const bool s = (lane >> 2) & 1;
        const double x = w_diag_terms(S, eint, cent, i, s ? w1 : w0, rsq, conf, ered);
        if (s) w1 = x;
        else w0 = x;
    }
}

// f(t, I, J, w0, w1) for every tile with W(R_ir) (HAMMAT + SUMLAM, hammat.f:85-113)
// of this lane's two elements.
template <int NT, class F>
__device__ __forceinline__ void w_each(const SysDev &S, const double *eint, const double *cent, int lane, int ir,
                                       double ered, F &&f)
{
    double rsq, conf;
    w_radial(S, ir, rsq, conf);
    w_sum_each<NT>(S, lane, ir, [&](int t, int I, int J, double w0, double w1) {
        if (I == J) w_diag_add(S, eint, cent, lane, I, rsq, conf, ered, w0, w1);
        f(t, I, J, w0, w1);
    });
}

// EINT and CENT into this warp's shared memory.
template <int NT>
__device__ __forceinline__ void stage_channels(const SysDev &S, int lane, double *eint, double *cent)
{
    for (int i = lane; i < G<NT>::NPAD; i += 32) {
        eint[i] = __ldg(S.eint + i);
        cent[i] = __ldg(S.cent + i);
    }
    __syncwarp();
}

// The coupling sum of W(R_ir)_ii for channel i.
template <int NT>
__device__ __forceinline__ double w_diag_sum_frag(const SysDev &S, int i, int ir)
{
    constexpr int NTL = G<NT>::NTL;
    const int I = i >> 3, r = pos_of(i & 7);
    const int lane = r * 4 + (r >> 1), s = r & 1;  // lane holding position (r, r) of tile (I, I)
    const size_t e = (size_t)tix(I, I) * 64 + lane * 2 + s;
    const double *P = S.ptab + (size_t)ir * S.nham;
    double x = 0.0;
    for (int l = 0; l < S.nham; ++l) {
        const double v = __ldg(S.vlt + (size_t)l * NTL * 64 + e);
        if (S.ivlfl <= 0) x = fma(v, __ldg(P + l), x);
        else if (v != 0.0) x = fma(v, __ldg(P + __ldg(S.ivt + (size_t)l * NTL * 64 + e)), x);
    }
    return x;
}

// W(R_2k-1)_ii (the DIAG array of HAMMAT) for the step loop, the coupling sum
// from the system's table when it has one.
template <int NT>
__device__ __forceinline__ double w_mid_diag_frag(const SysDev &S, const double *eint, const double *cent, int i, int k,
                                                  double ered)
{
    double rsq, conf;
    w_radial(S, 2 * k - 1, rsq, conf);
    const double x = S.wd != nullptr ? __ldg(S.wd + (size_t)(k - 1) * G<NT>::NPAD + i)
                                     : w_diag_sum_frag<NT>(S, i, 2 * k - 1);
    return w_diag_terms(S, eint, cent, i, x, rsq, conf, ered);
}

template <int NT>
__device__ __forceinline__ void load_lower_frag(const double *__restrict__ y, int n, int lane,
                                                double (&a)[G<NT>::NTL][2])
{
#pragma unroll
    for (int I = 0; I < NT; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int i = frow(I, lane), j = fcol(J, lane, s);
                const int lo = i < j ? i : j, hi = i < j ? j : i;
                a[tix(I, J)][s] = (i < n && j < n) ? y[(size_t)lo * n + hi] : 0.0;
            }
}

template <int NT>
__device__ __forceinline__ void store_full_frag(double *__restrict__ y, int n, int lane, double scale,
                                                const double (&a)[G<NT>::NTL][2])
{
#pragma unroll
    for (int I = 0; I < NT; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int i = frow(I, lane), j = fcol(J, lane, s);
                if (i < n && j <= i) {
                    const double x = scale * a[tix(I, J)][s];
                    y[(size_t)j * n + i] = x;
                    y[(size_t)i * n + j] = x;
                }
            }
}

// Resident CTAs (of kWPB warps) per SM the register budgets are set for.
#ifndef MGPU_FMB
#define MGPU_FMB 8, 6, 5, 4, 3, 2, 2, 2
#endif
constexpr int kFragBlocks[8] = {MGPU_FMB};
constexpr int frag_min_blocks(int nt) { return kFragBlocks[nt - 1]; }
// ---------------------------------------------------------------------------
// MDPROP energy-independent half on fragments: grid (ceil(NSTEP/kWPB), systems).
// ---------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(32 * kWPB, frag_min_blocks(NT))
ldmd_prep_frag_kernel(const SysDev *__restrict__ systems, const int *__restrict__ sys_list)
{
    constexpr int NTL = G<NT>::NTL;
    __shared__ __align__(16) double pans[kWPB][G<NT>::WSM];
    __shared__ SysDev s_sys;
    if (threadIdx.x == 0) s_sys = systems[sys_list[blockIdx.y]];
    __syncthreads();
    const SysDev &S = s_sys;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = blockIdx.x * kWPB + warp + 1;
    if (k > S.nstep) return;  // whole warp
    const double h = S.dr / 2.0;
    const double d1 = h * h / 3.0;
    const double d4 = -d1 / 16.0;
    if (S.wt != nullptr) {
        // the step loop's coupling sums: W at R_2k (and R_0 for the first
        // step) and the diagonal at R_2k-1, the same arithmetic as there
        for (int m = (k == 1 ? 0 : k); m <= k; ++m) {
            double *dst = S.wt + (size_t)m * NTL * 64 + lane * 2;
            w_sum_each<NT>(S, lane, 2 * m, [&](int t, int, int, double w0, double w1) {
                *reinterpret_cast<double2 *>(dst + t * 64) = make_double2(w0, w1);
            });
        }
    }
    double a[NTL][2];
    w_sum_each<NT>(S, lane, 2 * k - 1, [&](int t, int I, int J, double w0, double w1) {
        if (I == J && S.wd != nullptr && (lane & 3) == (lane >> 3))
            S.wd[(size_t)(k - 1) * G<NT>::NPAD + frow(I, lane)] = ((lane >> 2) & 1) ? w1 : w0;
        a[t][0] = (I == J && fdiag(lane, 0)) ? 0.125 : d4 * w0;
        a[t][1] = (I == J && fdiag(lane, 1)) ? 0.125 : d4 * w1;
    });
    int bad = SWEEP_OK;
    const int cnt = warp_sweep_invert<NT>(a, pans[warp], S.n, lane, bad);
    if (bad != SWEEP_OK) {
        if (lane == 0) {
            atomicMax(&S.prep[1], bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE);
            atomicMin(&S.prep[2], k);
        }
        return;
    }
    if (lane == 0 && cnt) atomicAdd(&S.prep[0], cnt);
    double *q = S.q + (size_t)(k - 1) * NTL * 64 + lane * 2;
#pragma unroll
    for (int I = 0; I < NT; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J) {
            double2 v;
            const int i = frow(I, lane);
            // a = -U^{-1};  2HQ(C) = U^{-1} - 8I
            const int j0 = fcol(J, lane, 0), j1 = fcol(J, lane, 1);
            v.x = (i >= S.n || j0 >= S.n) ? 0.0 : (i == j0 ? -a[tix(I, J)][0] - 8.0 : -a[tix(I, J)][0]);
            v.y = (i >= S.n || j1 >= S.n) ? 0.0 : (i == j1 ? -a[tix(I, J)][1] - 8.0 : -a[tix(I, J)][1]);
            *reinterpret_cast<double2 *>(q + tix(I, J) * 64) = v;
        }
}

// ---------------------------------------------------------------------------
// MDPROP step loop, one warp per job.
// ---------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(32 * kWPB, frag_min_blocks(NT))
ldmd_prop_frag_kernel(const SysDev *__restrict__ systems, const JobDev *__restrict__ jobs, int njobs,
                      double *__restrict__ y, int *__restrict__ nodes_out, int *__restrict__ status_out,
                      int *__restrict__ kfail_out)
{
    constexpr int NTL = G<NT>::NTL;
    constexpr int NPAD = G<NT>::NPAD;
    using W = WarpSmem<NT>;
    extern __shared__ __align__(16) double dsm[];
    __shared__ __align__(8) uint64_t qbar[kWPB];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int jix = blockIdx.x * kWPB + warp;
    if (jix >= njobs) return;  // whole warp; the kernel has no CTA-wide barrier
    const JobDev job = jobs[jix];
    const SysDev &S = systems[job.sys];
    double *pan = dsm + (size_t)warp * W::DOUBLES;
    double *s_y14 = pan + W::PAN;
    double *s_y14b = s_y14 + W::VEC;
    double *s_y23 = s_y14b + W::VEC;
    double *s_eint = s_y23 + W::VEC;
    double *s_cent = s_eint + W::VEC;
    double *qbuf = s_cent + W::VEC;
    const int n = S.n;
    const int nstep = S.nstep;
    const double ered = job.ered;
    const uint32_t qbytes = (uint32_t)(NTL * 64 * sizeof(double));
    uint64_t *bar = &qbar[warp];

    if (S.prep[1] != 0) {
        if (lane == 0) {
            status_out[job.out] = S.prep[1];
            kfail_out[job.out] = S.prep[2];
            nodes_out[job.out] = 0;
        }
        return;
    }
    // by position; a padding channel's diagonal is then 1 or 2 at every inversion
    for (int i = lane; i < NPAD; i += 32) {
        s_y14[i] = 0.5;
        s_y14b[i] = 1.0;
        s_y23[i] = 0.0;
    }
    stage_channels<NT>(S, lane, s_eint, s_cent);
    if (lane == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (lane == 0) bulk_load(qbuf, S.q, qbytes, bar);  // 2HQ(C_1); copy m completes phase m&1

    const double h = S.dr / 2.0;
    const double d1 = h * h / 3.0;
    const double d2 = 2.0 * d1;
    const double half = 0.5 * h;
    double *yj = y + job.yoff;

    double a[NTL][2];
    load_lower_frag<NT>(yj, n, lane, a);
    w_each<NT>(S, s_eint, s_cent, lane, 0, ered, [&](int t, int, int, double w0, double w1) {
        a[t][0] = fma(h, a[t][0], d1 * w0);  // mdprop.f:89-93
        a[t][1] = fma(h, a[t][1], d1 * w1);
    });
    const int r = lane >> 2, q = lane & 3;
    int nodes = 0, status = MGPU_OK, kfail = 0;
    int issued = 1, consumed = 0;
    const unsigned long long t0 = global_ns();
    const uint32_t wait_limit = g_step_wait_limit;
    const bool tabled = S.wt != nullptr;
    for (int k = 1; k <= nstep; ++k) {
        if (stop_poll_step(k)) {  // host cancel / time limit, lane 0's reading for the warp
            int stop = lane == 0 ? stop_requested(S.ctl, t0) : MGPU_OK;
            stop = __shfl_sync(0xffffffffu, stop, 0);
            if (stop != MGPU_OK) {
                status = stop;
                kfail = k;
                break;
            }
        }
        // reference-potential solutions in the sector (mdprop.f:143-164)
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            const double wref = w_mid_diag_frag<NT>(S, s_eint, s_cent, i, k, ered);
            double y14, y23;
            ref_solutions(wref, half, y14, y23);
            const int p = (i & ~7) + pos_of(i & 7);
            s_y14[p] = y14;
            s_y14b[p] = y14 - d1 * wref;
            s_y23[p] = y23;
        }
        __syncwarp();
#pragma unroll
        for (int I = 0; I < NT; ++I) {
            const double d = s_y14b[8 * I + r];
            if (fdiag(lane, 0)) a[tix(I, I)][0] += d;
            if (fdiag(lane, 1)) a[tix(I, I)][1] += d;
        }
        int bad = SWEEP_OK;
        nodes += warp_sweep_invert<NT>(a, pan, n, lane, bad);
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        // copy m of the run (2HQ(C_1), W(R_2), 2HQ(C_2), ..; without a table of
        // coupling sums only the former) completes phase (m - 1) & 1
        const bool landed = mbar_wait_bounded(bar, consumed & 1, wait_limit);
        if (__any_sync(0xffffffffu, !landed)) {
            status = MGPU_ERR_TIMEOUT;
            kfail = k;
            break;
        }
        ++consumed;
        {
            const double *qs = qbuf + lane * 2;
            // Y = 2HQ(C) + 2 Y14 - Y23 Y^-1 Y23   (a holds -Y^-1), mdprop.f:156,181-185
#pragma unroll
            for (int I = 0; I < NT; ++I) {
                const double yr = s_y23[8 * I + r];
#pragma unroll
                for (int J = 0; J <= I; ++J) {
                    const double2 qq = *reinterpret_cast<const double2 *>(qs + tix(I, J) * 64);
                    const double2 yc = *reinterpret_cast<const double2 *>(s_y23 + 8 * J + 2 * q);
                    a[tix(I, J)][0] = qq.x + yr * a[tix(I, J)][0] * yc.x;
                    a[tix(I, J)][1] = qq.y + yr * a[tix(I, J)][1] * yc.y;
                }
                const double d = 2.0 * s_y14[8 * I + r];
                if (fdiag(lane, 0)) a[tix(I, I)][0] += d;
                if (fdiag(lane, 1)) a[tix(I, I)][1] += d;
            }
        }
        // every lane has read 2HQ(C_k): the async proxy may refill the buffer,
        // with the coupling sums of this step's W while the second inversion runs
        __syncwarp();
        if (tabled || k + 1 <= nstep) {
            if (lane == 0) {
                fence_async_shared();
                bulk_load(qbuf, tabled ? S.wt + (size_t)k * NTL * 64 : S.q + (size_t)k * NTL * 64, qbytes, bar);
            }
            ++issued;
        }
        nodes += warp_sweep_invert<NT>(a, pan, n, lane, bad);
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        {
            const double dd = (k == nstep) ? d1 : d2;
            if (tabled) {
                const bool there = mbar_wait_bounded(bar, consumed & 1, wait_limit);
                if (__any_sync(0xffffffffu, !there)) {
                    status = MGPU_ERR_TIMEOUT;
                    kfail = k;
                    break;
                }
                ++consumed;
            }
            auto finish = [&](int t, int I, int J, double w0, double w1) {
                const double yr = s_y23[8 * I + r];
                const double2 yc = *reinterpret_cast<const double2 *>(s_y23 + 8 * J + 2 * q);
                a[t][0] = fma(dd, w0, yr * a[t][0] * yc.x);
                a[t][1] = fma(dd, w1, yr * a[t][1] * yc.y);
                if (I == J) {
                    const double d = s_y14b[8 * I + r];
                    if (fdiag(lane, 0)) a[t][0] += d;
                    if (fdiag(lane, 1)) a[t][1] += d;
                }
            };
            if (tabled) {
                double rsq, conf;
                w_radial(S, 2 * k, rsq, conf);
                const double *ws = qbuf + lane * 2;
#pragma unroll
                for (int I = 0; I < NT; ++I)
#pragma unroll
                    for (int J = 0; J <= I; ++J) {
                        const double2 x = *reinterpret_cast<const double2 *>(ws + tix(I, J) * 64);
                        double w0 = x.x, w1 = x.y;
                        if (I == J) w_diag_add(S, s_eint, s_cent, lane, I, rsq, conf, ered, w0, w1);
                        finish(tix(I, J), I, J, w0, w1);
                    }
                __syncwarp();
                if (k + 1 <= nstep) {
                    if (lane == 0) {
                        fence_async_shared();
                        bulk_load(qbuf, S.q + (size_t)k * NTL * 64, qbytes, bar);
                    }
                    ++issued;
                }
            } else {
                w_each<NT>(S, s_eint, s_cent, lane, 2 * k, ered, finish);
            }
        }
    }
    if (status != MGPU_OK && lane == 0 && issued > consumed) {
        // an early exit can leave one copy in flight: let it land (bounded)
        // before this warp's shared memory can be reused
        mbar_wait_bounded(bar, (issued - 1) & 1);
    }
    __syncwarp();
    if (status == MGPU_OK) store_full_frag<NT>(yj, n, lane, 1.0 / h, a);
    if (lane == 0) {
        status_out[job.out] = status;
        kfail_out[job.out] = kfail;
        nodes_out[job.out] = status == MGPU_OK ? nodes - S.prep[0] : 0;
    }
}

// ---------------------------------------------------------------------------
// LDPROP step loop, one warp per job (ldprop.f:46-147).
// ---------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(32 * kWPB, frag_min_blocks(NT))
ldj_prop_frag_kernel(const SysDev *__restrict__ systems, const JobDev *__restrict__ jobs, int njobs,
                     double *__restrict__ y, int *__restrict__ nodes_out, int *__restrict__ status_out,
                     int *__restrict__ kfail_out)
{
    constexpr int NTL = G<NT>::NTL;
    using W = WarpSmem<NT>;
    extern __shared__ __align__(16) double dsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int jix = blockIdx.x * kWPB + warp;
    if (jix >= njobs) return;
    const JobDev job = jobs[jix];
    const SysDev &S = systems[job.sys];
    double *pan = dsm + (size_t)warp * W::DOUBLES;
    double *s_eint = pan + W::PAN;
    double *s_cent = s_eint + W::VEC;
    // Z waits here while U is inverted: one matrix in registers leaves room for
    // the occupancy that hides the sweep's latency (two of them at N = 40 held
    // the kernel to two CTAs an SM, and above 40 do not fit)
    double *zs = pan + W::PAN + 5 * W::VEC + lane * 2;
    const int n = S.n;
    const double ered = job.ered;
    const double h = S.dr / 2.0;
    const double d1 = h * h / 3.0;
    const double d2 = 2.0 * d1;
    const double d4 = -d1 / 16.0;
    double *yj = y + job.yoff;
    const bool dg0 = fdiag(lane, 0), dg1 = fdiag(lane, 1);  // padding channels included
    stage_channels<NT>(S, lane, s_eint, s_cent);

    double a[NTL][2];
    load_lower_frag<NT>(yj, n, lane, a);
    w_each<NT>(S, s_eint, s_cent, lane, 0, ered, [&](int t, int I, int J, double w0, double w1) {
        a[t][0] = fma(h, a[t][0], d1 * w0) + (I == J && dg0 ? 1.0 : 0.0);  // ldprop.f:46-51
        a[t][1] = fma(h, a[t][1], d1 * w1) + (I == J && dg1 ? 1.0 : 0.0);
    });
    int nodes = 0, status = MGPU_OK, kfail = 0;
    const unsigned long long t0 = global_ns();
    for (int k = 1; k <= S.nstep; ++k) {
        if (stop_poll_step(k)) {
            int stop = lane == 0 ? stop_requested(S.ctl, t0) : MGPU_OK;
            stop = __shfl_sync(0xffffffffu, stop, 0);
            if (stop != MGPU_OK) {
                status = stop;
                kfail = k;
                break;
            }
        }
        int bad2 = SWEEP_OK;
        const int ncz = warp_sweep_invert<NT>(a, pan, n, lane, bad2);  // ldprop.f:83
#pragma unroll
        for (int t = 0; t < NTL; ++t) *reinterpret_cast<double2 *>(zs + t * 64) = make_double2(a[t][0], a[t][1]);
        w_each<NT>(S, s_eint, s_cent, lane, 2 * k - 1, ered, [&](int t, int I, int J, double w0, double w1) {
            a[t][0] = d4 * w0 + (I == J && dg0 ? 0.125 : 0.0);  // ldprop.f:67-72
            a[t][1] = d4 * w1 + (I == J && dg1 ? 0.125 : 0.0);
        });
        int bad = SWEEP_OK;
        const int ncu = warp_sweep_invert<NT>(a, pan, n, lane, bad);  // ldprop.f:78
        if (bad != SWEEP_OK || bad2 != SWEEP_OK) {
            status = (bad == SWEEP_ZERO || bad2 == SWEEP_ZERO) ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        nodes += ncz;
#pragma unroll
        for (int I = 0; I < NT; ++I)
#pragma unroll
            for (int J = 0; J <= I; ++J) {
                // Z = U^-1 - Z^-1 - 6I with a = -U^-1, z = -Z^-1 (ldprop.f:92-97)
                const double2 z = *reinterpret_cast<const double2 *>(zs + tix(I, J) * 64);
                a[tix(I, J)][0] = -a[tix(I, J)][0] + z.x - (I == J && dg0 ? 6.0 : 0.0);
                a[tix(I, J)][1] = -a[tix(I, J)][1] + z.y - (I == J && dg1 ? 6.0 : 0.0);
            }
        const int ncz2 = warp_sweep_invert<NT>(a, pan, n, lane, bad);  // ldprop.f:99
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        nodes += ncz2 - ncu;
        const double dd = (k == S.nstep) ? d1 : d2;
        w_each<NT>(S, s_eint, s_cent, lane, 2 * k, ered, [&](int t, int I, int J, double w0, double w1) {
            // Z = D2 W(B) + 2I - Z^-1 (ldprop.f:114-131)
            a[t][0] = dd * w0 + (I == J && dg0 ? 2.0 : 0.0) + a[t][0];
            a[t][1] = dd * w1 + (I == J && dg1 ? 2.0 : 0.0) + a[t][1];
        });
    }
    if (status == MGPU_OK) {
        // Y = Z/H - I/H (ldprop.f:140-147)
        const double hi = 1.0 / h;
#pragma unroll
        for (int I = 0; I < NT; ++I)
#pragma unroll
            for (int J = 0; J <= I; ++J) {
                a[tix(I, J)][0] = hi * a[tix(I, J)][0] - (I == J && dg0 ? hi : 0.0);
                a[tix(I, J)][1] = hi * a[tix(I, J)][1] - (I == J && dg1 ? hi : 0.0);
            }
        store_full_frag<NT>(yj, n, lane, 1.0, a);
    }
    if (lane == 0) {
        status_out[job.out] = status;
        kfail_out[job.out] = kfail;
        nodes_out[job.out] = status == MGPU_OK ? nodes : 0;
    }
}

// ---------------------------------------------------------------------------
// MGPROP step loop (the symplectic log-derivative propagator of Manolopoulos
// and Gray, mgprop.f:63-134), one warp per job.  Per sector, stage k forms
// X = Y + b_k h W(R) and, where a_k != 0, Y = [I - (I + a_k h X)^-1]/(a_k h)
// (the negative pivots of I + a_k h X added to NODES, subtracted where
// a_k < 0); R advances by a_k h.  W of stage k of sector s is row
// s*stride + k of the radial tables (stride = stages, or stages - 1 when
// a_M = 0 and the last stage's W serves as the next sector's first).
// ---------------------------------------------------------------------------
struct MGCoef {
    int m, stride;
    double a[6], b[6];
};
// Table I of D. E. Manolopoulos and S. K. Gray, J. Chem. Phys. 102, 9214
// (1995): [0] CS4 (IMGSEL = 4), [1] McLachlan and Atela's MA5 (IMGSEL = 5).
// The host lays out the radial tables from the same numbers.
#define MGPU_MG_COEFS { \
        {5, 4, \
         {0.20517766154229, 0.40302128160421, -0.12092087633891, 0.51272193319241, 0.0, 0.0}, \
         {0.061758858135626, 0.33897802655364, 0.61479130717558, -0.14054801465937, 0.12501982279453, 0.0}}, \
        {6, 6, \
         {0.33983962583911, -0.088601336903027, 0.58585647682596, -0.60303935653649, 0.32358079655470, \
          0.44236379421975}, \
         {0.11939002928757, 0.69892737038248, -0.17131235827160, 0.40126950225135, 0.010705081848236, \
          -0.058979625498031}}, \
    }
constexpr MGCoef kMGCoef[2] = MGPU_MG_COEFS;
// the device copy, initialised from the same literal list
__constant__ MGCoef c_mg[2] = MGPU_MG_COEFS;
#undef MGPU_MG_COEFS

template <int NT>
__global__ void __launch_bounds__(32 * kWPB, frag_min_blocks(NT))
ldmg_prop_frag_kernel(const SysDev *__restrict__ systems, const JobDev *__restrict__ jobs, int njobs, int method,
                      double *__restrict__ y, int *__restrict__ nodes_out, int *__restrict__ status_out,
                      int *__restrict__ kfail_out)
{
    constexpr int NTL = G<NT>::NTL;
    __shared__ __align__(16) double pans[kWPB][G<NT>::WSM];
    __shared__ double chan[kWPB][2 * G<NT>::NPAD];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int jix = blockIdx.x * kWPB + warp;
    if (jix >= njobs) return;
    const JobDev job = jobs[jix];
    const SysDev &S = systems[job.sys];
    const MGCoef &C = c_mg[method];
    double *pan = pans[warp];
    const int n = S.n;
    const double ered = job.ered;
    const double h = S.dr;
    double *yj = y + job.yoff;
    const bool dg0 = fdiag(lane, 0), dg1 = fdiag(lane, 1);  // padding channels included
    double *s_eint = chan[warp], *s_cent = s_eint + G<NT>::NPAD;
    stage_channels<NT>(S, lane, s_eint, s_cent);

    double a[NTL][2];
    load_lower_frag<NT>(yj, n, lane, a);
    int nodes = 0, status = MGPU_OK, kfail = 0;
    const unsigned long long t0 = global_ns();
    for (int sec = 0; sec < S.nstep; ++sec) {
        if (stop_poll_step(sec + 1)) {
            int stop = lane == 0 ? stop_requested(S.ctl, t0) : MGPU_OK;
            stop = __shfl_sync(0xffffffffu, stop, 0);
            if (stop != MGPU_OK) {
                status = stop;
                kfail = sec + 1;
                break;
            }
        }
#pragma unroll 1
        for (int k = 0; k < C.m; ++k) {
            const double bh = C.b[k] * h;
            w_each<NT>(S, s_eint, s_cent, lane, sec * C.stride + k, ered, [&](int t, int, int, double w0, double w1) {
                a[t][0] = fma(bh, w0, a[t][0]);  // X = Y + b_k h W
                a[t][1] = fma(bh, w1, a[t][1]);
            });
            const double ak = C.a[k];
            if (ak == 0.0) continue;  // Y = X
            const double ah = ak * h;
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J <= I; ++J) {
                    a[tix(I, J)][0] = ah * a[tix(I, J)][0] + (I == J && dg0 ? 1.0 : 0.0);  // I + a_k h X
                    a[tix(I, J)][1] = ah * a[tix(I, J)][1] + (I == J && dg1 ? 1.0 : 0.0);
                }
            int bad = SWEEP_OK;
            const int cnt = warp_sweep_invert<NT>(a, pan, n, lane, bad);  // a = -(I + a_k h X)^-1
            if (bad != SWEEP_OK) {
                status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
                kfail = sec + 1;
                break;
            }
            nodes += ak >= 0.0 ? cnt : -cnt;
            const double d1 = 1.0 / ah;
#pragma unroll
            for (int I = 0; I < NT; ++I)
#pragma unroll
                for (int J = 0; J <= I; ++J) {
                    a[tix(I, J)][0] = (a[tix(I, J)][0] + (I == J && dg0 ? 1.0 : 0.0)) * d1;  // [I - inverse]/(a_k h)
                    a[tix(I, J)][1] = (a[tix(I, J)][1] + (I == J && dg1 ? 1.0 : 0.0)) * d1;
                }
        }
        if (status != MGPU_OK) break;
    }
    if (status == MGPU_OK) store_full_frag<NT>(yj, n, lane, 1.0, a);
    if (lane == 0) {
        status_out[job.out] = status;
        kfail_out[job.out] = kfail;
        nodes_out[job.out] = status == MGPU_OK ? nodes : 0;
    }
}

}  // namespace wf
}  // namespace mgpu
