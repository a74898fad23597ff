// MAPROP (maprop.f:33-290), the quasi-adiabatic log-derivative propagator, and
// AIRY's sweep (aiprop.f:160-250) for the energies of one system: one CTA per
// energy (N <= 100).  Everything that does not depend on the energy -- for
// MAPROP the adiabatic bases at the sector midpoints and their eigenvalues, the
// basis changes Q_k = T_{k-1}^T U_k and the first-order corrections in the old
// basis -- comes from tables the host builds once per system (what the reference
// keeps on its ISCRU file after the first energy).  MAPROP per sector:
//   Y += C_k;  Y = Q_k^T Y Q_k;  Y_ii += y1_i;  Y = -y2 Y^-1 y2 + diag(y1)
// with the half-angle propagators of EIVAL - ERED (y3 = y2, y4 = y1), NODES
// from the inversion's negative pivots unless a channel is deeper than
// 24/DR^2; at the end Y = T Y T^T + Q_end.
//
// The matrix is held as the one-CTA kernels hold it (kernels_cta.cuh): lower 8x8
// tiles in DMMA fragments, the inversion is their sweep.  The basis change runs
// on DMMA too.  A warp takes a tile column J of the result:
//   S = Q[:, J]^T Y      (one tile row, in accumulators)
//   Y'(I, J) = sum_M Q[:, I]^T restricted to M . S(M)^T   for I >= J
// where S needs no exchange between lanes: a lane's accumulator element
// (row r, column 2q + s) is the B operand of k-slot q if slot (M, s) of the
// second product takes the rows 8M + 2q + s of Q, which is how Q is read.
// Before, one thread formed each element of both products with a modulo and a
// division per element and the matrix was inverted pivot by pivot with four
// barriers and two passes over it: 60 us a sector at N = 30.
// Included by propagator.cu.
#pragma once

namespace mgpu {
namespace ldma {

constexpr int kMaxN = 100;

struct Tables {
    int n, nstep, inward;
    double dr;
    const double *eival;  // [nstep][n]
    const double *q;      // [nstep][n*n] column-major
    const double *corr;   // [nstep][n*n]
    const double *tfin;   // [n*n]
    const double *qfin;   // [n*n]
};

// AIRY's sweep: per sector Z = T_k^T Z T_k (symmetrised), (Z + Y1)^-1 with its
// negative-pivot count (NODES += count outwards, N - count inwards),
// Z = -Y2 (Z + Y1)^-1 Y2 + Y4; at the end V Z V^T.  The sector functions (Y1, Y2,
// Y4) of every job, sector and channel come from the host:
// y124[job][sector][channel][3].
struct AiryTables {
    int n, nsect, inward;
    const double *tmat;  // [nsect][n*n] column-major
    const double *vfin;  // [n*n]
};

// Shared memory in doubles: the sweep's (kernels_cta.cuh, which includes two
// vectors per parity used here as y1 and y2), Q, Y before and after the basis change.
template <int NT, int W>
struct LSmem {
    static constexpr int QP = 8 * NT + 4;  // column pitch of Q: 4 mod 8, rows of the operand reads on distinct banks
    static constexpr int Q = cta::CSmem<NT, W>::PARK;
    static constexpr int YA = Q + 8 * NT * QP;
    static constexpr int YB = YA + cta::CG<NT, W>::TD;
    static constexpr size_t BYTES = (size_t)(YB + cta::CG<NT, W>::TD) * 8;
};

// Q (n x n, column-major; transposed if `tr`) into shared memory, zero padded.
template <int NT, int W>
__device__ __forceinline__ void load_q(const double *__restrict__ src, int n, bool tr, double *qs)
{
    constexpr int QP = LSmem<NT, W>::QP;
    const int lane = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < 8 * NT; j += W)
        for (int i = lane; i < 8 * NT; i += 32)
            qs[j * QP + i] = i < n && j < n ? __ldg(src + (tr ? j + (size_t)i * n : i + (size_t)j * n)) : 0.0;
}

// YB = Q^T YA Q on the lower tiles (both in fragment layout, tile after tile).
template <int NT, int W>
__device__ __forceinline__ void transform(const double *qs, const double *ya, double *yb, int nb)
{
    constexpr int QP = LSmem<NT, W>::QP;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    for (int J = warp; J < nb; J += W) {
        double s[NT][2];
#pragma unroll
        for (int M = 0; M < NT; ++M) s[M][0] = s[M][1] = 0.0;
        // S(M) += Q[K, J]^T Y[K, M], four rows of K at a time
#pragma unroll 1
        for (int K = 0; K < nb; ++K) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double a = qs[(8 * J + r) * QP + 8 * K + 4 * h + q];
#pragma unroll
                for (int M = 0; M < NT; ++M)
                    if (M < nb) {
                        // element (8K + 4h + q, 8M + r) from the lower triangle
                        const int t = M <= K ? cta::tix(K, M) : cta::tix(M, K);
                        const int e = M < K ? (4 * h + q) * 8 + r
                                            : M > K ? r * 8 + 4 * h + q
                                                    : (4 * h + q >= r ? (4 * h + q) * 8 + r : r * 8 + 4 * h + q);
                        wf::dmma(s[M][0], s[M][1], a, ya[t * 64 + e]);
                    }
            }
        }
#pragma unroll 1
        for (int I = J; I < nb; ++I) {
            double c0 = 0.0, c1 = 0.0;
#pragma unroll
            for (int M = 0; M < NT; ++M)
                if (M < nb) {
                    const double2 a = *reinterpret_cast<const double2 *>(qs + (8 * I + r) * QP + 8 * M + 2 * q);
                    wf::dmma(c0, c1, a.x, s[M][0]);
                    wf::dmma(c0, c1, a.y, s[M][1]);
                }
            *reinterpret_cast<double2 *>(yb + cta::tix(I, J) * 64 + lane * 2) = make_double2(c0, c1);
        }
    }
}

// The sector loop both propagators share.  `start(i, j)` is the first matrix,
// corr(k) the correction added in the old basis (or null), q(k) the basis
// change, funcs(k, i, y1, y2, y4) the sector functions of channel i (returns
// true when the sector counts no nodes), finish(i, j, v) takes the result.
template <int NT, int W, class Start, class Corr, class QK, class Funcs, class Finish>
__device__ __forceinline__ void sweep(int n, int nsect, int inward, const double *last, double *sm, int &nodes,
                                      int &status, Start &&start, Corr &&corr, QK &&qk, Funcs &&funcs, Finish &&finish)
{
    using C = cta::CG<NT, W>;
    using L = LSmem<NT, W>;
    __shared__ int cf[2];
    const cta::Own<NT, W> own(sm, n);
    const int tid = threadIdx.x, lane = own.lane, nb = own.nb;
    double *qs = sm + L::Q, *ya = sm + L::YA, *yb = sm + L::YB;
    double *y1 = sm + cta::CSmem<NT, W>::VEC, *y2 = y1 + C::NPAD, *y4 = y2 + C::NPAD;
    double a[C::TPW][2];
#pragma unroll
    for (int u = 0; u < C::TPW; ++u) a[u][0] = a[u][1] = 0.0;
    own.each(a, [&](int, int I, int J, bool, double &a0, double &a1) {
        const cta::Elem e(I, J, lane);
        a0 = e.i < n && e.j0 < n ? start(e.i, e.j0) : 0.0;
        a1 = e.i < n && e.j1 < n ? start(e.i, e.j1) : 0.0;
    });
    nodes = 0;
    status = MGPU_OK;
    for (int k = 0; k <= nsect; ++k) {
        const bool end = k == nsect;  // the last basis change
        const double *c = end ? nullptr : corr(k);
        own.each(a, [&](int t, int I, int J, bool real, double &a0, double &a1) {
            const cta::Elem e(I, J, lane);
            if (!real) return;
            double v0 = a0, v1 = a1;
            if (c != nullptr) {  // the correction in the old basis
                if (e.i < n && e.j0 < n) v0 += __ldg(c + e.i + (size_t)e.j0 * n);
                if (e.i < n && e.j1 < n) v1 += __ldg(c + e.i + (size_t)e.j1 * n);
            }
            *reinterpret_cast<double2 *>(ya + t * 64 + lane * 2) = make_double2(v0, v1);
        });
        load_q<NT, W>(end ? last : qk(k), n, end, qs);
        bool deep = false;
        if (!end)
            for (int i = tid; i < 8 * nb; i += C::NTHR) {
                double f1 = 1.0, f2 = 0.0, f4 = 0.0;  // padding: positive diagonal, nothing left of it
                if (i < n) deep = funcs(k, i, f1, f2, f4) || deep;
                y1[i] = f1;
                y2[i] = f2;
                y4[i] = f4;
            }
        const bool count = !__syncthreads_or(deep);
        transform<NT, W>(qs, ya, yb, nb);
        __syncthreads();
        if (end) break;
        own.each(a, [&](int t, int I, int J, bool real, double &a0, double &a1) {
            const cta::Elem e(I, J, lane);
            const double2 v = *reinterpret_cast<const double2 *>(yb + (real ? t : 0) * 64 + lane * 2);
            a0 = v.x + (e.d == 0 ? y1[e.i] : 0.0);
            a1 = v.y + (e.d == 1 ? y1[e.i] : 0.0);
        });
        int bad = SWEEP_OK;
        const int cnt = cta::cta_invert<NT, W>(a, own, sm, cf, bad);  // a = -(Y + y1)^-1
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            break;
        }
        if (count) nodes += inward ? n - cnt : cnt;
        own.each(a, [&](int, int I, int J, bool, double &a0, double &a1) {
            const cta::Elem e(I, J, lane);
            const double f = y2[e.i];
            a0 = f * a0 * y2[e.j0] + (e.d == 0 ? y4[e.i] : 0.0);
            a1 = f * a1 * y2[e.j1] + (e.d == 1 ? y4[e.i] : 0.0);
        });
        __syncthreads();  // the counters and the sector functions have been read
    }
    if (status == MGPU_OK)
        own.each(a, [&](int t, int I, int J, bool real, double &, double &) {
            const cta::Elem e(I, J, lane);
            if (!real) return;
            const double2 v = *reinterpret_cast<const double2 *>(yb + t * 64 + lane * 2);
            if (e.i < n && e.j0 <= e.i) finish(e.i, e.j0, v.x);
            if (e.i < n && e.j1 <= e.i) finish(e.i, e.j1, v.y);
        });
}

// CTAs an SM: registers for four of four warps, two of eight; the largest size one by shared memory
template <int NT, int W>
constexpr int min_ctas() { return W <= 4 ? 4 : NT <= 8 ? 2 : 1; }

template <int NT, int W>
__global__ void __launch_bounds__(32 * W, min_ctas<NT, W>())
ldma_kernel(Tables T, const double *__restrict__ ered, double *__restrict__ y, int *__restrict__ nodes_out,
            int *__restrict__ status_out)
{
    extern __shared__ __align__(16) double ldma_sm[];
    const int n = T.n, job = blockIdx.x;
    const size_t nn = (size_t)n * n;
    const double e = ered[job], wmax = 24.0 / (T.dr * T.dr);
    double *yj = y + (size_t)job * nn;
    int nodes, status;
    sweep<NT, W>(
        n, T.nstep, T.inward, T.tfin, ldma_sm, nodes, status,
        [&](int i, int j) { return 0.5 * (yj[i + (size_t)j * n] + yj[j + (size_t)i * n]); },
        [&](int k) { return T.corr + k * nn; }, [&](int k) { return T.q + k * nn; },
        [&](int k, int i, double &y1, double &y2, double &y4) {
            const double wref = __ldg(T.eival + (size_t)k * n + i) - e;
            const double flam = 0.5 * sqrt(fabs(wref));
            if (wref < 0.0) {
                const double tn = tan(flam * T.dr);
                y1 = flam / tn - flam * tn;
                y2 = flam / tn + flam * tn;
            } else {
                const double th = tanh(flam * T.dr);
                y1 = flam / th + flam * th;
                y2 = flam / th - flam * th;
            }
            y4 = y1;
            return wref > wmax;  // deeper than 24/DR^2: the sector's count is not used (maprop.f's NCHECK)
        },
        // back in the primitive basis, plus the end correction (maprop.f:281-287)
        [&](int i, int j, double v) {
            yj[i + (size_t)j * n] = v + __ldg(T.qfin + i + (size_t)j * n);
            if (i != j) yj[j + (size_t)i * n] = v + __ldg(T.qfin + j + (size_t)i * n);
        });
    if (threadIdx.x == 0) {
        status_out[job] = status;
        nodes_out[job] = status == MGPU_OK ? nodes : 0;
    }
}

template <int NT, int W>
__global__ void __launch_bounds__(32 * W, min_ctas<NT, W>())
airy_kernel(AiryTables T, const double *__restrict__ y124, double *__restrict__ z, int *__restrict__ nodes_out,
            int *__restrict__ status_out)
{
    extern __shared__ __align__(16) double airy_sm[];
    const int n = T.n, job = blockIdx.x;
    const size_t nn = (size_t)n * n;
    const double *yj = y124 + (size_t)job * T.nsect * n * 3;
    double *zj = z + (size_t)job * nn;
    int nodes, status;
    sweep<NT, W>(
        n, T.nsect, T.inward, T.vfin, airy_sm, nodes, status,
        [&](int i, int j) { return 0.5 * (zj[i + (size_t)j * n] + zj[j + (size_t)i * n]); },
        [&](int) { return (const double *)nullptr; }, [&](int k) { return T.tmat + k * nn; },
        [&](int k, int i, double &y1, double &y2, double &y4) {
            const double *f = yj + ((size_t)k * n + i) * 3;
            y1 = __ldg(f);
            y2 = __ldg(f + 1);
            y4 = __ldg(f + 2);
            return false;
        },
        [&](int i, int j, double v) {
            zj[i + (size_t)j * n] = v;
            zj[j + (size_t)i * n] = v;
        });
    if (threadIdx.x == 0) {
        status_out[job] = status;
        nodes_out[job] = status == MGPU_OK ? nodes : 0;
    }
}

// (NT, warps): N = 8 NT up to 104
#define MGPU_LDMA_BUCKETS(X) X(2, 4) X(3, 4) X(4, 4) X(5, 4) X(6, 8) X(8, 8) X(10, 8) X(13, 8)

static cudaError_t launch_ldma(const Tables &t, int njobs, const double *ered, double *y, int *nodes, int *status,
                               cudaStream_t st)
{
    cudaError_t e;
#define X(NT, W)                                                                                       \
    if (t.n <= 8 * NT) {                                                                               \
        if ((e = set_smem(ldma_kernel<NT, W>, LSmem<NT, W>::BYTES))) return e;                         \
        ldma_kernel<NT, W><<<njobs, 32 * W, LSmem<NT, W>::BYTES, st>>>(t, ered, y, nodes, status);     \
        return cudaGetLastError();                                                                     \
    }
    MGPU_LDMA_BUCKETS(X)
#undef X
    return cudaErrorInvalidValue;
}

static cudaError_t launch_airy(const AiryTables &t, int njobs, const double *y124, double *z, int *nodes, int *status,
                               cudaStream_t st)
{
    cudaError_t e;
#define X(NT, W)                                                                                       \
    if (t.n <= 8 * NT) {                                                                               \
        if ((e = set_smem(airy_kernel<NT, W>, LSmem<NT, W>::BYTES))) return e;                         \
        airy_kernel<NT, W><<<njobs, 32 * W, LSmem<NT, W>::BYTES, st>>>(t, y124, z, nodes, status);     \
        return cudaGetLastError();                                                                     \
    }
    MGPU_LDMA_BUCKETS(X)
#undef X
    return cudaErrorInvalidValue;
}

}  // namespace ldma
}  // namespace mgpu
