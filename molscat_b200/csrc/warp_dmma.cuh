// One warp per symmetric matrix, held in FP64 tensor-core (DMMA) fragments.
//
// The matrix (padded to NPAD = 8*NT) is cut into 8x8 tiles; the lower
// triangle of tiles, t = I*(I+1)/2 + J (I >= J), lives in registers in the
// accumulator layout of mma.sync.m8n8k4.f64: lane l holds the elements at
// positions (row l>>2, column 2(l&3) + s), s = 0,1, of a tile.  Diagonal tiles
// hold both triangles.
//
// Inversion is the symmetric Gauss-Jordan sweep done four pivots at a time
// (block sweep).  For the pivot block P = {p0..p0+3} with D = A_PP = L Delta L^T
// (unpivoted, the scalar sweep's own pivots delta_k) and Lam = L^{-1}:
//     c_k(i) = sum_m Lam[k][m] A_{i,p0+m}          (i not in P)
//     A_ij  -= sum_k c_k(i) c_k(j) / delta_k        (i, j not in P)
//     A_iP   = A_iP D^{-1} ,  A_PP = -D^{-1}
// which after all blocks leaves -A^{-1}.  The trailing update is the scalar
// sweep's own rank-one terms (the one-warp sweep adds a block's four in the
// order 3, 2, 1, 0, the others 0, 1, 2, 3), so the block sweep keeps its
// rounding behaviour; forming D^{-1} first and updating with A_iP D^{-1} A_Pj instead
// loses accuracy when a pivot is small next to its neighbours.  As in
// tiles.cuh the entries of row/column block P are zeroed first and the operands
// carry the pivot block, so every lower tile gets the same update
//     A_IJ += X_I B_J          (one m8n8k4 DMMA per lower tile)
// with X(i,k) = -c_k(i)/delta_k, B(j,k) = c_k(j) for rows outside P and
// X(p0+a,k) = Lam[k][a]/delta_k, B(p0+b,k) = -Lam[k][b] for rows of P, which
// writes A_iP D^{-1} into the columns of P and -D^{-1} into A_PP.  Every read of
// a diagonal tile takes the lower triangle, so the stored matrix is symmetric
// for the algorithm whatever rounding left in the upper triangle.
//
// The pivots delta_k are those of the unpivoted LDL^T SYMINV forms
// (syminv.f:27-49); their negative count is SYMINV's KOUNT (and DSYNEG's
// inertia by Sylvester's law); a zero pivot is the reference's IFAIL = N+1.
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "tiles.cuh"  // pivot_reciprocal, pivot_flags

namespace mgpu {
namespace wf {

template <int NT>
struct G {
    static constexpr int NTL = NT * (NT + 1) / 2;  // lower tiles
    static constexpr int NPAD = 8 * NT;
    // per-warp shared memory of the one-warp sweep (doubles): two pivot blocks,
    // then a transposition buffer of NT - 1 tiles (rows 10 doubles apart: no
    // bank conflict when a tile is read by columns)
    static constexpr int TPITCH = 10;
    static constexpr int WSM = 32 + (NT - 1) * 8 * TPITCH;
};

__host__ __device__ constexpr int tix(int I, int J) { return I * (I + 1) / 2 + J; }

// Not volatile: the result registers carry every dependency, and leaving
// the compiler free to schedule DMMAs between other work helps it overlap
// them with the look-ahead factorisation.
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// D = X B + C with C in other registers than D.
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b, double c0, double c1)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%5};"
                 : "=d"(d0), "=d"(d1)
                 : "d"(a), "d"(b), "d"(c0), "d"(c1));
}

// Unpivoted LDL^T of the symmetric 4x4 pivot block D, read from the lower
// triangle of d (the upper triangle is ignored), pivot by pivot as the scalar
// sweep meets them.  On return d holds the block's operands:
//     d[k][k] = 1/delta_k ,  d[i][k] = Lam[i][k] (i > k) ,  d[k][i] = 0
// with Lam = L^{-1} (unit lower).  Negative pivots are added to cnt.
__device__ __forceinline__ void ldl_block4(double d[4][4], int &cnt, int &flags)
{
    double l[4][4], rd[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double dk = d[k][k];
        flags |= pivot_flags(dk);
        cnt += (dk < 0.0);
        const double rk = pivot_reciprocal(dk);
        rd[k] = rk;
#pragma unroll
        for (int i = k + 1; i < 4; ++i) l[i][k] = d[i][k] * rk;
#pragma unroll
        for (int i = k + 1; i < 4; ++i)
#pragma unroll
            for (int j = k + 1; j <= i; ++j) d[i][j] = fma(-l[i][k], d[j][k], d[i][j]);
    }
    // Lam = L^{-1} by forward substitution
    double lam[4][4];
#pragma unroll
    for (int i = 1; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) {
            double s = -l[i][j];
#pragma unroll
            for (int m = j + 1; m < i; ++m) s = fma(-l[i][m], lam[m][j], s);
            lam[i][j] = s;
        }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) d[i][j] = (i == j) ? rd[i] : (i > j ? lam[i][j] : 0.0);
}

// ---- the one-warp sweep -----------------------------------------------------
// Which channel of a tile's eight sits at position p of its rows and columns:
// the even positions hold channels 3, 2, 1, 0 and the odd ones 7, 6, 5, 4.  A
// four-pivot block is then one slot s of every lane, and a lane's element
// A[i, P] (position 2q + s, pivot 3 - q of the block) is, as it stands in the
// accumulators, an A operand of the DMMA: the panel needs no exchange between
// lanes.  c = A[:, P] Lam^T is itself a DMMA (pivots in the order 3..0, so its
// chain of FMAs runs 3, 2, 1, 0 as the scalar formula
// fma(Lam0, A0, fma(Lam1, A1, fma(Lam2, A2, A3))) does, the leading terms being
// exact), and its result is in the layout of the update's X and B operands.
__host__ __device__ constexpr int chan_of(int p) { return 4 * (p & 1) + 3 - (p >> 1); }
__host__ __device__ constexpr int pos_of(int c) { return 2 * (3 - (c & 3)) + (c >> 2); }

// Pivots whose reciprocals need no scaling (and so are neither zero nor
// non-finite): 2^-1000 <= |d| < 2^1000 for all four, from the exponent bits.
__device__ __forceinline__ bool pivots_plain(double d0, double d1, double d2, double d3)
{
    const unsigned a = (__double2hiint(d0) & 0x7fffffffu) - 0x01700000u, b = (__double2hiint(d1) & 0x7fffffffu) - 0x01700000u;
    const unsigned c = (__double2hiint(d2) & 0x7fffffffu) - 0x01700000u, d = (__double2hiint(d3) & 0x7fffffffu) - 0x01700000u;
    return max(max(a, b), max(c, d)) < 0x7d000000u;
}

// ldl_block4 with the exact scaling and the pivot flags, for a block that holds
// an unusual pivot: blk[4i + j] (i >= j) in, the operands out in the same place.
// Returns the negative pivots | flags << 8.
__device__ __noinline__ int ldl_block4_any(double *blk)
{
    double d[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) d[i][j] = j <= i ? blk[4 * i + j] : 0.0;
    int cnt = 0, flags = 0;
    ldl_block4(d, cnt, flags);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) blk[4 * i + j] = d[i][j];
    }
    __syncwarp();
    return cnt | (flags << 8);
}

// What the rounds need of a factored pivot block, per lane: lam = Lam[r>>1][3-q],
// the B operand of c = A[:, P] Lam^T (its column 2k is pivot k), and
// nrd = -1/delta_q.
struct BlockOps {
    double lam, nrd;
};

// The operands of a factored 4x4 pivot block in registers: 1/delta_k and
// Lam = L^{-1} below the diagonal.
struct Block4 {
    double r0, r1, r2, r3, m10, m20, m21, m30, m31, m32;
};

// ldl_block4's arithmetic for a block whose four pivots are plain
// (pivots_plain); `neg` gets the negative ones.  Returns false when they are
// not: the caller then takes ldl_block4_any.
__device__ __forceinline__ bool ldl_block4_plain(double d00, double d10, double d11, double d20, double d21, double d22,
                                                 double d30, double d31, double d32, double d33, Block4 &o, int &neg)
{
    o.r0 = pivot_reciprocal_plain(d00);
    const double l10 = d10 * o.r0, l20 = d20 * o.r0, l30 = d30 * o.r0;
    d11 = fma(-l10, d10, d11);
    o.r1 = pivot_reciprocal_plain(d11);
    d21 = fma(-l20, d10, d21);
    d31 = fma(-l30, d10, d31);
    d22 = fma(-l20, d20, d22);
    d32 = fma(-l30, d20, d32);
    d33 = fma(-l30, d30, d33);
    const double l21 = d21 * o.r1, l31 = d31 * o.r1;
    d22 = fma(-l21, d21, d22);
    o.r2 = pivot_reciprocal_plain(d22);
    d32 = fma(-l31, d21, d32);
    d33 = fma(-l31, d31, d33);
    const double l32 = d32 * o.r2;
    d33 = fma(-l32, d32, d33);
    o.r3 = pivot_reciprocal_plain(d33);
    // Lam = L^{-1} by forward substitution
    o.m10 = -l10, o.m21 = -l21, o.m32 = -l32;
    o.m20 = fma(-l21, o.m10, -l20);
    o.m31 = fma(-l32, o.m21, -l31);
    o.m30 = fma(-l32, o.m20, fma(-l31, o.m10, -l30));
    neg = ((unsigned)__double2hiint(d00) >> 31) + ((unsigned)__double2hiint(d11) >> 31) +
          ((unsigned)__double2hiint(d22) >> 31) + ((unsigned)__double2hiint(d33) >> 31);
    return pivots_plain(d00, d11, d22, d33);
}

__device__ __forceinline__ void block4_from(const double *blk, Block4 &o)
{
    o.r0 = blk[0], o.m10 = blk[4], o.r1 = blk[5], o.m20 = blk[8], o.m21 = blk[9], o.r2 = blk[10];
    o.m30 = blk[12], o.m31 = blk[13], o.m32 = blk[14], o.r3 = blk[15];
}

// Factor the pivot block of slot H of the diagonal tile (v: this lane's element
// of that slot), ldl_block4's arithmetic in every lane.  The block reaches the
// lanes through shared memory: one store and six loads against twenty shuffles
// of four cycles each on the shared-memory pipe.  `live` = 0 (past the last
// block of the matrix): nothing is counted.
template <int H>
__device__ __forceinline__ void factor_block(double v, double *blk, int lane, bool live, BlockOps &o, int &cnt,
                                             int &flags)
{
    const int r = lane >> 2, q = lane & 3;
    if ((r & 1) == H) blk[4 * (3 - (r >> 1)) + 3 - q] = v;
    __syncwarp();
    const double2 b10 = *reinterpret_cast<const double2 *>(blk + 4);
    const double2 b20 = *reinterpret_cast<const double2 *>(blk + 8);
    const double2 b30 = *reinterpret_cast<const double2 *>(blk + 12);
    const double2 b32 = *reinterpret_cast<const double2 *>(blk + 14);
    Block4 b;
    int c;
    if (!ldl_block4_plain(blk[0], b10.x, b10.y, b20.x, b20.y, blk[10], b30.x, b30.y, b32.x, b32.y, b, c)) {
        const int cf = ldl_block4_any(blk);  // the same in every lane
        c = cf & 255;
        flags |= live ? cf >> 8 : 0;
        block4_from(blk, b);
    }
    cnt += live ? c : 0;
    const int j = r >> 1;  // row of Lam; this lane's column of it is 3 - q
    const double c0 = j == 3 ? b.m30 : j == 2 ? b.m20 : b.m10;
    const double c1 = j == 3 ? b.m31 : b.m21;
    const double x = q == 3 ? c0 : q == 2 ? c1 : b.m32;
    o.lam = j + q == 3 ? 1.0 : j + q > 3 ? x : 0.0;
    o.nrd = -(q == 0 ? b.r0 : q == 1 ? b.r1 : q == 2 ? b.r2 : b.r3);
}

// -A^{-1} in place; returns the negative-pivot count, `bad` as in tiles.cuh.
// Padding rows and columns are uncoupled and have a positive diagonal where a
// pivot block holds one beside a real channel.  A last half tile that is all
// padding is neither pivoted nor counted: its diagonal stays what it was,
// whatever that is.
// ws: G<NT>::WSM doubles of shared memory owned by this warp.
//
// The loop runs over the tile columns with the pivot tile always the first:
// after its two rounds every tile moves one place up and left (for nothing: the
// update's result registers are simply other ones than its addend's), the tiles
// of the first column become the last row, transposed through shared memory, and
// after NT turns the matrix stands in its own order again.  Every register index
// is fixed and the code is two rounds long, whatever NT: unrolled over the
// rounds it filled the instruction caches (7843 instructions a propagation step
// at NT = 5, N 33-36; this form issues 5561), and with the pivot tile first there
// is no row of tiles left of it, whose panel entries would need transposing.
// The next block is factored as soon as its tile has its update, beside the
// other DMMAs of the round.
template <int NT>
__device__ __forceinline__ int warp_sweep_invert(double (&a)[G<NT>::NTL][2], double *ws, int n, int lane, int &bad)
{
    const int r = lane >> 2, q = lane & 3;
    const bool odd = r & 1;
    const double unit = q == (r >> 1) ? -1.0 : 0.0;  // rows of P: c = Lam (-I), exactly -Lam[k][a]
    double *tb = ws + 32;
    int cnt = 0, flags = 0;
    BlockOps f;
    __syncwarp();
    factor_block<0>(a[0][0], ws, lane, true, f, cnt, flags);
#pragma unroll 1
    for (int K = 0; K < NT; ++K) {
        double B[NT], junk;
        // first half: pivots in slot 0 of tile column 0 (X_I = B_I nrd, formed where it is used)
        dmma(B[0], junk, odd ? a[0][0] : unit, f.lam, 0.0, 0.0);
        dmma(a[0][0], a[0][1], B[0] * f.nrd, B[0], 0.0, odd ? a[0][1] : 0.0);
#pragma unroll
        for (int I = 1; I < NT; ++I) dmma(B[I], junk, a[tix(I, 0)][0], f.lam, 0.0, 0.0);
        double nrd = f.nrd;
        factor_block<1>(a[0][1], ws + 16, lane, 8 * K + 4 < n, f, cnt, flags);
#pragma unroll
        for (int I = 1; I < NT; ++I) {
            const double X = B[I] * nrd;
            dmma(a[tix(I, 0)][0], a[tix(I, 0)][1], X, B[0], 0.0, a[tix(I, 0)][1]);
#pragma unroll
            for (int J = 1; J <= I; ++J) dmma(a[tix(I, J)][0], a[tix(I, J)][1], X, B[J]);
        }
        // second half: slot 1; the rows of the first half take A[i, P] from the
        // lower triangle, position (2q + 1, r)
        const bool more = K + 1 < NT;
        double e0, e1;  // the finished pivot tile
        if (8 * K + 4 < n) {
            const double up = __shfl_sync(0xffffffffu, a[0][0], (2 * q + 1) * 4 + (r >> 1));
            dmma(B[0], junk, odd ? unit : up, f.lam, 0.0, 0.0);
#pragma unroll
            for (int I = 1; I < NT; ++I) dmma(B[I], junk, a[tix(I, 0)][1], f.lam, 0.0, 0.0);
            nrd = f.nrd;
            if constexpr (NT > 1) {
                double d0, d1;  // the next pivot tile
                dmma(d0, d1, B[1] * nrd, B[1], a[tix(1, 1)][0], a[tix(1, 1)][1]);
                dmma(e0, e1, B[0] * nrd, B[0], odd ? 0.0 : a[0][0], 0.0);
                a[0][0] = d0;
                a[0][1] = d1;
                factor_block<0>(a[0][0], ws, lane, more, f, cnt, flags);
#pragma unroll
                for (int I = 1; I < NT; ++I) {
                    double t0, t1;
                    const double X = B[I] * nrd;
                    dmma(t0, t1, X, B[0], a[tix(I, 0)][0], 0.0);
                    *reinterpret_cast<double2 *>(tb + ((I - 1) * 8 + r) * G<NT>::TPITCH + 2 * q) = make_double2(t0, t1);
                    if (I > 1) {
#pragma unroll
                        for (int J = 1; J <= I; ++J)
                            dmma(a[tix(I - 1, J - 1)][0], a[tix(I - 1, J - 1)][1], X, B[J], a[tix(I, J)][0], a[tix(I, J)][1]);
                    }
                }
            } else {
                dmma(e0, e1, B[0] * nrd, B[0], odd ? 0.0 : a[0][0], 0.0);
            }
        } else {  // the last tile column, its second half all padding: only the move
            e0 = a[0][0];
            e1 = a[0][1];
            if constexpr (NT > 1) {
#pragma unroll
                for (int I = 1; I < NT; ++I)
                    *reinterpret_cast<double2 *>(tb + ((I - 1) * 8 + r) * G<NT>::TPITCH + 2 * q) =
                        make_double2(a[tix(I, 0)][0], a[tix(I, 0)][1]);
#pragma unroll
                for (int I = 1; I < NT; ++I)
#pragma unroll
                    for (int J = 1; J <= I; ++J) {
                        a[tix(I - 1, J - 1)][0] = a[tix(I, J)][0];
                        a[tix(I - 1, J - 1)][1] = a[tix(I, J)][1];
                    }
            }
        }
        if constexpr (NT > 1) {
            __syncwarp();
#pragma unroll
            for (int J = 0; J + 1 < NT; ++J) {
                a[tix(NT - 1, J)][0] = tb[(J * 8 + 2 * q) * G<NT>::TPITCH + r];
                a[tix(NT - 1, J)][1] = tb[(J * 8 + 2 * q + 1) * G<NT>::TPITCH + r];
            }
        }
        a[tix(NT - 1, NT - 1)][0] = e0;
        a[tix(NT - 1, NT - 1)][1] = e1;
    }
    bad = flags_to_status(flags);
    return cnt;
}

// ---- element bookkeeping ----------------------------------------------------
// Channel of the row, and of column slot s, of tile (I, J) held by `lane`.
__device__ __forceinline__ int frow(int I, int lane) { return 8 * I + chan_of(lane >> 2); }
__device__ __forceinline__ int fcol(int J, int lane, int s) { return 8 * J + chan_of(2 * (lane & 3) + s); }
// The lanes with (lane & 3) == lane >> 3 hold the diagonal of a diagonal tile, in slot (lane >> 2) & 1.
__device__ __forceinline__ bool fdiag(int lane, int s) { return (lane >> 2) == 2 * (lane & 3) + s; }

}  // namespace wf
}  // namespace mgpu
