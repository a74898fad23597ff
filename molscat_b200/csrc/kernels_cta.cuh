// LDMD / LDJ / LDMG kernels with one CTA per matrix: 64 < N <= 200.
// Included by propagator.cu after kernels_frag.cuh.
//
// The lower 8x8 tiles of the matrix stay with their warps for the whole
// propagation, in the DMMA accumulator layout: lane l holds positions
// (l>>2, 2(l&3) + s) of a tile.  The tile warps hold the off-diagonal tiles in
// registers, the last warp (the factoring warp) the diagonal ones in shared
// memory.  VL and the 2HQ(C) table are stored tile after tile in the same
// layout, the channels in their own order.
//
// The sweep takes the eight pivots of a tile row K at a time, as two blocks of
// four (P1, P2) with the arithmetic of warp_dmma.cuh:
//   a. the owners of tile column and row K publish the panel A[:, K], then zero
//      those tiles;                                                   barrier
//   b. thread i turns row i of the panel into the operands of both blocks:
//      c1 = Lam1 A[i, P1], x1 = -c1/delta; A[i, P2] += x1 . c1(P2) (what the
//      first block's update does to it); c2, x2.  Rows of P1 and P2 take -I for
//      their panel rows (so c = -Lam^T, x = Lam^T/delta), and zero in the first
//      block's operands for P2 (its rows and columns are zeroed between the
//      blocks);                                                        barrier
//   e. every tile: A_IJ += X1_I B1_J, then += X2_I B2_J, two DMMAs.  The
//      factoring warp does the next diagonal tile first and factors it (both
//      four-pivot blocks and the update between them) before its other tiles.
// So a tile row costs two CTA barriers, and the chain of pivot reciprocals runs
// beside the tile warps' DMMAs and their publishing of the next panel.
//
// What bounds it: the chain diagonal update -> 8x8 factor -> operand rows,
// against NT(NT+1)/2 * 2 * 16 / 4 cycles of DMMA a tile row; two CTAs an SM
// overlap the two.  No loop over a warp's tiles branches on a tile: a test, a
// table read and a skip per tile serialised their latencies (150 cycles a tile
// to publish, 190 to update).  The form before this one took four pivots a
// round and 3900 cycles for it at N = 106 with two CTAs an SM.
#pragma once
#include "kernels_frag.cuh"

namespace mgpu {
namespace cta {

using wf::tix;

// NT tile rows, W warps in all: W - 1 tile warps and the factoring warp.
template <int NT, int W>
struct CG {
    static constexpr int NTL = NT * (NT + 1) / 2;
    static constexpr int NPAD = 8 * NT;
    static constexpr int NTHR = 32 * W;
    static constexpr int TW = W - 1;                                // tile warps
    // The factoring warp's chain of DFMAs waits for the DMMAs of the other warps on its
    // scheduler's FP64 pipe.  At NT = 14 and 20 those warps (3, 7, .. of 4n) take LN / LDEN of
    // the others' tiles.  It costs registers (spill loads of the step kernels at NT = 14: LDMD
    // 168 -> 624 bytes a thread, LDPROP 68 -> 812, LDMG 28 -> 376) and is the faster all the
    // same, us a step without -> with: N = 106, 1184 jobs, LDMD 430 -> 401, LDMG 1221 -> 1143,
    // LDPROP 703 -> 709 (no difference; 296 jobs 176 -> 171), 96 jobs LDMD 82.5 -> 81.8, LDMG 251
    // -> 247; N = 150, 1184 jobs, LDMD 1189 -> 1138, LDMG 3299 -> 3189, 48 jobs LDMD 147 -> 141.
    // Not so elsewhere: N = 90 (any number of jobs) no difference, N = 128, 1184 jobs, LDMD 610
    // -> 623, LDMG 1555 -> 1562 (but LDPROP 1314 -> 1262), N = 199, 592 jobs, LDMD 1236 -> 1292.
    // N = 72 in its shape of eight warps for few jobs would gain 2 %.
    static constexpr int LIGHT = NT == 14 || NT == 20 ? TW / 4 : 0;
    static constexpr int LN = W <= 8 ? 2 : 4, LDEN = W <= 8 ? 3 : 5;
    // tiles of one of the other warps when there are `ntiles` off the diagonal
    __host__ __device__ static constexpr int heavy(int ntiles)
    {
        const int parts = LDEN * (TW - LIGHT) + LN * LIGHT;
        return (LDEN * ntiles + parts - 1) / parts;
    }
    static constexpr int TPW = heavy(NT * (NT - 1) / 2);            // tile slots of a warp
    static constexpr int TD = NTL * 64;                             // doubles of one tiled matrix
    // pitch of the panel and operand columns in 16-byte pairs: 2 mod 8, so that the
    // eight lanes of an access phase meet eight bank groups; eight rows past the
    // matrix, always zero, for the slots that hold no tile (and read past the last tile
    // row where the diagonal tiles are taken by twos and their number is odd)
    static constexpr int LD = NPAD + 10;
};

// The factored 8x8 block in shared memory: [0..9] Block4 of P1, [10..19] of P2,
// [20..35] c1 of the rows of P2, [36..51] x1 of them, [52..67] a block on its
// way through ldl_block4_any.
struct Fact {
    static constexpr int P1 = 0, P2 = 10, C = 20, X = 36, ANY = 52, SIZE = 68;
};

// Shared memory of one CTA, in doubles.
template <int NT, int W>
struct CSmem {
    using C = CG<NT, W>;
    static constexpr int PAN = 0;                       // panel [4][LD] pairs of columns
    static constexpr int XS = PAN + 8 * C::LD;          // X operands [4][LD] pairs (block 1, block 2)
    static constexpr int BS = XS + 8 * C::LD;           // B operands
    static constexpr int DG = BS + 8 * C::LD;           // the diagonal tiles and room for one more (rounded up to four)
    static constexpr int FB = DG + 64 * ((NT + 3) / 4 * 4);             // Fact
    static constexpr int VEC = FB + Fact::SIZE;         // y14, y14', y23 by channel, twice (step parity)
    static constexpr int PARK = VEC + 6 * C::NPAD + 8;  // LDJ: the parked Z (eight doubles of slack for empty slots' reads)
    __host__ __device__ static constexpr size_t bytes(bool park) { return (size_t)(PARK + (park ? C::TD : 0)) * 8; }
};

// What a warp holds: the off-diagonal tiles e0 .. e0 + ntw - 1 of the row-major
// list (tile slots; rc = 128 I | 128 J << 16, the byte offsets of its operand
// rows, I = J = NT for an empty slot), or the
// diagonal tiles (the factoring warp).
template <int NT, int W>
struct Own {
    using C = CG<NT, W>;
    int warp, lane, nb, e0, ntw;
    unsigned rc[C::TPW];
    double *dg;

    // also clears the operand rows past the matrix; ends with a barrier
    __device__ __forceinline__ Own(double *sm, int n)
    {
        warp = threadIdx.x >> 5;
        lane = threadIdx.x & 31;
        nb = (n + 7) >> 3;
        const int nact = nb * (nb - 1) / 2, hv = C::heavy(nact);
        const int lt = C::LIGHT ? max(0, nact - (C::TW - C::LIGHT) * hv + C::LIGHT - 1) / max(1, C::LIGHT) : hv;
        e0 = (warp - warp / 4) * hv + warp / 4 * lt;
        ntw = warp < C::TW ? max(0, min(C::LIGHT && (warp & 3) == 3 ? lt : hv, nact - e0)) : 0;
        dg = sm + CSmem<NT, W>::DG;
#pragma unroll
        for (int u = 0; u < C::TPW; ++u) {
            int I = 1, e = e0 + u;
            while (I * (I + 1) / 2 <= e) ++I;  // row I of the strict lower triangle starts at I(I-1)/2
            rc[u] = u < ntw ? (unsigned)(128 * I | (128 * (e - I * (I - 1) / 2)) << 16) : 128u * NT | (128u * NT) << 16;
        }
        for (int i = threadIdx.x; i < 64; i += C::NTHR) {
            const int o = 2 * ((i >> 4) * C::LD + C::NPAD) + (i & 15);
            sm[CSmem<NT, W>::XS + o] = sm[CSmem<NT, W>::BS + o] = 0.0;
        }
        __syncthreads();
    }
    // f(t, I, J, real, a0, a1) for every tile of this warp; a slot without a tile is passed with real =
    // false, a valid t and I = J = NT.
    template <class F>
    __device__ __forceinline__ void each(double (&acc)[C::TPW][2], F &&f) const
    {
        if (warp == C::TW) {
#pragma unroll 2
            for (int I = 0; I < nb; ++I) {
                double2 *d = reinterpret_cast<double2 *>(dg + 64 * I) + lane;
                double2 v = *d;
                f(tix(I, I), I, I, true, v.x, v.y);
                *d = v;
            }
        } else {
#pragma unroll
            for (int g = 0; g < C::TPW; g += 5) {
                if (g < ntw) {
#pragma unroll
                    for (int u = g; u < (g + 5 < C::TPW ? g + 5 : C::TPW); ++u) {
                        const int I = (rc[u] & 0xffff) >> 7, J = rc[u] >> 23;
                        const bool real = u < ntw;
                        f(real ? tix(I, J) : 0, I, J, real, acc[u][0], acc[u][1]);
                    }
                }
            }
        }
    }
};

__device__ __forceinline__ void put_block4(double *d, const wf::Block4 &b)
{
    double2 *p = reinterpret_cast<double2 *>(d);
    p[0] = make_double2(b.r0, b.r1);
    p[1] = make_double2(b.r2, b.r3);
    p[2] = make_double2(b.m10, b.m20);
    p[3] = make_double2(b.m21, b.m30);
    p[4] = make_double2(b.m31, b.m32);
}

__device__ __forceinline__ void get_block4(const double *d, wf::Block4 &b)
{
    const double2 *p = reinterpret_cast<const double2 *>(d);
    double2 v;
    v = p[0], b.r0 = v.x, b.r1 = v.y;
    v = p[1], b.r2 = v.x, b.r3 = v.y;
    v = p[2], b.m10 = v.x, b.m20 = v.y;
    v = p[3], b.m21 = v.x, b.m30 = v.y;
    v = p[4], b.m31 = v.x, b.m32 = v.y;
}

// c = Lam v, x = -c / delta
__device__ __forceinline__ void row_operands(const wf::Block4 &b, const double (&v)[4], double (&c)[4], double (&x)[4])
{
    c[0] = v[0];
    c[1] = fma(b.m10, v[0], v[1]);
    c[2] = fma(b.m20, v[0], fma(b.m21, v[1], v[2]));
    c[3] = fma(b.m30, v[0], fma(b.m31, v[1], fma(b.m32, v[2], v[3])));
    x[0] = c[0] * -b.r0;
    x[1] = c[1] * -b.r1;
    x[2] = c[2] * -b.r2;
    x[3] = c[3] * -b.r3;
}

// The factoring warp: the 8x8 block of the diagonal tile dt (lower triangle)
// into fb, the four-pivot chains in every lane, the rows of P2 and its update
// (written back into dt) spread over the lanes.
__device__ __forceinline__ void factor8(double *dt, double *fb, int lane, int &cnt, int &flags)
{
    auto factor4 = [&](int o, double *out) {  // the 4x4 block from channel o
        auto at = [&](int i, int j) { return dt[8 * (o + i) + o + j]; };
        wf::Block4 b;
        int c;
        const double d00 = at(0, 0), d10 = at(1, 0), d11 = at(1, 1), d20 = at(2, 0), d21 = at(2, 1), d22 = at(2, 2);
        const double d30 = at(3, 0), d31 = at(3, 1), d32 = at(3, 2), d33 = at(3, 3);
        if (!wf::ldl_block4_plain(d00, d10, d11, d20, d21, d22, d30, d31, d32, d33, b, c)) {
            double *blk = fb + Fact::ANY;
            __syncwarp();
            if (lane == 0) {
                blk[0] = d00, blk[4] = d10, blk[5] = d11, blk[8] = d20, blk[9] = d21, blk[10] = d22;
                blk[12] = d30, blk[13] = d31, blk[14] = d32, blk[15] = d33;
            }
            __syncwarp();
            const int cf = wf::ldl_block4_any(blk);
            c = cf & 255;
            flags |= cf >> 8;
            wf::block4_from(blk, b);
        }
        cnt += c;
        if (lane == 0) put_block4(out, b);
        return b;
    };
    __syncwarp();
    const wf::Block4 b1 = factor4(0, fb + Fact::P1);
    {
        const int m = lane & 3;  // every group of four lanes the same: no divergence
        const double *row = dt + 8 * (4 + m);
        const double v[4] = {row[0], row[1], row[2], row[3]};
        double c[4], x[4];
        row_operands(b1, v, c, x);
        if (lane < 4) {
            double2 *pc = reinterpret_cast<double2 *>(fb + Fact::C + 4 * m), *px = reinterpret_cast<double2 *>(fb + Fact::X + 4 * m);
            pc[0] = make_double2(c[0], c[1]);
            pc[1] = make_double2(c[2], c[3]);
            px[0] = make_double2(x[0], x[1]);
            px[1] = make_double2(x[2], x[3]);
        }
    }
    __syncwarp();
    {
        const int i = (lane >> 2) & 3, j = lane & 3;  // element (i, j) of P2 (the upper triangle is not read)
        const double2 *px = reinterpret_cast<const double2 *>(fb + Fact::X + 4 * i), *pc = reinterpret_cast<const double2 *>(fb + Fact::C + 4 * j);
        const double2 x01 = px[0], x23 = px[1], c01 = pc[0], c23 = pc[1];
        double *d = dt + 8 * (4 + i) + 4 + j;
        const double v = fma(x23.y, c23.y, fma(x23.x, c23.x, fma(x01.y, c01.y, fma(x01.x, c01.x, *d))));
        __syncwarp();
        if (lane < 16) *d = v;
    }
    __syncwarp();
    factor4(4, fb + Fact::P2);
}

// Shared-memory accesses of the tile loops by 32-bit address, the predicated
// ones without a branch.
__device__ __forceinline__ double2 lds2(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void lds2_if(bool p, double2 &v, uint32_t a)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p ld.shared.v2.f64 {%0, %1}, [%3];\n\t}"
                 : "+d"(v.x), "+d"(v.y)
                 : "r"((int)p), "r"(a)
                 : "memory");
}
__device__ __forceinline__ void sts2_if(bool p, uint32_t a, double v0, double v1)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p st.shared.v2.f64 [%1], {%2, %3};\n\t}" ::"r"((int)p), "r"(a),
                 "d"(v0), "d"(v1)
                 : "memory");
}
__device__ __forceinline__ void sts_if(bool p, uint32_t a, double v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %0, 0;\n\t@p st.shared.f64 [%1], %2;\n\t}" ::"r"((int)p), "r"(a), "d"(v)
                 : "memory");
}

// -A^{-1} of the CTA's matrix in place; returns the negative-pivot count, `bad`
// as in tiles.cuh.  Every thread of the CTA calls it together.  Padding channels
// up to the next multiple of eight have a positive diagonal.  N > 8 (two tile
// rows): then the first CTA barrier of an inversion lies before the store of its
// counters, and no barrier is needed between two of them.
template <int NT, int W>
__device__ __forceinline__ int cta_invert(double (&acc)[CG<NT, W>::TPW][2], const Own<NT, W> &own, double *sm, int *cf,
                                          int &bad)
{
    using C = CG<NT, W>;
    using M = CSmem<NT, W>;
    const int tid = threadIdx.x, lane = own.lane, r = lane >> 2, q = lane & 3;
    const bool factoring = own.warp == C::TW;
    double *pan = sm + M::PAN, *fb = sm + M::FB;
    double2 *xs = reinterpret_cast<double2 *>(sm + M::XS), *bs = reinterpret_cast<double2 *>(sm + M::BS);
    const double2 *xr = xs + q * C::LD + r, *br = bs + q * C::LD + r;
    // byte addresses: this lane's operands of tile row 0, and where its elements of a tile of the
    // panel's column (row 8I + r) or row (transposed) go
    const uint32_t xa = smem_u32(xr), ba = smem_u32(br);
    const uint32_t pc = smem_u32(pan + 2 * (q * C::LD + r));
    const uint32_t pr = smem_u32(pan + 2 * ((r >> 1) * C::LD + 2 * q) + (r & 1));
    const int nb = own.nb;
    int cnt = 0, flags = 0;
    if (factoring) factor8(own.dg, fb, lane, cnt, flags);
#pragma unroll 1
    for (int K = 0; K < nb; ++K) {
        if (!factoring) {
            // a. publish tile column K below the diagonal and tile row K left of it; zero them
            const unsigned kk = 128u * K;
#pragma unroll
            for (int u = 0; u < C::TPW; ++u) {
                const unsigned oi = own.rc[u] & 0xffff, oj = own.rc[u] >> 16;
                const bool col = oj == kk, row = oi == kk;
                sts2_if(col, pc + oi, acc[u][0], acc[u][1]);
                sts_if(row, pr + oj, acc[u][0]);
                sts_if(row, pr + 16 + oj, acc[u][1]);
                acc[u][0] = col || row ? 0.0 : acc[u][0];
                acc[u][1] = col || row ? 0.0 : acc[u][1];
            }
        } else if (K + 1 == nb && lane == 0) {
            cf[0] = cnt;
            cf[1] = flags;
        }
        __syncthreads();
        // b. operand rows, the same code for the rows of P1 and P2 with other inputs
        for (int i = tid; i < 8 * nb; i += C::NTHR) {
            double *xi = reinterpret_cast<double *>(xs + i), *bi = reinterpret_cast<double *>(bs + i);
            const int a = i - 8 * K;
            const bool p1 = a >= 0 && a < 4, p2 = a >= 4 && a < 8;
            const double2 *p = reinterpret_cast<const double2 *>(pan) + i;
            const double2 t0 = p[0], t1 = p[C::LD], t2 = p[2 * C::LD], t3 = p[3 * C::LD];
            const bool own_row = p1 || p2;
            double v[4] = {own_row ? (a == 0 ? -1.0 : 0.0) : t0.x, own_row ? (a == 1 ? -1.0 : 0.0) : t0.y,
                           own_row ? (a == 2 ? -1.0 : 0.0) : t1.x, own_row ? (a == 3 ? -1.0 : 0.0) : t1.y};
            double w[4] = {own_row ? 0.0 : t2.x, own_row ? 0.0 : t2.y, own_row ? 0.0 : t3.x, own_row ? 0.0 : t3.y};
            double c[4], x[4];
            wf::Block4 b;
            get_block4(fb + Fact::P1, b);
            row_operands(b, v, c, x);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                xi[2 * k * C::LD] = x[k];
                bi[2 * k * C::LD] = c[k];
            }
            // A[i, P2]'s update is x1(P2) . c1(i), row P2 of the lower triangle, for rows above it, else x1(i) . c1(P2)
            const bool swap = p1 || a < 0;
            const double *o = fb + (swap ? Fact::X : Fact::C);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double f = swap ? c[k] : x[k];
#pragma unroll
                for (int m = 0; m < 4; ++m) w[m] = fma(f, o[4 * m + k], w[m]);
            }
            if (p2) {
#pragma unroll
                for (int m = 0; m < 4; ++m) w[m] = a == 4 + m ? -1.0 : 0.0;
            }
            get_block4(fb + Fact::P2, b);
            row_operands(b, w, c, x);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                xi[2 * k * C::LD + 1] = x[k];
                bi[2 * k * C::LD + 1] = c[k];
            }
        }
        __syncthreads();
        // e. the update, the next diagonal tile first
        if (factoring) {
            auto diag = [&](int I0, auto count) {  // `count` tiles from I0, their loads first
                constexpr int NC = decltype(count)::value;
                double2 x[NC], b[NC], v[NC];
#pragma unroll
                for (int m = 0; m < NC; ++m) {
                    x[m] = lds2(xa + 128 * (I0 + m));
                    b[m] = lds2(ba + 128 * (I0 + m));
                    v[m] = *(reinterpret_cast<const double2 *>(own.dg + 64 * (I0 + m)) + lane);
                    if (I0 + m == K) v[m] = make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int m = 0; m < NC; ++m) wf::dmma(v[m].x, v[m].y, x[m].x, b[m].x);
#pragma unroll
                for (int m = 0; m < NC; ++m) {
                    wf::dmma(v[m].x, v[m].y, x[m].y, b[m].y);
                    if (NC == 1 || I0 + m != K + 1) *(reinterpret_cast<double2 *>(own.dg + 64 * (I0 + m)) + lane) = v[m];
                }
            };
            if (K + 1 < nb) {
                diag(K + 1, std::integral_constant<int, 1>());
                factor8(own.dg + 64 * (K + 1), fb, lane, cnt, flags);
            }
            // the others (tile K + 1's second update is dropped)
#pragma unroll 1
            for (int I = 0; I < nb; I += 2) diag(I, std::integral_constant<int, 2>());
        } else {
            unsigned held = ~0u;  // the row operand in x
            double2 x = make_double2(0.0, 0.0);
#pragma unroll
            for (int g = 0; g < C::TPW; g += 5) {
                constexpr int GW = 5;
                if (g < own.ntw) {
                    double2 b[GW];
#pragma unroll
                    for (int u = g; u < g + GW; ++u)
                        if (u < C::TPW) {
                            b[u - g] = lds2(ba + (own.rc[u] >> 16));
                        }
#pragma unroll
                    for (int u = g; u < g + GW; ++u)
                        if (u < C::TPW) {
                            const unsigned at = xa + (own.rc[u] & 0xffff);
                            lds2_if(at != held, x, at);
                            held = at;
                            wf::dmma(acc[u][0], acc[u][1], x.x, b[u - g].x);
                            wf::dmma(acc[u][0], acc[u][1], x.y, b[u - g].y);
                        }
                }
            }
        }
    }
    bad = flags_to_status(cf[1]);
    return cf[0];
}

// The coupling sum of this lane's two elements of tile t at P (SUMLAM).
__device__ __forceinline__ double2 w_sum(const SysDev &S, const double *__restrict__ P, int t, int lane)
{
    const size_t td = (size_t)S.ntiles * 64, x = (size_t)t * 64 + lane * 2;
    double w0 = 0.0, w1 = 0.0;
    if (S.ivlfl <= 0) {
        for (int l = 0; l < S.nham; ++l) {
            const double2 v = __ldg(reinterpret_cast<const double2 *>(S.vlt + l * td + x));
            const double pl = __ldg(P + l);
            w0 = fma(v.x, pl, w0);
            w1 = fma(v.y, pl, w1);
        }
    } else {
        for (int l = 0; l < S.nham; ++l) {
            const double2 v = __ldg(reinterpret_cast<const double2 *>(S.vlt + l * td + x));
            const int2 ix = __ldg(reinterpret_cast<const int2 *>(S.ivt + l * td + x));
            if (v.x != 0.0) w0 = fma(v.x, __ldg(P + ix.x), w0);
            if (v.y != 0.0) w1 = fma(v.y, __ldg(P + ix.y), w1);
        }
    }
    return make_double2(w0, w1);
}

// The diagonal terms of W(R) for channel i < N (HAMMAT, hammat.f:85-113).
__device__ __forceinline__ double w_diag(const SysDev &S, int i, int ir, double ered, double w)
{
    const double R = __ldg(S.rtab + ir);
    const double rsq = fmin(1.0 / (R * R), 1.0e16);
    if (S.nrsq == 0) w += rsq * S.cent[i];
    if (S.nconst == 0) w += S.eint[i];
    if (S.conlen > 0.0) {
        const double c2 = S.conlen * S.conlen;
        w += R * R / (c2 * c2);
    }
    return w - ered;
}

// W(R_ir) of element x, (i, j) of a tiled matrix in channel order (the large-N
// kernels), optionally with the diagonal terms.
__device__ __forceinline__ double w_elem(const SysDev &S, const double *__restrict__ P, int x, int i, int j, int ir,
                                         double ered, bool diag_terms)
{
    const size_t td = (size_t)S.ntiles * 64;
    double w = 0.0;
    if (S.ivlfl <= 0) {
        for (int l = 0; l < S.nham; ++l) w = fma(__ldg(S.vlt + l * td + x), __ldg(P + l), w);
    } else {
        for (int l = 0; l < S.nham; ++l) {
            const double v = __ldg(S.vlt + l * td + x);
            if (v != 0.0) w = fma(v, __ldg(P + __ldg(S.ivt + l * td + x)), w);
        }
    }
    if (diag_terms && i == j && i < S.n) w = w_diag(S, i, ir, ered, w);
    return w;
}

// One lane's view of a tile: its row channel, its two column channels, and
// which of the two elements is on the diagonal (-1: none).
struct Elem {
    int i, j0, j1, d;
    __device__ __forceinline__ Elem(int I, int J, int lane)
    {
        i = 8 * I + (lane >> 2);
        j0 = 8 * J + 2 * (lane & 3);
        j1 = 8 * J + 2 * (lane & 3) + 1;
        d = i == j0 ? 0 : i == j1 ? 1 : -1;
    }
};

// f(t, e, real, a0, a1, w0, w1) for every tile of this warp, with W(R_ir) of its elements.
template <int NT, int W, class F>
__device__ __forceinline__ void each_w(const SysDev &S, const Own<NT, W> &own, double (&acc)[CG<NT, W>::TPW][2], int ir,
                                       double ered, F &&f)
{
    const double *P = S.ptab + (size_t)ir * S.nham;
    own.each(acc, [&](int t, int I, int J, bool real, double &a0, double &a1) {
        const Elem e(I, J, own.lane);
        double2 w = w_sum(S, P, t, own.lane);
        if (real && e.d >= 0 && e.i < S.n) {
            if (e.d == 0) w.x = w_diag(S, e.i, ir, ered, w.x);
            else w.y = w_diag(S, e.i, ir, ered, w.y);
        }
        f(t, e, real, a0, a1, w.x, w.y);
    });
}

// The lower triangle of the caller's Y into the tiles, and the tiles (times
// `scale`) into both triangles of it.
template <int NT, int W>
__device__ __forceinline__ void load_y(const double *__restrict__ y, int n, const Own<NT, W> &own,
                                       double (&acc)[CG<NT, W>::TPW][2])
{
#pragma unroll
    for (int u = 0; u < CG<NT, W>::TPW; ++u) acc[u][0] = acc[u][1] = 0.0;
    own.each(acc, [&](int, int I, int J, bool, double &a0, double &a1) {
        const Elem e(I, J, own.lane);
        const int lo0 = min(e.i, e.j0), hi0 = max(e.i, e.j0), lo1 = min(e.i, e.j1), hi1 = max(e.i, e.j1);
        a0 = hi0 < n ? y[(size_t)lo0 * n + hi0] : 0.0;
        a1 = hi1 < n ? y[(size_t)lo1 * n + hi1] : 0.0;
    });
}

template <int NT, int W>
__device__ __forceinline__ void store_y(double *__restrict__ y, int n, const Own<NT, W> &own, double scale,
                                        double (&acc)[CG<NT, W>::TPW][2])
{
    own.each(acc, [&](int, int I, int J, bool, double &a0, double &a1) {
        const Elem e(I, J, own.lane);
        if (e.i < n && e.j0 <= e.i) {
            const double v = scale * a0;
            y[(size_t)e.j0 * n + e.i] = v;
            y[(size_t)e.i * n + e.j0] = v;
        }
        if (e.i < n && e.j1 <= e.i) {
            const double v = scale * a1;
            y[(size_t)e.j1 * n + e.i] = v;
            y[(size_t)e.i * n + e.j1] = v;
        }
    });
}

// CTAs an SM the register budget is set for: two of eight warps, one of sixteen.
// Most step kernels spill at it (spill loads a thread, LDMD: <25, 16> 2844 bytes,
// <16, 8> 1928, <10, 4> 964, <20, 12> 628, <14, 8> 624; at N = 106 that is 2.5 % of
// the instructions executed).
template <int W>
constexpr int min_ctas() { return W <= 4 ? 4 : W <= 8 ? 2 : 1; }

// ---------------------------------------------------------------------------
// MDPROP energy-independent half: one CTA per (step, system).
// ---------------------------------------------------------------------------
template <int NT, int W>
__global__ void __launch_bounds__(32 * W, min_ctas<W>())
ldmd_prep_cta_kernel(const SysDev *__restrict__ systems, const int *__restrict__ sys_list)
{
    using C = CG<NT, W>;
    extern __shared__ __align__(16) double sm[];
    __shared__ int cf[2];
    __shared__ SysDev s_sys;
    if (threadIdx.x == 0) s_sys = systems[sys_list[blockIdx.y]];
    __syncthreads();
    const SysDev &S = s_sys;
    const int k = blockIdx.x + 1;
    if (k > S.nstep) return;  // whole CTA
    const Own<NT, W> own(sm, S.n);
    const int lane = own.lane;
    const double h = S.dr / 2.0;
    const double d1 = h * h / 3.0;
    const double d4 = -d1 / 16.0;
    const double *P = S.ptab + (size_t)(2 * k - 1) * S.nham;
    double a[C::TPW][2];
    own.each(a, [&](int t, int I, int J, bool real, double &a0, double &a1) {
        const Elem e(I, J, lane);
        const double2 w = w_sum(S, P, t, lane);
        a0 = e.d == 0 ? 0.125 : d4 * w.x;
        a1 = e.d == 1 ? 0.125 : d4 * w.y;
    });
    int bad = SWEEP_OK;
    const int cnt = cta_invert<NT, W>(a, own, sm, cf, bad);
    if (bad != SWEEP_OK) {
        if (threadIdx.x == 0) {
            atomicMax(&S.prep[1], bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE);
            atomicMin(&S.prep[2], k);
        }
        return;
    }
    if (threadIdx.x == 0 && cnt) atomicAdd(&S.prep[0], cnt);
    double *qk = S.q + (size_t)(k - 1) * C::TD;
    own.each(a, [&](int t, int I, int J, bool real, double &a0, double &a1) {
        const Elem e(I, J, lane);
        // a = -U^{-1};  2HQ(C) = U^{-1} - 8I; zero in the padding
        double2 v;
        v.x = (e.i >= S.n || e.j0 >= S.n) ? 0.0 : (e.d == 0 ? -a0 - 8.0 : -a0);
        v.y = (e.i >= S.n || e.j1 >= S.n) ? 0.0 : (e.d == 1 ? -a1 - 8.0 : -a1);
        if (real) *reinterpret_cast<double2 *>(qk + (size_t)t * 64 + lane * 2) = v;
    });
}

// ---------------------------------------------------------------------------
// MDPROP step loop, one CTA per job.
// ---------------------------------------------------------------------------
template <int NT, int W>
__global__ void __launch_bounds__(32 * W, min_ctas<W>())
ldmd_prop_cta_kernel(const SysDev *__restrict__ systems, const JobDev *__restrict__ jobs, double *__restrict__ y,
                     int *__restrict__ nodes_out, int *__restrict__ status_out, int *__restrict__ kfail_out)
{
    using C = CG<NT, W>;
    extern __shared__ __align__(16) double sm[];
    __shared__ int cf[2];
    __shared__ int s_stop;
    __shared__ SysDev s_sys;
    const JobDev job = jobs[blockIdx.x];
    if (threadIdx.x == 0) s_sys = systems[job.sys];
    __syncthreads();
    const SysDev &S = s_sys;
    const Own<NT, W> own(sm, S.n);
    const int tid = threadIdx.x, lane = own.lane;
    const int n = S.n;
    const int nstep = S.nstep;
    const double ered = job.ered;
    if (S.prep[1] != 0) {
        if (tid == 0) {
            status_out[job.out] = S.prep[1];
            kfail_out[job.out] = S.prep[2];
            nodes_out[job.out] = 0;
        }
        return;
    }
    const double h = S.dr / 2.0;
    const double d1 = h * h / 3.0;
    const double d2 = 2.0 * d1;
    const double half = 0.5 * h;
    double *yj = y + job.yoff;
    // padding channels: diagonal 1 or 2 at every inversion
    for (int i = tid; i < 2 * C::NPAD; i += C::NTHR) {
        double *v = sm + CSmem<NT, W>::VEC + (i / C::NPAD) * 3 * C::NPAD + i % C::NPAD;
        v[0] = 0.5;
        v[C::NPAD] = 1.0;
        v[2 * C::NPAD] = 0.0;
    }
    double a[C::TPW][2];
    load_y<NT, W>(yj, n, own, a);
    each_w<NT, W>(S, own, a, 0, ered, [&](int, const Elem &, bool, double &a0, double &a1, double w0, double w1) {
        a0 = fma(h, a0, d1 * w0);  // mdprop.f:89-93
        a1 = fma(h, a1, d1 * w1);
    });
    __syncthreads();
    int nodes = 0, status = MGPU_OK, kfail = 0;
    const unsigned long long t0 = global_ns();
    for (int k = 1; k <= nstep; ++k) {
        if (stop_poll_step(k)) {  // host cancel / time limit: thread 0's reading for the CTA
            if (tid == 0) s_stop = stop_requested(S.ctl, t0);
            __syncthreads();  // the next write comes kStopPoll steps (and their barriers) later
            const int stop = s_stop;
            if (stop != MGPU_OK) {
                status = stop;
                kfail = k;
                break;
            }
        }
        // reference-potential solutions (mdprop.f:143-164), in the buffer of this step's
        // parity: the other one may still be read by the last step's tile warps
        double *s_y14 = sm + CSmem<NT, W>::VEC + (k & 1) * 3 * C::NPAD;
        double *s_y14b = s_y14 + C::NPAD, *s_y23 = s_y14b + C::NPAD;
        for (int i = tid; i < n; i += C::NTHR) {
            const int p = i & 7;
            const size_t td = (size_t)S.ntiles * 64, e = (size_t)tix(i >> 3, i >> 3) * 64 + (p * 4 + (p >> 1)) * 2 + (p & 1);
            const double *P = S.ptab + (size_t)(2 * k - 1) * S.nham;
            double x = 0.0;
            for (int l = 0; l < S.nham; ++l) {
                const double v = __ldg(S.vlt + l * td + e);
                if (S.ivlfl <= 0) x = fma(v, __ldg(P + l), x);
                else if (v != 0.0) x = fma(v, __ldg(P + __ldg(S.ivt + l * td + e)), x);
            }
            const double wref = w_diag(S, i, 2 * k - 1, ered, x);
            double y14, y23;
            ref_solutions(wref, half, y14, y23);
            s_y14[i] = y14;
            s_y14b[i] = y14 - d1 * wref;
            s_y23[i] = y23;
        }
        __syncthreads();
        own.each(a, [&](int, int I, int J, bool real, double &a0, double &a1) {
            if (I != J) return;
            const Elem e(I, J, lane);
            const double d = s_y14b[e.i];
            if (e.d == 0) a0 += d;
            if (e.d == 1) a1 += d;
        });
        int bad = SWEEP_OK;
        nodes += cta_invert<NT, W>(a, own, sm, cf, bad);
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        const double *qk = S.q + (size_t)(k - 1) * C::TD + lane * 2;
        own.each(a, [&](int t, int I, int J, bool real, double &a0, double &a1) {
            const Elem e(I, J, lane);
            // Y = 2HQ(C) + 2 Y14 - Y23 Y^-1 Y23  (a holds -Y^-1), mdprop.f:156,181-185
            const double2 qq = __ldg(reinterpret_cast<const double2 *>(qk + (size_t)t * 64));
            const double yr = s_y23[e.i];
            a0 = qq.x + yr * a0 * s_y23[e.j0];
            a1 = qq.y + yr * a1 * s_y23[e.j1];
            if (I == J) {
                const double d = 2.0 * s_y14[e.i];
                if (e.d == 0) a0 += d;
                if (e.d == 1) a1 += d;
            }
        });
        nodes += cta_invert<NT, W>(a, own, sm, cf, bad);
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        const double dd = (k == nstep) ? d1 : d2;
        each_w<NT, W>(S, own, a, 2 * k, ered, [&](int, const Elem &e, bool, double &a0, double &a1, double w0, double w1) {
            // Y = D2 W(B) - Y23 Y^-1 Y23 + Y14'  (mdprop.f:196-230)
            const double yr = s_y23[e.i];
            a0 = fma(dd, w0, yr * a0 * s_y23[e.j0]);
            a1 = fma(dd, w1, yr * a1 * s_y23[e.j1]);
            const double d = s_y14b[e.i];
            if (e.d == 0) a0 += d;
            if (e.d == 1) a1 += d;
        });
    }
    if (status == MGPU_OK) store_y<NT, W>(yj, n, own, 1.0 / h, a);
    if (tid == 0) {
        status_out[job.out] = status;
        kfail_out[job.out] = kfail;
        nodes_out[job.out] = status == MGPU_OK ? nodes - S.prep[0] : 0;
    }
}

// ---------------------------------------------------------------------------
// LDPROP step loop, one CTA per job; Z waits in shared memory while U is
// inverted.
// ---------------------------------------------------------------------------
template <int NT, int W>
__global__ void __launch_bounds__(32 * W, min_ctas<W>())
ldj_prop_cta_kernel(const SysDev *__restrict__ systems, const JobDev *__restrict__ jobs, double *__restrict__ y,
                    int *__restrict__ nodes_out, int *__restrict__ status_out, int *__restrict__ kfail_out)
{
    using C = CG<NT, W>;
    extern __shared__ __align__(16) double sm[];
    __shared__ int cf[2];
    __shared__ int s_stop;
    __shared__ SysDev s_sys;
    const JobDev job = jobs[blockIdx.x];
    if (threadIdx.x == 0) s_sys = systems[job.sys];
    __syncthreads();
    const SysDev &S = s_sys;
    const Own<NT, W> own(sm, S.n);
    const int tid = threadIdx.x, lane = own.lane;
    double *park = sm + CSmem<NT, W>::PARK + lane * 2;  // only this thread reads what it wrote
    const int n = S.n;
    const double ered = job.ered;
    const double h = S.dr / 2.0;
    const double d1 = h * h / 3.0;
    const double d2 = 2.0 * d1;
    const double d4 = -d1 / 16.0;
    double *yj = y + job.yoff;
    double a[C::TPW][2];
    load_y<NT, W>(yj, n, own, a);
    // the unit matrices cover the padding channels too
    each_w<NT, W>(S, own, a, 0, ered, [&](int, const Elem &e, bool, double &a0, double &a1, double w0, double w1) {
        a0 = fma(h, a0, d1 * w0) + (e.d == 0 ? 1.0 : 0.0);  // ldprop.f:46-51
        a1 = fma(h, a1, d1 * w1) + (e.d == 1 ? 1.0 : 0.0);
    });
    int nodes = 0, status = MGPU_OK, kfail = 0;
    const unsigned long long t0 = global_ns();
    for (int k = 1; k <= S.nstep; ++k) {
        if (stop_poll_step(k)) {
            if (tid == 0) s_stop = stop_requested(S.ctl, t0);
            __syncthreads();  // the next write comes kStopPoll steps (and their barriers) later
            const int stop = s_stop;
            if (stop != MGPU_OK) {
                status = stop;
                kfail = k;
                break;
            }
        }
        int bad = SWEEP_OK, bad2 = SWEEP_OK;
        const int ncz = cta_invert<NT, W>(a, own, sm, cf, bad2);  // ldprop.f:83
        own.each(a, [&](int t, int, int, bool real, double &a0, double &a1) {
            if (real) *reinterpret_cast<double2 *>(park + (size_t)t * 64) = make_double2(a0, a1);
        });
        each_w<NT, W>(S, own, a, 2 * k - 1, ered, [&](int, const Elem &e, bool, double &a0, double &a1, double w0, double w1) {
            a0 = d4 * w0 + (e.d == 0 ? 0.125 : 0.0);  // ldprop.f:67-72
            a1 = d4 * w1 + (e.d == 1 ? 0.125 : 0.0);
        });
        const int ncu = cta_invert<NT, W>(a, own, sm, cf, bad);  // ldprop.f:78
        if (bad != SWEEP_OK || bad2 != SWEEP_OK) {
            status = (bad == SWEEP_ZERO || bad2 == SWEEP_ZERO) ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        nodes += ncz;
        own.each(a, [&](int t, int I, int J, bool real, double &a0, double &a1) {
            const Elem e(I, J, lane);
            const double2 z = *reinterpret_cast<const double2 *>(park + (size_t)t * 64);
            // Z = U^-1 - Z^-1 - 6I (ldprop.f:92-97)
            a0 = -a0 + z.x - (e.d == 0 ? 6.0 : 0.0);
            a1 = -a1 + z.y - (e.d == 1 ? 6.0 : 0.0);
        });
        const int ncz2 = cta_invert<NT, W>(a, own, sm, cf, bad);  // ldprop.f:99
        if (bad != SWEEP_OK) {
            status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
            kfail = k;
            break;
        }
        nodes += ncz2 - ncu;
        const double dd = (k == S.nstep) ? d1 : d2;
        each_w<NT, W>(S, own, a, 2 * k, ered, [&](int, const Elem &e, bool, double &a0, double &a1, double w0, double w1) {
            // Z = D2 W(B) + 2I - Z^-1 (ldprop.f:114-131)
            a0 = dd * w0 + (e.d == 0 ? 2.0 : 0.0) + a0;
            a1 = dd * w1 + (e.d == 1 ? 2.0 : 0.0) + a1;
        });
    }
    if (status == MGPU_OK) {
        // Y = Z/H - I/H (ldprop.f:140-147)
        const double hi = 1.0 / h;
        own.each(a, [&](int, int I, int J, bool real, double &a0, double &a1) {
            const Elem e(I, J, lane);
            a0 = hi * a0 - (e.d == 0 ? hi : 0.0);
            a1 = hi * a1 - (e.d == 1 ? hi : 0.0);
        });
        store_y<NT, W>(yj, n, own, 1.0, a);
    }
    if (tid == 0) {
        status_out[job.out] = status;
        kfail_out[job.out] = kfail;
        nodes_out[job.out] = status == MGPU_OK ? nodes : 0;
    }
}

// ---------------------------------------------------------------------------
// MGPROP step loop on one CTA per job: the stages of the one-warp kernel
// (kernels_frag.cuh, ldmg_prop_frag_kernel).
// ---------------------------------------------------------------------------
template <int NT, int W>
__global__ void __launch_bounds__(32 * W, min_ctas<W>())
ldmg_prop_cta_kernel(const SysDev *__restrict__ systems, const JobDev *__restrict__ jobs, int method,
                     double *__restrict__ y, int *__restrict__ nodes_out, int *__restrict__ status_out,
                     int *__restrict__ kfail_out)
{
    using C = CG<NT, W>;
    extern __shared__ __align__(16) double sm[];
    __shared__ int cf[2];
    __shared__ int s_stop;
    __shared__ SysDev s_sys;
    const JobDev job = jobs[blockIdx.x];
    if (threadIdx.x == 0) s_sys = systems[job.sys];
    __syncthreads();
    const SysDev &S = s_sys;
    const Own<NT, W> own(sm, S.n);
    const wf::MGCoef &M = wf::c_mg[method];
    const int tid = threadIdx.x, lane = own.lane;
    const int n = S.n;
    const double ered = job.ered;
    const double h = S.dr;
    double *yj = y + job.yoff;
    double a[C::TPW][2];
    load_y<NT, W>(yj, n, own, a);
    int nodes = 0, status = MGPU_OK, kfail = 0;
    const unsigned long long t0 = global_ns();
    for (int sec = 0; sec < S.nstep && status == MGPU_OK; ++sec) {
        if (stop_poll_step(sec + 1)) {
            if (tid == 0) s_stop = stop_requested(S.ctl, t0);
            __syncthreads();  // the next write comes kStopPoll sectors (and their barriers) later
            const int stop = s_stop;
            if (stop != MGPU_OK) {
                status = stop;
                kfail = sec + 1;
                break;
            }
        }
#pragma unroll 1
        for (int k = 0; k < M.m; ++k) {
            const int ir = sec * M.stride + k;
            const double bh = M.b[k] * h, ak = M.a[k], ah = ak * h;
            each_w<NT, W>(S, own, a, ir, ered, [&](int, const Elem &e, bool, double &a0, double &a1, double w0, double w1) {
                const double x0 = fma(bh, w0, a0), x1 = fma(bh, w1, a1);  // X = Y + b_k h W
                a0 = ak == 0.0 ? x0 : ah * x0 + (e.d == 0 ? 1.0 : 0.0);        // I + a_k h X
                a1 = ak == 0.0 ? x1 : ah * x1 + (e.d == 1 ? 1.0 : 0.0);
            });
            if (ak == 0.0) continue;
            int bad = SWEEP_OK;
            const int cnt = cta_invert<NT, W>(a, own, sm, cf, bad);
            if (bad != SWEEP_OK) {
                status = bad == SWEEP_ZERO ? MGPU_ERR_INVERSION : MGPU_ERR_NONFINITE;
                kfail = sec + 1;
                break;
            }
            nodes += ak >= 0.0 ? cnt : -cnt;
            const double d1 = 1.0 / ah;
            own.each(a, [&](int, int I, int J, bool real, double &a0, double &a1) {
                const Elem e(I, J, lane);
                a0 = (a0 + (e.d == 0 ? 1.0 : 0.0)) * d1;  // [I - inverse]/(a_k h)
                a1 = (a1 + (e.d == 1 ? 1.0 : 0.0)) * d1;
            });
        }
    }
    if (status == MGPU_OK) store_y<NT, W>(yj, n, own, 1.0, a);
    if (tid == 0) {
        status_out[job.out] = status;
        kfail_out[job.out] = kfail;
        nodes_out[job.out] = status == MGPU_OK ? nodes : 0;
    }
}

}  // namespace cta
}  // namespace mgpu
