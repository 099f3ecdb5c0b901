// dev_potrf128.cuh -- Cholesky factor of one 128x128 diagonal block and its
// inverse, by eight warps on a block that stays in shared memory.
//
// The serial chain of the tile Cholesky runs through this routine once per
// 128 columns, so it is built for latency:
//   - the block is read from L2 once and written once; every panel, update
//     and inverse in between is shared-memory traffic;
//   - warp 0 factors a 32x32 diagonal block column by column (chol32_col) with
//     nothing on the chain from one pivot to the next but the reciprocal root, a
//     product and a multiply-add;
//   - the rows below are solved by substitution, one row per lane (sweep32),
//     which needs the factor only.  The inverse of the diagonal block is the
//     same sweep on the unit vectors, beside it on another warp, so no inverse is
//     on the chain but the last block's;
//   - while warp 0 updates and factors the next diagonal block the others update
//     the rest, assemble the finished rows of the inverse and store what is done.
// Measured on one SM: 49,000 cycles (25 us) with load and stores; the form it
// replaces (block in L2, inverse on the chain, a panel per barrier) took 123 us
// where its code was cold and about 75 us warm.
#pragma once
#include "dev_common.cuh"
#include "dev_chol32.cuh"

namespace db2 {

constexpr int P128_SP = 132;                              // pitch of the block's columns (= 4 mod 16)
constexpr int P128_DP = 36;                               // pitch of the 32x32 inverses (= 4 mod 16)
constexpr int P128_S = 128 * P128_SP;                     // the block; W's off-diagonal blocks in its upper part
constexpr int P128_D = 4 * 32 * P128_DP;                  // inverses of the 32x32 diagonal blocks, row-major
constexpr int P128_LB = 1024 + 32;                        // blocked copy of the current 32x32 factor, 1/diagonal
constexpr int P128_DOUBLES = P128_S + P128_D + P128_LB;   // shared scratch in doubles

// 1 / sqrt(x) without a branch, x within the range the caller checks: the
// hardware's approximation and two Newton steps y += y (1/2 - x/2 y^2).
__device__ __forceinline__ double rsqrt_newton(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = 0.5 * x;
    y = fma(y, fma(-h * y, y, 0.5), y);
    y = fma(y, fma(-h * y, y, 0.5), y);
    return y;
}

// Columns J0 .. J0+15 of the 32x32 factorization (frame: d[k] = A(i, j + k) at
// column j); LIVE columns of the frame are kept up to date.
template <int LIVE>
__device__ __forceinline__ void chol32_half(double (&d)[32], int J0, int lane, double &dg, double &lp, double &piv,
                                            double &rdiag, bool &ok, double *Sd, int sp, double *Lb)
{
#pragma unroll
    for (int jj = 0; jj < 16; ++jj) {
        const int j = J0 + jj;
        // what the next pivot needs from lane j + 1, before the pivot's root is known
        const double dn = __shfl_sync(0xffffffffu, dg, j + 1);       // its diagonal entry
        const double an = __shfl_sync(0xffffffffu, d[0], j + 1);     // A(j+1, j)
        ok = ok && piv > 1e-280 && piv < 1e280;
        const double r = rsqrt_newton(piv);
        // column j - 1 applied to the columns beyond j
        if (j > 0) {
            // (16-byte pairs where row j + k is even)
            const double *Lp = Sd + (j - 1) * sp + j;
            if (jj & 1) {
#pragma unroll
                for (int k = 1; k < LIVE; k += 2) {
                    const double2 v = *reinterpret_cast<const double2 *>(Lp + k);
                    d[k] = fma(-lp, v.x, d[k]);
                    if (k + 1 < LIVE) d[k + 1] = fma(-lp, v.y, d[k + 1]);
                }
            } else {
                d[1] = fma(-lp, Lp[1], d[1]);
#pragma unroll
                for (int k = 2; k < LIVE; k += 2) {
                    const double2 v = *reinterpret_cast<const double2 *>(Lp + k);
                    d[k] = fma(-lp, v.x, d[k]);
                    if (k + 1 < LIVE) d[k + 1] = fma(-lp, v.y, d[k + 1]);
                }
            }
        }
        const double ln = an * r;                                     // L(j+1, j)
        const double pn = fma(-ln, ln, dn);
        double l = d[0] * r;
        const double s = fma(fma(-l, l, piv), 0.5 * r, l);            // lane j: sqrt, corrected
        dg = fma(-l, l, dg);
        const double d0 = fma(-l, ln, d[1]);
        if (lane == j) {
            l = s;
            rdiag = r;
        }
        if (lane >= j) Sd[j * sp + lane] = l;
        Lb[(j >> 2) * 128 + lane * 4 + (j & 3)] = lane >= j ? l : 0.0;
        __syncwarp();
        lp = l;
        piv = pn;
#pragma unroll
        for (int k = 1; k < LIVE - 1; ++k) d[k] = d[k + 1];
        d[0] = d0;
    }
}

// Cholesky factor of the 32x32 block at Sd (column c, row r at c * sp + r) in
// place by one warp, lane i owning row i.  Also the blocked copy Lb
// ([8][32][4]) and rd[c] = 1 / L(c,c).  Returns false when a pivot leaves the
// range in which the branch-free root is good (or is not positive): the block
// is then spoilt below the diagonal.
__device__ __forceinline__ bool chol32_col(double (&d)[32], int lane, double *Sd, int sp, double *Lb, double *rd)
{
    double dg = 0.0, lp = 0.0, rdiag = 0.0;
#pragma unroll
    for (int c = 0; c < 32; ++c)
        if (lane == c) dg = d[c];
    double piv = __shfl_sync(0xffffffffu, dg, 0);
    bool ok = true;
    chol32_half<32>(d, 0, lane, dg, lp, piv, rdiag, ok, Sd, sp, Lb);
    chol32_half<16>(d, 16, lane, dg, lp, piv, rdiag, ok, Sd, sp, Lb);
    rd[lane] = rdiag;
    __syncwarp();
    return ok;
}

// Solve L x = b for one right-hand side per lane (b[c], c = 0..31), L in the
// blocked copy Lb and rd[c] = 1 / L(c,c): steps of four columns in a rotating
// frame, out(c, x) receives x_c.
template <class Out>
__device__ __forceinline__ void sweep32(const double *Lb, const double *rd, double (&b)[32], Out out)
{
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        const double *Lk = Lb + (j >> 2) * 128;
        double r4[4];
        c32_load4(rd + j, r4);
        const double l10 = Lk[(j + 1) * 4], l20 = Lk[(j + 2) * 4], l21 = Lk[(j + 2) * 4 + 1];
        const double l30 = Lk[(j + 3) * 4], l31 = Lk[(j + 3) * 4 + 1], l32 = Lk[(j + 3) * 4 + 2];
        double x[4];
        x[0] = b[0] * r4[0];
        x[1] = (b[1] - l10 * x[0]) * r4[1];
        b[2] -= l20 * x[0];
        b[3] -= l30 * x[0];
        x[2] = (b[2] - l21 * x[1]) * r4[2];
        b[3] -= l31 * x[1];
        x[3] = (b[3] - l32 * x[2]) * r4[3];
#pragma unroll
        for (int r = 0; r < 4; ++r) out(j + r, x[r]);
#pragma unroll
        for (int c = 4; c < 32; ++c) {
            if (j + c < 32) {
                double v[4];
                c32_load4(Lk + (j + c) * 4, v);
                b[c] -= v[0] * x[0];
                b[c] -= v[1] * x[1];
                b[c] -= v[2] * x[2];
                b[c] -= v[3] * x[3];
            }
        }
#pragma unroll
        for (int q = 0; q < 28; ++q) b[q] = b[q + 4];
    }
}

// acc (MI*16 x NI*8 fragments of one warp) += (-) A B over one 32-deep block:
// A(m, k) at Ap[k * ak + m * am], B(k, n) at Bp[k * bk + n * bn].
template <int MI, int NI>
__device__ __forceinline__ void mma32(double (&acc)[MI][NI][4], const double *Ap, int ak, int am, const double *Bp,
                                      int bk, int bn, bool neg, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int kk = 0; kk < 32; kk += 4) {
        double af[MI][2], bf[NI];
#pragma unroll
        for (int mi = 0; mi < MI; ++mi) {
            af[mi][0] = Ap[(kk + t) * ak + (mi * 16 + g) * am];
            af[mi][1] = Ap[(kk + t) * ak + (mi * 16 + g + 8) * am];
            if (neg) {
                af[mi][0] = -af[mi][0];
                af[mi][1] = -af[mi][1];
            }
        }
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) bf[ni] = Bp[(kk + t) * bk + (ni * 8 + g) * bn];
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < NI; ++ni) dmma_16x8x4(acc[mi][ni], af[mi][0], af[mi][1], bf[ni]);
    }
}
// fragments <-> memory, element (r, c) at p[r * rs + c * cs]
template <int MI, int NI>
__device__ __forceinline__ void frag_load(double (&acc)[MI][NI][4], const double *p, int rs, int cs, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                acc[mi][ni][q] = p[(mi * 16 + g + ((q & 2) ? 8 : 0)) * rs + (ni * 8 + 2 * t + (q & 1)) * cs];
}
template <int MI, int NI>
__device__ __forceinline__ void frag_store(const double (&acc)[MI][NI][4], double *p, int rs, int cs, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                p[(mi * 16 + g + ((q & 2) ? 8 : 0)) * rs + (ni * 8 + 2 * t + (q & 1)) * cs] = acc[mi][ni][q];
}
template <int MI, int NI>
__device__ __forceinline__ void frag_zero(double (&acc)[MI][NI][4])
{
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;
}

__device__ __forceinline__ void named_bar_arrive(int id, int nthreads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Assembly of W's blocks below the diagonal, in units of a column half h (16
// columns) of block (i, c):
//   G_ic += sum_{l=l0}^{l1-1} L_il W_lc (W_cc = D_c), kept at the block's place,
//   then, when dg is set, W_ic = -D_i G_ic, to its place and to global memory.
// P128_UNITS[phase][warp] lists up to two units per warp; phase 2 j is the one
// in which warp 0 factors diagonal block j, 2 j + 1 the sweeps of that step,
// 8 the last products.  Row i needs D_i (phase 2 i + 1) and the rows above.
constexpr uint16_t p128_unit(int i, int c, int h, int l0, int l1, int first, int dg)
{
    return (uint16_t)(1 | i << 1 | c << 3 | h << 5 | l0 << 6 | l1 << 8 | first << 10 | dg << 11);
}
static __constant__ uint16_t P128_UNITS[5][8][2] = {
    // phase 4: row 1
    {{0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {p128_unit(1, 0, 0, 0, 1, 1, 1), 0}, {p128_unit(1, 0, 1, 0, 1, 1, 1), 0}},
    {{0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
    // phase 6: row 2, and the sums of row 3 over rows 0 and 1
    {{0, 0},
     {p128_unit(2, 0, 0, 0, 2, 1, 1), p128_unit(3, 1, 0, 1, 2, 1, 0)},
     {p128_unit(2, 0, 1, 0, 2, 1, 1), p128_unit(3, 1, 1, 1, 2, 1, 0)},
     {p128_unit(2, 1, 0, 1, 2, 1, 1), 0},
     {0, 0},
     {p128_unit(3, 0, 0, 0, 2, 1, 0), 0},
     {p128_unit(3, 0, 1, 0, 2, 1, 0), 0},
     {p128_unit(2, 1, 1, 1, 2, 1, 1), 0}},
    // phase 7: the terms of row 3 with row 2
    {{0, 0},
     {p128_unit(3, 0, 0, 2, 3, 0, 0), 0},
     {p128_unit(3, 0, 1, 2, 3, 0, 0), 0},
     {p128_unit(3, 1, 0, 2, 3, 0, 0), 0},
     {0, 0},
     {p128_unit(3, 1, 1, 2, 3, 0, 0), 0},
     {p128_unit(3, 2, 0, 2, 3, 1, 0), 0},
     {p128_unit(3, 2, 1, 2, 3, 1, 0), 0}},
    // phase 8: row 3
    {{p128_unit(3, 0, 0, 0, 0, 0, 1), 0}, {p128_unit(3, 0, 1, 0, 0, 0, 1), 0}, {p128_unit(3, 1, 0, 0, 0, 0, 1), 0},
     {p128_unit(3, 1, 1, 0, 0, 0, 1), 0}, {p128_unit(3, 2, 0, 0, 0, 0, 1), 0}, {p128_unit(3, 2, 1, 0, 0, 0, 1), 0},
     {0, 0}, {0, 0}}};

__device__ __forceinline__ void p128_run_unit(uint32_t u, double *S, const double *D, double *Wb, int lane)
{
    constexpr int SP = P128_SP, DP = P128_DP;
    const int i = (u >> 1) & 3, c = (u >> 3) & 3, h = (u >> 5) & 1, l0 = (u >> 6) & 3, l1 = (u >> 8) & 3;
    double acc[2][2][4];
    double *Wp = S + i * 32 * SP + c * 32 + 16 * h;
    if ((u >> 10) & 1) frag_zero(acc);
    else frag_load(acc, Wp, SP, 1, lane);
#pragma unroll 1
    for (int l = l0; l < l1; ++l) {
        const double *Bp = (l == c) ? D + l * 32 * DP : S + l * 32 * SP + c * 32;
        mma32(acc, S + l * 32 * SP + i * 32, SP, 1, Bp + 16 * h, l == c ? DP : SP, 1, false, lane);
    }
    frag_store(acc, Wp, SP, 1, lane);
    __syncwarp();
    if ((u >> 11) & 1) {
        frag_zero(acc);
        mma32(acc, D + i * 32 * DP, 1, DP, Wp, SP, 1, true, lane);
        __syncwarp();
        frag_store(acc, Wp, SP, 1, lane);
        frag_store(acc, Wb + (c * 32 + 16 * h) * 128 + i * 32, 1, 128, lane);
    }
}

// diagonal block i of W to global memory, coalesced by rows (zero above the diagonal)
__device__ __forceinline__ void p128_put_d(const double *D, int i, double *Wb, int lane)
{
    const double *Di = D + (i * 32 + lane) * P128_DP;
    double *o = Wb + (i * 32) * 128 + i * 32 + lane;
#pragma unroll 8
    for (int c = 0; c < 32; ++c) o[c * 128] = c <= lane ? Di[c] : 0.0;
}
// columns 32 jj + w, + nw, ... of the factor to T
__device__ __forceinline__ void p128_put_l(const double *S, int jj, double *T, int ld, int w, int nw, int lane)
{
#pragma unroll 2
    for (int c = 32 * jj + w; c < 32 * jj + 32; c += nw)
#pragma unroll
        for (int r0 = 0; r0 < 128; r0 += 32)
            if (r0 + lane >= c) T[(int64_t)c * ld + r0 + lane] = S[c * P128_SP + r0 + lane];
}

// The 32x32 diagonal block j again, from the stored matrix (its block columns
// from j on are still untouched at T) and the rows solved so far, by the
// general routine: any pivot the full square root takes, and the exact failing
// column.  Returns that column of the block, or -1.
static __device__ __noinline__ int p128_diag_general(double *S, const double *T, int ld, int j, double *Lb, double *rd,
                                              int lane)
{
    constexpr int SP = P128_SP;
    const int p0 = 32 * j;
    double *Sd = S + p0 * SP + p0;
    {
        double acc[2][4][4];
        frag_load(acc, T + (int64_t)p0 * ld + p0, 1, ld, lane);
        for (int l = 0; l < j; ++l) mma32(acc, S + l * 32 * SP + p0, SP, 1, S + l * 32 * SP + p0, SP, 1, true, lane);
        __syncwarp();
        frag_store(acc, Sd, 1, SP, lane);
        __syncwarp();
    }
    double d[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) d[c] = (c <= lane) ? Sd[c * SP + lane] : 0.0;
    double rdiag = 0.0;
    const int f = chol32_blk<double>(d, lane, rdiag, Lb);
    rd[lane] = rdiag;
    __syncwarp();
#pragma unroll 1
    for (int c = 0; c <= lane; ++c) Sd[c * SP + lane] = Lb[(c >> 2) * 128 + lane * 4 + (c & 3)];
    __syncwarp();
    return f;
}

// Factor the block in S (column c, row r at S[c * P128_SP + r], lower part)
// and form W = L^-1, by the 256 threads of barrier `bar` (bar + 1 is used
// inside); S must be complete (the caller's barrier) and T is the block it was
// loaded from, leading dimension ld.  The factor's lower triangle goes to T and
// W (zero above the diagonal) to the 128x128 block Wb; S keeps the factor, with
// W's off-diagonal 32x32 blocks transposed in its upper part (W(r, c) at
// S[r * P128_SP + c]) and the diagonal ones row-major behind it (P128_S).
// Returns the failing column, the same in every thread, or -1; *fail is a
// shared word.
__device__ __forceinline__ int potrf128_smem(double *S, int *fail, double *T, int ld, double *Wb, int warp, int lane,
                                             int bar)
{
    constexpr int SP = P128_SP, DP = P128_DP;
    double *D = S + P128_S, *Lb = D + P128_D, *rd = Lb + 1024;
    const int w = warp < 4 ? warp - 1 : warp - 2;       // 0..5 for the helpers
    const bool helper = warp != 0 && warp != 4;         // warp 4 shares warp 0's sub-partition
#pragma unroll 1
    for (int ph = 0; ph < 9; ++ph) {
        const int j = ph >> 1, p0 = j * 32;
        int put_jj = -1, put_w = 0, put_n = 1, put_d = -1;
        if (ph & 1) {
            // rows below (one 32-row block per warp) and the inverse of the diagonal block
            const int nrow = 3 - j;
            if (warp <= nrow) {
                const bool inv = warp == nrow;
                double b[32];
                double *Xp = S + p0 * SP + (j + 1 + warp) * 32 + lane;
#pragma unroll
                for (int c = 0; c < 32; ++c) b[c] = inv ? (c == lane ? 1.0 : 0.0) : Xp[c * SP];
                double *o = inv ? D + j * 32 * DP + lane : Xp;
                const int os = inv ? DP : SP;
                sweep32(Lb, rd, b, [&](int c, double x) { o[c * os] = x; });
            }
        } else if (j < 4) {
            double *Sd = S + p0 * SP + p0;
            if (j > 0 && warp < 3) {
                // the next diagonal block, one lower 16x16 quarter per warp
                const int qr = warp == 0 ? 0 : 16, qc = warp == 2 ? 16 : 0;
                double acc[1][2][4];
                double *C = Sd + qc * SP + qr;
                frag_load(acc, C, 1, SP, lane);
                const double *X = S + (p0 - 32) * SP + p0;
                mma32(acc, X + qr, SP, 1, X + qc, SP, 1, true, lane);
                frag_store(acc, C, 1, SP, lane);
                if (warp > 0) named_bar_arrive(bar + 1, 96);
            }
            if (warp == 0) {
                if (j > 0) named_bar_sync(bar + 1, 96);
                double d[32];
#pragma unroll
                for (int c = 0; c < 32; ++c) d[c] = (c <= lane) ? Sd[c * SP + lane] : 0.0;
                int f = -1;
                if (!chol32_col(d, lane, Sd, SP, Lb, rd)) f = p128_diag_general(S, T, ld, j, Lb, rd, lane);
                if (lane == 0) *fail = f >= 0 ? p0 + f : -1;
            } else if (helper && j > 0) {
                // trailing blocks (bi, bk), j <= bk <= bi, but (j, j)
                const int q = 4 - j, nit = q * (q + 1) / 2 - 1;
                const double *X = S + (p0 - 32) * SP;
#pragma unroll 1
                for (int it = w; it < nit; it += 6) {
                    int bk = 0, rem = it + 1;
                    while (rem >= q - bk) {
                        rem -= q - bk;
                        ++bk;
                    }
                    const int bi = j + bk + rem;
                    bk += j;
                    double acc[2][4][4];
                    double *C = S + bk * 32 * SP + bi * 32;
                    frag_load(acc, C, 1, SP, lane);
                    mma32(acc, X + bi * 32, SP, 1, X + bk * 32, SP, 1, true, lane);
                    frag_store(acc, C, 1, SP, lane);
                }
                put_jj = j - 1;
                put_w = 5 - w;
                put_n = 6;
                if (w == 3) put_d = j - 1;
                if (j == 1 && w == 5) {
                    // W is zero above its diagonal blocks
#pragma unroll 1
                    for (int c = 32; c < 128; ++c)
#pragma unroll
                        for (int r0 = 0; r0 < 96; r0 += 32)
                            if (r0 + 32 <= (c & ~31)) Wb[c * 128 + r0 + lane] = 0.0;
                }
            }
        } else {
            if (warp == 7) put_jj = 3;
            if (warp == 6) put_d = 3;
        }
        if (ph >= 4) {
#pragma unroll 1
            for (int q = 0; q < 2; ++q) {
                const uint32_t u = P128_UNITS[ph - 4][warp][q];
                if (u) p128_run_unit(u, S, D, Wb, lane);
            }
        }
        if (put_jj >= 0) p128_put_l(S, put_jj, T, ld, put_w, put_n, lane);
        if (put_d >= 0) p128_put_d(D, put_d, Wb, lane);
        named_bar_sync(bar, 256);
        // read where no warp can be writing it: the next write follows the next barrier
        if (!(ph & 1) && *fail >= 0) return *fail;
    }
    return -1;
}

// Load the lower 32-blocks (whole: all) of the 128x128 block at T (leading
// dimension ld), 256 threads.
__device__ __forceinline__ void p128_load(double *S, const double *T, int ld, bool whole, int tid)
{
    const int r = (tid & 63) * 2, c0 = tid >> 6;
#pragma unroll 1
    for (int cc = 0; cc < 128; cc += 64) {
        double2 v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int c = cc + c0 + 4 * q;
            if (whole || r + 2 > (c & ~31)) v[q] = __ldcg(reinterpret_cast<const double2 *>(T + (int64_t)c * ld + r));
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int c = cc + c0 + 4 * q;
            if (whole || r + 2 > (c & ~31)) *reinterpret_cast<double2 *>(S + c * P128_SP + r) = v[q];
        }
    }
}

// One 128x128x128 product inside a diagonal tile, 16 rows per warp, all 128
// columns (64 accumulators a thread), A from L2 and B from S:
//   strip   C = A W^T with the inverse as potrf128_smem left it in S (K block
//           kb reaches the column blocks >= kb only); C may be A;
//   update  C -= A X^T with X whole in S (column k at S[k * SP]); diag: only
//           the lower triangle of C.
__device__ __forceinline__ void p128_rows(bool strip, bool diag, const double *S, const double *A, double *C, int ld,
                                          int warp, int lane)
{
    constexpr int SP = P128_SP, DP = P128_DP;
    const int g = lane >> 2, t = lane & 3;
    double acc[16][4];
#pragma unroll
    for (int ni = 0; ni < 16; ++ni)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[ni][q] = 0.0;
    const double *Ar = A + warp * 16 + g;
    const int last = diag ? warp >> 1 : 3;                       // column blocks beyond it are above the diagonal
#pragma unroll 1
    for (int kb = 0; kb < 4; ++kb) {
        double a[16];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            a[2 * q] = __ldcg(Ar + (int64_t)(32 * kb + 4 * q + t) * ld);
            a[2 * q + 1] = __ldcg(Ar + (int64_t)(32 * kb + 4 * q + t) * ld + 8);
        }
#pragma unroll
        for (int ng = 0; ng < 4; ++ng) {
            if (strip ? ng >= kb : ng <= last) {
                const double *Bp = strip ? (ng == kb ? S + P128_S + kb * 32 * DP : S + ng * 32 * SP + kb * 32)
                                         : S + kb * 32 * SP + ng * 32;
                const int bn = strip ? (ng == kb ? DP : SP) : 1, bk = strip ? 1 : SP;
                const double *Bl = Bp + g * bn + t * bk;
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int n4 = 0; n4 < 4; ++n4)
                        dmma_16x8x4(acc[4 * ng + n4], a[2 * q], a[2 * q + 1], Bl[(8 * n4) * bn + 4 * q * bk]);
            }
        }
    }
    double *Cr = C + warp * 16 + g;
#pragma unroll
    for (int ng = 0; ng < 4; ++ng) {
        if (ng > last) break;
        double old[16];
        if (!strip) {
#pragma unroll
            for (int e = 0; e < 16; ++e)
                old[e] = __ldcg(Cr + (int64_t)(32 * ng + 8 * (e >> 2) + 2 * t + (e & 1)) * ld + ((e & 2) ? 8 : 0));
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int c = 32 * ng + 8 * (e >> 2) + 2 * t + (e & 1), r = (e & 2) ? 8 : 0;
            const double v = acc[4 * ng + (e >> 2)][e & 3];
            if (!diag || warp * 16 + g + r >= c) Cr[(int64_t)c * ld + r] = strip ? v : old[e] - v;
        }
    }
}

}  // namespace db2
