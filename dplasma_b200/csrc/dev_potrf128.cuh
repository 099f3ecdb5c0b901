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
//   - every panel's products are summed by themselves and subtracted once:
//     accumulated onto the block, each would be rounded at the block's size (a
//     factor of 256 columns 2.1e-16 off instead of 1.2e-16, diagonally dominant);
//   - while warp 0 updates and factors the next diagonal block the others update
//     the rest, assemble the finished rows of the inverse and store what is done.
// Measured in place: 35 us with load and stores; the form it replaces (block in
// L2, inverse on the chain, a panel per barrier) took 123 us where its code was
// cold and about 75 us warm.
#pragma once
#include "dev_common.cuh"
#include "dev_chol32.cuh"
#include "dev_frag.cuh"

namespace db2 {

constexpr int P128_SP = 132;                              // pitch of the block's columns (= 4 mod 16)
constexpr int P128_DP = 36;                               // pitch of the 32x32 inverses (= 4 mod 16)
constexpr int P128_S = 128 * P128_SP;                     // the block; W's off-diagonal blocks in its upper part
constexpr int P128_D = 4 * 32 * P128_DP;                  // inverses of the 32x32 diagonal blocks, row-major
constexpr int P128_LB = C32_LB;                           // blocked copy of the current 32x32 factor, 1/diagonal
constexpr int P128_DOUBLES = P128_S + P128_D + P128_LB;   // shared scratch in doubles

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
__host__ __device__ constexpr uint16_t p128_unit(int i, int c, int h, int l0, int l1, int first, int dg)
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
        // panel by panel, as the updates of potrf128_smem
        double acc[2][4][4];
        frag_load(acc, T + (int64_t)p0 * ld + p0, 1, ld, lane);
        __syncwarp();
        frag_store(acc, Sd, 1, SP, lane);
        for (int l = 0; l < j; ++l) {
            frag_zero(acc);
            mma32(acc, S + l * 32 * SP + p0, SP, 1, S + l * 32 * SP + p0, SP, 1, false, lane);
            frag_sub(acc, Sd, 1, SP, lane);
        }
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
// inside); the first 32 columns of S must be there (the caller's barrier), the
// threads' copies of the others may be in flight; T is the block it was loaded
// from, leading dimension ld.  The factor's lower triangle goes to T and
// W (zero above the diagonal) to the 128x128 block Wb; S keeps the factor, with
// W's off-diagonal 32x32 blocks transposed in its upper part (W(r, c) at
// S[r * P128_SP + c]) and the diagonal ones row-major behind it (P128_S).
// Returns the failing column, the same in every thread, or -1; *fail is a
// shared word.  VEC: as chol32_col.
template <bool VEC>
__device__ __forceinline__ int potrf128_smem(double *S, int *fail, double *T, int ld, double *Wb, int warp, int lane,
                                             int bar)
{
    constexpr int SP = P128_SP, DP = P128_DP;
    double *D = S + P128_S, *Lb = D + P128_D, *rd = Lb + C32_RD;
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
                double *Xp = S + p0 * SP + (inv ? 0 : (j + 1 + warp) * 32) + lane;
                double *o = inv ? D + j * 32 * DP + lane : Xp;
                const int os = inv ? DP : SP;
                sweep32_sums<double>(Lb, rd, [&](int c) { return inv ? (c == lane ? 1.0 : 0.0) : Xp[c * SP]; },
                                     [&](int c, double x) { o[c * os] = x; });
            }
        } else if (j < 4) {
            double *Sd = S + p0 * SP + p0;
            if (j > 0 && warp < 3) {
                // the next diagonal block, one lower 16x16 quarter per warp
                const int qr = warp == 0 ? 0 : 16, qc = warp == 2 ? 16 : 0;
                double old[1][2][4], acc[1][2][4];
                double *C = Sd + qc * SP + qr;
                frag_load(old, C, 1, SP, lane);
                const double *X = S + (p0 - 32) * SP + p0;
                frag_zero(acc);
                mma32(acc, X + qr, SP, 1, X + qc, SP, 1, false, lane);
#pragma unroll
                for (int e = 0; e < 8; ++e) old[0][e >> 2][e & 3] -= acc[0][e >> 2][e & 3];
                frag_store(old, C, 1, SP, lane);
                if (warp > 0) named_bar_arrive(bar + 1, 96);
            }
            if (warp == 0) {
                if (j > 0) named_bar_sync(bar + 1, 96);
                double d[32];
#pragma unroll
                for (int c = 0; c < 32; ++c) d[c] = (c <= lane) ? Sd[c * SP + lane] : 0.0;
                int f = -1;
                if (!chol32_col<double, VEC>(d, lane, Sd, SP, Lb, rd)) f = p128_diag_general(S, T, ld, j, Lb, rd, lane);
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
                    frag_zero(acc);
                    mma32(acc, X + bi * 32, SP, 1, X + bk * 32, SP, 1, false, lane);
                    frag_sub(acc, S + bk * 32 * SP + bi * 32, 1, SP, lane);
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
        if (ph == 0) cp_async_wait(0);
        if (put_jj >= 0) p128_put_l(S, put_jj, T, ld, put_w, put_n, lane);
        if (put_d >= 0) p128_put_d(D, put_d, Wb, lane);
        named_bar_sync(bar, 256);
        // read where no warp can be writing it: the next write follows the next barrier
        if (!(ph & 1) && *fail >= 0) return *fail;
    }
    return -1;
}

// Inverse of the lower triangular block in S (unit: diagonal taken as 1) to
// the 128x128 block Wb, zero above the diagonal, by the 256 threads of barrier
// `bar`; LB4 is scratch of 4 P128_LB doubles, S keeps the layout above.
__device__ __forceinline__ void p128_invert(double *S, double *LB4, int unit, double *Wb, int warp, int lane, int bar)
{
    constexpr int SP = P128_SP, DP = P128_DP;
    double *D = S + P128_S;
    if (warp < 4) {
        // the four diagonal blocks: blocked copy, then the unit vectors
        double *Lb = LB4 + warp * P128_LB, *rd = Lb + C32_RD;
        const double *Sd = S + warp * 32 * SP + warp * 32 + lane;
#pragma unroll 8
        for (int c = 0; c < 32; ++c) Lb[(c >> 2) * 128 + lane * 4 + (c & 3)] = c <= lane ? Sd[c * SP] : 0.0;
        rd[lane] = unit ? 1.0 : 1.0 / Sd[lane * SP];
        __syncwarp();
        double *o = D + warp * 32 * DP + lane;
        sweep32_sums<double>(Lb, rd, [&](int c) { return c == lane ? 1.0 : 0.0; },
                             [&](int c, double x) { o[c * DP] = x; });
    } else {
        // W is zero above its diagonal blocks
#pragma unroll 1
        for (int c = 32 + (warp - 4); c < 128; c += 4)
#pragma unroll
            for (int r0 = 0; r0 < 96; r0 += 32)
                if (r0 + 32 <= (c & ~31)) Wb[c * 128 + r0 + lane] = 0.0;
    }
    named_bar_sync(bar, 256);
    // block row i: W_ic = -D_i sum_{l=c}^{i-1} L_il W_lc, a column half per warp
#pragma unroll 1
    for (int i = 1; i < 4; ++i) {
        if (warp < 2 * i) p128_run_unit(p128_unit(i, warp >> 1, warp & 1, warp >> 1, i, 1, 1), S, D, Wb, lane);
        if (warp >= 6 && i < 3) p128_put_d(D, 2 * (i - 1) + (warp - 6), Wb, lane);
        named_bar_sync(bar, 256);
    }
}
constexpr int P128_INV_DOUBLES = P128_S + P128_D + 4 * P128_LB;

// Load the lower 32-blocks (whole: all) of the 128x128 block at T (leading
// dimension ld), 256 threads: two groups of asynchronous copies, the first 32
// columns and the rest, which the caller waits for (through registers, in two
// rounds, the chain waited 6,400 cycles for the whole block; 38 -> 35 us per
// POTRF).
__device__ __forceinline__ void p128_load(double *S, const double *T, int ld, bool whole, int tid)
{
    const int r = (tid & 63) * 2;
#pragma unroll 4
    for (int c = tid >> 6; c < 128; c += 4) {
        if (whole || r + 2 > (c & ~31)) cp_async16(S + c * P128_SP + r, T + (int64_t)c * ld + r);
        if ((c & ~3) == 28 || (c & ~3) == 124) cp_async_commit();
    }
}

// A = A L^-T in place for 128 rows beside a factored block, 16 rows per warp, by
// substitution over the four 32-wide blocks of L as potrf128_smem left it in S (X_p =
// (A_p - sum_{q<p} X_q L_pq^T) D_p^T).  A product with the 128-wide inverse is faster
// (p128_rows; a 256-wide tile takes 132 us with it, 142 with this), but its error grows
// with the condition of 128 columns; the FP64 tiles of the task pools and the
// allocation-free entry take this one.  X goes through L2 between the steps; only this
// warp touches its rows.
__device__ __forceinline__ void p128_solve_rows(const double *S, double *A, int ld, int warp, int lane)
{
    constexpr int SP = P128_SP, DP = P128_DP;
    const int g = lane >> 2, t = lane & 3;
    double *Ar = A + warp * 16 + g;
#pragma unroll 1
    for (int p = 0; p < 4; ++p) {
        double acc[4][4], a[8][2];
        double *Ap = Ar + (int64_t)(32 * p) * ld;
        auto at = [&](int n4, int e) { return Ap + (int64_t)(8 * n4 + 2 * t + (e & 1)) * ld + ((e & 2) ? 8 : 0); };
        auto operand = [&](int b) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) a[q][h] = __ldcg(Ar + (int64_t)(32 * b + 4 * q + t) * ld + 8 * h);
        };
#pragma unroll
        for (int n4 = 0; n4 < 4; ++n4)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n4][e] = 0.0;
#pragma unroll 1
        for (int b = 0; b < p; ++b) {
            operand(b);
            const double *Bl = S + (32 * b + t) * SP + 32 * p + g;
#pragma unroll
            for (int q = 0; q < 8; ++q)
#pragma unroll
                for (int n4 = 0; n4 < 4; ++n4) dmma_16x8x4(acc[n4], a[q][0], a[q][1], Bl[4 * q * SP + 8 * n4]);
        }
        if (p > 0) {
#pragma unroll
            for (int n4 = 0; n4 < 4; ++n4)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[n4][e] = __ldcg(at(n4, e)) - acc[n4][e];
#pragma unroll
            for (int n4 = 0; n4 < 4; ++n4)
#pragma unroll
                for (int e = 0; e < 4; ++e) *at(n4, e) = acc[n4][e];
            __syncwarp();
        }
        operand(p);
        __syncwarp();
        const double *Dl = S + P128_S + (32 * p + g) * DP + t;
#pragma unroll
        for (int n4 = 0; n4 < 4; ++n4) {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n4][e] = 0.0;
#pragma unroll
            for (int q = 0; q < 2 * n4 + 2; ++q)             // D is lower triangular
                dmma_16x8x4(acc[n4], a[q][0], a[q][1], Dl[8 * n4 * DP + 4 * q]);
#pragma unroll
            for (int e = 0; e < 4; ++e) *at(n4, e) = acc[n4][e];
        }
        __syncwarp();
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
