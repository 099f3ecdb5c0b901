// batched.cu -- many independent small SPD systems in one persistent launch:
// Cholesky factorization, solve and log-determinant of each, FP64 or FP32.
//
// There is no batched interface in dplasma; each problem follows the
// reference's own single-tile path (the POTRF / TRSM / SYRK task bodies of
// src/zpotrf_L.jdf applied to one matrix) with the same INFO convention.
// CTAs take problems from an atomic work queue in decreasing order of n
// (longest first), so one launch balances sizes from 1 to 512.  A problem is
// factored right-looking in 32-column panels:
//   1. warp 0 factors the 32x32 diagonal block (chol32_col);
//   2. the rows below are solved by substitution, one row per lane (sweep32), to
//      global memory and to a shared panel; the right-hand sides are one more set
//      of rows of the same solve, the inverse of the diagonal block (for the
//      backward solve) one more sweep on the unit vectors, so neither is on the
//      chain;
//   3. the lower triangle of the trailing matrix is updated from the shared
//      panel in 32x32 tiles, one warp per tile (FP64 tensor cores; FP32 on
//      the FMA pipes), the next diagonal block first so that warp 0 factors
//      it while the others finish the update.
// What bounds a problem is the latency of these steps, so several problems
// share an SM where there are enough of them (bt_choose).  The solve ends with the backward sweep on the
// factor in 32-row blocks; the log-determinant is 2 * sum log L(i,i).
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <functional>
#include <numeric>
#include <vector>

#include "dev_common.cuh"
#include "internal.h"
#include "dev_chol32.cuh"

namespace db2 {

constexpr int BT_NB = 32;
constexpr int BT_DP = 33;          // pitch of a diagonal block in shared memory
constexpr int BT_NMAX = 4096;      // largest n of one problem
constexpr int BT_MAXRHS = 16;      // right-hand sides per problem

template <typename T>
struct BatchArgs {
    int batch;
    const int *n;
    const int *lda;
    T *const *A;
    T *const *B;          // may be null: factor only
    int nrhs;
    double *logdet;       // may be null
    int *info;            // per problem
    const int *order;     // problems by decreasing n
    int *ticket;
    T *dscr;              // per CTA (dstride): inverses of the 32x32 diagonal blocks of its current problem
    int64_t dstride;
    int prow;             // panel rows kept in shared memory
};

// Diagonal block j0 (jb <= 32 columns) of one problem by one warp: factor,
// write L back, accumulate log det; the blocked copy Lb and the reciprocal
// diagonal rd serve the sweeps.  in_sm: the block lies in Lb's place already
// (column c, row r at c * BT_DP + r; also in the matrix).  Returns the failing
// column within the block or -1.
template <typename T>
__device__ __forceinline__ int bt_diag(T *A, int lda, int j0, int jb, bool in_sm, T *Lb, T *rd, double &ld_acc, int lane)
{
    T d[32];
    // padding rows are the identity (a running pointer: 32 addresses would take the registers)
    auto load = [&](const T *p, int ld) {
        p += lane;
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            d[c] = (lane < jb && c < jb) ? ((c <= lane) ? *p : T(0)) : (c == lane ? T(1) : T(0));
            p += ld;
        }
    };
    T *Aj = A + (int64_t)j0 * lda + j0;
    if (in_sm) load(Lb, BT_DP);
    else load(Aj, lda);
    __syncwarp();
    int f = -1;
    if (!chol32_col<T>(d, lane, (T *)nullptr, 0, Lb, rd)) {
        // a pivot outside the fast root's range, or not positive
        load(Aj, lda);
        T rdiag = T(0);
        f = chol32_blk<T>(d, lane, rdiag, Lb);
        rd[lane] = rdiag;
        __syncwarp();
        if (f >= jb) f = -1;
        if (f >= 0) return f;
    }
    if (lane < jb) {
        T *p = Aj + lane;
#pragma unroll 8
        for (int c = 0; c < 32; ++c) {
            if (c <= lane && c < jb) *p = Lb[(c >> 2) * 128 + lane * 4 + (c & 3)];
            p += lda;
        }
        ld_acc -= 2.0 * log((double)rd[lane]);   // rd = 1 / L(i,i)
    }
    return -1;
}

// The next diagonal block (tile (0,0) of the trailing matrix) before it is
// factored, C -= P P^T in lower 16x16 quarters q = 0 (top), 1 (below), 2: to the
// matrix and to shared memory at Sd (pitch BT_DP).  The products are summed by
// themselves and subtracted once, here and in bt_tile: accumulated onto C, every
// product is rounded at the size of C (factors of 256 diagonally dominant FP64
// columns 2.5e-16 off instead of 1.0e-16, FP32 1.4e-7 instead of 5.4e-8).
__device__ __forceinline__ void bt_quarter(double *C, int lda, int m, const double *Pr, int sr, double *Sd, int q,
                                           int lane)
{
    const int g = lane >> 2, t = lane & 3;
    const int qr = q == 0 ? 0 : 16, qc = q == 2 ? 16 : 0;
    double old[2][4], acc[2][4];
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = qr + g + ((e & 2) ? 8 : 0), c = qc + ni * 8 + 2 * t + (e & 1);
            old[ni][e] = (r < m && c <= r) ? C[(int64_t)c * lda + r] : 0.0;
            acc[ni][e] = 0.0;
        }
#pragma unroll
    for (int kk = 0; kk < 32; kk += 4) {
        const double *pk = Pr + (int64_t)(kk + t) * sr + g;
        const double a0 = qr + g < m ? pk[qr] : 0.0, a1 = qr + g + 8 < m ? pk[qr + 8] : 0.0;
#pragma unroll
        for (int ni = 0; ni < 2; ++ni)
            dmma_16x8x4(acc[ni], a0, a1, qc + ni * 8 + g < m ? pk[qc + ni * 8] : 0.0);
    }
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = qr + g + ((e & 2) ? 8 : 0), c = qc + ni * 8 + 2 * t + (e & 1);
            const double v = old[ni][e] - acc[ni][e];
            Sd[c * BT_DP + r] = v;
            if (r < m && c <= r) C[(int64_t)c * lda + r] = v;
        }
}
__device__ __forceinline__ void bt_quarter(float *C, int lda, int m, const float *Pr, int sr, float *Sd, int q, int lane)
{
    // half the columns of a row per lane: quarter q has rows qr + (lane / 2), eight columns each
    const int qr = q == 0 ? 0 : 16, qc = (q == 2 ? 16 : 0) + 8 * (lane & 1), r = qr + (lane >> 1);
    float old[8], acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        old[j] = (r < m && qc + j <= r) ? C[(int64_t)(qc + j) * lda + r] : 0.f;
        acc[j] = 0.f;
    }
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
        const float pr = Pr[k * sr + r];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = fmaf(pr, Pr[k * sr + qc + j], acc[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float v = old[j] - acc[j];
        Sd[(qc + j) * BT_DP + r] = v;
        if (r < m && qc + j <= r) C[(int64_t)(qc + j) * lda + r] = v;
    }
}

// One 32x32 tile (rb, cb), rb >= cb, of the trailing update C -= P P^T by one
// warp; C is the trailing matrix (origin at A(o, o)), m its order, P the panel
// (rows beyond m zero) with k stride RP.  The C values are on their way while the
// products are formed.
// FULL: all 32 x 32 elements exist (below the diagonal block, inside m).  NI: 8-column
// groups of the tile formed at a time (two where the registers are limited).
template <bool FULL, int NI>
__device__ __forceinline__ void bt_tile_f64(double *A, int lda, int o, int m, const double *P, int RP, int rb, int cb,
                                            int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int n0 = 0; n0 < 32; n0 += 8 * NI) {
        double *C = A + (int64_t)(o + cb * 32 + n0 + 2 * t) * lda + o + rb * 32 + g;
        const int mr = m - rb * 32 - g, mc = m - cb * 32 - n0 - 2 * t, dd = rb == cb ? g - n0 - 2 * t : 1 << 20;
        // element (row 16 mi + 8 h, column 8 ni + e) of this thread
        auto in = [&](int r, int c) { return FULL || (r < mr && c < mc && r - c + dd >= 0); };
        double old[2][NI][4], acc[2][NI][4];
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) {
            const double *p0 = C + (int64_t)(ni * 8) * lda, *p1 = p0 + lda;
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = mi * 16 + ((q & 2) ? 8 : 0), c = ni * 8 + (q & 1);
                    old[mi][ni][q] = in(r, c) ? ((q & 1) ? p1 : p0)[r] : 0.0;
                    acc[mi][ni][q] = 0.0;
                }
        }
        const double *a0 = P + t * RP + rb * 32 + g, *b0 = P + t * RP + cb * 32 + n0 + g;
#pragma unroll
        for (int kk = 0; kk < 32; kk += 4) {
            double af[2][2], bf[NI];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
                af[mi][0] = a0[mi * 16];
                af[mi][1] = a0[mi * 16 + 8];
            }
#pragma unroll
            for (int ni = 0; ni < NI; ++ni) bf[ni] = b0[ni * 8];
            a0 += 4 * RP;
            b0 += 4 * RP;
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < NI; ++ni) dmma_16x8x4(acc[mi][ni], af[mi][0], af[mi][1], bf[ni]);
        }
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) {
            double *p0 = C + (int64_t)(ni * 8) * lda, *p1 = p0 + lda;
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = mi * 16 + ((q & 2) ? 8 : 0), c = ni * 8 + (q & 1);
                    if (in(r, c)) ((q & 1) ? p1 : p0)[r] = old[mi][ni][q] - acc[mi][ni][q];
                }
        }
    }
}
template <int NI>
__device__ __forceinline__ void bt_tile(double *A, int lda, int o, int m, const double *P, int RP, int rb, int cb,
                                        int lane)
{
    if (rb > cb && rb * 32 + 32 <= m) bt_tile_f64<true, NI>(A, lda, o, m, P, RP, rb, cb, lane);
    else bt_tile_f64<false, NI>(A, lda, o, m, P, RP, rb, cb, lane);
}
// FP32: lane = row of the tile, 8 NI columns per lane at a time (the panel values
// of the columns are broadcasts)
template <int NI>
__device__ __forceinline__ void bt_tile(float *A, int lda, int o, int m, const float *P, int RP, int rb, int cb,
                                        int lane)
{
    const int r = rb * 32 + lane;
#pragma unroll 1
    for (int c0 = cb * 32; c0 < cb * 32 + 32; c0 += 8 * NI) {
        float old[8 * NI], acc[8 * NI];
#pragma unroll
        for (int j = 0; j < 8 * NI; ++j) {
            const int c = c0 + j;
            old[j] = (r < m && c < m && r >= c) ? A[(int64_t)(o + c) * lda + o + r] : 0.f;
            acc[j] = 0.f;
        }
#pragma unroll 4
        for (int k = 0; k < 32; ++k) {
            const float pr = P[k * RP + r];
#pragma unroll
            for (int j = 0; j < 8 * NI; j += 4) {
                float v[4];
                c32_load4(P + k * RP + c0 + j, v);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[j + e] = fmaf(pr, v[e], acc[j + e]);
            }
        }
#pragma unroll
        for (int j = 0; j < 8 * NI; ++j) {
            const int c = c0 + j;
            if (r < m && c < m && r >= c) A[(int64_t)(o + c) * lda + o + r] = old[j] - acc[j];
        }
    }
}

// One problem, whole CTA.  Right-looking in 32-column panels with one step of
// look-ahead: after the panel, three warps update the next diagonal block; then
// warp 0 factors it while the other warps update the rest of the trailing matrix.
// P: the panel, RP its k stride.  Returns INFO (0 or the 1-based failing column).
template <typename T, int NT, int NI>
__device__ int bt_factor(T *A, int n, int lda, T *Lb, T *P, int RP, int *sflag, double *logdet_out,
                         T *B, int nrhs, T *dscr, T *ybuf)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int NW = NT / 32;
    T *rd = Lb + C32_RD;
    double ld_acc = 0.0;
    if (warp == 0) {
        const int f = bt_diag<T>(A, lda, 0, min(BT_NB, n), false, Lb, rd, ld_acc, lane);
        if (lane == 0) sflag[0] = f;
    }
    __syncthreads();
    int info = sflag[0] >= 0 ? sflag[0] + 1 : 0;
    for (int j0 = 0; j0 < n && info == 0; j0 += BT_NB) {
        const int jb = min(BT_NB, n - j0);
        const int o = j0 + jb, m = n - o, mb = (m + 31) / 32;
        // (P) rows below, the right-hand sides and the inverse of the diagonal
        // block, each 32 vectors of the same substitution (the inverse and the
        // right-hand sides also after the last block)
        const int nit = mb + (B ? 2 : 0);
#pragma unroll 1
        for (int it = NW > 1 ? NW - 1 - warp : 0; it < nit; it += NW) {
            T b[32];
            const int rr = it * 32 + lane;
            const bool rows = it < mb, rhs = it == mb;
            T *src = A + (int64_t)j0 * lda + o + rr;
            int64_t stride = lda;
            bool live = rows && rr < m;
            if (rhs) {
                src = B + (int64_t)lane * n + j0;
                stride = 1;
                live = lane < nrhs;
            }
            const T *q = src;
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                b[c] = (live && c < jb) ? *q : T(0);
                q += stride;
            }
            if (!rows && !rhs) {
#pragma unroll
                for (int c = 0; c < 32; ++c) b[c] = c == lane ? T(1) : T(0);
            }
            T *Dk = dscr + (int64_t)(j0 / BT_NB) * 32 * 32 + lane;
            T *Pp = P + rr;
            sweep32<T>(Lb, rd, b, [&](int c, T x) {               // in order of c
                if (live && c < jb) *src = x;
                src += stride;
                if (rows) *Pp = x;
                Pp += RP;
                if (rhs && lane < nrhs) ybuf[lane * 32 + c] = c < jb ? x : T(0);
                if (!rows && !rhs) Dk[c * 32] = x;            // D^-1(c, lane)
            });
        }
        __syncthreads();
        if (m <= 0) break;
        // the next diagonal block, in quarters on three warps; then warp 0
        // factors it while the others do all other tiles and the right-hand
        // sides below, b_r -= L(r, panel) y_panel
        T *C00 = A + (int64_t)o * lda + o;
        if (NW >= 4 ? warp < 3 : warp == 0) {
#pragma unroll 1
            for (int q = NW >= 4 ? warp : 0; q < 3; q += NW >= 4 ? 3 : 1)
                bt_quarter(C00, lda, m, P, RP, Lb, q, lane);
            if (NW >= 4) {
                if (warp > 0) asm volatile("bar.arrive 1, 96;" ::: "memory");
                else asm volatile("bar.sync 1, 96;" ::: "memory");
            } else {
                __syncwarp();
            }
        }
        if (warp == 0) {
            const int f = bt_diag<T>(A, lda, o, min(BT_NB, m), true, Lb, rd, ld_acc, lane);
            if (lane == 0) sflag[0] = f;
        }
        const int ntile = mb * (mb + 1) / 2;
        // warp 4 shares warp 0's sub-partition (and its FP64 pipe): it helps only
        // where the tiles outlast the diagonal block
        const bool spare = NW == 8 && ntile < 24;
        if ((warp > 0 && !(spare && warp == 4)) || NW == 1) {
            const int w = NW == 1 ? 0 : warp - 1 - (spare && warp > 4);
            const int NH = NW == 1 ? 1 : NW - 1 - spare;
#pragma unroll 1
            for (int it = 1 + w; it < ntile; it += NH) {
                // tiles enumerated column by column
                int cb = 0, rem = it;
                while (rem >= mb - cb) {
                    rem -= mb - cb;
                    ++cb;
                }
                const int rb = cb + rem;
                bt_tile<NI>(A, lda, o, m, P, RP, rb, cb, lane);
            }
            if (B) {
#pragma unroll 1
                for (int it = NH - 1 - w; it < mb; it += NH) {
                    const int rr = it * 32 + lane;
                    if (rr >= m) continue;
                    const T *pr = P + rr;
                    T pv[32];
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        pv[c] = *pr;
                        pr += RP;
                    }
                    for (int col = 0; col < nrhs; ++col) {
                        T s = T(0);
#pragma unroll
                        for (int c = 0; c < 32; ++c) s = fma(pv[c], ybuf[col * 32 + c], s);
                        B[(int64_t)col * n + o + rr] -= s;
                    }
                }
            }
        }
        __syncthreads();
        if (sflag[0] >= 0) info = o + sflag[0] + 1;
    }
    // log-determinant: lanes of warp 0 hold the pieces
    if (warp == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ld_acc += __shfl_xor_sync(0xffffffffu, ld_acc, o);
        if (lane == 0 && logdet_out) *logdet_out = info ? (double)NAN : ld_acc;
    }
    return info;
}

// Backward solve L^T X = Y in place (Y from the fused forward solve), whole
// CTA, with the stored inverses of the diagonal blocks: for each block j from
// the last, s = L(below, j)^T x_below (lanes over rows, four columns of a warp
// at a time so that their loads overlap), then x_j = D_j^-T (y_j - s).  x
// stays in shared memory (xs, n values); red holds 32.
template <typename T, int NT>
__device__ void bt_backward(const T *A, int n, int lda, T *B, int nrhs, const T *dscr, T *red, T *xs)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int NW = NT / 32;
    for (int col = 0; col < nrhs; ++col) {
        T *b = B + (int64_t)col * n;
        __syncthreads();
        for (int i = tid; i < n; i += NT) xs[i] = b[i];
        __syncthreads();
        const int nblk = (n + BT_NB - 1) / BT_NB;
        for (int bk = nblk - 1; bk >= 0; --bk) {
            const int j0 = bk * BT_NB, jb = min(BT_NB, n - j0), o = j0 + jb;
            T dk[32];
            if (warp == 0) {
                const T *Dk = dscr + (int64_t)bk * 32 * 32 + lane;   // Dk[i * 32 + c] = D^-1(i, c)
#pragma unroll
                for (int i = 0; i < 32; ++i) dk[i] = Dk[i * 32];
            }
            for (int c = 4 * warp; c < jb; c += 4 * NW) {
                T s[4] = {T(0), T(0), T(0), T(0)};
                const T *Lc[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) Lc[q] = A + (int64_t)(j0 + min(c + q, jb - 1)) * lda;
#pragma unroll 2
                for (int r = o + lane; r < n; r += 32) {
                    const T x = xs[r];
#pragma unroll
                    for (int q = 0; q < 4; ++q) s[q] = fma(Lc[q][r], x, s[q]);
                }
#pragma unroll
                for (int w = 16; w > 0; w >>= 1)
#pragma unroll
                    for (int q = 0; q < 4; ++q) s[q] += __shfl_xor_sync(0xffffffffu, s[q], w);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (lane == q) red[c + q] = s[q];
            }
            __syncthreads();
            if (warp == 0) {
                const T tl = lane < jb ? xs[j0 + lane] - red[lane] : T(0);
                T x0 = T(0), x1 = T(0);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    x0 = fma(dk[i], __shfl_sync(0xffffffffu, tl, i), x0);
                    x1 = fma(dk[i + 1], __shfl_sync(0xffffffffu, tl, i + 1), x1);
                }
                if (lane < jb) {
                    xs[j0 + lane] = x0 + x1;
                    b[j0 + lane] = x0 + x1;
                }
            }
            __syncthreads();
        }
    }
}

template <typename T, int NT, int OCC>
__global__ void __launch_bounds__(NT, OCC) batched_posv_kernel(BatchArgs<T> a)
{
    extern __shared__ __align__(16) unsigned char bsm[];
    T *Lb = reinterpret_cast<T *>(bsm);       // blocked copy of the diagonal factor, 1 / diagonal
    T *P = Lb + C32_LB;                       // panel, k stride prow + 4
    __shared__ int sflag[2];
    __shared__ T ybuf[32 * BT_MAXRHS];
    T *dscr = a.dscr + (int64_t)blockIdx.x * a.dstride;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) sflag[1] = atomicAdd(a.ticket, 1);
        __syncthreads();
        const int slot = sflag[1];
        if (slot >= a.batch) break;
        const int i = a.order[slot];
        const int n = a.n[i], lda = a.lda[i];
        int info = 0;
        if (n > 0) {
            T *Bi = (a.B && a.nrhs > 0) ? a.B[i] : nullptr;
            info = bt_factor<T, NT, NT * OCC <= 256 ? 4 : 2>(a.A[i], n, lda, Lb, P, a.prow + 4, sflag,
                                    a.logdet ? a.logdet + i : nullptr, Bi, a.nrhs, dscr, ybuf);
            if (info == 0 && Bi) bt_backward<T, NT>(a.A[i], n, lda, Bi, a.nrhs, dscr, Lb, P);
        } else if (threadIdx.x == 0 && a.logdet) {
            a.logdet[i] = 0.0;
        }
        if (threadIdx.x == 0) a.info[i] = info;
    }
}

// ---------------------------------------------------------------------------
// host: launch shapes
// ---------------------------------------------------------------------------
template <typename T>
using BtLaunch = int (*)(Context *, BatchArgs<T> &, int nmax);

// OCC: CTAs of an SM the registers are limited for
template <typename T, int NT, int OCC>
static int bt_launch(Context *ctx, BatchArgs<T> &a, int nmax)
{
    // the panel's rows: those below the first block
    a.prow = std::max(32, (nmax - 1) / 32 * 32);
    const size_t smem = (C32_LB + 32 * (size_t)(a.prow + 4)) * sizeof(T);
    CK(cudaFuncSetAttribute(batched_posv_kernel<T, NT, OCC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int occ = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batched_posv_kernel<T, NT, OCC>, NT, smem));
    if (occ < 1) {
        ctx->set_error("batched kernel does not fit (n max %d)", nmax);
        return DPLASMA_ERR_INTERNAL_LIMIT;
    }
    const int grid = std::min(a.batch, ctx->sms * occ);
    // inverses of the diagonal blocks of the CTA's problem
    a.dstride = (int64_t)((nmax + BT_NB - 1) / BT_NB) * 32 * 32;
    a.dscr = (T *)ctx->buffer(BUF_BATCH_SCR, (size_t)grid * a.dstride * sizeof(T));
    if (!a.dscr) return DPLASMA_ERR_OUT_OF_RESOURCES;
    CK(cudaMemsetAsync(a.ticket, 0, sizeof(int), ctx->stream));
    batched_posv_kernel<T, NT, OCC><<<grid, NT, smem, ctx->stream>>>(a);
    CK(cudaGetLastError());
    ctx->launches++;
    return 0;
}

template <typename T>
struct BtVariant {
    const char *name;
    BtLaunch<T> fn;
};
// FP64 has the first three
template <typename T>
static const BtVariant<T> *bt_variants();
template <>
const BtVariant<double> *bt_variants<double>()
{
    static const BtVariant<double> v[] = {{"1 warp per problem", bt_launch<double, 32, 8>},
                                          {"4 warps per problem", bt_launch<double, 128, 3>},
                                          {"8 warps per problem", bt_launch<double, 256, 1>}};
    return v;
}
template <>
const BtVariant<float> *bt_variants<float>()
{
    static const BtVariant<float> v[] = {{"1 warp per problem", bt_launch<float, 32, 8>},
                                         {"4 warps per problem", bt_launch<float, 128, 3>},
                                         {"8 warps per problem", bt_launch<float, 256, 1>},
                                         {"8 warps per problem, two per SM", bt_launch<float, 256, 2>}};
    return v;
}

// Warps per problem: a problem's latency falls with its warps, the work in flight on
// an SM rises with the problems that share it.  The launch ends with whichever is
// later, its largest problem or the last of its work:
//   largest: `one` when it has the SM to itself, `full` when `per` like it share the
//            SM, in between by the problems per SM of the batch;
//   work:    sum of full / per over the problems, shared by the SMs.
// The table holds kernel times in us of 148 problems of order 32, 64, 128, .. on 148
// SMs and of per x 148.  On 419 batches (one order or uniform up to one, 1 to 4096
// problems, many small ones with a few large) the choice costs 0.5 % on average and
// 19 % at most over the best shape of each, where a rule by the largest order alone
// cost up to 2.5 times (FP64, 500 of order 64 and 20 of 256: 294 us with four warps,
// 115 with eight; FP32, 297 of 8 to 768: 2.97 ms with eight warps two per SM, 1.57
// one per SM; FP32, 8192 of 8 to 96: 0.31 ms with one warp, 0.96 with eight).
struct BtTimes {
    int per;
    float one[6], full[6];
};
constexpr float BT_LAUNCH = 6.f;              // of each time, once per launch
static const BtTimes BT_TIMES_F64[] = {
    {8, {24.4f, 44.f, 109.f, 394.f, 2370.f}, {33.9f, 64.8f, 241.f, 1390.f, 18800.f}},
    {3, {24.2f, 41.6f, 77.5f, 207.f, 1080.f}, {26.3f, 45.2f, 97.9f, 342.f, 3210.f}},
    {1, {18.1f, 28.4f, 49.3f, 115.f, 571.f}, {18.1f, 28.4f, 49.3f, 115.f, 571.f}}};
static const BtTimes BT_TIMES_F32[] = {
    {8, {20.f, 37.3f, 92.3f, 386.f, 2240.f, 16200.f}, {24.5f, 48.6f, 131.f, 854.f, 7280.f, 130000.f}},
    {3, {16.6f, 24.2f, 42.9f, 136.f, 764.f, 5520.f}, {18.f, 28.1f, 59.5f, 231.f, 1410.f, 16500.f}},
    {1, {16.2f, 22.5f, 38.8f, 106.f, 520.f, 3590.f}, {16.2f, 22.5f, 38.8f, 106.f, 520.f, 3590.f}},
    {2, {16.4f, 24.f, 43.f, 144.f, 742.f, 5260.f}, {17.9f, 26.2f, 51.1f, 181.f, 983.f, 10500.f}}};

// a row of the table at an order of b 32-wide blocks, by powers between its points
static double bt_time(const float *y, int points, int b)
{
    const double x = log2((double)std::max(b, 1));
    const int i = std::min((int)x, points - 2);
    return y[i] * pow((double)y[i + 1] / y[i], x - i);
}

// order(i): the i-th largest order
template <class Order>
static int bt_choose(bool fp64, int batch, int sms, Order order)
{
    const BtTimes *t = fp64 ? BT_TIMES_F64 : BT_TIMES_F32;
    const int nv = fp64 ? 3 : 4, points = fp64 ? 5 : 6;
    // problems by their 32-wide blocks
    int count[BT_NMAX / BT_NB + 1] = {0};
    const int top = batch > 0 ? (order(0) + BT_NB - 1) / BT_NB : 0;
    for (int b = top, from = 0; b >= 0; --b) {
        int lo = from, hi = batch;                 // the first beyond those of b blocks
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (order(mid) > (b - 1) * BT_NB) lo = mid + 1;
            else hi = mid;
        }
        count[b] = lo - from;
        from = lo;
    }
    int best = 0;
    double best_us = 0.0;
    for (int v = 0; v < nv; ++v) {
        const double share = std::min((double)t[v].per, std::max(1.0, (double)batch / sms));
        const double one = bt_time(t[v].one, points, top), full = bt_time(t[v].full, points, top);
        const double largest = t[v].per > 1 ? one + (full - one) * (share - 1.0) / (t[v].per - 1) : one;
        double work = 0.0;
        for (int b = 0; b <= top; ++b)
            if (count[b]) work += count[b] * (bt_time(t[v].full, points, b) - BT_LAUNCH);
        const double us = std::max(largest, BT_LAUNCH + work / ((double)sms * t[v].per));
        if (v == 0 || us < best_us) {
            best = v;
            best_us = us;
        }
    }
    return best;
}

template <typename T>
int batched_posv(Context *ctx, int batch, const int *d_n, const int *d_lda, T *const *d_A, T *const *d_B, int nrhs,
                 double *d_logdet, int *d_info)
{
    if (batch <= 0) return 0;
    cudaStream_t st = ctx->stream;
    // sizes to the host for the work order (longest first) and the smem size
    std::vector<int> hn(batch);
    CK(cudaMemcpyAsync(hn.data(), d_n, batch * sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    int nmax = 0;
    for (int v : hn) {
        if (v < 0) {
            ctx->set_error("negative order in the batch");
            return DPLASMA_ERR_ILLEGAL_VALUE;
        }
        nmax = std::max(nmax, v);
    }
    if (nmax > BT_NMAX || (size_t)(nmax + 96) * 36 * sizeof(T) > 220 * 1024) {
        ctx->set_error("batched problems of order %d exceed the limit", nmax);
        return DPLASMA_ERR_INTERNAL_LIMIT;
    }
    std::vector<int> order(batch);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return hn[x] > hn[y]; });
    int *dord = (int *)ctx->buffer(BUF_BATCH, ((size_t)batch + 64) * sizeof(int));
    if (!dord) return DPLASMA_ERR_OUT_OF_RESOURCES;
    CK(cudaMemcpyAsync(dord, order.data(), batch * sizeof(int), cudaMemcpyHostToDevice, st));

    if (nrhs > BT_MAXRHS) {
        ctx->set_error("batched solve takes at most %d right-hand sides (got %d)", BT_MAXRHS, nrhs);
        return DPLASMA_ERR_NOT_SUPPORTED;
    }
    BatchArgs<T> a;
    a.batch = batch;
    a.n = d_n;
    a.lda = d_lda;
    a.A = d_A;
    a.B = d_B;
    a.nrhs = nrhs;
    a.logdet = d_logdet;
    a.info = d_info;
    a.order = dord;
    a.ticket = dord + batch + 32;
    const int choice = bt_choose(sizeof(T) == 8, batch, ctx->sms, [&](int i) { return hn[order[i]]; });
    const BtVariant<T> &shape = bt_variants<T>()[choice];
    CK(cudaEventRecord(ctx->ev0, st));
    const int rc = shape.fn(ctx, a, nmax);
    if (rc) return rc;
    ctx->bt_last_variant = shape.name;
    CK(cudaEventRecord(ctx->ev1, st));
    CK(cudaStreamSynchronize(st));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    ctx->last_factor_ms = ms;
    return 0;
}

// ---------------------------------------------------------------------------
// batched inverse from the factors: A_i = L_i (lower) -> A_i^-1 (lower)
// (dplasma's potri = trtri + lauum, src/zpotri_wrapper.c, per problem), the
// backward step of a batch of GP likelihoods.  One CTA per problem from the
// same work queue; 32x32 tiles, one warp per tile, FP64 tensor cores, the
// factor and W = L^-1 in per-CTA scratch (padded to a multiple of 32 with the
// identity).
//   W_jj = L_jj^-1 (warp 0);  W_ij = -(sum_{k=j+1}^{i} W_ik L_kj) W_jj,  j from the last
//   A^-1 = W^T W:  (i >= j)  sum_{k >= i} W_ki^T W_kj
// ---------------------------------------------------------------------------
constexpr int BI_PP = 36;

// acc(32x32) += op(X) op(Y) over one 32-deep K block; X, Y in global memory
// (column-major, L2 reads), op = transpose when tx / ty
__device__ __forceinline__ void bi_mma(double (&acc)[2][4][4], const double *X, int ldx, bool tx, const double *Y,
                                       int ldy, bool ty, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int kk = 0; kk < 32; kk += 4) {
        double af[2][2], bf[4];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = mi * 16 + g + 8 * h, k = kk + t;
                af[mi][h] = tx ? __ldcg(X + (int64_t)r * ldx + k) : __ldcg(X + (int64_t)k * ldx + r);
            }
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
            const int k = kk + t, c = ni * 8 + g;
            bf[ni] = ty ? __ldcg(Y + (int64_t)k * ldy + c) : __ldcg(Y + (int64_t)c * ldy + k);
        }
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) dmma_16x8x4(acc[mi][ni], af[mi][0], af[mi][1], bf[ni]);
    }
}

struct BatchInvArgs {
    int batch;
    const int *n;
    const int *lda;
    double *const *A;
    int *info;
    const int *order;
    int *ticket;
    double *scr;      // per CTA: padded factor and W, each nmax32^2
    int nmax32;
    // GP gradient (null: the inverse goes to A's lower triangle): the factor
    // stays, out_i (both triangles, leading dimension lda_i) = g_i / 2 (alpha_i
    // alpha_i^T - K_i^-1)
    const double *const *alpha;
    const double *g;
    double *const *out;
};

__global__ void __launch_bounds__(256) batched_potri_kernel(BatchInvArgs a)
{
    extern __shared__ __align__(16) double bism[];
    double *Wd = bism;                       // W_jj, 32 x BI_PP
    double *Ls = Wd + 32 * BI_PP;            // staging of L_jj
    double *Tw = Ls + 32 * BI_PP;            // per warp 32 x BI_PP
    __shared__ int slot_s, bad_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int64_t ss = (int64_t)a.nmax32 * a.nmax32;
    double *Lp = a.scr + (int64_t)blockIdx.x * 2 * ss;
    double *W = Lp + ss;
    while (true) {
        __syncthreads();
        if (tid == 0) slot_s = atomicAdd(a.ticket, 1);
        __syncthreads();
        if (slot_s >= a.batch) break;
        const int pi = a.order[slot_s];
        const int n = a.n[pi], lda = a.lda[pi];
        double *A = a.A[pi];
        if (n <= 0) {
            if (tid == 0) a.info[pi] = 0;
            continue;
        }
        const int nb = (n + 31) / 32, ld = nb * 32;
        // padded factor: lower part of L, identity beyond n, zero above
        for (int64_t e = tid; e < (int64_t)ld * ld; e += 256) {
            const int r = (int)(e % ld), c = (int)(e / ld);
            double v = 0.0;
            if (r >= c) v = (r < n && c < n) ? A[(int64_t)c * lda + r] : (r == c ? 1.0 : 0.0);
            Lp[e] = v;
        }
        __syncthreads();
        int info = 0;
        for (int j = nb - 1; j >= 0 && info == 0; --j) {
            // W_jj = L_jj^-1 by warp 0 (lane c forms column c)
            if (warp == 0) {
                const double *Lj = Lp + (int64_t)(32 * j) * ld + 32 * j;
#pragma unroll
                for (int c = 0; c < 32; ++c) Ls[lane * BI_PP + c] = (c <= lane) ? __ldcg(Lj + (int64_t)c * ld + lane) : 0.0;
                __syncwarp();
                const double dl = Ls[lane * BI_PP + lane];
                const double rd = 1.0 / dl;
                const int bad = __ballot_sync(0xffffffffu, dl == 0.0);
                if (lane == 0) bad_s = bad ? 32 * j + __ffs(bad) : 0;   // INFO of a zero pivot
                double x[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    double s0 = 0.0, s1 = 0.0;
#pragma unroll
                    for (int l = 0; l + 1 < i; l += 2) {
                        s0 = fma(Ls[i * BI_PP + l], x[l], s0);
                        s1 = fma(Ls[i * BI_PP + l + 1], x[l + 1], s1);
                    }
                    if (i & 1) s0 = fma(Ls[i * BI_PP + i - 1], x[i - 1], s0);
                    const double ri = __shfl_sync(0xffffffffu, rd, i);
                    x[i] = (i < lane) ? 0.0 : ((i == lane) ? ri : -(s0 + s1) * ri);
                }
                double *Wj = W + (int64_t)(32 * j) * ld + 32 * j;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    Wd[i * BI_PP + lane] = x[i];
                    Wj[(int64_t)lane * ld + i] = x[i];
                }
            }
            __syncthreads();
            if (bad_s != 0) {
                info = bad_s;
                break;
            }
            // block rows below: W_ij = -(sum_{k=j+1}^{i} W_ik L_kj) W_jj
            double *T = Tw + warp * 32 * BI_PP;
            for (int i = j + 1 + warp; i < nb; i += 8) {
                double acc[2][4][4];
#pragma unroll
                for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;
                for (int k = j + 1; k <= i; ++k)
                    bi_mma(acc, W + (int64_t)(32 * k) * ld + 32 * i, ld, false, Lp + (int64_t)(32 * j) * ld + 32 * k, ld,
                           false, lane);
#pragma unroll
                for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int r = mi * 16 + g + ((q & 2) ? 8 : 0), c = ni * 8 + 2 * t + (q & 1);
                            T[r * BI_PP + c] = acc[mi][ni][q];
                            acc[mi][ni][q] = 0.0;
                        }
                __syncwarp();
#pragma unroll
                for (int kk = 0; kk < 32; kk += 4) {
                    double af[2][2], bf[4];
#pragma unroll
                    for (int mi = 0; mi < 2; ++mi) {
                        af[mi][0] = T[(mi * 16 + g) * BI_PP + kk + t];
                        af[mi][1] = T[(mi * 16 + g + 8) * BI_PP + kk + t];
                    }
#pragma unroll
                    for (int ni = 0; ni < 4; ++ni) bf[ni] = Wd[(kk + t) * BI_PP + ni * 8 + g];
#pragma unroll
                    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                        for (int ni = 0; ni < 4; ++ni) dmma_16x8x4(acc[mi][ni], af[mi][0], af[mi][1], bf[ni]);
                }
                double *Wij = W + (int64_t)(32 * j) * ld + 32 * i;
#pragma unroll
                for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int r = mi * 16 + g + ((q & 2) ? 8 : 0), c = ni * 8 + 2 * t + (q & 1);
                            Wij[(int64_t)c * ld + r] = -acc[mi][ni][q];
                        }
                __syncwarp();
            }
            __syncthreads();
        }
        if (info == 0) {
            // A^-1 = W^T W, lower tiles (i >= j), into A, or straight into the
            // likelihood's gradient: the tile and its mirror, from registers
            // (the inverse, its symmetric copy and the rank-1 term as whole-batch
            // passes took 2.8 ms of the 1024-problem gradient's 4.7)
            const double *al = a.alpha ? a.alpha[pi] : nullptr;
            const double hg = a.alpha ? 0.5 * a.g[pi] : 0.0;
            double *O = a.alpha ? a.out[pi] : nullptr;
            const int ntile = nb * (nb + 1) / 2;
            for (int it = warp; it < ntile; it += 8) {
                int bi = (int)((sqrtf(8.0f * it + 1.0f) - 1.0f) * 0.5f);
                while ((bi + 1) * (bi + 2) / 2 <= it) ++bi;
                while (bi * (bi + 1) / 2 > it) --bi;
                const int bj = it - bi * (bi + 1) / 2;
                double acc[2][4][4];
#pragma unroll
                for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;
                for (int k = bi; k < nb; ++k)
                    bi_mma(acc, W + (int64_t)(32 * bi) * ld + 32 * k, ld, true, W + (int64_t)(32 * bj) * ld + 32 * k, ld,
                           false, lane);
#pragma unroll
                for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int r = 32 * bi + mi * 16 + g + ((q & 2) ? 8 : 0);
                            const int c = 32 * bj + ni * 8 + 2 * t + (q & 1);
                            if (O) {
                                if (r < n && c < n) {
                                    const double v = hg * (__ldg(al + r) * __ldg(al + c) - acc[mi][ni][q]);
                                    O[(int64_t)c * lda + r] = v;
                                    if (bi != bj) O[(int64_t)r * lda + c] = v;
                                }
                            } else if (r < n && c < n && r >= c) {
                                A[(int64_t)c * lda + r] = acc[mi][ni][q];
                            }
                        }
            }
        }
        __syncthreads();
        if (tid == 0) a.info[pi] = info;
    }
}

int batched_potri(Context *ctx, int batch, const int *d_n, const int *d_lda, double *const *d_A, int *d_info,
                  const double *const *d_alpha, const double *d_g, double *const *d_out)
{
    if (batch <= 0) return 0;
    cudaStream_t st = ctx->stream;
    std::vector<int> hn(batch);
    CK(cudaMemcpyAsync(hn.data(), d_n, batch * sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    int nmax = 0;
    for (int v : hn) nmax = std::max(nmax, v);
    if (nmax > BT_NMAX) return DPLASMA_ERR_INTERNAL_LIMIT;
    std::vector<int> order(batch);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return hn[x] > hn[y]; });
    int *dord = (int *)ctx->buffer(BUF_BATCH, ((size_t)batch + 64) * sizeof(int));
    if (!dord) return DPLASMA_ERR_OUT_OF_RESOURCES;
    int *ticket = dord + batch + 32;
    CK(cudaMemcpyAsync(dord, order.data(), batch * sizeof(int), cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(ticket, 0, sizeof(int), st));
    const int nmax32 = std::max(32, (nmax + 31) & ~31);
    const size_t smem = (size_t)(2 * 32 * BI_PP + 8 * 32 * BI_PP) * sizeof(double);
    CK(cudaFuncSetAttribute(batched_potri_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int occ = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batched_potri_kernel, 256, smem));
    const int grid = ctx->sms * std::max(1, std::min(occ, 2));
    double *scr = (double *)ctx->buffer(BUF_BATCH_W, (size_t)grid * 2 * nmax32 * nmax32 * sizeof(double));
    if (!scr) return DPLASMA_ERR_OUT_OF_RESOURCES;
    BatchInvArgs a;
    a.batch = batch;
    a.n = d_n;
    a.lda = d_lda;
    a.A = d_A;
    a.info = d_info;
    a.order = dord;
    a.ticket = ticket;
    a.scr = scr;
    a.nmax32 = nmax32;
    a.alpha = d_alpha;
    a.g = d_g;
    a.out = d_out;
    CK(cudaEventRecord(ctx->ev0, st));
    batched_potri_kernel<<<grid, 256, smem, st>>>(a);
    CK(cudaGetLastError());
    CK(cudaEventRecord(ctx->ev1, st));
    ctx->launches++;
    CK(cudaStreamSynchronize(st));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    ctx->last_solve_ms = ms;
    return 0;
}

template int batched_posv<double>(Context *, int, const int *, const int *, double *const *, double *const *, int,
                                  double *, int *);
template int batched_posv<float>(Context *, int, const int *, const int *, float *const *, float *const *, int,
                                 double *, int *);

}  // namespace db2

// Test hook (not part of the public header): the launch shape of a batch of orders n
extern "C" int dplasma_b200_debug_batched_choice(int fp64, int sms, int batch, const int *n)
{
    std::vector<int> sorted(n, n + batch);
    std::sort(sorted.begin(), sorted.end(), std::greater<int>());
    return db2::bt_choose(fp64 != 0, batch, sms, [&](int i) { return sorted[i]; });
}
