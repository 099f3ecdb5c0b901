// adjoint.cu -- reverse-mode derivative of the Cholesky factorization.
//
// For A = L L^T and the adjoint Lbar = dF/dL of a scalar F, the adjoint of A
// (symmetric) is
//     Abar = sym( L^-T Phi(L^T Lbar) L^-1 ),   sym(X) = (X + X^T) / 2,
// with Phi(X) the lower triangle of X with its diagonal halved (the
// blocked form of the reverse Cholesky sweep, Murray 2016, "Differentiation
// of the Cholesky decomposition").  It is computed with W = L^-1 as
//     W                 diagonal 128-blocks inverted in shared memory, then
//                       W_ij = -W_ii sum_{k=j}^{i-1} L_ik W_kj, block row by row
//     Y = Phi(L^T Lbar) lower tiles, k >= i
//     Z = Y W           lower tiles, j <= k <= i
//     Abar = sym(W^T Z) lower tiles: (W^T Z + Z^T W) / 2, k >= i
// on dense column-major copies in the padded index space of the device
// tiles (padding rows: identity in L, zero in Lbar, hence zero in Abar).
// Every product runs on one FP64 tensor-core GEMM kernel over 128x128 output
// tiles whose K range follows the triangular structure.
//
// The same products give the inverse of the factor and of A (dplasma's
// dtrtri / dlauum / dpotri / dpoinv, src/zpotri_wrapper.c: trtri then lauum):
//     trtri  W = L^-1;  lauum  L^T L;  potri  A^-1 = W^T W  (lower part).
//
// The log-determinant and solve adjoints reduce to it or to rank updates:
// log det A = 2 sum log L(i,i) gives Lbar(i,i) = 2 / L(i,i) and Abar = A^-1;
// x = A^-1 b gives Abar = -A^-1 xbar x^T (symmetrized) and bbar = A^-1 xbar.
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "dev_potrf128.cuh"
#include "internal.h"

namespace db2 {

constexpr int AG_T = 128;     // output tile
constexpr int AG_K = 16;      // K chunk
constexpr int AG_P = 132;     // shared pitch of a chunk stored by columns of A (= 4 mod 16)
constexpr int AG_KP = 20;     // of one stored by rows, K contiguous as in memory (= 4 mod 16)
constexpr int AG_NST = 4;     // chunks of A and B in shared memory

// Tile sets and K ranges (block indices):
//   LOWER_KGE_I   tiles i >= j                 k in [i, P-1]
//   LOWER_JKI     tiles i >= j                 k in [j, i]
//   SYM_KGE_I     tiles i >= j                 k in [i, P-1], A^T B + B^T A
//   GRAD          as LOWER_KGE_I, its result straight into a GP gradient
//   LVL_T, LVL_W  one level of the recursive triangular inverse: for every
//                 diagonal block [o, o+2h) of 2h tiles, with W11 = the inverse
//                 of its first half and W22 of its second (previous level),
//                   LVL_T: Y21 = L21 W11     tiles (o+h+i, o+j), k in [o+j, o+h)
//                   LVL_W: W21 = -W22 Y21    tiles (o+h+i, o+j), k in [o+h, o+h+i]
//                 (h = rowblk; the last block's second half may be short)
// Blocks run in order, so every mode starts with its longest K ranges: the last
// wave is then made of short ones (N = 4096: JKI 1224 us in row order).
enum : int { AG_LOWER_KGE_I = 1, AG_LOWER_JKI = 2, AG_SYM_KGE_I = 3, AG_GRAD = 4, AG_LVL_T = 5, AG_LVL_W = 6 };

struct AgArgs {
    int mode, P, rowblk, nblk;
    const double *A;
    int lda;
    const double *B;
    int ldb;
    double *C;
    int ldc;
    double alpha;
    // GRAD: out (n x n, both triangles, ld n) = g / 2 (al al^T - nal * product);
    // alt (null: al al^T in the epilogue): al^T, K contiguous, padded with zeros to
    // nk = 16 ceil(nal / 16) by whole tiles, for al al^T as a product of its own
    const double *al, *g;
    int nal, n;
    double *out;
    const double *alt;
    int nk;
};

// C(i,j) = alpha * sum_{k in range} op(A)(i,k) B(k,j), 128x128 tiles; op is the
// transpose when TA.  Chunks stay as they lie in memory (B, and A when TA, with K
// contiguous), so they arrive by 16-byte asynchronous copies three ahead and the
// fragments are read without bank conflicts either way.  Bound: DMMA, and the last
// wave (N = 4096: L^T Lbar 828 us of 620 at the DMMA peak, Y W 835, W^T Z + Z^T W
// 1634 of 1240; through registers, stored transposed and two chunks deep, 995, 933
// and 1963).
constexpr int AG_OP = 128 * AG_KP;                              // doubles of one operand's chunk
constexpr size_t AG_SMEM = AG_NST * 2 * AG_OP * sizeof(double);
static_assert(AG_K * AG_P <= AG_OP, "either form fits");

// COLS: GRAD with alt (al al^T first).
template <bool TA, bool COLS>
__global__ void __launch_bounds__(256, 1) ag_gemm_kernel(AgArgs a)
{
    extern __shared__ __align__(16) double agsm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int wm = warp & 1, wn = warp >> 1;
    // tile and K range; A(i, ako + k), B(bko + k, j)
    int i, j, k0, k1, ako = 0, bko = 0;
    const int tix = blockIdx.x;
    if (a.mode == AG_LVL_T || a.mode == AG_LVL_W) {
        const int h = a.rowblk;
        const int b = tix % a.nblk, rem = tix / a.nblk;
        const int o = b * 2 * h;
        int ii, jj;
        if (a.mode == AG_LVL_T) {
            ii = rem % h;
            jj = rem / h;
        } else {
            ii = h - 1 - rem / h;
            jj = rem % h;
        }
        if (ii >= min(h, a.P - o - h)) return;   // beyond a short last block
        i = o + h + ii;
        j = o + jj;
        if (a.mode == AG_LVL_T) {
            ako = bko = o;
            k0 = jj;
            k1 = h - 1;
        } else {
            ako = bko = o + h;
            k0 = 0;
            k1 = ii;
        }
    } else if (a.mode == AG_LOWER_JKI) {
        // by diagonals i - j = P-1, P-2, ..: the d-th from the corner holds d + 1 tiles
        int d = (int)((sqrtf(8.0f * tix + 1.0f) - 1.0f) * 0.5f);
        while ((d + 1) * (d + 2) / 2 <= tix) ++d;
        while (d * (d + 1) / 2 > tix) --d;
        j = tix - d * (d + 1) / 2;
        i = j + a.P - 1 - d;
        k0 = j;
        k1 = i;
    } else {
        int bi = (int)((sqrtf(8.0f * tix + 1.0f) - 1.0f) * 0.5f);
        while ((bi + 1) * (bi + 2) / 2 <= tix) ++bi;
        while (bi * (bi + 1) / 2 > tix) --bi;
        i = bi;
        j = tix - bi * (bi + 1) / 2;
        k0 = i;
        k1 = a.P - 1;
    }
    double acc[4][4][4];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;

    const int kbeg = k0 * AG_T, kend = (k1 + 1) * AG_T;
    const double *Aop = a.A, *Bop = a.B;
    int lda = a.lda, ldb = a.ldb;
    auto load = [&](int slot, int kc) {
        double *As = agsm + slot * 2 * AG_OP, *Bs = As + AG_OP;
        // four 16-byte pieces of each operand a thread
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!TA) {
                const int r = 2 * (tid & 63), kk = (tid >> 6) + 4 * q;
                cp_async16(As + kk * AG_P + r, Aop + (int64_t)(ako * AG_T + kc + kk) * lda + i * AG_T + r);
            }
            const int kk = 2 * (tid & 7), r = (tid >> 3) + 32 * q;
            if (TA) cp_async16(As + r * AG_KP + kk, Aop + (int64_t)(i * AG_T + r) * lda + ako * AG_T + kc + kk);
            cp_async16(Bs + r * AG_KP + kk, Bop + (int64_t)(j * AG_T + r) * ldb + bko * AG_T + kc + kk);
        }
    };
    // one pass over K, or two with the operands exchanged (SYM), after nal chunks of
    // al^T (GRAD with many columns)
    const int len = kend - kbeg, nal = COLS ? a.nk / AG_K : 0;
    const int nch = nal + (a.mode == AG_SYM_KGE_I ? 2 * len : len) / AG_K;
    auto stage = [&](int ch) {
        if (COLS && ch < nal) {
            Aop = Bop = a.alt;
            lda = ldb = a.nk;
            load(ch % AG_NST, ch * AG_K);
        } else if (ch < nch) {
            const int at = (ch - nal) * AG_K;
            if (COLS && at == 0) {
                Aop = a.A;
                Bop = a.B;
                lda = a.lda;
                ldb = a.ldb;
            }
            if (at >= len) {
                Aop = a.B;
                Bop = a.A;
            }
            load(ch % AG_NST, kbeg + (at >= len ? at - len : at));
        }
        cp_async_commit();                     // (empty at the end: the count of groups stays even)
    };
    constexpr int ar = TA ? AG_KP : 1, ak = TA ? 1 : AG_P;      // strides of a chunk of A
#pragma unroll 1
    for (int ch = 0; ch < AG_NST - 1; ++ch) stage(ch);
    // element (mi, ni, q) of this thread in the result
    auto row = [&](int mi, int q) { return i * AG_T + wm * 64 + mi * 16 + g + ((q & 2) ? 8 : 0); };
    auto col = [&](int ni, int q) { return j * AG_T + wn * 32 + ni * 8 + 2 * t + (q & 1); };
#pragma unroll 1
    for (int ch = 0; ch < nch; ++ch) {
        cp_async_wait(AG_NST - 2);
        __syncthreads();                       // chunk ch is there, chunk ch - 1 is free
        if (COLS && ch == nal) {
            // al al^T is complete: it waits in the result's place (read back below by
            // the thread that wrote it)
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int r = row(mi, q), c = col(ni, q);
                        if (r < a.n && c < a.n) a.out[(int64_t)c * a.n + r] = acc[mi][ni][q];
                        acc[mi][ni][q] = 0.0;
                    }
        }
        stage(ch + AG_NST - 1);
        const double *Ab = agsm + (ch % AG_NST) * 2 * AG_OP + (wm * 64 + g) * ar + t * ak;
        const double *Bb = agsm + (ch % AG_NST) * 2 * AG_OP + AG_OP + (wn * 32 + g) * AG_KP + t;
#pragma unroll
        for (int kk = 0; kk < AG_K; kk += 4) {
            double af[4][2], bf[4];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) {
                af[mi][0] = Ab[kk * ak + mi * 16 * ar];
                af[mi][1] = Ab[kk * ak + (mi * 16 + 8) * ar];
            }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) bf[ni] = Bb[kk + ni * 8 * AG_KP];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma_16x8x4(acc[mi][ni], af[mi][0], af[mi][1], bf[ni]);
        }
    }
    if (a.mode == AG_GRAD) {
        // the tile and its mirror from registers: the inverse, its symmetric copy
        // and the rank-m term as passes of their own took 1.1 ms of 14 at n = 6001
        const double hg = 0.5 * *a.g;
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) {
            // (the stores below may not be passed by loads: those of 16 values first)
            double s[4][4];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = row(mi, q), c = col(ni, q);
                    s[ni][q] = COLS && r < a.n && c < a.n ? a.out[(int64_t)c * a.n + r] : 0.0;
                }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = row(mi, q), c = col(ni, q);
                    if (r >= a.n || c >= a.n) continue;
                    double v = fma(-(double)a.nal, acc[mi][ni][q], s[ni][q]);
                    if (!COLS)
                        for (int l = 0; l < a.nal; ++l)
                            v = fma(__ldg(a.al + (int64_t)l * a.n + r), __ldg(a.al + (int64_t)l * a.n + c), v);
                    a.out[(int64_t)c * a.n + r] = hg * v;
                    if (i != j) a.out[(int64_t)r * a.n + c] = hg * v;
                }
        }
        return;
    }
    double *C = a.C + (int64_t)(j * AG_T) * a.ldc + i * AG_T;
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = wm * 64 + mi * 16 + g + ((q & 2) ? 8 : 0);
                const int c = wn * 32 + ni * 8 + 2 * t + (q & 1);
                C[(int64_t)c * a.ldc + r] = a.alpha * acc[mi][ni][q];
            }
}

struct AgGrad {
    const double *al, *g;
    int nal, n;
    double *out;
    const double *alt;
    int nk;
};
static int ag_gemm(Context *ctx, int mode, int P, int rowblk, const double *A, int lda, int transA, const double *B,
                   int ldb, double *C, int ldc, double alpha, const AgGrad *gr = nullptr)
{
    AgArgs a;
    a.al = gr ? gr->al : nullptr;
    a.g = gr ? gr->g : nullptr;
    a.nal = gr ? gr->nal : 0;
    a.n = gr ? gr->n : 0;
    a.out = gr ? gr->out : nullptr;
    a.alt = gr ? gr->alt : nullptr;
    a.nk = gr ? gr->nk : 0;
    a.mode = mode;
    a.P = P;
    a.rowblk = rowblk;
    a.nblk = rowblk > 0 ? (P + 2 * rowblk - 1) / (2 * rowblk) : 0;
    a.A = A;
    a.lda = lda;
    a.B = B;
    a.ldb = ldb;
    a.C = C;
    a.ldc = ldc;
    a.alpha = alpha;
    int ntile;
    if (mode == AG_LVL_T || mode == AG_LVL_W) ntile = a.nblk * rowblk * rowblk;
    else ntile = P * (P + 1) / 2;
    if (ntile <= 0) return 0;
    auto fn = !transA ? ag_gemm_kernel<false, false>
                      : a.alt ? ag_gemm_kernel<true, true> : ag_gemm_kernel<true, false>;
    CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AG_SMEM));
    fn<<<ntile, 256, AG_SMEM, ctx->stream>>>(a);
    CK(cudaGetLastError());
    ctx->launches++;
    return 0;
}

// ---------------------------------------------------------------------------
// layout helpers (padded index space of the device tiles, ld = Np)
// ---------------------------------------------------------------------------
// Lower tiles <-> the dense lower part, one CTA per 64x64 piece; the part above
// the diagonal of a diagonal tile is zero in the dense form, the tiles above it
// are never read.
constexpr int AG_M = 64;
template <bool TO_DENSE>
__global__ void __launch_bounds__(256) ag_move(double *T, int mt, int nbi, double *D, int ld)
{
    const int m = blockIdx.x, n = blockIdx.y;
    if (m < n) return;
    const int per = nbi / AG_M, r = (blockIdx.z % per) * AG_M + (threadIdx.x & (AG_M - 1));
    const int c0 = (blockIdx.z / per) * AG_M + threadIdx.x / AG_M;
    double *Tt = T + lower_tile_index(m, n, mt) * (int64_t)nbi * nbi + r;
    double *Dt = D + (int64_t)(n * nbi) * ld + m * nbi + r;
#pragma unroll 8
    for (int c = c0; c < c0 + AG_M; c += 256 / AG_M) {
        if (TO_DENSE) Dt[(int64_t)c * ld] = (m == n && r < c) ? 0.0 : Tt[(int64_t)c * nbi];
        else if (m != n || r >= c) Tt[(int64_t)c * nbi] = Dt[(int64_t)c * ld];
    }
}

// Phi: keep the lower triangle, halve the diagonal (diagonal 128-blocks only;
// the GEMM wrote lower tiles and never the strictly upper ones)
__global__ void ag_phi(double *Y, int ld, int P)
{
    const int b = blockIdx.x;
    double *Yb = Y + (int64_t)(b * AG_T) * ld + b * AG_T;
    for (int e = threadIdx.x; e < AG_T * AG_T; e += blockDim.x) {
        const int r = e % AG_T, c = e / AG_T;
        double &v = Yb[(int64_t)c * ld + r];
        if (r < c) v = 0.0;
        else if (r == c) v *= 0.5;
    }
}

// inverses of the 128x128 diagonal blocks of a dense lower factor, written
// into the diagonal blocks of W (ld = ldw); W's other blocks untouched.
// 76 -> 14 us at 32 blocks with the blocks in shared memory
__global__ void __launch_bounds__(256) ag_trtri_diag(const double *L, int ld, double *W, int ldw, double *scratch,
                                                     int unit_diag)
{
    extern __shared__ __align__(16) double tsm[];
    const int b = blockIdx.x;
    const int tid = threadIdx.x;
    const double *T = L + (int64_t)(b * AG_T) * ld + b * AG_T;
    double *Wk = scratch + (int64_t)b * AG_T * AG_T;   // 128x128, ld 128
    p128_load(tsm, T, ld, false, tid);
    cp_async_wait(0);
    __syncthreads();
    p128_invert(tsm, tsm + P128_S + P128_D, unit_diag, Wk, tid >> 5, tid & 31, 1);
    double *Wb = W + (int64_t)(b * AG_T) * ldw + b * AG_T;
    for (int e = tid; e < AG_T * AG_T; e += 256) {
        const int r = e % AG_T, c = e / AG_T;
        Wb[(int64_t)c * ldw + r] = Wk[e];
    }
}

// W = L^-1 into W (dense, ld), from the dense L; unit: diagonal taken as 1.
// Recursive by levels: the 128x128 diagonal inverses, then for blocks of 2,
// 4, 8, ... tiles W21 = -W22 (L21 W11) from the two half-blocks' inverses,
// every block of a level in one launch (log2(P) levels of two launches).
static int ag_inverse(Context *ctx, const double *L, double *W, double *Y, double *scr, int P, int ld, int unit)
{
    cudaStream_t st = ctx->stream;
    int rc;
    const size_t tsmem = P128_INV_DOUBLES * sizeof(double);
    CK(cudaFuncSetAttribute(ag_trtri_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem));
    ag_trtri_diag<<<P, 256, tsmem, st>>>(L, ld, W, ld, scr, unit);
    CK(cudaGetLastError());
    ctx->launches++;
    for (int h = 1; h < P; h *= 2) {
        if ((rc = ag_gemm(ctx, AG_LVL_T, P, h, L, ld, 0, W, ld, Y, ld, 1.0))) return rc;
        if ((rc = ag_gemm(ctx, AG_LVL_W, P, h, W, ld, 0, Y, ld, W, ld, -1.0))) return rc;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// driver: L and Lbar as device tiles (lower, padded), Abar (lower tiles) out
// ---------------------------------------------------------------------------
int potrf_adjoint_tiles(Context *ctx, const double *Lt, double *Lbt, const Geom &g)
{
    const int Np = g.mt * g.nbi, P = Np / AG_T, ld = Np;
    const size_t nn = (size_t)Np * Np;
    double *D = (double *)ctx->buffer(BUF_ADJ, 4 * nn * sizeof(double) + (size_t)P * AG_T * AG_T * sizeof(double));
    if (!D) return DPLASMA_ERR_OUT_OF_RESOURCES;
    double *L = D, *W = D + nn, *Y = D + 2 * nn, *Z = D + 3 * nn, *scr = D + 4 * nn;
    cudaStream_t st = ctx->stream;
    int rc;
    const dim3 tg(g.mt, g.mt, (g.nbi / AG_M) * (g.nbi / AG_M));
    ag_move<true><<<tg, 256, 0, st>>>(const_cast<double *>(Lt), g.mt, g.nbi, L, ld);
    CK(cudaGetLastError());
    ag_move<true><<<tg, 256, 0, st>>>(Lbt, g.mt, g.nbi, Z, ld);   // Lbar (lower) into Z for now
    CK(cudaGetLastError());
    ctx->launches += 2;
    // W = L^-1
    if ((rc = ag_inverse(ctx, L, W, Y, scr, P, ld, 0))) return rc;
    // Y = Phi(L^T Lbar), lower tiles, k >= i
    if ((rc = ag_gemm(ctx, AG_LOWER_KGE_I, P, 0, L, ld, 1, Z, ld, Y, ld, 1.0))) return rc;
    ag_phi<<<P, 256, 0, st>>>(Y, ld, P);
    CK(cudaGetLastError());
    ctx->launches++;
    // Z = Y W, lower tiles, j <= k <= i
    if ((rc = ag_gemm(ctx, AG_LOWER_JKI, P, 0, Y, ld, 0, W, ld, Z, ld, 1.0))) return rc;
    // Abar = sym(W^T Z), lower tiles
    if ((rc = ag_gemm(ctx, AG_SYM_KGE_I, P, 0, W, ld, 1, Z, ld, Y, ld, 0.5))) return rc;
    ag_move<false><<<tg, 256, 0, st>>>(Lbt, g.mt, g.nbi, Y, ld);
    CK(cudaGetLastError());
    ctx->launches++;
    CK(cudaStreamSynchronize(st));
    return 0;
}

// ---------------------------------------------------------------------------
// inverses: trtri, lauum, potri on the device tiles (lower, padded), in place
// ---------------------------------------------------------------------------
// first zero pivot of the diagonal (1-based, 0 if none): LAPACK dtrtri INFO
__global__ void ag_zero_pivot(const double *L, int ld, int n, int *info)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (L[(int64_t)i * ld + i] == 0.0) atomicMin(info, i + 1);
}

// op: 0 trtri (L -> L^-1), 1 lauum (L -> L^T L), 2 potri (L -> (L L^T)^-1), on whole
// tiles (work_geom: nb == nbi, row i of the caller is row i of the tiles).
// gr (op 2, may be null): the GP gradient is written instead of Lt.
static int inverse_or_gradient(Context *ctx, double *Lt, const Geom &g, int op, int unit, int *info, const AgGrad *gr)
{
    const int Np = g.mt * g.nbi, P = Np / AG_T, ld = Np;
    const size_t nn = (size_t)Np * Np;
    double *D = (double *)ctx->buffer(BUF_ADJ, 4 * nn * sizeof(double) + (size_t)P * AG_T * AG_T * sizeof(double));
    if (!D) return DPLASMA_ERR_OUT_OF_RESOURCES;
    double *L = D, *W = D + nn, *Y = D + 2 * nn, *scr = D + 4 * nn;
    cudaStream_t st = ctx->stream;
    int rc;
    const dim3 tg(g.mt, g.mt, (g.nbi / AG_M) * (g.nbi / AG_M));
    ag_move<true><<<tg, 256, 0, st>>>(Lt, g.mt, g.nbi, L, ld);
    CK(cudaGetLastError());
    ctx->launches++;
    *info = 0;
    if (op != 1 && !unit) {
        int *dinfo = (int *)(scr);
        const int big = 0x7fffffff;
        CK(cudaMemcpyAsync(dinfo, &big, sizeof(int), cudaMemcpyHostToDevice, st));
        ag_zero_pivot<<<ctx->sms, 256, 0, st>>>(L, ld, g.n, dinfo);
        CK(cudaGetLastError());
        int h = big;
        CK(cudaMemcpyAsync(&h, dinfo, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        ctx->launches++;
        if (h != big) {
            *info = h;
            return 0;
        }
    }
    const double *src = L;
    if (op != 1) {
        if ((rc = ag_inverse(ctx, L, W, Y, scr, P, ld, unit))) return rc;
        src = W;
    }
    if (gr) {
        if ((rc = ag_gemm(ctx, AG_GRAD, P, 0, W, ld, 1, W, ld, Y, ld, 1.0, gr))) return rc;
        CK(cudaStreamSynchronize(st));
        return 0;
    }
    double *out = W;
    if (op != 0) {
        // src^T src, lower tiles only (k >= i >= j): the result is symmetric
        if ((rc = ag_gemm(ctx, AG_LOWER_KGE_I, P, 0, src, ld, 1, src, ld, Y, ld, 1.0))) return rc;
        out = Y;
    }
    ag_move<false><<<tg, 256, 0, st>>>(Lt, g.mt, g.nbi, out, ld);
    CK(cudaGetLastError());
    ctx->launches++;
    CK(cudaStreamSynchronize(st));
    return 0;
}

int inverse_tiles(Context *ctx, double *Lt, const Geom &g, int op, int unit, int *info)
{
    return inverse_or_gradient(ctx, Lt, g, op, unit, info, nullptr);
}

// al^T (row l of alt's K is column l of al), zero beyond n rows and nal columns
__global__ void __launch_bounds__(256) ag_transpose_pad(const double *al, int n, int nal, double *alt, int nk, int np)
{
    __shared__ double sm[32][33];
    const int r0 = blockIdx.x * 32, l0 = blockIdx.y * 32, x = threadIdx.x & 31;
    for (int y = threadIdx.x >> 5; y < 32; y += 8)
        sm[y][x] = r0 + x < n && l0 + y < nal ? al[(int64_t)(l0 + y) * n + r0 + x] : 0.0;
    __syncthreads();
    for (int y = threadIdx.x >> 5; y < 32; y += 8)
        if (r0 + y < np && l0 + x < nk) alt[(int64_t)(r0 + y) * nk + l0 + x] = sm[x][y];
}

// Columns of al from which al al^T is a product of its own.  In the epilogue each
// column costs two loads and a multiply-add per element outside the tensor cores;
// gradient of n = 4096 with 1 / 4 / 64 / 1024 columns, ms: in the epilogue 2.42 /
// 2.66 / 2.84 / 8.04, as a product 2.45 / 2.41 / 2.50 / 3.04 (n = 1000: 0.68 / 0.73 /
// 0.83 / 2.07 and 0.68 / 0.68 / 0.69 / 0.83).
constexpr int AG_GRAD_COLS = 4;
int gp_gradient_tiles(Context *ctx, double *Lt, const Geom &g, const double *al, int nal, const double *dg, double *out,
                      int *info)
{
    AgGrad gr = {al, dg, nal, g.n, out, nullptr, 0};
    if (nal >= AG_GRAD_COLS) {
        const int np = g.mt * g.nbi;
        gr.nk = (nal + AG_K - 1) / AG_K * AG_K;
        double *alt = (double *)ctx->buffer(BUF_B, (size_t)np * gr.nk * sizeof(double));
        if (!alt) return DPLASMA_ERR_OUT_OF_RESOURCES;
        ag_transpose_pad<<<dim3(np / 32, (gr.nk + 31) / 32), 256, 0, ctx->stream>>>(al, g.n, nal, alt, gr.nk, np);
        CK(cudaGetLastError());
        ctx->launches++;
        gr.alt = alt;
    }
    return inverse_or_gradient(ctx, Lt, g, 2, 0, info, &gr);
}

}  // namespace db2
