// dev_chol32.cuh -- factorization of a 32x32 diagonal block by one warp and
// substitution with it (FP64 for the tile Cholesky, FP64 or FP32 for the batched
// solver).
#pragma once
#include <cuda_runtime.h>

namespace db2 {

__device__ __forceinline__ double c32_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float c32_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double c32_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float c32_rsqrt(float x) { return rsqrtf(x); }

// four consecutive values, 16-byte aligned, as vector accesses
__device__ __forceinline__ void c32_load4(const double *p, double (&v)[4])
{
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}
__device__ __forceinline__ void c32_load4(const float *p, float (&v)[4])
{
    const float4 a = *reinterpret_cast<const float4 *>(p);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = a.z;
    v[3] = a.w;
}
// 16 bytes
__device__ __forceinline__ void c32_loadv(const double *p, double (&v)[2])
{
    const double2 a = *reinterpret_cast<const double2 *>(p);
    v[0] = a.x;
    v[1] = a.y;
}
__device__ __forceinline__ void c32_loadv(const float *p, float (&v)[4]) { c32_load4(p, v); }
__device__ __forceinline__ void c32_store4(double *p, const double (&v)[4])
{
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void c32_store4(float *p, const float (&v)[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// Cholesky of a 32x32 block by one warp, lane i owning row i, in steps of
// four columns.  The row lives in registers in a frame that rotates by four
// columns per step (d[c] = A(i, J + c) at step J), so the rolled loop body
// uses compile-time register indices (POTRF runs once per step on one SM
// between update tasks; a fully unrolled form is thousands of instructions
// executed once each, paced by instruction fetch).  Per step: every lane
// gathers the 4x4 diagonal block by shuffles and factors it redundantly, forms
// its row of the 4-column panel, publishes it in the blocked copy Lb
// ([8][32][4]: Lb[J/4][i][k] = L(i, J+k)), and applies the rank-4 update to
// its remaining columns, reading the panel rows back from Lb with 16-byte
// broadcasts.  Every element receives the operations of LAPACK dpotf2's
// right-looking order (the same subtractions in the same order).  sqrt and
// 1/sqrt are independent, so a pivot costs one of them rather than a square
// root and a division.  A non-positive pivot (or NaN) marks the column and
// the remaining steps run on harmless values.  Returns the first failing
// column or -1; rdiag (lane j) = 1 / L(j,j).
template <typename T>
__device__ __forceinline__ int chol32_blk(T (&d)[32], int lane, T &rdiag, T *Lb)
{
    int failcol = -1;
#pragma unroll 1
    for (int J = 0; J < 32; J += 4) {
        T a[4][4], l[4][4], rr[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c <= r; ++c) a[r][c] = __shfl_sync(0xffffffffu, d[c], J + r);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            T piv = a[j][j];
            if (!(piv > T(0))) {   // LAPACK dpotf2: ajj <= 0 or NaN stops the factorization
                if (failcol < 0) failcol = J + j;
                piv = T(1);
            }
            l[j][j] = c32_sqrt(piv);
            rr[j] = c32_rsqrt(piv);
#pragma unroll
            for (int r = j + 1; r < 4; ++r) l[r][j] = a[r][j] * rr[j];
#pragma unroll
            for (int c = j + 1; c < 4; ++c)
#pragma unroll
                for (int r = c; r < 4; ++r) a[r][c] -= l[r][j] * l[c][j];
        }
        // this lane's row of the 4-column panel
        const int rb = lane - J;
        T x[4];
        {
            T y1 = d[1], y2 = d[2], y3 = d[3];
            x[0] = d[0] * rr[0];
            y1 -= x[0] * l[1][0];
            y2 -= x[0] * l[2][0];
            y3 -= x[0] * l[3][0];
            x[1] = y1 * rr[1];
            y2 -= x[1] * l[2][1];
            y3 -= x[1] * l[3][1];
            x[2] = y2 * rr[2];
            y3 -= x[2] * l[3][2];
            x[3] = y3 * rr[3];
        }
        if (rb < 0) {
#pragma unroll
            for (int c = 0; c < 4; ++c) x[c] = T(0);            // above the block: upper part of L
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (rb == r) {
#pragma unroll
                for (int c = 0; c < 4; ++c) x[c] = (c <= r) ? l[r][c] : T(0);
                rdiag = rr[r];
            }
        c32_store4(Lb + ((J >> 2) * 32 + lane) * 4, x);
        __syncwarp();
        // rank-4 update of the columns J+4.. (the values of lanes above the
        // diagonal are never read)
        const T *Lr = Lb + (J >> 2) * 128;
#pragma unroll
        for (int c0 = 4; c0 < 32; c0 += 4) {
            if (J + c0 < 32) {
#pragma unroll
                for (int c = c0; c < c0 + 4; ++c) {
                    T v[4];
                    c32_load4(Lr + (J + c) * 4, v);
                    d[c] -= x[0] * v[0];
                    d[c] -= x[1] * v[1];
                    d[c] -= x[2] * v[2];
                    d[c] -= x[3] * v[3];
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 28; ++c) d[c] = d[c + 4];
    }
    return failcol;
}

// ---------------------------------------------------------------------------
// The latency form, column by column: 5,400 cycles for FP64 against 11,400 of
// chol32_blk (6,400 with a load per value of the last column); 2,000 for a sweep
// against 4,900 of an inverse in steps of four rows.
// ---------------------------------------------------------------------------
// the pivots for which the branch-free root is good
template <typename T>
struct c32_range;
template <>
struct c32_range<double> {
    static constexpr double lo = 1e-280, hi = 1e280;
};
template <>
struct c32_range<float> {
    static constexpr float lo = 1e-30f, hi = 1e30f;
};
// Columns per unrolled body: 16 is the fastest alone but its code is four times as
// long, and every caller runs it between other code: the factorizations are alike
// for 4, 8 and 16 and the batched solver is 5 to 15 % faster with 4.
constexpr int C32_U = 4;
constexpr int C32_RD = 1024;        // 1 / diagonal, 32 values behind the blocked copy
constexpr int C32_CB = 1024 + 32;   // the last two columns, 48 values each (rows past the block are read)
constexpr int C32_LB = C32_CB + 96;
// 1 / sqrt(x) without a branch, x within the range the caller checks: the
// hardware's approximation and two Newton steps y += y (1/2 - x/2 y^2).
__device__ __forceinline__ float rsqrt_newton(float x) { return rsqrtf(x); }
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
template <typename T, int LIVE, bool VEC>
__device__ __forceinline__ void chol32_half(T (&d)[32], int J0, int lane, T &dg, T &lp, T &piv, T &rdiag, bool &ok,
                                            T *Sd, int sp, T *Lb)
{
    T *Cb = Lb + C32_CB;
    constexpr int V = 16 / sizeof(T);
    static_assert(C32_U == 4, "column j0 + u starts at the vector boundary u & (V - 1)");
#pragma unroll 1
    for (int j0 = J0; j0 < J0 + 16; j0 += C32_U)
#pragma unroll
    for (int u = 0; u < C32_U; ++u) {
        const int j = j0 + u;
        // what the next pivot needs from lane j + 1, before the pivot's root is known
        const T dn = __shfl_sync(0xffffffffu, dg, j + 1);       // its diagonal entry
        const T an = __shfl_sync(0xffffffffu, d[0], j + 1);     // A(j+1, j)
        ok = ok && piv > c32_range<T>::lo && piv < c32_range<T>::hi;
        const T r = rsqrt_newton(piv);
        // column j - 1 applied to the columns beyond j
        if (j > 0) {
            // (rows past the block, k >= 32 - j, feed columns that are never used)
            if (VEC) {
                // from its contiguous copy, 16 bytes a load
                const T *Lp = Cb + ((u + 1) & 1) * 48 + j0;
#pragma unroll
                for (int r = (u + 1) / V * V; r < u + LIVE; r += V) {
                    T v[V];
                    c32_loadv(Lp + r, v);
#pragma unroll
                    for (int e = 0; e < V; ++e)
                        if (r + e > u && r + e < u + LIVE) d[r + e - u] = fma(-lp, v[e], d[r + e - u]);
                }
            } else {
                const T *Lp = Lb + ((j - 1) >> 2) * 128 + j * 4 + ((j - 1) & 3);
#pragma unroll
                for (int k = 1; k < LIVE; ++k) d[k] = fma(-lp, Lp[4 * k], d[k]);
            }
        }
        const T ln = an * r;                                     // L(j+1, j)
        const T pn = fma(-ln, ln, dn);
        T l = d[0] * r;
        const T s = fma(fma(-l, l, piv), T(0.5) * r, l);            // lane j: sqrt, corrected
        dg = fma(-l, l, dg);
        const T d0 = fma(-l, ln, d[1]);
        if (lane == j) {
            l = s;
            rdiag = r;
        }
        if (Sd && lane >= j) Sd[j * sp + lane] = l;
        if (VEC) Cb[(u & 1) * 48 + lane] = l;
        Lb[(j >> 2) * 128 + lane * 4 + (j & 3)] = lane >= j ? l : T(0);
        __syncwarp();
        lp = l;
        piv = pn;
#pragma unroll
        for (int k = 1; k < LIVE - 1; ++k) d[k] = d[k + 1];
        d[0] = d0;
    }
}

// Cholesky factor of a 32x32 block by one warp, lane i owning row i (d[c] =
// A(i, c), zero above the diagonal): the blocked copy Lb ([8][32][4], C32_LB
// values), rd[c] = 1 / L(c,c) (may lie behind the copy, C32_RD) and, unless Sd
// is null, the lower triangle at Sd (column c, row r at c * sp + r).  Returns
// false when a pivot leaves the range in which the branch-free root is good (or
// is not positive): the results are then useless.
// VEC: 5,400 cycles (FP64) against 6,400; the FP64 scheduler kernel goes without, as
// the loads' registers made it spill 196 bytes instead of 20 (a POTRF 36.7 us
// against 34.5).
template <typename T, bool VEC = true>
__device__ __forceinline__ bool chol32_col(T (&d)[32], int lane, T *Sd, int sp, T *Lb, T *rd)
{
    T dg = T(0), lp = T(0), rdiag = T(0);
#pragma unroll
    for (int c = 0; c < 32; ++c)
        if (lane == c) dg = d[c];
    T piv = __shfl_sync(0xffffffffu, dg, 0);
    bool ok = true;
    chol32_half<T, 32, VEC>(d, 0, lane, dg, lp, piv, rdiag, ok, Sd, sp, Lb);
    chol32_half<T, 16, VEC>(d, 16, lane, dg, lp, piv, rdiag, ok, Sd, sp, Lb);
    rd[lane] = rdiag;
    __syncwarp();
    return ok;
}

// Four of the eight steps of sweep32, columns J0 .. J0+15; LIVE columns of the
// frame (b[c] = b_{j+c} at step j) are kept up to date, those past the block
// with values that are never used.
template <typename T, int LIVE, class Out>
__device__ __forceinline__ void sweep32_half(const T *Lb, const T *rd, T (&b)[32], int J0, Out &out)
{
#pragma unroll 1
    for (int j = J0; j < J0 + 16; j += 4) {
        const T *Lk = Lb + (j >> 2) * 128 + j * 4;
        T r4[4];
        c32_load4(rd + j, r4);
        const T l10 = Lk[4], l20 = Lk[8], l21 = Lk[9], l30 = Lk[12], l31 = Lk[13], l32 = Lk[14];
        T x[4];
        x[0] = b[0] * r4[0];
        x[1] = (b[1] - l10 * x[0]) * r4[1];
        b[2] -= l20 * x[0];
        b[3] -= l30 * x[0];
        x[2] = (b[2] - l21 * x[1]) * r4[2];
        b[3] -= l31 * x[1];
        x[3] = (b[3] - l32 * x[2]) * r4[3];
#pragma unroll
        for (int c = 4; c < LIVE; ++c) {
            T v[4];
            c32_load4(Lk + c * 4, v);
            T s = v[0] * x[0];
            s += v[1] * x[1];
            s += v[2] * x[2];
            s += v[3] * x[3];
            b[c - 4] = b[c] - s;               // one rounding at the size of b per four columns
        }
        // (after the loads of this step, which could not pass the stores)
#pragma unroll
        for (int r = 0; r < 4; ++r) out(j + r, x[r]);
    }
}
// Solve L x = b for one right-hand side per lane (b[c], c = 0..31), L in the
// blocked copy Lb and rd[c] = 1 / L(c,c), four columns per step in a rotating
// frame; out(c, x) receives x_c, c ascending.  Two rolled halves: 2,000 cycles
// as when fully unrolled, in a third of the code.
template <typename T, class Out>
__device__ __forceinline__ void sweep32(const T *Lb, const T *rd, T (&b)[32], Out out)
{
    sweep32_half<T, 32>(Lb, rd, b, 0, out);
    sweep32_half<T, 16>(Lb, rd, b, 16, out);
}

// The same for right-hand sides that lie in shared memory (in(c) = b_c, read when
// column c is reached): the frame holds the sums s_c = sum_k L(c,k) x_k from zero,
// x_c = b_c / L(c,c) - s_c / L(c,c), so no product is rounded at the size of b and
// nothing is added to the chain.
template <typename T, int LIVE, class In, class Out>
__device__ __forceinline__ void sweep32_sums_half(const T *Lb, const T *rd, T (&s)[32], int J0, In &in, Out &out)
{
#pragma unroll 1
    for (int j = J0; j < J0 + 16; j += 4) {
        const T *Lk = Lb + (j >> 2) * 128 + j * 4;
        T r4[4], br[4];
        c32_load4(rd + j, r4);
#pragma unroll
        for (int r = 0; r < 4; ++r) br[r] = in(j + r) * r4[r];
        const T l10 = Lk[4], l20 = Lk[8], l21 = Lk[9], l30 = Lk[12], l31 = Lk[13], l32 = Lk[14];
        T x[4];
        x[0] = fma(-s[0], r4[0], br[0]);
        x[1] = fma(-fma(l10, x[0], s[1]), r4[1], br[1]);
        s[2] = fma(l20, x[0], s[2]);
        s[3] = fma(l30, x[0], s[3]);
        x[2] = fma(-fma(l21, x[1], s[2]), r4[2], br[2]);
        s[3] = fma(l31, x[1], s[3]);
        x[3] = fma(-fma(l32, x[2], s[3]), r4[3], br[3]);
#pragma unroll
        for (int c = 4; c < LIVE; ++c) {
            T v[4];
            c32_load4(Lk + c * 4, v);
            T y = s[c];
            y = fma(v[0], x[0], y);
            y = fma(v[1], x[1], y);
            y = fma(v[2], x[2], y);
            s[c - 4] = fma(v[3], x[3], y);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) out(j + r, x[r]);
    }
}
template <typename T, class In, class Out>
__device__ __forceinline__ void sweep32_sums(const T *Lb, const T *rd, In in, Out out)
{
    T s[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) s[c] = T(0);
    sweep32_sums_half<T, 32>(Lb, rd, s, 0, in, out);
    sweep32_sums_half<T, 16>(Lb, rd, s, 16, in, out);
}

}  // namespace db2
