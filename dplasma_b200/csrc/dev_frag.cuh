// dev_frag.cuh -- one warp's FP64 tensor-core products on fragments of 16 x 8
// blocks: 32-deep multiply-accumulate from strided operands (shared or global
// memory) and moves between fragments and memory.
#pragma once
#include "dev_common.cuh"

namespace db2 {

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
// element (r, c) at p[r * rs + c * cs] -= acc
template <int MI, int NI>
__device__ __forceinline__ void frag_sub(const double (&acc)[MI][NI][4], double *p, int rs, int cs, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mi = 0; mi < MI; ++mi) {
        double old[NI][4];             // the loads may not pass the stores
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                old[ni][q] = p[(mi * 16 + g + ((q & 2) ? 8 : 0)) * rs + (ni * 8 + 2 * t + (q & 1)) * cs];
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                p[(mi * 16 + g + ((q & 2) ? 8 : 0)) * rs + (ni * 8 + 2 * t + (q & 1)) * cs] = old[ni][q] - acc[mi][ni][q];
    }
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

}  // namespace db2
