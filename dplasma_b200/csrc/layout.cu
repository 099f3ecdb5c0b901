// layout.cu -- moves matrices between the caller's descriptor layout (TILE
// or LAPACK storage, host or device) and the device tile layout the kernels
// use, and the seeded generators dplasma_dplgsy / dplasma_dplrnt.
#include <cuda_runtime.h>
#include <string.h>

#include "dev_common.cuh"
#include "internal.h"

namespace db2 {

Geom make_geom(int n, int nb)
{
    Geom g;
    g.n = n;
    g.nb = nb;
    g.nbi = ((nb + 127) / 128) * 128;
    g.mt = (n + nb - 1) / nb;
    return g;
}

// Tiles of 128 where the caller's edge is no multiple of it (the matrix is
// copied anyway): padded tile by tile, an edge of 93 costs (128/93)^3 = 2.6 times
// the flops and 1.4 times the steps of the chain, 320 (384/320)^3 = 1.7 times
// (N = 378 in 93-wide tiles: 5 steps, 0.37 ms, now 3, 0.22 ms; N = 7000 in
// 320-wide ones: 9.0 ms, now 5.8 ms).
Geom work_geom(int n, int nb) { return make_geom(n, nb % 128 == 0 ? nb : 128); }

// ---------------------------------------------------------------------------
// caller layout description, usable on the device
// ---------------------------------------------------------------------------
struct DescView {
    double *mat;
    int storage;   // PARSEC_MATRIX_TILE / PARSEC_MATRIX_LAPACK
    int sym;       // 0 whole grid, 1 lower tiles packed, 2 upper tiles packed
    int mb, nb, lmt, lda;
    int m, n, mt, nt;
    int64_t bsiz;
};

static DescView view_of(const parsec_tiled_matrix_t *A, double *mat)
{
    DescView v;
    v.mat = mat;
    v.storage = A->storage;
    v.sym = (A->storage == PARSEC_MATRIX_TILE) ? (A->uplo == dplasmaLower ? 1 : (A->uplo == dplasmaUpper ? 2 : 0)) : 0;
    v.mb = A->mb;
    v.nb = A->nb;
    v.lmt = A->lmt;
    v.lda = A->lda;
    v.m = A->m;
    v.n = A->n;
    v.mt = A->mt;
    v.nt = A->nt;
    v.bsiz = (int64_t)A->bsiz;
    return v;
}

__host__ __device__ __forceinline__ int64_t view_tile_offset(const DescView &v, int m, int n)
{
    if (v.storage == PARSEC_MATRIX_LAPACK) return (int64_t)m * v.mb + (int64_t)n * v.nb * v.lda;
    if (v.sym == 1) return (m < n) ? -1 : ((int64_t)n * v.lmt - ((int64_t)n * (n - 1)) / 2 + (m - n)) * v.bsiz;
    if (v.sym == 2) return (m > n) ? -1 : (((int64_t)n * (n + 1)) / 2 + m) * v.bsiz;
    return ((int64_t)m + (int64_t)n * v.lmt) * v.bsiz;
}
__host__ __device__ __forceinline__ int view_ld(const DescView &v) { return v.storage == PARSEC_MATRIX_LAPACK ? v.lda : v.mb; }

int64_t tile_offset(const parsec_tiled_matrix_t *A, int m, int n)
{
    DescView v = view_of(A, nullptr);
    return view_tile_offset(v, m, n);
}

size_t desc_elems(const parsec_tiled_matrix_t *A)
{
    if (A->storage == PARSEC_MATRIX_LAPACK) return (size_t)A->lda * (size_t)A->ln;
    return A->bsiz * A->nb_local_tiles;
}

// Element (r,c) of internal tile `idx` = (m,n), m >= n.  Thread block per tile.
__device__ __forceinline__ void tile_of_index(int64_t idx, int mt, int &m, int &n)
{
    // column n holds mt - n tiles
    int nn = 0;
    int64_t rem = idx;
    // binary search on the column start offset
    int lo = 0, hi = mt - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) / 2;
        int64_t start = (int64_t)mid * mt - ((int64_t)mid * (mid - 1)) / 2;
        if (start <= idx) lo = mid; else hi = mid - 1;
    }
    nn = lo;
    rem = idx - ((int64_t)nn * mt - ((int64_t)nn * (nn - 1)) / 2);
    n = nn;
    m = nn + (int)rem;
}

// Caller's storage <-> device tiles, TO the tiles or back.  Internal tile (m,n)
// element (r,c) is matrix element (i,j) = (m nb + r, n nb + c), whatever the
// caller's own tile edge; only i >= j is moved (the stored triangle; upper
// storage holds its mirror (j,i)).  The rest of a diagonal tile is zero and the
// padding the identity.  One CTA per 64x64 piece, sixteen elements a thread;
// an upper matrix is transposed through shared memory so that both sides are
// read and written in runs of 64.  (One CTA per tile with an index division per
// element took 137 us for N = 4096 in 256-wide tiles, 378 for the strided side
// of an upper N = 7000.)
constexpr int LM = 64;
__device__ __forceinline__ int64_t view_elem(const DescView &v, int a, int b)
{
    if (v.storage == PARSEC_MATRIX_LAPACK) return (int64_t)b * v.lda + a;
    const int ta = a / v.mb, tb = b / v.nb;
    return view_tile_offset(v, ta, tb) + (a - ta * v.mb) + (int64_t)(b - tb * v.nb) * v.mb;
}

template <bool TO>
__global__ void __launch_bounds__(256) sym_move_kernel(DescView v, int upper, int n_user, int nb, int nbi, int mt,
                                                       double *dA)
{
    __shared__ double sm[LM][LM + 1];
    int m, n;
    tile_of_index(blockIdx.x, mt, m, n);
    const int per = nbi / LM, r0 = (blockIdx.y % per) * LM, c0 = (blockIdx.y / per) * LM;
    const int tm = (m == mt - 1) ? n_user - m * nb : nb;
    const int tn = (n == mt - 1) ? n_user - n * nb : nb;
    double *T = dA + (int64_t)blockIdx.x * nbi * nbi + (int64_t)c0 * nbi + r0;
    const int x = threadIdx.x & (LM - 1), y = threadIdx.x / LM;
    constexpr int NY = 256 / LM;
    // element (r, c) of the piece: moved, or what the tile holds instead
    auto moved = [&](int r, int c) { return r0 + r < tm && c0 + c < tn && m * nb + r0 + r >= n * nb + c0 + c; };
    auto filler = [&](int r, int c) {
        return m == n && r0 + r == c0 + c && !(r0 + r < tm && c0 + c < tn) ? 1.0 : 0.0;
    };
    if (!upper) {
        const int i = m * nb + r0 + x;
#pragma unroll 8
        for (int c = y; c < LM; c += NY) {
            const int j = n * nb + c0 + c;
            if (TO) T[(int64_t)c * nbi + x] = moved(x, c) ? v.mat[view_elem(v, i, j)] : filler(x, c);
            else if (moved(x, c)) v.mat[view_elem(v, i, j)] = T[(int64_t)c * nbi + x];
        }
        return;
    }
    // caller's side: runs along c (rows of its column i)
    if (TO) {
#pragma unroll 8
        for (int r = y; r < LM; r += NY)
            sm[x][r] = moved(r, x) ? v.mat[view_elem(v, n * nb + c0 + x, m * nb + r0 + r)] : filler(r, x);
        __syncthreads();
#pragma unroll 8
        for (int c = y; c < LM; c += NY) T[(int64_t)c * nbi + x] = sm[c][x];
    } else {
#pragma unroll 8
        for (int c = y; c < LM; c += NY) sm[c][x] = T[(int64_t)c * nbi + x];
        __syncthreads();
#pragma unroll 8
        for (int r = y; r < LM; r += NY)
            if (moved(r, x)) v.mat[view_elem(v, n * nb + c0 + x, m * nb + r0 + r)] = sm[x][r];
    }
}

template <bool TO>
static int sym_move(Context *ctx, const DescView &v, dplasma_enum_t uplo, const Geom &g, double *dA)
{
    const int per = g.nbi / LM;
    sym_move_kernel<TO><<<dim3((unsigned)g.ntiles(), per * per), 256, 0, ctx->stream>>>(v, uplo == dplasmaUpper, g.n,
                                                                                       g.nb, g.nbi, g.mt, dA);
    CK(cudaGetLastError());
    ctx->launches++;
    return 0;
}

static bool fast_path(const parsec_tiled_matrix_t *A, dplasma_enum_t uplo, const Geom &g)
{
    return A->storage == PARSEC_MATRIX_TILE && A->uplo == dplasmaLower && uplo == dplasmaLower &&
           g.nbi == g.nb && g.nb == A->mb && (g.n % g.nb) == 0 && A->lmt == g.mt && A->mb == A->nb;
}

int upload_sym(Context *ctx, const parsec_tiled_matrix_t *A, dplasma_enum_t uplo, const Geom &g, double *dA)
{
    cudaStream_t st = ctx->stream;
    const size_t bytes = desc_elems(A) * sizeof(double);
    if (fast_path(A, uplo, g)) {
        CK(cudaMemcpyAsync(dA, A->mat, g.elems() * sizeof(double),
                           A->location == DPLASMA_B200_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, st));
        return 0;
    }
    double *src = (double *)A->mat;
    if (A->location != DPLASMA_B200_DEVICE) {
        src = (double *)ctx->buffer(BUF_STAGE, bytes);
        if (!src) return DPLASMA_ERR_OUT_OF_RESOURCES;
        CK(cudaMemcpyAsync(src, A->mat, bytes, cudaMemcpyHostToDevice, st));
    }
    return sym_move<true>(ctx, view_of(A, src), uplo, g, dA);
}

int download_sym(Context *ctx, parsec_tiled_matrix_t *A, dplasma_enum_t uplo, const Geom &g, const double *dA)
{
    cudaStream_t st = ctx->stream;
    const size_t bytes = desc_elems(A) * sizeof(double);
    if (fast_path(A, uplo, g)) {
        CK(cudaMemcpyAsync(A->mat, dA, g.elems() * sizeof(double),
                           A->location == DPLASMA_B200_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        return 0;
    }
    double *dst = (double *)A->mat;
    if (A->location != DPLASMA_B200_DEVICE) dst = (double *)ctx->buffer(BUF_STAGE, 0);   // filled by upload_sym
    const int rc = sym_move<false>(ctx, view_of(A, dst), uplo, g, const_cast<double *>(dA));
    if (rc) return rc;
    if (A->location != DPLASMA_B200_DEVICE) CK(cudaMemcpyAsync(A->mat, dst, bytes, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return 0;
}

// ---------------------------------------------------------------------------
// right-hand sides: caller N x NRHS matrix <-> padded column-major npad x nrhs
// ---------------------------------------------------------------------------
// Device right-hand sides live in the padded row space of the tiles: row
// m*nbi + r holds global row m*nb + r for r < (rows of tile m), zero otherwise.
__global__ void rhs_in_kernel(DescView src, int nb, int nbi, int npad, int nrhs, double *dB)
{
    const int64_t total = (int64_t)npad * nrhs;
    const int ld = view_ld(src);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int ip = (int)(e % npad), j = (int)(e / npad);
        const int t = ip / nbi, r = ip % nbi;
        const int64_t i = (int64_t)t * nb + r;
        double v = 0.0;
        if (r < nb && i < src.m && j < src.n) {
            const int64_t off = view_tile_offset(src, (int)(i / src.mb), j / src.nb);
            v = src.mat[off + (i % src.mb) + (int64_t)(j % src.nb) * ld];
        }
        dB[e] = v;
    }
}
__global__ void rhs_out_kernel(DescView dst, int nb, int nbi, int npad, int nrhs, const double *dB)
{
    const int64_t total = (int64_t)npad * nrhs;
    const int ld = view_ld(dst);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int ip = (int)(e % npad), j = (int)(e / npad);
        const int t = ip / nbi, r = ip % nbi;
        const int64_t i = (int64_t)t * nb + r;
        if (r < nb && i < dst.m && j < dst.n) {
            const int64_t off = view_tile_offset(dst, (int)(i / dst.mb), j / dst.nb);
            dst.mat[off + (i % dst.mb) + (int64_t)(j % dst.nb) * ld] = dB[e];
        }
    }
}

int upload_rhs(Context *ctx, const parsec_tiled_matrix_t *B, int nb, int nbi, int npad, int nrhs, double *dB)
{
    cudaStream_t st = ctx->stream;
    double *src = (double *)B->mat;
    if (B->location != DPLASMA_B200_DEVICE) {
        const size_t bytes = desc_elems(B) * sizeof(double);
        src = (double *)ctx->buffer(BUF_BSTAGE, bytes);
        if (!src) return DPLASMA_ERR_OUT_OF_RESOURCES;
        CK(cudaMemcpyAsync(src, B->mat, bytes, cudaMemcpyHostToDevice, st));
    }
    DescView v = view_of(B, src);
    rhs_in_kernel<<<ctx->sms * 4, 256, 0, st>>>(v, nb, nbi, npad, nrhs, dB);
    CK(cudaGetLastError());
    ctx->launches++;
    return 0;
}

int download_rhs(Context *ctx, parsec_tiled_matrix_t *B, int nb, int nbi, int npad, int nrhs, const double *dB)
{
    cudaStream_t st = ctx->stream;
    double *dst = (B->location != DPLASMA_B200_DEVICE) ? (double *)ctx->buffer(BUF_BSTAGE, desc_elems(B) * sizeof(double))
                                                       : (double *)B->mat;
    if (!dst) return DPLASMA_ERR_OUT_OF_RESOURCES;
    DescView v = view_of(B, dst);
    rhs_out_kernel<<<ctx->sms * 4, 256, 0, st>>>(v, nb, nbi, npad, nrhs, dB);
    CK(cudaGetLastError());
    ctx->launches++;
    if (B->location != DPLASMA_B200_DEVICE)
        CK(cudaMemcpyAsync(B->mat, dst, desc_elems(B) * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return 0;
}

// ---------------------------------------------------------------------------
// Generators.  64-bit LCG with jump-ahead (src/cores/random.h:19-41); each
// value is formed in single precision, `0.5f - ran * RndF_Mul`
// (src/cores/core_zplgsy.c:89), with the conversion, multiply and subtract
// each rounded to nearest (no contraction), then stored as double.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t rnd64_jump(uint64_t n, uint64_t seed)
{
    uint64_t a_k = 6364136223846793005ULL, c_k = 1ULL, ran = seed;
    while (n) {
        if (n & 1ULL) ran = a_k * ran + c_k;
        c_k *= (a_k + 1ULL);
        a_k *= a_k;
        n >>= 1;
    }
    return ran;
}
__device__ __forceinline__ uint64_t rnd64_next(uint64_t ran) { return 6364136223846793005ULL * ran + 1ULL; }
__device__ __forceinline__ double rnd_value(uint64_t ran)
{
    const float r = __ull2float_rn(ran);
    const float p = __fmul_rn(r, 5.4210108624275222e-20f);
    return (double)__fsub_rn(0.5f, p);
}

constexpr int GEN_CHUNK = 32;

// One thread per (tile column, chunk of GEN_CHUNK rows) of every generated
// tile.  sym != 0: symmetric (dplgsy), value(i,j) from jump max(i,j) +
// min(i,j)*gM, bump on the diagonal.  sym == 0: general (dplrnt), value(i,j)
// from jump i + j*gM, `bump` added on the local diagonal of tiles (m,m).
__global__ void gen_kernel(DescView d, int sym, int region, double bump, uint64_t seed, int gM)
{
    const int ext = max(d.mb, d.nb);
    const int chunks = (ext + GEN_CHUNK - 1) / GEN_CHUNK;
    const int64_t per_tile = (int64_t)chunks * ext;
    const int64_t total = per_tile * d.mt * d.nt;
    const int ld = view_ld(d);
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
        const int64_t tile = w / per_tile;
        const int rem = (int)(w % per_tile);
        const int a = rem / chunks, ch = rem % chunks;
        const int m = (int)(tile % d.mt), n = (int)(tile / d.mt);
        if (region == dplasmaLower && m < n) continue;
        if (region == dplasmaUpper && m > n) continue;
        const int tm = (m == d.mt - 1) ? d.m - m * d.mb : d.mb;
        const int tn = (n == d.nt - 1) ? d.n - n * d.nb : d.nb;
        const int64_t off = view_tile_offset(d, m, n);
        if (off < 0) continue;
        double *T = d.mat + off;
        const int64_t i0 = (int64_t)m * d.mb, j0 = (int64_t)n * d.nb;
        if (sym && i0 + tm <= j0) {
            // tile strictly above the diagonal: value(i,j) = LCG at j + i*gM,
            // consecutive along a row -> walk row `a`, columns of chunk ch
            const int r = a, c0 = ch * GEN_CHUNK;
            if (r >= tm || c0 >= tn) continue;
            const int c1 = min(tn, c0 + GEN_CHUNK);
            uint64_t ran = rnd64_jump((uint64_t)(j0 + c0) + (uint64_t)(i0 + r) * (uint64_t)gM, seed);
            for (int c = c0; c < c1; ++c) {
                T[r + (int64_t)c * ld] = rnd_value(ran);
                ran = rnd64_next(ran);
            }
            continue;
        }
        const int c = a, r0 = ch * GEN_CHUNK;
        if (c >= tn || r0 >= tm) continue;
        const int r1 = min(tm, r0 + GEN_CHUNK);
        double *col = T + (int64_t)c * ld;
        const int64_t j = j0 + c;
        if (!sym) {
            uint64_t ran = rnd64_jump((uint64_t)(i0 + r0) + (uint64_t)j * (uint64_t)gM, seed);
            for (int r = r0; r < r1; ++r) {
                double v = rnd_value(ran);
                if (m == n && r == c) v += bump;
                col[r] = v;
                ran = rnd64_next(ran);
            }
        } else {
            // rows above the diagonal: mirrored values, one jump each
            int r = r0;
            for (; r < r1 && i0 + r < j; ++r)
                col[r] = rnd_value(rnd64_jump((uint64_t)j + (uint64_t)(i0 + r) * (uint64_t)gM, seed));
            if (r < r1) {
                uint64_t ran = rnd64_jump((uint64_t)(i0 + r) + (uint64_t)j * (uint64_t)gM, seed);
                for (; r < r1; ++r) {
                    double v = rnd_value(ran);
                    if (i0 + r == j) v += bump;
                    col[r] = v;
                    ran = rnd64_next(ran);
                }
            }
        }
    }
}

static bool generates_everything(const parsec_tiled_matrix_t *A, int region)
{
    if (A->storage != PARSEC_MATRIX_TILE) return false;
    if (region == dplasmaUpperLower) return A->uplo == dplasmaUpperLower || A->uplo == dplasmaLower || A->uplo == dplasmaUpper;
    return A->uplo == region;
}

static int run_generator(Context *ctx, parsec_tiled_matrix_t *A, int sym, int region, double bump, unsigned long long seed)
{
    cudaStream_t st = ctx->stream;
    const size_t bytes = desc_elems(A) * sizeof(double);
    double *dst = (double *)A->mat;
    if (A->location != DPLASMA_B200_DEVICE) {
        dst = (double *)ctx->buffer(BUF_STAGE, bytes);
        if (!dst) return DPLASMA_ERR_OUT_OF_RESOURCES;
        if (!generates_everything(A, region)) CK(cudaMemcpyAsync(dst, A->mat, bytes, cudaMemcpyHostToDevice, st));
    }
    DescView v = view_of(A, dst);
    gen_kernel<<<ctx->sms * 8, 256, 0, st>>>(v, sym, region, bump, seed, A->m);
    CK(cudaGetLastError());
    ctx->launches++;
    if (A->location != DPLASMA_B200_DEVICE) CK(cudaMemcpyAsync(A->mat, dst, bytes, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return 0;
}

int generate_plgsy(Context *ctx, double bump, dplasma_enum_t uplo, parsec_tiled_matrix_t *A, unsigned long long seed)
{
    return run_generator(ctx, A, 1, uplo, bump, seed);
}

int generate_plrnt(Context *ctx, int diagdom, parsec_tiled_matrix_t *A, unsigned long long seed)
{
    const double alpha = diagdom ? (double)(A->m > A->n ? A->m : A->n) : 0.0;
    return run_generator(ctx, A, 0, dplasmaUpperLower, alpha, seed);
}

}  // namespace db2
