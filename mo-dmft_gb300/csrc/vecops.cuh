// vecops.cuh -- kernels over sets of sector vectors, shared by the
// eigensolvers (krylov.cu, eigs.cu).
//
// Vectors are padded to a multiple of 32 elements and 256-byte aligned, so
// every access covers 4 consecutive elements (16 bytes and up).  Sums are
// per-block partials added in a fixed order (run-to-run deterministic).
// Per-element work of FP32 vectors stays in FP32: GB300 issues an FP64 warp
// instruction every 64 cycles per sub-partition.
#pragma once

#include <algorithm>
#include <cstring>

#include "krylov.cuh"

namespace moed {

constexpr int kVecThreads = 256;

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v)
{
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}
__device__ __forceinline__ float warp_sum(float v)
{
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}

// block-wide sum, result valid in thread 0
__device__ __forceinline__ double block_sum(double v, double *sred)
{
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sred[wid] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sred[w];
    return t;
}

// fixed-order sums of a[0 .. na) (warps 0-3) and b[0 .. nb) (warps 4-7) in out[0], out[1]
// (out: 10 doubles)
__device__ __forceinline__ void two_sums(const double *a, int na, const double *b, int nb, double *out)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double *p = wid < 4 ? a : b;
    const int n = wid < 4 ? na : nb;
    double s = 0.0;
#pragma unroll 4
    for (int i = 32 * (wid & 3) + lane; i < n; i += 128) s += p[i];
    s = warp_sum(s);
    if (lane == 0) out[2 + wid] = s;
    __syncthreads();
    if (threadIdx.x < 2) {
        const double *q = out + 2 + 4 * threadIdx.x;
        out[threadIdx.x] = (q[0] + q[1]) + (q[2] + q[3]);
    }
    __syncwarp();   // read by thread 0
}

// block_sum by one warp from a buffer of kVecThreads doubles: 13 FP64 warp
// instructions per block instead of 48, each 64 cycles of a sub-partition's
// pipe; for kernels with a block per few elements
__device__ __forceinline__ double block_sum_few(double v, double *buf)
{
    __syncthreads();
    buf[threadIdx.x] = v;
    __syncthreads();
    double s[kVecThreads / 32];
    if (threadIdx.x >= 32) return 0.0;
#pragma unroll
    for (int i = 0; i < kVecThreads / 32; ++i) s[i] = buf[threadIdx.x + 32 * i];
#pragma unroll
    for (int h = kVecThreads / 64; h; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) s[i] += s[i + h];
    return warp_sum(s[0]);
}

template <typename TX, typename TY>
__global__ void k_dot_part(const TX *__restrict__ x, const TY *__restrict__ y, long long n,
                           double *part)
{
    __shared__ double sred[32];
    double acc = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    // products and sums in FP64 (an FP32 x FP32 product is exact in FP64)
    for (; i + 3 * stride < n; i += 4 * stride) {
        acc += (double)x[i] * (double)y[i] + (double)x[i + stride] * (double)y[i + stride] +
               (double)x[i + 2 * stride] * (double)y[i + 2 * stride] +
               (double)x[i + 3 * stride] * (double)y[i + 3 * stride];
    }
    for (; i < n; i += stride) acc += (double)x[i] * (double)y[i];
    double t = block_sum(acc, sred);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

static __global__ void k_sum_parts(const double *part, int n, double *out)
{
    __shared__ double sred[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
    double t = block_sum(acc, sred);
    if (threadIdx.x == 0) *out = t;
}

// 16-byte vector access to 4 consecutive elements (vectors are padded to a
// multiple of 32 elements and 256-byte aligned)
template <typename T>
__device__ __forceinline__ void vload4(const T *p, T (&r)[4])
{
    if constexpr (sizeof(T) == 4) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
        r[0] = a.x;
        r[1] = a.y;
        r[2] = a.z;
        r[3] = a.w;
    } else {
        const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
        const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
        r[0] = a.x;
        r[1] = a.y;
        r[2] = b.x;
        r[3] = b.y;
    }
}

template <typename T>
__device__ __forceinline__ void vstore4(T *p, const T (&r)[4])
{
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(r[0], r[1], r[2], r[3]);
    } else {
        reinterpret_cast<double2 *>(p)[0] = make_double2(r[0], r[1]);
        reinterpret_cast<double2 *>(p)[1] = make_double2(r[2], r[3]);
    }
}

constexpr int kMaxNcv = 496;   // most vectors in one call of the kernels below

template <typename T>
struct VPtrs {
    const T *p[kMaxNcv + 1];
};

template <typename T>
static VPtrs<T> make_ptrs(const std::vector<DevBuf *> &v, int n)
{
    VPtrs<T> p;
    memset(&p, 0, sizeof(p));
    for (int i = 0; i < n; ++i) p.p[i] = (const T *)v[i]->p;
    return p;
}


// ---------------------------------------------------------------------------
// dots of a vector with many others
// ---------------------------------------------------------------------------
// part[row][b nv + l] = a share of V_l . w_b for l < nv, b < NW.  Bound by
// reading the V_l once (FP32) or by the FP64 pipe (FP64).  The 8 warps of a
// CTA split the vectors among them (vw of them; the other factor ew of 8 / vw
// splits the elements), LU vectors at a time, each warp walking Q * 128
// elements per step: a lane keeps LU sums per w instead of one per vector, and
// the warps' copies of w meet in L1.  A row is a CTA and an element share.
// FP32 products are summed in FP32 over 8 quads (32 elements), then in FP64;
// a lane's sum that never got that far (small sectors) is added over the warp
// in FP32 and widened once.  31 vectors of 15 million FP32 elements: 404 us
// with every thread keeping a sum per vector, 280 us so.
template <typename T>
struct WPtrs {
    T *p[2];
};

template <typename T, int Q, int LU, int NW>
__global__ void __launch_bounds__(kVecThreads)
k_dots(const __grid_constant__ VPtrs<T> V, int nv, int vw, const __grid_constant__ WPtrs<T> w, long long D, double *part)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ew = kVecThreads / 32 / vw, vi = wid % vw, ei = wid / vw;
    const long long row = (long long)blockIdx.x * ew + ei, nrow = (long long)gridDim.x * ew;
    for (int l0 = vi * LU; l0 < nv; l0 += vw * LU) {
        double acc[NW][LU];
        T s[NW][LU];
        const T *p[LU];
#pragma unroll
        for (int l = 0; l < LU; ++l) {
#pragma unroll
            for (int b = 0; b < NW; ++b) {
                acc[b][l] = 0.0;
                s[b][l] = T(0);
            }
            p[l] = V.p[min(l0 + l, nv - 1)];   // past the end: the last vector again, not written
        }
        int cnt = 0;
        bool flushed = false;
        for (long long i0 = row * (Q * 128) + 4 * lane; i0 < D; i0 += nrow * (Q * 128)) {
            T x[NW][Q][4], a[Q][LU][4];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const long long i = i0 + 128 * q;
                if (i < D) {
#pragma unroll
                    for (int b = 0; b < NW; ++b) vload4(w.p[b] + i, x[b][q]);
#pragma unroll
                    for (int l = 0; l < LU; ++l) vload4(p[l] + i, a[q][l]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
#pragma unroll
                        for (int b = 0; b < NW; ++b) x[b][q][e] = T(0);
#pragma unroll
                        for (int l = 0; l < LU; ++l) a[q][l][e] = T(0);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int l = 0; l < LU; ++l)
#pragma unroll
                    for (int b = 0; b < NW; ++b)
                        s[b][l] += a[q][l][0] * x[b][q][0] + a[q][l][1] * x[b][q][1] + a[q][l][2] * x[b][q][2] +
                                   a[q][l][3] * x[b][q][3];
            if constexpr (sizeof(T) == 4) {
                if (++cnt == 8 / Q) {
#pragma unroll
                    for (int l = 0; l < LU; ++l)
#pragma unroll
                        for (int b = 0; b < NW; ++b) {
                            acc[b][l] += (double)s[b][l];
                            s[b][l] = T(0);
                        }
                    cnt = 0;
                    flushed = true;
                }
            }
        }
        const bool wide = sizeof(T) == 8 || __any_sync(0xffffffffu, flushed);
#pragma unroll
        for (int b = 0; b < NW; ++b)
#pragma unroll
            for (int l = 0; l < LU; ++l) {
                const double v = wide ? warp_sum(sizeof(T) == 8 ? (double)s[b][l] : acc[b][l] + (double)s[b][l])
                                      : (double)warp_sum(s[b][l]);
                if (lane == 0 && l0 + l < nv) part[((size_t)row * NW + b) * nv + l0 + l] = v;
            }
    }
}

// out[l] = sum of column l of part[rows][nv] in a fixed order, one warp per column
static __global__ void __launch_bounds__(kVecThreads)
k_sum_cols(const double *__restrict__ part, int rows, int nv, double *__restrict__ out)
{
    const int l = (blockIdx.x * kVecThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (l >= nv) return;
    double s = 0.0;
    for (int r = lane; r < rows; r += 32) s += part[(size_t)r * nv + l];
    s = warp_sum(s);
    if (lane == 0) out[l] = s;
}

// rows of part a call of dots() may write, and its doubles for up to kMaxNcv vectors
inline int dots_blocks(const mo_ed_ctx *ctx, long long D, int Q, int ew)
{
    return (int)std::max(1LL, std::min((D + (long long)Q * ew * 128 - 1) / ((long long)Q * ew * 128),
                                       (long long)ctx->num_sms * 4));
}
inline size_t dots_part_doubles(const mo_ed_ctx *ctx) { return (size_t)ctx->num_sms * 4 * 2 * (kMaxNcv + 8); }
// up to this many rows the consumer adds them itself (axpys); beyond, k_sum_cols does
constexpr int kFuseRows = 32;

// V_l . w_b for l < nv, b < NW: *src is [*rows][NW nv] partials, or the sums (*rows = 1)
template <typename T, int NW>
int dots(mo_ed_ctx *ctx, const VPtrs<T> &P, int nv, const WPtrs<T> &w, long long D, double *part, double *sums,
         const double **src, int *rows)
{
    constexpr int Q = 2, LU = sizeof(T) == 4 ? 4 : 2;
    const int groups = (nv + LU - 1) / LU;   // warps the vectors can occupy
    const int vw = groups >= 5 ? 8 : groups >= 3 ? 4 : groups;
    const int ew = kVecThreads / 32 / vw;
    const int g = dots_blocks(ctx, D, Q, ew);
    k_dots<T, Q, LU, NW><<<g, kVecThreads, 0, ctx->stream>>>(P, nv, vw, w, D, part);
    MOED_CHECK_LAUNCH(ctx);
    *src = part;
    *rows = g * ew;
    if (*rows > kFuseRows) {
        k_sum_cols<<<(NW * nv + 7) / 8, kVecThreads, 0, ctx->stream>>>(part, *rows, NW * nv, sums);
        MOED_CHECK_LAUNCH(ctx);
        *src = sums;
        *rows = 1;
    }
    return MO_ED_OK;
}

// w_b -= sum_l c_l V_l, b < NW, with c_l = inv[l]^2 (sum of column b nv + l
// of src[rows][NW nv]) (inv: reciprocal norms of the V_l, or null for unit
// vectors); hout[b hstride + l] (block 0, optional) = inv[l] times that sum,
// the dot with the unit vector; norm_part (optional): partials of ||w||^2 of
// the last w.  4 consecutive elements per thread, 4 vectors' loads in flight.
// VS warps of a CTA share the elements of one and split the vectors among
// them: VS = 1 where the elements fill the chip; VS = 8 in small sectors,
// whose time is the chain of nv / 4 dependent L2 round trips (130 vectors of
// 4,900 FP32 elements, two w: 13.6 us with VS = 1).
template <typename T, int NW, int VS>
__global__ void __launch_bounds__(kVecThreads)
k_axpys(const __grid_constant__ VPtrs<T> V, int nv, const double *__restrict__ src, int rows,
        const double *__restrict__ inv, const __grid_constant__ WPtrs<T> w, long long D, double *norm_part, double *hout,
        int hstride)
{
    constexpr int EW = kVecThreads / 32 / VS;   // warps along the elements
    __shared__ T sh[NW][kMaxNcv + 4];
    __shared__ double sred[32];
    __shared__ T sx[VS > 1 ? VS - 1 : 1][NW][4][EW * 32 + 1];
    for (int k = threadIdx.x; k < NW * (nv + 4); k += blockDim.x) {
        const int b = k / (nv + 4), l = k - b * (nv + 4);
        double h = 0.0;
        if (l < nv) {
            for (int r = 0; r < rows; ++r) h += src[((size_t)r * NW + b) * nv + l];
            const double v = inv ? inv[l] : 1.0;
            h *= v;
            if (hout && blockIdx.x == 0) hout[(size_t)b * hstride + l] = h;
            h *= v;
        }
        sh[b][l] = (T)h;
    }
    __syncthreads();
    const int vs = (threadIdx.x >> 5) / EW, te = threadIdx.x - vs * EW * 32;   // vector share, thread along the elements
    const int per = ((nv + VS - 1) / VS + 3) & ~3, l_end = min(nv, (vs + 1) * per);
    // ||w||^2: partials of 4 squares in T, added in FP64 every 8 iterations
    double acc = 0.0;
    T sacc = T(0);
    int cnt = 0;
    // one trip count for all threads of the CTA (barriers inside)
    for (long long i0 = 4 * (blockIdx.x * (long long)(EW * 32)); i0 < D; i0 += 4 * (long long)gridDim.x * (EW * 32)) {
        const long long i = i0 + 4 * te;
        const bool in = i < D;
        T s[NW][4];
#pragma unroll
        for (int b = 0; b < NW; ++b)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[b][e] = T(0);
        if (in)
            for (int l = vs * per; l < l_end; l += 4) {
                T a[4][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (l + q < nv) vload4(V.p[l + q] + i, a[q]);
                    else a[q][0] = a[q][1] = a[q][2] = a[q][3] = T(0);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int b = 0; b < NW; ++b)
#pragma unroll
                        for (int e = 0; e < 4; ++e) s[b][e] += a[q][e] * sh[b][l + q];
            }
        if constexpr (VS > 1) {
            __syncthreads();   // the previous iteration's sums have been read
            if (vs > 0) {
#pragma unroll
                for (int b = 0; b < NW; ++b)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sx[vs - 1][b][e][te] = s[b][e];
            }
            __syncthreads();
            if (vs == 0)
                for (int q = 0; q < VS - 1; ++q)
#pragma unroll
                    for (int b = 0; b < NW; ++b)
#pragma unroll
                        for (int e = 0; e < 4; ++e) s[b][e] += sx[q][b][e][te];
        }
        if (in && vs == 0) {
#pragma unroll
            for (int b = 0; b < NW; ++b) {
                T x[4];
                vload4(w.p[b] + i, x);
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] -= s[b][e];
                if (b == NW - 1) sacc += (x[0] * x[0] + x[1] * x[1]) + (x[2] * x[2] + x[3] * x[3]);
                vstore4(w.p[b] + i, x);
            }
            if (++cnt == 8) {
                acc += (double)sacc;
                sacc = T(0);
                cnt = 0;
            }
        }
    }
    acc += (double)sacc;
    if (norm_part) {
        double t = block_sum(acc, sred);
        if (threadIdx.x == 0) norm_part[blockIdx.x] = t;
    }
}

// blocks of axpys over D elements: its norm partials
inline bool axpys_split(const mo_ed_ctx *ctx, long long D) { return D < 4 * kVecThreads * (long long)ctx->num_sms; }
inline int axpys_blocks(const mo_ed_ctx *ctx, long long D)
{
    const long long per = axpys_split(ctx, D) ? 128 : 4 * kVecThreads;
    return (int)std::max(1LL, std::min((D + per - 1) / per, (long long)ctx->num_sms * 4));
}

template <typename T, int NW>
int axpys(mo_ed_ctx *ctx, const VPtrs<T> &P, int nv, const double *src, int rows, const double *inv, const WPtrs<T> &w,
          long long D, double *norm_part, double *hout, int hstride)
{
    const int g = axpys_blocks(ctx, D);
    if (axpys_split(ctx, D))
        k_axpys<T, NW, 8><<<g, kVecThreads, 0, ctx->stream>>>(P, nv, src, rows, inv, w, D, norm_part, hout, hstride);
    else
        k_axpys<T, NW, 1><<<g, kVecThreads, 0, ctx->stream>>>(P, nv, src, rows, inv, w, D, norm_part, hout, hstride);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

// deterministic pseudo-random start vector in [-1, 1) (zero in the row pads)
template <typename T>
__global__ void k_random(T *x, long long n, int ld, int nu, unsigned long long seed)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        if ((int)(i % ld) >= nu) {
            x[i] = T(0);
            continue;
        }
        unsigned long long z = (unsigned long long)i + seed * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        x[i] = (T)((double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0);
    }
}

// X_c = sum_l V_l Y[l][c] for c in [c0, c0+KC).  Accumulated in the vector
// precision (FP32 vectors: FP32; GB300 runs FP64 at a small fraction of the
// FP32 rate), coefficients from shared memory, 4 vectors' loads in flight.
template <typename T, int KC>
__global__ void __launch_bounds__(kVecThreads)
k_rotate(const __grid_constant__ VPtrs<T> V, int nv, const double *__restrict__ Y, int ldy, int c0,
         int nc, const __grid_constant__ VPtrs<T> X, long long D)
{
    __shared__ __align__(16) T sy[(kMaxNcv + 4) * KC];
    for (int idx = threadIdx.x; idx < (nv + 4) * KC; idx += blockDim.x) {
        int l = idx / KC, c = idx - l * KC;
        sy[idx] = (c < nc && l < nv) ? (T)Y[(size_t)(c0 + c) * ldy + l] : T(0);
    }
    __syncthreads();
    // 4 consecutive elements per thread (16-byte accesses; D is a multiple
    // of 32 and the vectors are 256-byte aligned)
    for (long long i = 4 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); i < D;
         i += 4 * (long long)gridDim.x * blockDim.x) {
        T acc[KC][4];
#pragma unroll
        for (int c = 0; c < KC; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[c][e] = T(0);
        for (int l = 0; l < nv; l += 4) {
            T v[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (l + q < nv) vload4(V.p[l + q] + i, v[q]);
                else v[q][0] = v[q][1] = v[q][2] = v[q][3] = T(0);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int c = 0; c < KC; ++c) {
                    const T y = sy[(l + q) * KC + c];
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[c][e] += v[q][e] * y;
                }
        }
#pragma unroll
        for (int c = 0; c < KC; ++c)
            if (c < nc) vstore4(const_cast<T *>(X.p[c]) + i, acc[c]);
    }
}

// k_rotate of nc <= 8 columns.  FP64 is bound by its pipe, so exactly nc columns
// (6 of 290 vectors of 0.86 million elements: 3.4 ms with 8, 2.6 with 6); FP32
// reads at HBM speed either way.
template <typename T>
int rotate(mo_ed_ctx *ctx, int G, const VPtrs<T> &V, int nv, const double *Y, int ldy, int c0, int nc, const VPtrs<T> &X,
           long long D)
{
    constexpr bool f64 = sizeof(T) == 8;
    auto go = [&](auto kern) { kern<<<G, kVecThreads, 0, ctx->stream>>>(V, nv, Y, ldy, c0, nc, X, D); };
    if (f64 && nc == 1) go(k_rotate<T, f64 ? 1 : 8>);
    else if (f64 && nc == 2) go(k_rotate<T, f64 ? 2 : 8>);
    else if (f64 && nc == 3) go(k_rotate<T, f64 ? 3 : 8>);
    else if (f64 && nc == 4) go(k_rotate<T, f64 ? 4 : 8>);
    else if (f64 && nc == 5) go(k_rotate<T, f64 ? 5 : 8>);
    else if (f64 && nc == 6) go(k_rotate<T, f64 ? 6 : 8>);
    else go(k_rotate<T, 8>);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

}  // namespace moed
