// eigs.cu -- the lowest eigenpairs of a sector (diag, ed_solver.F90:107-191):
// one long Lanczos run with periodic reorthogonalisation, and the FP64
// Rayleigh-Ritz that ends every eigensolve.
//
// Reorthogonalising every step against every earlier vector is what a
// thick-restart Lanczos spends its time on (two Gram-Schmidt passes of ~30
// vectors per H*v: 80 % of an FP32 eigensolve of 15 million elements, 92 % of
// an FP64 one of 0.85 million).  Here a step is the three-term recurrence
// alone, and only every `period` steps the last two vectors are
// orthogonalised against all earlier ones, both in one pass (Simon, Math.
// Comp. 42, 1984: a recurrence whose vectors stay orthogonal to the square
// root of the rounding unit finds the eigenvalues of the projected operator
// to the rounding unit).  Rounding errors grow by the ratio at which Ritz
// values converge; the period follows the components measured at each
// reorthogonalisation, towards 2e-5 (FP32) / 1e-11 (FP64) (kryhost.h).
//
// The components h that a reorthogonalisation takes out belong to the
// projected matrix (KryRun::vectors): H Q = Q (T + h) + beta q e^T holds to
// rounding whatever their size.  Convergence is judged on the symmetric
// tridiagonal T; the returned vectors are the right eigenvectors of T + h
// where h matters, and their true residual decides whether they are returned.
//
// The run is not restarted while its vectors fit (kKryMax, and half the free
// memory), so it also takes fewer H*v.  A run that fills the room continues
// from the wanted Ritz space: the kept basis is chosen so that the projected
// matrix stays tridiagonal (Lanczos on diag(theta) started from the residual
// couplings), and the recurrence goes on unchanged.
//
// Vectors are stored unnormalised, U_j = ||U_j|| q_j, as in the reference
// recurrence (k_lz_update): the norm is needed one launch later than the
// vector, so no pass over it is spent on scaling.
#include <cfloat>
#include <cmath>
#include <cstring>

#include <cooperative_groups.h>

#include "hvrow.cuh"
#include "kryhost.h"
#include "math64.cuh"
#include "symeig.h"
#include "vecops.cuh"

namespace moed {

namespace cg = cooperative_groups;

// Krylov vectors of one run and their memory (at most half of what is free): a
// run of some 350 to 480 steps restarted at 352 spent half of its time on the
// rotation and on steps taken again (FP64, 0.86 million elements, 413 steps:
// 83 -> 44 ms; 41 million, 344 steps, 145 vectors in 48 GB: 2.4 -> 1.3 s)
constexpr int kKryMax = 488, kKryWide = 117;           // more vectors than kKryWide to start with: thick restarts
constexpr size_t kKryRunBytes = (size_t)128 << 30;
constexpr long long kKryMinDim = 128;                  // smaller sectors: thick restarts (krylov.cu)
constexpr size_t kKryAskBytes = (size_t)4 << 30;       // runs that may need more look at the free memory first
constexpr size_t kRrPoolBytes = (size_t)64 << 20;      // largest FP64 vector of the pooled Rayleigh-Ritz workspace
constexpr size_t kSlabBytes = (size_t)1 << 20;         // returned vectors up to this size share one allocation
// k_kry_cluster: sectors up to these sizes, shared memory of a CTA.  4 states
// by launches / by clusters, ms: FP32 4,900 elements 2.5 / 1.5, 10,584 4.3 / 3.3,
// 15,876 3.1 / 2.7; FP64 4,900 3.8 / 3.0, 7,056 4.9 / 4.4, 10,584 6.2 / 6.9
// (8 SMs' FP64 pipes are the limit there).
constexpr long long kKcMaxDimF32 = 16384, kKcMaxDimF64 = 8192;
constexpr int kKcSmem = 80 * 1024;
// partial sums that the next step's blocks add themselves (1.2 us with four warps
// per sum and no square root); with more, a one-block launch does (6.5 us)
constexpr int kKryFuseParts = 4096;

// device scalars of a run: alpha[j] = q_j H q_j, beta[j] couples q_{j-1} and
// q_j, inv[j] = 1 / ||U_j||
struct KryScal {
    double *alpha, *beta, *inv;
};

// the scalars of step j from ||U_j||^2 and U_j . H U_j (zeros where the Krylov
// space has closed: the vectors to come are zero then)
__device__ __forceinline__ void kry_store(const KryScal &sc, int j, double n2, double d)
{
    const double inv = n2 > 0.0 ? rsqrt_pos(n2) : 0.0;
    sc.inv[j] = inv;
    sc.beta[j] = n2 * inv;
    sc.alpha[j] = n2 > 0.0 ? div_by(d, n2, rcp_pos(n2)) : 0.0;
}

// the same from the partials of step j
__global__ void __launch_bounds__(kVecThreads)
k_kry_scalars(KryScal sc, int j, const double *__restrict__ norm_part, int gn, const double *__restrict__ dot_part, int gd)
{
    __shared__ double sums[10];
    two_sums(norm_part, gn, dot_part, gd, sums);
    if (threadIdx.x == 0) kry_store(sc, j, sums[0], sums[1]);
}

// U_j = (w - alpha_{j-1} U_{j-1}) / ||U_{j-1}|| - beta_{j-1} q_{j-2} with
// w = H U_{j-1}, and the partials of ||U_j||^2.  FUSED: every block first adds
// step j-1's partials (block 0 stores the scalars): one launch less per step.
template <typename T, bool FUSED>
__global__ void __launch_bounds__(kVecThreads)
k_kry_update(KryScal sc, int j, const double *__restrict__ norm_part, int gn, const double *__restrict__ dot_part,
             int gd, const T *__restrict__ w, const T *__restrict__ uc, const T *__restrict__ up, T *__restrict__ un,
             long long D, double *__restrict__ norm_out)
{
    __shared__ double sred[kVecThreads];
    __shared__ T coef[3];
    // square roots and divisions are tens of FP64 instructions: one thread's
    if (FUSED) two_sums(norm_part, gn, dot_part, gd, sred);
    if (threadIdx.x == 0) {
        double v[3];   // alpha, beta, inv of step j - 1
        if (FUSED) {
            const KryScal mine{v, v + 1, v + 2};
            kry_store(mine, 0, sred[0], sred[1]);
            if (blockIdx.x == 0) {
                sc.alpha[j - 1] = v[0];
                sc.beta[j - 1] = v[1];
                sc.inv[j - 1] = v[2];
            }
        } else {
            v[0] = sc.alpha[j - 1];
            v[1] = sc.beta[j - 1];
            v[2] = sc.inv[j - 1];
        }
        coef[0] = (T)v[2];
        coef[1] = (T)v[0];
        coef[2] = up ? (T)(v[1] * sc.inv[j - 2]) : T(0);
    }
    __syncthreads();
    const T s = coef[0], a = coef[1], c = coef[2];
    double acc = 0.0;
    T sacc = T(0);
    int cnt = 0;
    for (long long i = 4 * (blockIdx.x * (long long)kVecThreads + threadIdx.x); i < D;
         i += 4 * (long long)gridDim.x * kVecThreads) {
        T wv[4], cv[4], pv[4] = {T(0), T(0), T(0), T(0)}, v[4];
        vload4(w + i, wv);
        vload4(uc + i, cv);
        if (up) vload4(up + i, pv);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = s * (wv[e] - a * cv[e]) - c * pv[e];
        // ||U_j||^2: partials of 4 squares in T, added in FP64 every 8 iterations
        sacc += (v[0] * v[0] + v[1] * v[1]) + (v[2] * v[2] + v[3] * v[3]);
        if (++cnt == 8) {
            acc += widen(sacc);
            sacc = T(0);
            cnt = 0;
        }
        vstore4(un + i, v);
    }
    acc += widen(sacc);
    const double t = block_sum_few(acc, sred);
    if (threadIdx.x == 0) norm_out[blockIdx.x] = t;
}

// ---------------------------------------------------------------------------
// small sectors: many steps in one launch
// ---------------------------------------------------------------------------
// Steps j0 .. j1 of a run by one cluster; U[i] is U_{j0-2+i}.
struct KrySeg {
    static constexpr int most = 32;      // steps
    int j0, j1;
    bool update0, hv1;                   // U_{j0} is to be formed; w = H U_{j1} as well
    const double *norm_part;             // !update0: partials of ||U_{j0}||^2
    int gn;
    void *U[most + 2];
    void *w;
};

// The recurrence of k_kry_update and k_hv_row for sectors that a cluster of up
// to 8 CTAs holds: a launch per 2 x steps becomes one per segment between
// reorthogonalisations.  A thread keeps its EPT elements of w, U_{j-1}, U_{j-2}
// in registers; U_j goes to every CTA's shared memory, so the gathers of H*v
// are local; two cluster barriers per step.  What bounds a step is its chain of
// latencies (barriers, two FP64 sums, the scalars), not work: 4,900 FP32
// elements, 10 us per step as two launches, 4.8 us so.
constexpr int kKcThreads = 512, kKcMaxEpt = 4;
template <typename T, int EPT>
__global__ void __launch_bounds__(kKcThreads)
k_kry_cluster(const __grid_constant__ HvJobT<T> jb, const ModelDev *__restrict__ mdl, KryScal sc,
              const __grid_constant__ KrySeg seg, int ld)
{
    constexpr int NT = kKcThreads;
    extern __shared__ double raw[];
    double *const red = raw;                               // [2][NT]
    T *const xs = (T *)(red + 2 * NT);                     // U_j without its pads (jb.ld = nu)
    __shared__ T s_cross[kMaxImp * kMaxImp];
    __shared__ unsigned s_pmask[kMaxImp];
    __shared__ int s_t4[kMaxPair * kMaxImp];
    __shared__ double s_slot[2 * 8], s_part[4], s_n0;
    __shared__ T s_coef[3];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, C = gridDim.x, rank = blockIdx.x;
    const int nimp = mdl->nimp, npair = mdl->npair, nu = jb.nu, n = nu * jb.nd;
    for (int i = tid; i < npair * nimp; i += NT) s_t4[i] = mdl->t4[i];
    for (int i = tid; i < nimp; i += NT) s_pmask[i] = mdl->pairmask[i];
    for (int i = tid; i < nimp * nimp; i += NT) s_cross[i] = (T)mdl->cross[i];
    const T Jc = (T)mdl->J;
    if (!seg.update0 && wid == 0) {
        double a = 0.0;
        for (int i = lane; i < seg.gn; i += 32) a += seg.norm_part[i];
        a = warp_sum(a);
        if (lane == 0) s_n0 = a;
    }
    __syncthreads();
    // this thread's elements: address, column and row information, diagonal
    int at[EPT], col[EPT], row[EPT], inf[EPT], dinf[EPT];
    T diag[EPT], w[EPT], uc[EPT], up[EPT];
    const T *gw = (const T *)seg.w, *g1 = (const T *)seg.U[1], *g2 = (const T *)seg.U[0], *g0 = (const T *)seg.U[2];
#pragma unroll
    for (int k = 0; k < EPT; ++k) {
        const int e = (k * C + rank) * NT + tid;
        at[k] = -1;
        w[k] = uc[k] = up[k] = T(0);
        if (e < n) {
            const int d = e / nu, u = e - d * nu;
            at[k] = d * ld + u;
            row[k] = d;
            col[k] = u;
            inf[k] = __ldg(jb.up_info + u);
            dinf[k] = __ldg(jb.dn_info + d);
            diag[k] = __ldg(jb.up_diag + u) + __ldg(jb.dn_diag + d) +
                      s_cross[((inf[k] >> 8) & 0xff) * nimp + ((dinf[k] >> 8) & 0xff)];
            if (seg.update0) {
                w[k] = gw[at[k]];
                uc[k] = g1[at[k]];
                if (seg.j0 >= 2) up[k] = g2[at[k]];
            } else {
                uc[k] = g0[at[k]];
                if (seg.j0 >= 1) up[k] = g1[at[k]];
            }
        }
    }
    double inv1 = 0.0;   // thread 0: inv of the step before the one to come
    if (tid == 0) {
        const int j = seg.j0 - 1;
        if (j >= 0) inv1 = sc.inv[j];
        if (seg.update0) {
            s_coef[0] = (T)inv1;
            s_coef[1] = (T)sc.alpha[j];
            s_coef[2] = j >= 1 ? (T)(sc.beta[j] * sc.inv[j - 1]) : T(0);
        }
    }
    cl.sync();           // every CTA runs; the coefficients are there
    for (int j = seg.j0;; ++j) {
        const bool given = j == seg.j0 && !seg.update0;
        T sq = T(0);
        if (!given) {
            const T s = s_coef[0], a = s_coef[1], c = s_coef[2];
            T *un = (T *)seg.U[j - seg.j0 + 2];
#pragma unroll
            for (int k = 0; k < EPT; ++k)
                if (at[k] >= 0) {
                    const T v = s * (w[k] - a * uc[k]) - c * up[k];
                    up[k] = uc[k];
                    uc[k] = v;
                    sq += v * v;
                    un[at[k]] = v;
                }
            for (int d = rank * (NT / 32) + wid; d < jb.nd; d += C * (NT / 32))
                for (int u = nu + lane; u < ld; u += 32) un[d * ld + u] = T(0);
        }
        if (j == seg.j1 && !seg.hv1) break;
        for (int r = 0; r < C; ++r) {
            T *peer = cl.map_shared_rank(xs, r);
#pragma unroll
            for (int k = 0; k < EPT; ++k)
                if (at[k] >= 0) peer[(k * C + rank) * NT + tid] = uc[k];
        }
        cl.sync();
        double dot = 0.0;
#pragma unroll
        for (int k = 0; k < EPT; ++k)
            if (at[k] >= 0) {
                w[k] = hv_moves<T, T, false>(jb, mdl, xs, row[k], col[k], inf[k], dinf[k], s_pmask, s_t4, nimp, Jc,
                                             diag[k] * uc[k]);
                const double p = widen(uc[k] * w[k]);
                dot = k == 0 ? p : dot + p;
            }
        // sums over the cluster in a fixed order: halves of each by a warp
        red[tid] = widen(sq);
        red[NT + tid] = dot;
        __syncthreads();
        if (wid < 4) {
            const double *p = red + wid * (NT / 2) + lane;
            double v = 0.0;
#pragma unroll
            for (int i = 0; i < NT / 2; i += 32) v += p[i];
            v = warp_sum(v);
            if (lane == 0) s_part[wid] = v;
        }
        __syncthreads();
        if (tid < 2 * C) cl.map_shared_rank(s_slot, tid >> 1)[2 * rank + (tid & 1)] = s_part[2 * (tid & 1)] + s_part[2 * (tid & 1) + 1];
        cl.sync();
        if (wid == 0) {
            double v = lane < 2 * C ? s_slot[lane] : 0.0;
#pragma unroll
            for (int o = 8; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const double d = __shfl_sync(0xffffffffu, v, 1), n2 = given ? s_n0 : v;
            if (lane == 0) {
                double al, be, in;
                kry_store(KryScal{&al, &be, &in}, 0, n2, d);
                if (rank == 0) {
                    sc.alpha[j] = al;
                    sc.beta[j] = be;
                    sc.inv[j] = in;
                }
                s_coef[0] = (T)in;
                s_coef[1] = (T)al;
                s_coef[2] = j >= 1 ? (T)(be * inv1) : T(0);
                inv1 = in;
            }
        }
        __syncthreads();
        if (j == seg.j1) {
            T *gwo = (T *)seg.w;
#pragma unroll
            for (int k = 0; k < EPT; ++k)
                if (at[k] >= 0) gwo[at[k]] = w[k];
            break;
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 Rayleigh-Ritz
// ---------------------------------------------------------------------------
// part[block][pair * 18 + ...]: shares of S_ab = X_a . X_b and P_ab = X_a .
// (H X_b) for the 3 x 3 tile (a, b) = (3 bi .., 3 bj ..) of pair blockIdx.y,
// bi <= bj, products and sums in FP64 (an FP32 x FP32 product is exact).
// Bound by the FP64 pipe: 18 FMAs per element and tile, values widened with
// integer operations; one pass per tile instead of two per column.  6 vectors
// of 15 million FP32 elements: 18.6 ms as column-wise multi-dots.
template <typename T>
__global__ void __launch_bounds__(kVecThreads)
k_gram(const __grid_constant__ VPtrs<T> X, const __grid_constant__ VPtrs<double> HX, int n, int ntile, long long D,
       double *__restrict__ part)
{
    __shared__ double sred[kVecThreads / 32][18];
    int bi = 0, bj = blockIdx.y;
    while (bj >= ntile - bi) bj -= ntile - bi, ++bi;
    bj += bi;
    const T *xa[3], *xb[3];
    const double *hb[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {   // past the end: the last vector again, not read by the host
        xa[q] = X.p[min(3 * bi + q, n - 1)];
        xb[q] = X.p[min(3 * bj + q, n - 1)];
        hb[q] = HX.p[min(3 * bj + q, n - 1)];
    }
    double s[9], p[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = p[k] = 0.0;
    for (long long i = blockIdx.x * (long long)kVecThreads + threadIdx.x; i < D; i += (long long)gridDim.x * kVecThreads) {
        double a[3], b[3], h[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            a[q] = widen(xa[q][i]);
            h[q] = hb[q][i];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) b[q] = bi == bj ? a[q] : widen(xb[q][i]);
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                s[3 * q + r] = fma(a[q], b[r], s[3 * q + r]);
                p[3 * q + r] = fma(a[q], h[r], p[3 * q + r]);
            }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const double vs = warp_sum(s[k]), vp = warp_sum(p[k]);
        if (lane == 0) {
            sred[wid][k] = vs;
            sred[wid][9 + k] = vp;
        }
    }
    __syncthreads();
    if (threadIdx.x < 18) {
        double t = 0.0;
        for (int q = 0; q < kVecThreads / 32; ++q) t += sred[q][threadIdx.x];
        part[((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 18 + threadIdx.x] = t;
    }
}

// The refined vectors O_c = sum_l X_l C[c * n + l] (accumulated in T) and the
// partials of ||H O_c - E_c O_c||^2 (H O_c from the FP64 images) and ||O_c||^2,
// for the columns 6 blockIdx.y ..  One pass: the images of the refined vectors
// are not written.
constexpr int kOutCols = 6;
template <typename T>
__global__ void __launch_bounds__(kVecThreads)
k_ritz_out(const __grid_constant__ VPtrs<T> X, const __grid_constant__ VPtrs<double> HX, int n,
           const double *__restrict__ C, const double *__restrict__ E, const __grid_constant__ VPtrs<T> O, long long D,
           double *__restrict__ part)
{
    __shared__ double ch[kMaxNcv * kOutCols];
    __shared__ T cx[kMaxNcv * kOutCols];
    __shared__ double sred[32];
    const int c0 = blockIdx.y * kOutCols, nc = min(kOutCols, n - c0);
    for (int i = threadIdx.x; i < n * kOutCols; i += kVecThreads) {
        const int l = i / kOutCols, c = i - l * kOutCols;
        const double v = c < nc ? C[(size_t)(c0 + c) * n + l] : 0.0;
        ch[i] = v;
        cx[i] = (T)v;
    }
    __syncthreads();
    double rr[kOutCols], xx[kOutCols];
#pragma unroll
    for (int c = 0; c < kOutCols; ++c) rr[c] = xx[c] = 0.0;
    for (long long i = blockIdx.x * (long long)kVecThreads + threadIdx.x; i < D; i += (long long)gridDim.x * kVecThreads) {
        T o[kOutCols];
        double h[kOutCols];
#pragma unroll
        for (int c = 0; c < kOutCols; ++c) {
            o[c] = T(0);
            h[c] = 0.0;
        }
        for (int l = 0; l < n; ++l) {
            const T x = X.p[l][i];
            const double y = HX.p[l][i];
#pragma unroll
            for (int c = 0; c < kOutCols; ++c) {
                o[c] += x * cx[l * kOutCols + c];
                h[c] = fma(y, ch[l * kOutCols + c], h[c]);
            }
        }
#pragma unroll
        for (int c = 0; c < kOutCols; ++c)
            if (c < nc) {
                const_cast<T *>(O.p[c0 + c])[i] = o[c];
                const double x = widen(o[c]), r = fma(-E[c0 + c], x, h[c]);
                rr[c] = fma(r, r, rr[c]);
                xx[c] = fma(x, x, xx[c]);
            }
    }
#pragma unroll
    for (int c = 0; c < kOutCols; ++c)
        if (c < nc) {   // nc is uniform over the CTA
            const double a = block_sum(rr[c], sred), b = block_sum(xx[c], sred);
            if (threadIdx.x == 0) {
                part[(size_t)blockIdx.x * 2 * n + c0 + c] = a;
                part[(size_t)blockIdx.x * 2 * n + n + c0 + c] = b;
            }
        }
}

// See krylov.cuh.  P = X^T H X with H applied in FP64 accumulation, S = X^T X
// (X in the vector precision), P c = lambda S c on the host: eigenvalues of a
// cluster of near-degenerate states are accurate to ~res^2 / (gap to the rest
// of the spectrum), whatever the mixing inside the cluster.
template <typename T>
int ritz_pairs(mo_ed_ctx *ctx, const Sector &s, const VPtrs<T> &V, int m, const double *d_Y, int nout, int nev,
               long long matvecs, std::vector<double> &vals, std::vector<DevBuf> *vecs)
{
    const long long Dp = s.Dpad();
    const size_t vb = sizeof(T) * (size_t)Dp, vb64 = sizeof(double) * (size_t)Dp;
    std::vector<DevBuf> local;
    std::vector<DevBuf> &rp = vb64 <= kRrPoolBytes ? ctx->rr_pool : local;
    if (rp.size() < (size_t)(2 * nout + 2)) rp.resize(2 * nout + 2);
    DevBuf &dpart = rp[2 * nout], &dsmall = rp[2 * nout + 1];
    for (int i = 0; i < nout; ++i) {
        if (int rc = ensure(ctx, rp[i], vb)) return rc;
        if (int rc = ensure(ctx, rp[nout + i], vb64)) return rc;
    }
    const int ntile = (nout + 2) / 3, npair = ntile * (ntile + 1) / 2;
    const int G = (int)std::max(1LL, std::min((Dp + kVecThreads - 1) / kVecThreads, (long long)ctx->num_sms * 4));
    const int Gg = std::min(G, std::max(1, ctx->num_sms * 4 / npair));
    if (int rc = ensure(ctx, dpart, sizeof(double) * std::max((size_t)Gg * npair * 18, (size_t)G * 2 * nout))) return rc;
    const int nsum = std::max(npair * 18, 2 * nout);
    if (int rc = ensure(ctx, dsmall, sizeof(double) * ((size_t)nout * nout + nout + nsum))) return rc;
    double *dC = (double *)dsmall.p, *dE = dC + (size_t)nout * nout, *dsum = dE + nout;

    VPtrs<T> X;
    VPtrs<double> HX;
    memset(&X, 0, sizeof(X));
    memset(&HX, 0, sizeof(HX));
    std::vector<const void *> px(nout);
    std::vector<void *> ph(nout);
    for (int i = 0; i < nout; ++i) {
        X.p[i] = (const T *)(px[i] = rp[i].p);
        HX.p[i] = (const double *)(ph[i] = rp[nout + i].p);
    }
    for (int c0 = 0; c0 < nout; c0 += 8) {
        VPtrs<T> Xp;
        memset(&Xp, 0, sizeof(Xp));
        const int nc = std::min(8, nout - c0);
        for (int c = 0; c < nc; ++c) Xp.p[c] = X.p[c0 + c];
        if (int rc = rotate<T>(ctx, G, V, m, d_Y, m, c0, nc, Xp, Dp)) return rc;
    }
    const int hk = sizeof(T) == 4 ? HV_MIXED : HV_F64;
    if (int rc = hv_multi(ctx, s, hk, nout, px.data(), ph.data())) return rc;
    matvecs += nout;
    k_gram<T><<<dim3(Gg, npair), kVecThreads, 0, ctx->stream>>>(X, HX, nout, ntile, Dp, (double *)dpart.p);
    MOED_CHECK_LAUNCH(ctx);
    k_sum_cols<<<(npair * 18 + 7) / 8, kVecThreads, 0, ctx->stream>>>((const double *)dpart.p, Gg, npair * 18, dsum);
    MOED_CHECK_LAUNCH(ctx);
    std::vector<double> g(npair * 18);
    MOED_CUDA(ctx, cudaMemcpyAsync(g.data(), dsum, sizeof(double) * g.size(), cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    std::vector<double> P((size_t)nout * nout), S((size_t)nout * nout), ev(nout), C((size_t)nout * nout);
    int pair = 0;
    for (int bi = 0; bi < ntile; ++bi)
        for (int bj = bi; bj < ntile; ++bj, ++pair)
            for (int q = 0; q < 3; ++q)
                for (int r = 0; r < 3; ++r) {
                    const int a = 3 * bi + q, b = 3 * bj + r;
                    if (a > b || b >= nout) continue;
                    const double ps = g[pair * 18 + 3 * q + r];
                    double pp = g[pair * 18 + 9 + 3 * q + r];
                    if (bi == bj) pp = 0.5 * (pp + g[pair * 18 + 9 + 3 * r + q]);
                    S[(size_t)a * nout + b] = S[(size_t)b * nout + a] = ps;
                    P[(size_t)a * nout + b] = P[(size_t)b * nout + a] = pp;
                }
    if (!gen_sym_eig(nout, P, S, ev.data(), C.data()))
        return fail(ctx, MO_ED_ERR_NOCONV, "Ritz vectors numerically dependent");
    MOED_CUDA(ctx, cudaMemcpyAsync(dC, C.data(), sizeof(double) * C.size(), cudaMemcpyHostToDevice, ctx->stream));
    MOED_CUDA(ctx, cudaMemcpyAsync(dE, ev.data(), sizeof(double) * nout, cudaMemcpyHostToDevice, ctx->stream));
    std::vector<DevBuf> X2(nout);
    if (vb <= kSlabBytes) {
        if (int rc = dev_alloc_slab(ctx, X2.data(), nout, vb)) return rc;
    } else {
        for (auto &b : X2)
            if (int rc = dev_alloc(ctx, b, vb)) return rc;
    }
    VPtrs<T> O;
    memset(&O, 0, sizeof(O));
    for (int i = 0; i < nout; ++i) O.p[i] = (const T *)X2[i].p;
    k_ritz_out<T><<<dim3(G, (nout + kOutCols - 1) / kOutCols), kVecThreads, 0, ctx->stream>>>(X, HX, nout, dC, dE, O, Dp,
                                                                                              (double *)dpart.p);
    MOED_CHECK_LAUNCH(ctx);
    k_sum_cols<<<(2 * nout + 7) / 8, kVecThreads, 0, ctx->stream>>>((const double *)dpart.p, G, 2 * nout, dsum);
    MOED_CHECK_LAUNCH(ctx);
    std::vector<double> sq(2 * nout);
    MOED_CUDA(ctx, cudaMemcpyAsync(sq.data(), dsum, sizeof(double) * sq.size(), cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    vals.assign(nev, DBL_MAX);
    double res_true = 0.0;
    for (int i = 0; i < nout; ++i) {
        vals[i] = ev[i];
        res_true = std::max(res_true, std::sqrt(sq[i] / sq[nout + i]));
    }
    ctx->diag_matvecs = matvecs;
    ctx->diag_res_true = res_true;
    if (vecs) *vecs = std::move(X2);
    return MO_ED_OK;
}
template int ritz_pairs<float>(mo_ed_ctx *, const Sector &, const VPtrs<float> &, int, const double *, int, int,
                               long long, std::vector<double> &, std::vector<DevBuf> *);
template int ritz_pairs<double>(mo_ed_ctx *, const Sector &, const VPtrs<double> &, int, const double *, int, int,
                                long long, std::vector<double> &, std::vector<DevBuf> *);

// ---------------------------------------------------------------------------
// the run
// ---------------------------------------------------------------------------
namespace {

// Krylov vectors in chunks, allocated as the run reaches them: the first kHold
// bytes stay with the context (the sectors of a solve of many small ones), the
// next come from its pool, up to what that keeps, and the rest from cudaMalloc: 46
// GB for 41 million FP32 elements, 251 ms; all of it from the pool 260
struct KryVectors {
    static constexpr size_t kHold = (size_t)64 << 20;
    mo_ed_ctx *ctx;
    size_t vb, held = 0, pooled = 0;
    int per;                             // vectors per chunk
    size_t nheld = 0;
    std::vector<DevBuf> chunks;
    std::vector<void *> p;               // vector j
    KryVectors(mo_ed_ctx *c, size_t bytes) : ctx(c), vb((bytes + 255) & ~(size_t)255)
    {
        per = (int)std::max<size_t>(1, std::min<size_t>(32, ((size_t)1 << 30) / vb));
    }
    KryVectors(const KryVectors &) = delete;
    int grow(int n)                      // vectors 0 .. n-1 exist
    {
        while ((int)p.size() < n) {
            const size_t need = vb * (size_t)per;
            void *base;
            if (held + need <= kHold) {
                std::vector<DevBuf> &h = ctx->kry_hold;
                if (h.size() <= nheld) h.resize(nheld + 1);
                if (int rc = ensure(ctx, h[nheld], need)) return rc;
                base = h[nheld++].p;
                held += need;
            } else {
                DevBuf b;
                if (int rc = pooled + need <= pool_keep(ctx) ? pool_alloc(ctx, b, need) : dev_alloc(ctx, b, need)) return rc;
                pooled += need;
                base = b.p;
                chunks.push_back(std::move(b));
            }
            for (int i = 0; i < per; ++i) p.push_back((char *)base + vb * i);
        }
        return MO_ED_OK;
    }
};

// One Lanczos run in a sector: its vectors, device scalars and host state.
// `front`: unit vectors (the states found so far) that the run stays
// orthogonal to; their projections are not part of its projected matrix.
template <typename T>
struct KryRun {
    static constexpr bool f32 = sizeof(T) == 4;
    static constexpr int ns = kKryMax + 2;
    mo_ed_ctx *ctx;
    const Sector &s;
    int nwant, mmax, least;
    double tol;
    long long Dp;
    size_t vb;
    int kind, G, Gr, gmax, gd = 0;
    bool fused = false;
    bool clustered = false;       // segments of steps by k_kry_cluster
    int csize = 1, ept = 1;
    HvJobT<T> job;
    KryVectors U;
    DevBuf wlocal;
    T *w = nullptr;
    KryScal sc;
    double *npart[2], *dpart, *mpart, *msums, *hcol;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    std::vector<const T *> front;

    // of the current run
    unsigned long long seed = 0;
    int base = 0;                 // kept vectors of the last restart (0: none)
    int gn = 0;                   // norm partials of the last step
    KryPeriod ctl;
    int next_re = 0, last_re = -1;
    std::vector<KryClean> re;     // since the last restart
    size_t nread_re = 0;          // of them, on their way to the host
    long long matvecs = 0;
    int cycles = 0, m = 0, redo = -1;
    double anorm = 0.0;
    std::vector<double> al, be, inv, th, y;

    KryRun(mo_ed_ctx *c, const Sector &sec, int nw, int most, int lo, double tl)
        : ctx(c), s(sec), nwant(nw), mmax(most), least(lo), tol(tl), Dp(sec.Dpad()), vb(sizeof(T) * (size_t)sec.Dpad()),
          kind(f32 ? HV_F32 : HV_F64), U(c, sizeof(T) * (size_t)sec.Dpad()), ctl(f32, sec.D()), al(ns), be(ns), inv(ns),
          th(nw), y(ns)
    {
        // FP64: 8 elements per thread, as every block adds the last step's partials
        // on the FP64 pipe (0.86 million elements: 18.8 -> 14.4 us)
        G = (int)std::max(1LL, std::min((Dp / (f32 ? 4 : 8) + kVecThreads - 1) / kVecThreads, (long long)ctx->num_sms * 8));
        Gr = (int)std::max(1LL, std::min((Dp + kVecThreads - 1) / kVecThreads, (long long)ctx->num_sms * 4));
        gmax = std::max(std::max(G, Gr), axpys_blocks(ctx, Dp));
    }
    ~KryRun()
    {
        for (cudaEvent_t x : ev)
            if (x) cudaEventDestroy(x);
    }
    KryRun(const KryRun &) = delete;

    int setup()
    {
        if (int rc = hv_dot_parts(ctx, s, kind, &gd)) return rc;
        fused = gmax + gd <= kKryFuseParts;
        if (s.D() <= (f32 ? kKcMaxDimF32 : kKcMaxDimF64)) {
            if (int rc = hv_row_job<T>(ctx, s, kind, &job, &clustered)) return rc;
            job.ld = job.nu;
            while (csize < 8 && s.D() > (long long)csize * kKcThreads) csize *= 2;
            ept = (int)((s.D() + (long long)csize * kKcThreads - 1) / ((long long)csize * kKcThreads));
            const void *k = ept == 1 ? (const void *)k_kry_cluster<T, 1>
                                     : ept == 2 ? (const void *)k_kry_cluster<T, 2> : (const void *)k_kry_cluster<T, kKcMaxEpt>;
            MOED_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kKcSmem));
        }
        std::vector<DevBuf> &sm = ctx->kry_small;
        if (sm.size() < 4) sm.resize(4);
        // scalars, two sets of norm partials, dot partials; multi-dot partials and sums; h columns; w
        if (int rc = ensure(ctx, sm[0], sizeof(double) * (4 * ns + 2 * (size_t)gmax + gd))) return rc;
        if (int rc = ensure(ctx, sm[1], sizeof(double) * (dots_part_doubles(ctx) + 2 * kMaxNcv + 2))) return rc;
        if (int rc = ensure(ctx, sm[2], sizeof(double) * (size_t)ns * ns)) return rc;
        DevBuf &W = vb <= kRrPoolBytes ? sm[3] : wlocal;
        if (int rc = ensure(ctx, W, vb)) return rc;
        if (int rc = ensure_pinned(ctx, sizeof(double) * 2 * (3 + kReadRe) * ns)) return rc;
        sc.alpha = (double *)sm[0].p;
        sc.beta = sc.alpha + ns;
        sc.inv = sc.beta + 2 * ns;   // after ns doubles that hold 1 for the front vectors, read at negative offsets
        npart[0] = sc.inv + ns;
        npart[1] = npart[0] + gmax;
        dpart = npart[1] + gmax;
        mpart = (double *)sm[1].p;
        msums = mpart + dots_part_doubles(ctx);
        hcol = (double *)sm[2].p;
        w = (T *)W.p;
        std::vector<double> one(ns, 1.0);
        MOED_CUDA(ctx, cudaMemcpyAsync(sc.inv - ns, one.data(), sizeof(double) * ns, cudaMemcpyHostToDevice, ctx->stream));
        for (cudaEvent_t &x : ev) MOED_CUDA(ctx, cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
        return MO_ED_OK;
    }

    // the front vectors and U_0 .. U_{n-1}
    VPtrs<T> basis(int n) const
    {
        VPtrs<T> P;
        memset(&P, 0, sizeof(P));
        int k = 0;
        for (const T *f : front) P.p[k++] = f;
        for (int l = 0; l < n; ++l) P.p[k++] = (const T *)U.p[l];
        return P;
    }

    // take the components along the front vectors and U_0 .. U_{n-1} out of
    // NW vectors; their dots with the unit vectors go to h, h + ns (and gn counts
    // the norm partials)
    template <int NW>
    int clean(int n, const WPtrs<T> &x, double *norm_out, double *h)
    {
        const int nf = (int)front.size();
        const VPtrs<T> P = basis(n);
        const double *src;
        int rows;
        if (int rc = dots<T, NW>(ctx, P, nf + n, x, Dp, mpart, msums, &src, &rows)) return rc;
        gn = axpys_blocks(ctx, Dp);
        return axpys<T, NW>(ctx, P, nf + n, src, rows, sc.inv - nf, x, Dp, norm_out, h, ns);
    }

    // U_0: a random vector, orthogonal to the front vectors
    int first()
    {
        if (int rc = U.grow(1)) return rc;
        T *un = (T *)U.p[0];
        k_random<T><<<Gr, kVecThreads, 0, ctx->stream>>>(un, Dp, s.ld(), s.up->n, seed);
        MOED_CHECK_LAUNCH(ctx);
        if (front.empty()) {
            gn = Gr;
            k_dot_part<T, T><<<Gr, kVecThreads, 0, ctx->stream>>>(un, un, Dp, npart[0]);
            MOED_CHECK_LAUNCH(ctx);
        } else {
            for (int pass = 0; pass < 2; ++pass)
                if (int rc = clean<1>(0, WPtrs<T>{{un, nullptr}}, npart[0], hcol)) return rc;
        }
        return MO_ED_OK;
    }

    // U_{j-1} and U_j together: one pass over the others for both
    int reorthogonalise(int j)
    {
        if (int rc = clean<2>(j - 1, WPtrs<T>{{(T *)U.p[j - 1], (T *)U.p[j]}}, npart[j & 1], hcol + (size_t)(j - 1) * ns))
            return rc;
        re.push_back({j, j - std::max(last_re, base)});
        last_re = j;
        next_re = j + ctl.period;
        return MO_ED_OK;
    }

    int step(int j)
    {
        if (int rc = U.grow(j + 1)) return rc;
        T *un = (T *)U.p[j];
        if (j == 0) {
            if (int rc = first()) return rc;
        } else {
            T *uc = (T *)U.p[j - 1];
            const T *up = j >= 2 ? (const T *)U.p[j - 2] : nullptr;
            // right after a restart or a step back the scalars of j - 1 are stored
            if (fused && !(base > 0 && j == base + 1) && j != redo)
                k_kry_update<T, true><<<G, kVecThreads, 0, ctx->stream>>>(sc, j, npart[(j - 1) & 1], gn, dpart, gd, w, uc,
                                                                          up, un, Dp, npart[j & 1]);
            else
                k_kry_update<T, false><<<G, kVecThreads, 0, ctx->stream>>>(sc, j, nullptr, 0, nullptr, 0, w, uc, up, un, Dp,
                                                                           npart[j & 1]);
            MOED_CHECK_LAUNCH(ctx);
            gn = G;
            if (j >= next_re)
                if (int rc = reorthogonalise(j)) return rc;
        }
        if (int rc = hv_single_dot(ctx, s, kind, un, w, dpart)) return rc;
        ++matvecs;
        if (!fused) {
            k_kry_scalars<<<1, kVecThreads, 0, ctx->stream>>>(sc, j, npart[j & 1], gn, dpart, gd);
            MOED_CHECK_LAUNCH(ctx);
        }
        redo = -1;
        return MO_ED_OK;
    }

    size_t kc_smem() const { return sizeof(double) * 2 * kKcThreads + sizeof(T) * (size_t)s.D(); }

    template <int EPT>
    int segment(const KrySeg &seg)
    {
        const size_t smem = kc_smem();
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)csize;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)csize);
        cfg.blockDim = dim3(kKcThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = ctx->stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        MOED_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_kry_cluster<T, EPT>, job, (const ModelDev *)ctx->d_mdl, sc, seg, s.ld()));
        MOED_CHECK_LAUNCH(ctx);
        return MO_ED_OK;
    }

    // steps j .. stop - 1 in segments: up to the next vector to be
    // reorthogonalised, and on from its H*v
    int run_to(int &j, int stop)
    {
        bool formed = false;             // U_j is there and its H*v is not
        while (j < stop) {
            if (j == 0 && !formed) {
                if (int rc = first()) return rc;
                formed = true;
            }
            KrySeg seg;
            memset(&seg, 0, sizeof(seg));
            const bool clean_last = !formed ? std::max(j, next_re) < std::min(stop, j + KrySeg::most)
                                            : std::max(j + 1, next_re) < std::min(stop, j + KrySeg::most);
            const int last = clean_last ? std::max(formed ? j + 1 : j, next_re) : std::min(stop, j + KrySeg::most) - 1;
            if (int rc = U.grow(last + 1)) return rc;
            seg.j0 = j;
            seg.j1 = last;
            seg.update0 = !formed;
            seg.hv1 = !clean_last;
            seg.norm_part = npart[j & 1];
            seg.gn = gn;
            for (int i = 0; i < last - j + 3; ++i)
                if (j - 2 + i >= 0) seg.U[i] = U.p[j - 2 + i];
            seg.w = w;
            if (int rc = ept == 1 ? segment<1>(seg) : ept == 2 ? segment<2>(seg) : segment<kKcMaxEpt>(seg)) return rc;
            matvecs += last - j + (clean_last ? 0 : 1);
            if (clean_last) {
                if (int rc = reorthogonalise(last)) return rc;
                j = last;
                formed = true;
            } else {
                j = last + 1;
                formed = false;
            }
        }
        redo = -1;
        return MO_ED_OK;
    }

    // go back to step j (a reorthogonalised one): w = H U_j again; its scalars
    // are stored already
    int go_back(int j)
    {
        if (int rc = hv_single_dot(ctx, s, kind, U.p[j], w, dpart)) return rc;
        ++matvecs;
        while (!re.empty() && re.back().j > j) re.pop_back();
        nread_re = re.size();
        last_re = j;
        next_re = j + ctl.period;
        redo = j + 1;
        return MO_ED_OK;
    }

    // after step j: its scalars, and the components that the reorthogonalisations
    // since the last read have found, to pinned memory.  At most 117 steps (the
    // first) lie between two reads, every sixth of them with one, then 44, every
    // second; what there is no room for goes with the next read.
    static constexpr int kReadRe = 24;
    int read_j[2];
    std::vector<KryClean> read_re[2];
    double *read_at(int slot) const { return (double *)ctx->pinned + (size_t)slot * (3 + kReadRe) * ns; }
    int read_back(int slot, int j)
    {
        if (fused && !clustered) {
            k_kry_scalars<<<1, kVecThreads, 0, ctx->stream>>>(sc, j, npart[j & 1], gn, dpart, gd);
            MOED_CHECK_LAUNCH(ctx);
        }
        double *h = read_at(slot);
        MOED_CUDA(ctx, cudaMemcpyAsync(h, sc.alpha, sizeof(double) * 2 * ns, cudaMemcpyDeviceToHost, ctx->stream));
        MOED_CUDA(ctx, cudaMemcpyAsync(h + 2 * ns, sc.inv, sizeof(double) * ns, cudaMemcpyDeviceToHost, ctx->stream));
        read_re[slot].clear();
        for (; nread_re < re.size() && read_re[slot].size() < (size_t)kReadRe; ++nread_re) {
            h += read_re[slot].empty() ? 3 * ns : ns;
            read_re[slot].push_back(re[nread_re]);
            MOED_CUDA(ctx, cudaMemcpyAsync(h, hcol + (size_t)re[nread_re].j * ns, sizeof(double) * ns, cudaMemcpyDeviceToHost,
                                           ctx->stream));
        }
        MOED_CUDA(ctx, cudaEventRecord(ev[slot], ctx->stream));
        read_j[slot] = j;
        return MO_ED_OK;
    }

    // The run from a random vector.  cut null: until the nwant lowest Ritz
    // pairs have converged.  cut: until every Ritz value below *cut has
    // converged and the next one is known to kSettled of its distance from the
    // cut (*nlow = how many lie below).  *ok = false: gave up.
    //
    // A Ritz value above the cut can stand still for a while before it falls to
    // a level below that the start vector has a small share of.  Its residual
    // then is that share's angle times the distance, so kSettled bounds the
    // angle; random shares a tenth of their neighbours' are common.
    static constexpr double kSettled = 1e-3;
    int go(unsigned long long seed_, const double *cut, int *nlow, bool *ok)
    {
        *ok = false;
        seed = seed_;
        base = cycles = m = gn = 0;
        redo = -1;
        ctl = KryPeriod(f32, s.D());
        next_re = 3;
        last_re = -1;
        re.clear();
        nread_re = 0;
        anorm = 0.0;
        double last_res = 0.0;
        int last_m = 0;
        int j = 0;                    // next step
        int stop = cut ? 24 : least;  // steps 0 .. stop - 1 before the next read
        bool full = false;
        int nread = 0, ndone = 0;     // reads issued, reads judged
        for (;;) {
            if (!full) {
                if (clustered)
                    if (int rc = run_to(j, stop)) return rc == MO_ED_ERR_NOMEM ? (int)MO_ED_OK : rc;
                for (; j < stop; ++j)
                    if (int rc = step(j)) {
                        if (rc != MO_ED_ERR_NOMEM || j < least + 8) return rc == MO_ED_ERR_NOMEM ? (int)MO_ED_OK : rc;
                        mmax = j - 1;   // no room for vector j: the run ends at the ones it has
                        break;
                    }
                full = j > mmax || j < stop;
                if (int rc = read_back(nread & 1, j - 1)) return rc;
                ++nread;
                stop = std::min(j + 4, mmax + 1);
            }
            if (nread - ndone < 2 && !full) continue;   // judge one read while the next steps run
            const int slot = ndone & 1;
            ++ndone;
            MOED_CUDA(ctx, cudaEventSynchronize(ev[slot]));
            const double *h = read_at(slot);
            m = read_j[slot];   // alpha[0 .. m), and U_m is the residual vector
            for (int i = 0; i <= m; ++i) {
                al[i] = h[i];
                be[i] = h[ns + i];
                inv[i] = h[2 * ns + i];
                if (!std::isfinite(al[i]) || !std::isfinite(be[i]) || !std::isfinite(inv[i])) return MO_ED_OK;
            }
            // the norm that tolerances are relative to; scalars of steps that are
            // about to be discarded can be of any size and must not stay in it
            double an = anorm;
            bool closed = false;   // the Krylov space ends at U_{m-1}
            for (int i = base; i < m && !closed; ++i) {
                an = std::max(an, std::fabs(al[i]) + be[i + 1]);
                if (be[i + 1] > (f32 ? 1e-5 : 1e-12) * std::max(an, 1.0)) continue;
                if (!cut) return MO_ED_OK;   // an invariant subspace: thick restarts go on from there
                // it has a vector of every eigenspace but the found states': the
                // search ends here
                m = i + 1;
                closed = true;
            }
            KryPeriod::Verdict verdict = KryPeriod::kept;
            for (size_t r = 0; r < read_re[slot].size() && verdict == KryPeriod::kept; ++r) {
                const KryClean &cl = read_re[slot][r];
                if (cl.j >= m + !closed) break;
                double c = 0.0;
                for (int l = 0; l < cl.j - 1 + (int)front.size(); ++l)
                    c = std::max(c, std::fabs(h[(3 + r) * ns + l]));
                verdict = ctl.judge(cl, c * inv[cl.j], base > 0);
            }
            if (verdict == KryPeriod::lost) return MO_ED_OK;
            if (verdict == KryPeriod::back) {
                if (int rc = go_back(ctl.good)) return rc;
                j = ctl.good + 1;
                full = false;
                stop = std::min(j + 4, mmax + 1);
                nread = ndone = 0;
                last_m = 0;
                continue;
            }
            anorm = an;
            const double want = tol * std::max(anorm, 1.0);
            double res = 0.0, aim = want;
            if (!cut) {
                tri_lowest(m, al.data(), be.data() + 1, nwant, th.data());
                for (int i = 0; i < nwant; ++i) {
                    tri_eigvec(m, al.data(), be.data() + 1, th[i], y.data());
                    res = std::max(res, std::fabs(be[m] * y[m - 1]));
                }
                ctx->diag_res_est = res;
                if (res <= want) {
                    *ok = true;
                    return MO_ED_OK;
                }
            } else {
                const int k = std::min(nwant + 1, m);
                th.resize(k);
                tri_lowest(m, al.data(), be.data() + 1, k, th.data());
                int n = 0;
                while (n < k && th[n] < *cut) ++n;
                *nlow = std::min(n, nwant);
                for (int i = 0; i < *nlow; ++i) {
                    tri_eigvec(m, al.data(), be.data() + 1, th[i], y.data());
                    res = std::max(res, std::fabs(be[m] * y[m - 1]));
                }
                bool settled = res <= want;
                if (n < k) {   // the first value above the cut
                    tri_eigvec(m, al.data(), be.data() + 1, th[n], y.data());
                    const double r = std::fabs(be[m] * y[m - 1]), lim = std::max(kSettled * (th[n] - *cut), want);
                    if (r > lim) settled = false;
                    if (n == 0) {
                        res = r;
                        aim = lim;
                    }
                }
                if (settled || closed) {
                    *ok = settled;
                    return MO_ED_OK;
                }
            }
            // steps to the tolerance at the rate since the last read, 70 % of them before the next
            int ahead = 4;
            if (last_m > 0 && m > last_m && res < last_res && res > aim)
                ahead = (int)(0.7 * (m - last_m) * std::log(res / aim) / std::log(last_res / res));
            last_m = m;
            last_res = res;
            if (!full) {
                stop = std::min(std::max(j + 4, m + std::min(ahead, 40)), mmax + 1);
            } else if (ndone == nread) {
                if (++cycles >= ctx->opt.gs_maxcycles)
                    return cut ? (int)MO_ED_OK : fail(ctx, MO_ED_ERR_NOCONV, "eigensolver did not converge");
                bool again = false;
                if (int rc = restart(&again)) return rc == MO_ED_ERR_NOMEM ? (int)MO_ED_OK : rc;
                if (!again) return MO_ED_OK;
                j = base + 1;
                full = false;
                last_m = 0;
                stop = std::min(base + 12, mmax + 1);
                nread = ndone = 0;
            }
        }
    }

    // The run is full: go on from the lowest Ritz vectors (of T alone; h is
    // kept small by the shorter period)
    int restart(bool *again)
    {
        const int kk = nwant + 20;
        std::vector<double> Z((size_t)m * m, 0.0), d(al.begin(), al.begin() + m), e(be.begin() + 1, be.begin() + m);
        for (int i = 0; i < m; ++i) Z[(size_t)i * m + i] = 1.0;
        e.push_back(0.0);
        if (!tri_qr(m, d.data(), e.data(), m, Z.data())) return MO_ED_OK;
        std::vector<int> ord(m);
        for (int i = 0; i < m; ++i) ord[i] = i;
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return d[a] < d[b]; });
        // Lanczos on diag(theta) from the couplings to U_m, last kept vector first
        std::vector<double> Q((size_t)kk * kk, 0.0), r(kk), ka(kk), kb(kk + 1, 0.0);
        double nr = 0.0;
        for (int i = 0; i < kk; ++i) {
            r[i] = be[m] * Z[(size_t)(m - 1) * m + ord[i]];
            nr += r[i] * r[i];
        }
        kb[kk] = std::sqrt(nr);
        for (int c = kk - 1; c >= 0; --c) {
            double *q = &Q[(size_t)c * kk];
            if (!(kb[c + 1] > 1e-14 * std::max(anorm, 1.0))) return MO_ED_OK;   // decoupled: thick restarts
            for (int i = 0; i < kk; ++i) q[i] = r[i] / kb[c + 1];
            ka[c] = 0.0;
            for (int i = 0; i < kk; ++i) ka[c] += q[i] * q[i] * d[ord[i]];
            for (int i = 0; i < kk; ++i) r[i] = (d[ord[i]] - ka[c]) * q[i];
            for (int pass = 0; pass < 2; ++pass)
                for (int c2 = c; c2 < kk; ++c2) {
                    double t = 0.0;
                    for (int i = 0; i < kk; ++i) t += r[i] * Q[(size_t)c2 * kk + i];
                    for (int i = 0; i < kk; ++i) r[i] -= t * Q[(size_t)c2 * kk + i];
                }
            nr = 0.0;
            for (int i = 0; i < kk; ++i) nr += r[i] * r[i];
            kb[c] = std::sqrt(nr);
        }
        std::vector<double> Y((size_t)m * kk, 0.0);   // kept vector c = sum_l U_l Y[c * m + l]
        for (int c = 0; c < kk; ++c) {
            for (int i = 0; i < kk; ++i) {
                const double f = Q[(size_t)c * kk + i];
                for (int l = 0; l < m; ++l) Y[(size_t)c * m + l] += f * Z[(size_t)l * m + ord[i]];
            }
            for (int l = 0; l < m; ++l) Y[(size_t)c * m + l] *= inv[l];
        }
        DevBuf dY;
        if (int rc = dev_alloc(ctx, dY, sizeof(double) * Y.size())) return rc;
        MOED_CUDA(ctx, cudaMemcpyAsync(dY.p, Y.data(), sizeof(double) * Y.size(), cudaMemcpyHostToDevice, ctx->stream));
        VPtrs<T> V;
        memset(&V, 0, sizeof(V));
        for (int l = 0; l < m; ++l) V.p[l] = (const T *)U.p[l];
        std::vector<DevBuf> kept(kk);
        for (int c = 0; c < kk; ++c)
            if (int rc = dev_alloc(ctx, kept[c], vb)) return rc;
        for (int c0 = 0; c0 < kk; c0 += 8) {
            VPtrs<T> O;
            memset(&O, 0, sizeof(O));
            const int nc = std::min(8, kk - c0);
            for (int c = 0; c < nc; ++c) O.p[c] = (const T *)kept[c0 + c].p;
            if (int rc = rotate<T>(ctx, Gr, V, m, (const double *)dY.p, m, c0, nc, O, Dp)) return rc;
        }
        for (int c = 0; c < kk; ++c)
            MOED_CUDA(ctx, cudaMemcpyAsync(U.p[c], kept[c].p, vb, cudaMemcpyDeviceToDevice, ctx->stream));
        std::swap(U.p[kk], U.p[m]);
        for (int c = 0; c < kk; ++c) {
            al[c] = ka[c];
            be[c] = kb[c];
            inv[c] = 1.0;
        }
        al[kk] = al[m];
        be[kk] = kb[kk];
        inv[kk] = inv[m];
        const size_t nb = sizeof(double) * (size_t)(kk + 1);
        MOED_CUDA(ctx, cudaMemcpyAsync(sc.alpha, al.data(), nb, cudaMemcpyHostToDevice, ctx->stream));
        MOED_CUDA(ctx, cudaMemcpyAsync(sc.beta, be.data(), nb, cudaMemcpyHostToDevice, ctx->stream));
        MOED_CUDA(ctx, cudaMemcpyAsync(sc.inv, inv.data(), nb, cudaMemcpyHostToDevice, ctx->stream));
        MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));   // kept and the host arrays go
        base = kk;
        next_re = base + 1;
        last_re = -1;
        re.clear();
        nread_re = 0;
        ctl.restart();
        *again = true;
        return MO_ED_OK;
    }

    // Coefficients of the n lowest Ritz vectors over the stored vectors
    // U_0 .. U_{m-1}, Y[i * ld + off + l]: eigenvectors of T, or of T + h where
    // h is above rounding.
    int vectors(int n, std::vector<double> &Y, int ld, int off)
    {
        std::vector<double> Hp;
        if (ctl.hmax > (f32 ? 1e-6 : 1e-12)) {
            const int nf = (int)front.size();
            std::vector<double> hall((size_t)ns * (m + 1));
            MOED_CUDA(ctx, cudaMemcpyAsync(hall.data(), hcol, sizeof(double) * hall.size(), cudaMemcpyDeviceToHost,
                                           ctx->stream));
            MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            kry_projected(m, al.data(), be.data(), inv.data(), re, hall.data() + nf, ns, Hp);
        }
        // Ritz values that agree to rounding (copies of a degenerate level that
        // rounding has brought into the run): any independent vectors of them
        const double same = (f32 ? 1e-6 : 1e-9) * std::max(anorm, 1.0);
        std::vector<const double *> prev;
        for (int i = 0; i < n; ++i) {
            double *yi = &Y[(size_t)i * ld + off];
            if (i > 0 && th[i] - th[i - 1] > same) prev.clear();
            if (Hp.empty())
                tri_eigvec(m, al.data(), be.data() + 1, th[i], yi, prev.data(), (int)prev.size());
            else
                hess_eigvec(m, Hp.data(), m, th[i], anorm, yi, prev.data(), (int)prev.size());
            prev.push_back(yi);
        }
        for (int i = 0; i < n; ++i)
            for (int l = 0; l < m; ++l) Y[(size_t)i * ld + off + l] *= inv[l];
        return MO_ED_OK;
    }
};

}  // namespace

template <typename T>
int plz_solve(mo_ed_ctx *ctx, const Sector &s, int nev, std::vector<double> &vals, std::vector<DevBuf> *vecs,
              bool *done)
{
    *done = false;
    constexpr bool f32 = sizeof(T) == 4;
    const long long D = s.D();
    const int least = 2 * nev + 24;       // vectors below which a run is not worth restarting
    if (ctx->opt.gs_ncv > 0 || D < kKryMinDim || D < 4LL * least || least > kKryWide) return MO_ED_OK;
    const double tol = ctx->opt.gs_tol > 0 ? ctx->opt.gs_tol : (f32 ? 1e-7 : 1e-11);
    const size_t vb = sizeof(T) * (size_t)s.Dpad();
    // room for the front vectors of the search below: nev
    int mmax = (int)std::min<long long>(kKryMax - nev, 3 * D / 4);
    if (vb * (size_t)mmax > kKryAskBytes) {
        size_t fr = 0, tot = 0;
        MOED_CUDA(ctx, cudaMemGetInfo(&fr, &tot));
        if (ctx->mem_pool) {   // what idles in the pool is free
            unsigned long long held = 0, used = 0;
            MOED_CUDA(ctx, cudaMemPoolGetAttribute(ctx->mem_pool, cudaMemPoolAttrReservedMemCurrent, &held));
            MOED_CUDA(ctx, cudaMemPoolGetAttribute(ctx->mem_pool, cudaMemPoolAttrUsedMemCurrent, &used));
            fr += (size_t)(held - used);
        }
        mmax = (int)std::min<size_t>(mmax, std::min(kKryRunBytes, fr / 2) / vb);
        if (mmax < least + 40) return MO_ED_OK;
    }
    KryRun<T> run(ctx, s, nev, mmax, least, tol);
    if (int rc = run.setup()) return rc == MO_ED_ERR_NOMEM ? (int)MO_ED_OK : rc;
    const unsigned long long seed = 0x5eedULL + 977ULL * (unsigned)s.ne_up + 131ULL * (unsigned)s.ne_down;
    bool ok = false;
    if (int rc = run.go(seed, nullptr, nullptr, &ok)) return rc;
    if (!ok) return MO_ED_OK;
    std::vector<double> Y((size_t)run.m * nev);
    if (int rc = run.vectors(nev, Y, run.m, 0)) return rc;
    MOED_CUDA(ctx, cudaMemcpyAsync(run.hcol, Y.data(), sizeof(double) * Y.size(), cudaMemcpyHostToDevice, ctx->stream));
    std::vector<DevBuf> X;
    const int cycles = run.cycles;
    int rc = ritz_pairs<T>(ctx, s, run.basis(run.m), run.m, run.hcol, nev, nev, run.matvecs, vals,
                           vecs || ctx->degenerate ? &X : nullptr);
    if (rc == MO_ED_ERR_NOCONV || rc == MO_ED_ERR_NOMEM) return MO_ED_OK;   // the thick restarts try
    if (rc) return rc;
    if (!(ctx->diag_res_true <= kry_residual_limit(f32, tol, run.anorm))) return MO_ED_OK;
    // A Krylov space holds one vector of each eigenspace.  Where the model can
    // have exactly degenerate levels, runs orthogonal to the states found look
    // for others below the highest of them, until one finds none.  A run that
    // gives up says nothing: others from other vectors take its place, and after
    // three of them the thick restarts do.
    const double norm = std::max(run.anorm, 1.0);
    bool complete = !ctx->degenerate;
    for (int round = 1, lost = 0; !complete && lost < 3 && round <= 2 * nev + 5; ++round) {
        run.front.clear();
        for (const DevBuf &b : X) run.front.push_back((const T *)b.p);
        const double cut = vals[nev - 1] - 10 * tol * norm;
        int nlow = 0;
        run.matvecs = 0;
        if (int r2 = run.go(seed + 7919ULL * round, &cut, &nlow, &ok)) return r2;
        const long long mv = ctx->diag_matvecs + run.matvecs;
        const double res = ctx->diag_res_true;
        ctx->diag_matvecs = mv;
        if (!ok) {
            ++lost;
            continue;
        }
        if (nlow == 0) {
            complete = true;
            break;
        }
        const int n = nev + nlow, mm = nev + run.m;
        Y.assign((size_t)mm * n, 0.0);
        for (int i = 0; i < nev; ++i) Y[(size_t)i * mm + i] = 1.0;
        std::vector<double> Yl((size_t)mm * nlow, 0.0);
        if (int r2 = run.vectors(nlow, Yl, mm, nev)) return r2;
        std::copy(Yl.begin(), Yl.end(), Y.begin() + (size_t)nev * mm);
        MOED_CUDA(ctx, cudaMemcpyAsync(run.hcol, Y.data(), sizeof(double) * Y.size(), cudaMemcpyHostToDevice, ctx->stream));
        std::vector<double> v2;
        std::vector<DevBuf> X2;
        rc = ritz_pairs<T>(ctx, s, run.basis(run.m), mm, run.hcol, n, n, mv, v2, &X2);
        if (rc == MO_ED_ERR_NOMEM) break;
        if (rc && rc != MO_ED_ERR_NOCONV) return rc;
        if (rc || !(ctx->diag_res_true <= kry_residual_limit(f32, tol, norm))) {
            ++lost;
            ctx->diag_res_true = res;
            continue;
        }
        X2.resize(nev);
        X = std::move(X2);
        vals.assign(v2.begin(), v2.begin() + nev);
    }
    if (!complete) return MO_ED_OK;
    ctx->diag_cycles = cycles + 1;
    if (vecs) *vecs = std::move(X);
    *done = true;
    return MO_ED_OK;
}
template int plz_solve<float>(mo_ed_ctx *, const Sector &, int, std::vector<double> &, std::vector<DevBuf> *, bool *);
template int plz_solve<double>(mo_ed_ctx *, const Sector &, int, std::vector<double> &, std::vector<DevBuf> *, bool *);

}  // namespace moed
