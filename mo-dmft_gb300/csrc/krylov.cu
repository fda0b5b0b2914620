// krylov.cu -- Lanczos on the device.
//
//  * lz_* : the reference three-term recurrence (ed_lanczos.F90:14-68) as
//    batched kernels: update -> H*v (fused alpha partials) -> finalize, so
//    that every excitation vector of the Green's function advances in the
//    same three launches per step and no host round trip occurs.
//  * diag_sector : replaces the PARPACK 'SA' solve of diag()
//    (ed_solver.F90:107-191).  Sectors of some size go to the solver of
//    eigs.cu; here is a thick-restart Lanczos with full reorthogonalisation
//    (classical Gram-Schmidt, two passes) for small sectors, for a given
//    Krylov dimension (gs_ncv) and for what the other solver hands back.
//    Eigenvalues are returned as FP64 Rayleigh quotients of the Ritz vectors
//    (FP64-accumulated H*v for FP32 vectors; ritz_pairs in eigs.cu).
// All reductions are per-block partials summed in a fixed order (run-to-run
// deterministic).  Per-element work of FP32 vectors stays in FP32; FP64 is
// used once per 4-8 elements in the partial sums.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "hvrow.cuh"
#include "krylov.cuh"
#include "math64.cuh"
#include "symeig.h"
#include "vecops.cuh"

namespace moed {

static int dot_grid(mo_ed_ctx *ctx, long long n)
{
    long long g = (n + kVecThreads * 4 - 1) / (kVecThreads * 4);
    return (int)std::max(1LL, std::min(g, (long long)ctx->num_sms * 4));
}

int dot_dev(mo_ed_ctx *ctx, int prec_x, const void *x, int prec_y, const void *y, long long n,
            double *d_out)
{
    const int g = dot_grid(ctx, n);
    if (int rc = ensure(ctx, ctx->scratch_part, sizeof(double) * g)) return rc;
    double *part = (double *)ctx->scratch_part.p;
    if (prec_x == MO_ED_FP32 && prec_y == MO_ED_FP32)
        k_dot_part<float, float><<<g, kVecThreads, 0, ctx->stream>>>((const float *)x, (const float *)y, n, part);
    else if (prec_x == MO_ED_FP32)
        k_dot_part<float, double><<<g, kVecThreads, 0, ctx->stream>>>((const float *)x, (const double *)y, n, part);
    else if (prec_y == MO_ED_FP32)
        k_dot_part<double, float><<<g, kVecThreads, 0, ctx->stream>>>((const double *)x, (const float *)y, n, part);
    else
        k_dot_part<double, double><<<g, kVecThreads, 0, ctx->stream>>>((const double *)x, (const double *)y, n, part);
    MOED_CHECK_LAUNCH(ctx);
    k_sum_parts<<<1, kVecThreads, 0, ctx->stream>>>(part, g, d_out);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

template <typename TI, typename TO>
__global__ void k_convert(const TI *__restrict__ in, TO *__restrict__ out, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = (TO)in[i];
}

int convert_f64_to_f32(mo_ed_ctx *ctx, const double *in, float *out, long long n)
{
    if (n <= 0) return MO_ED_OK;
    k_convert<double, float><<<dot_grid(ctx, n), kVecThreads, 0, ctx->stream>>>(in, out, n);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

int convert_f32_to_f64(mo_ed_ctx *ctx, const float *in, double *out, long long n)
{
    if (n <= 0) return MO_ED_OK;
    k_convert<float, double><<<dot_grid(ctx, n), kVecThreads, 0, ctx->stream>>>(in, out, n);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

// ---------------------------------------------------------------------------
// reference recurrence, batched
// ---------------------------------------------------------------------------
__device__ __forceinline__ int find_run_upd(const LzBatchDev &b, int item)
{
    int r = 0;
    while (r + 1 < b.nrun && item >= b.run[r + 1].upd_item0) ++r;
    return r;
}

// step j = 0: partial sums of ||u_0||^2
template <typename T>
__global__ void k_lz_norm0(const __grid_constant__ LzBatchDev b)
{
    __shared__ double sred[32];
    for (int item = blockIdx.x; item < b.total_items; item += gridDim.x) {
        const int r = find_run_upd(b, item);
        const LzRunDev &R = b.run[r];
        const int it = item - R.upd_item0;
        const long long i0 = (long long)it * R.chunk, i1 = min(R.D, i0 + R.chunk);
        const T *u = (const T *)R.u[0];
        double acc = 0.0;
        for (long long i = i0 + threadIdx.x; i < i1; i += blockDim.x) acc += (double)u[i] * (double)u[i];
        double t = block_sum(acc, sred);
        if (threadIdx.x == 0) R.upd_part[it] = t;
    }
}

// step j >= 1: u_j = s (w - a_{j-1} u_{j-1}) - c u_{j-2},  s = 1/sqrt(b_{j-1}),
// c = sqrt(b_{j-1}/b_{j-2}) -- ed_lanczos.F90:38 (j = 1) and :54 (j >= 2)
// with the reference's normalized vectors written as scaled stored ones.
// 4 consecutive elements per thread (16-byte accesses; run lengths are
// multiples of 32 elements).
template <typename T>
__global__ void k_lz_update(const __grid_constant__ LzBatchDev b, int j)
{
    __shared__ double sred[kVecThreads];
    for (int item = blockIdx.x; item < b.total_items; item += gridDim.x) {
        const int r = find_run_upd(b, item);
        const LzRunDev &R = b.run[r];
        if (*R.active == 0) continue;
        const int it = item - R.upd_item0;
        const long long i0 = (long long)it * R.chunk, i1 = min(R.D, i0 + R.chunk);
        const T s = (T)R.inv[j - 1], a = (T)R.a[j - 1], c = (j >= 2) ? (T)R.cpl[j - 1] : T(0);
        const T *w = (const T *)R.w;
        const T *uc = (const T *)R.u[(j - 1) % 3];
        const T *up = (const T *)R.u[(j + 1) % 3];   // (j-2) mod 3
        T *un = (T *)R.u[j % 3];
        // ||u_j||^2: partials of 4 squares in T, added to the FP64 sum every
        // 8 iterations (per-element FP64 work would bound the kernel on GB300)
        double acc = 0.0;
        T sacc = T(0);
        int cnt = 0;
        for (long long i = i0 + 4 * threadIdx.x; i < i1; i += 4 * blockDim.x) {
            T wv[4], cv[4], pv[4], v[4];
            vload4(w + i, wv);
            vload4(uc + i, cv);
            if (j >= 2) {
                vload4(up + i, pv);
            } else {
                pv[0] = pv[1] = pv[2] = pv[3] = T(0);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                v[e] = (j >= 2) ? s * (wv[e] - a * cv[e]) - c * pv[e] : s * (wv[e] - a * cv[e]);
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
        if (threadIdx.x == 0) R.upd_part[it] = t;
    }
}

// nrm_j and a_j from the partials; the reference's stop test b(j) < 1.e-12
// (a default-REAL literal, ed_lanczos.F90:62) -- applied from j = 1 on.
__global__ void k_lz_finalize(const __grid_constant__ LzBatchDev b, int j, int nstep)
{
    __shared__ double sums[10];
    const LzRunDev &R = b.run[blockIdx.x];
    if (*R.active == 0) return;
    two_sums(R.upd_part, R.upd_nitems, R.hv_part, R.hv_nitems, sums);
    __syncthreads();
    if (threadIdx.x == 32) {               // next to warp 0, on another sub-partition's FP64 pipe
        double c = 0.0;
        if (j > 0) {
            const double last = R.nrm[j - 1], q = div_by(sums[0], last, rcp_pos(last));
            c = sqrt_by(q, rsqrt_pos(q));
        }
        R.cpl[j] = c;
    }
    if (threadIdx.x == 0) {
        const double nrm = sums[0], dot = sums[1];
        R.nrm[j] = nrm;
        if (j == 0 && nrm == 0.0) {        // zero start vector: no contribution
            R.a[0] = 0.0;
            *R.nstep_calc = 0;
            *R.active = 0;
            return;
        }
        R.a[j] = dot / nrm;
        // for the next update: square roots and divisions are tens of FP64
        // instructions, so not in its threads
        R.inv[j] = rsqrt_by(nrm, rsqrt_pos(nrm));
        const double tiny = (double)1.e-12f;
        if (j >= 1 && nrm < tiny) {
            *R.nstep_calc = j;
            *R.active = 0;
        } else if (j == nstep) {
            *R.nstep_calc = nstep;
            *R.active = 0;
        }
    }
}

void *lz_start_vector(LzBatch &b, int r) { return b.vecs[4 * r]; }

static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

int lz_setup(mo_ed_ctx *ctx, LzBatch &b, const std::vector<Sector> &secs, int prec, int nstep)
{
    const int nrun = (int)secs.size();
    if (nrun > kLzMaxRuns) return fail(ctx, MO_ED_ERR_ARG, "too many Lanczos runs in one batch");
    b.prec = prec;
    b.nstep = nstep;
    b.sec = secs;
    b.upd_item0.resize(nrun);
    b.upd_nitems.resize(nrun);
    b.hv_item0.resize(nrun);
    b.hv_nitems.resize(nrun);
    b.upd_total = b.hv_total = 0;
    const int kind = prec == MO_ED_FP32 ? HV_F32 : HV_F64;
    // one tile shape for the whole batch: the one tuned for its largest sector
    int big = 0;
    for (int r = 1; r < nrun; ++r)
        if (secs[r].D() > secs[big].D()) big = r;
    if (int rc = hv_prepare(ctx, secs[big], kind, &b.hv_variant, &b.hv_rows)) return rc;
    const size_t es = prec == MO_ED_FP32 ? sizeof(float) : sizeof(double);
    size_t vbytes = 0;
    for (int r = 0; r < nrun; ++r) {
        if (int rc = hv_prepare_rows(ctx, secs[r], kind, b.hv_variant)) return rc;
        const int chunk = vec_chunk(secs[r].Dpad());
        b.upd_item0[r] = b.upd_total;
        b.upd_nitems[r] = (int)((secs[r].Dpad() + chunk - 1) / chunk);
        b.upd_total += b.upd_nitems[r];
        b.hv_item0[r] = b.hv_total;
        b.hv_nitems[r] = secs[r].dn->nitems.at(b.hv_rows);
        b.hv_total += b.hv_nitems[r];
        vbytes += 4 * up256(es * (size_t)secs[r].Dpad());
    }
    // one workspace: the context's up to kLzHoldBytes, then from its pool (a
    // cudaMalloc costs more than several steps of a small sector)
    const size_t ncoef = (size_t)4 * (nstep + 1) * nrun;
    const size_t ocoef = vbytes, oflags = ocoef + up256(sizeof(double) * ncoef), oupd = oflags + up256(sizeof(int) * 2 * nrun);
    const size_t ohv = oupd + up256(sizeof(double) * std::max(1, b.upd_total));
    const size_t total = ohv + up256(sizeof(double) * std::max(1, b.hv_total));
    const bool hold = total <= kLzHoldBytes;
    if (int rc = hold ? ensure(ctx, ctx->lz_hold, total)
                      : total <= pool_keep(ctx) ? pool_alloc(ctx, b.own, total) : dev_alloc(ctx, b.own, total))
        return rc;
    char *base = (char *)(hold ? ctx->lz_hold.p : b.own.p);
    b.vecs.clear();
    size_t o = 0;
    for (int r = 0; r < nrun; ++r)
        for (int k = 0; k < 4; ++k) {
            b.vecs.push_back(base + o);
            o += up256(es * (size_t)secs[r].Dpad());
        }
    b.coef = (double *)(base + ocoef);
    b.flags = (int *)(base + oflags);
    b.upd_part = (double *)(base + oupd);
    b.hv_part = (double *)(base + ohv);
    MOED_CUDA(ctx, cudaMemsetAsync(b.coef, 0, sizeof(double) * ncoef, ctx->stream));
    std::vector<int> fl(2 * nrun);
    for (int r = 0; r < nrun; ++r) {
        fl[2 * r] = 1;
        fl[2 * r + 1] = 0;
    }
    MOED_CUDA(ctx, cudaMemcpyAsync(b.flags, fl.data(), sizeof(int) * 2 * nrun, cudaMemcpyHostToDevice, ctx->stream));
    return MO_ED_OK;
}

static void lz_fill_dev(LzBatch &b, LzBatchDev &d)
{
    const int nrun = (int)b.sec.size();
    memset(&d, 0, sizeof(d));
    d.nrun = nrun;
    d.total_items = b.upd_total;
    for (int r = 0; r < nrun; ++r) {
        LzRunDev &R = d.run[r];
        for (int k = 0; k < 3; ++k) R.u[k] = b.vecs[4 * r + k];
        R.w = b.vecs[4 * r + 3];
        R.D = b.sec[r].Dpad();
        R.chunk = vec_chunk(R.D);
        R.upd_item0 = b.upd_item0[r];
        R.upd_nitems = b.upd_nitems[r];
        R.hv_item0 = b.hv_item0[r];
        R.hv_nitems = b.hv_nitems[r];
        R.a = b.coef + (size_t)4 * (b.nstep + 1) * r;
        R.nrm = R.a + (b.nstep + 1);
        R.inv = R.nrm + (b.nstep + 1);
        R.cpl = R.inv + (b.nstep + 1);
        R.active = b.flags + 2 * r;
        R.nstep_calc = b.flags + 2 * r + 1;
        R.upd_part = b.upd_part + b.upd_item0[r];
        R.hv_part = b.hv_part + b.hv_item0[r];
    }
}

// All nstep+1 steps of a batch: 3 launches per step (4 with a split H*v), no
// host round trip (runs stop on the device through their active flags).  The
// launches go out faster than the kernels run, so a graph of them, used once,
// only adds its instantiation (50 FP64 steps of 0.73 million elements: 0.6 ms
// of 5.1 ms).
template <typename T>
static int lz_steps(mo_ed_ctx *ctx, LzBatch &b, LzBatchDev &d)
{
    const int nrun = d.nrun;
    const int kind = sizeof(T) == 4 ? HV_F32 : HV_F64;
    std::vector<HvJobT<T>> jobs[3];
    for (int k = 0; k < 3; ++k) {
        jobs[k].resize(nrun);
        for (int r = 0; r < nrun; ++r) {
            hv_fill_job<T>(ctx, b.sec[r], b.hv_rows, d.run[r].u[k], d.run[r].w, jobs[k][r]);
            jobs[k][r].dot_partial = d.run[r].hv_part;
            jobs[k][r].active = d.run[r].active;
        }
    }
    const int gv = std::max(1, std::min(d.total_items, ctx->num_sms * 8));
    for (int j = 0; j <= b.nstep; ++j) {
        if (j == 0) {
            k_lz_norm0<T><<<gv, kVecThreads, 0, ctx->stream>>>(d);
        } else {
            k_lz_update<T><<<gv, kVecThreads, 0, ctx->stream>>>(d, j);
        }
        MOED_CHECK_LAUNCH(ctx);
        int rc = (sizeof(T) == 4)
                     ? hv_launch_f32(ctx, b.hv_variant, (const HvJobT<float> *)jobs[j % 3].data(), nrun)
                     : hv_launch_f64(ctx, HV_F64, b.hv_variant, (const HvJobT<double> *)jobs[j % 3].data(), nrun);
        if (rc) return rc;
        k_lz_finalize<<<nrun, kVecThreads, 0, ctx->stream>>>(d, j, b.nstep);
        MOED_CHECK_LAUNCH(ctx);
    }
    return MO_ED_OK;
}

int lz_run(mo_ed_ctx *ctx, LzBatch &b, std::vector<std::vector<double>> &a,
           std::vector<std::vector<double>> &bb, std::vector<int> &nstep_calc)
{
    LzBatchDev d;
    lz_fill_dev(b, d);
    const int nrun = d.nrun;
    int rc = (b.prec == MO_ED_FP32) ? lz_steps<float>(ctx, b, d) : lz_steps<double>(ctx, b, d);
    if (rc) return rc;
    std::vector<double> coef((size_t)4 * (b.nstep + 1) * nrun);
    std::vector<int> fl(2 * nrun);
    MOED_CUDA(ctx, cudaMemcpyAsync(coef.data(), b.coef, sizeof(double) * coef.size(),
                                   cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaMemcpyAsync(fl.data(), b.flags, sizeof(int) * fl.size(),
                                   cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    a.assign(nrun, std::vector<double>(b.nstep + 1, 0.0));
    bb.assign(nrun, std::vector<double>(b.nstep + 1, 0.0));
    nstep_calc.assign(nrun, 0);
    for (int r = 0; r < nrun; ++r) {
        const double *ar = coef.data() + (size_t)4 * (b.nstep + 1) * r;
        const double *nr = ar + (b.nstep + 1);
        nstep_calc[r] = fl[2 * r + 1];
        for (int j = 0; j <= b.nstep; ++j) {
            a[r][j] = ar[j];
            bb[r][j] = (j == 0) ? 0.0 : nr[j];
        }
    }
    return MO_ED_OK;
}

int lanczos_reference(mo_ed_ctx *ctx, const Sector &s, const double *h_vec, int nstep,
                      int *nstep_calc, double *a, double *b)
{
    LzBatch lb;
    const int prec = ctx->opt.precision;
    if (int rc = lz_setup(ctx, lb, {s}, prec, nstep)) return rc;
    const long long Dp = s.Dpad();
    if (prec == MO_ED_FP32) {
        if (int rc = ensure(ctx, ctx->scratch_a, sizeof(double) * Dp)) return rc;
        if (int rc = upload_padded(ctx, s, h_vec, ctx->scratch_a.p, sizeof(double))) return rc;
        if (int rc = convert_f64_to_f32(ctx, (const double *)ctx->scratch_a.p,
                                        (float *)lz_start_vector(lb, 0), Dp))
            return rc;
    } else {
        if (int rc = upload_padded(ctx, s, h_vec, lz_start_vector(lb, 0), sizeof(double))) return rc;
    }
    std::vector<std::vector<double>> A, B;
    std::vector<int> nc;
    if (int rc = lz_run(ctx, lb, A, B, nc)) return rc;
    *nstep_calc = nc[0];
    for (int j = 0; j <= nstep; ++j) {
        a[j] = A[0][j];
        b[j] = B[0][j];
    }
    return MO_ED_OK;
}

// The same recurrence inside a caller-provided device region.  Layout, each
// part starting on a 256-byte boundary: a, nrm, inv, cpl [nstep+1] each, the two
// flags, the update and H*v partial sums, u_0, u_1 u_2 (adjacent; for FP32
// runs they first hold the FP64 start vector before its conversion) and w.
namespace {
struct LzRegion {
    size_t coef, flags, upd, hv, u0, u12, w, end;
};

LzRegion lz_region(const Sector &s, int prec, int nstep, int hv_rows)
{
    const size_t es = prec == MO_ED_FP32 ? sizeof(float) : sizeof(double);
    const size_t Dp = (size_t)s.Dpad();
    const size_t upd_n = (Dp + vec_chunk((long long)Dp) - 1) / vec_chunk((long long)Dp);
    const size_t hv_n = (size_t)std::max(1, s.dn->nitems.at(hv_rows));
    LzRegion r;
    r.coef = 0;
    r.flags = up256(r.coef + sizeof(double) * 4 * (size_t)(nstep + 1));
    r.upd = up256(r.flags + sizeof(int) * 2);
    r.hv = up256(r.upd + sizeof(double) * upd_n);
    r.u0 = up256(r.hv + sizeof(double) * hv_n);
    r.u12 = up256(r.u0 + es * Dp);
    r.w = up256(r.u12 + std::max(2 * es * Dp, prec == MO_ED_FP32 ? sizeof(double) * Dp : 0));
    r.end = up256(r.w + es * Dp);
    return r;
}

// a = nrm = 0, active = 1, nstep_calc = 0 (the region keeps an earlier call's contents)
__global__ void k_lz_reset(const __grid_constant__ LzBatchDev b, int nstep)
{
    const LzRunDev &R = b.run[blockIdx.x];
    for (int j = threadIdx.x; j <= nstep; j += blockDim.x) {
        R.a[j] = 0.0;
        R.nrm[j] = 0.0;
    }
    if (threadIdx.x == 0) {
        *R.active = 1;
        *R.nstep_calc = 0;
    }
}
}  // namespace

// Load the kernel only the region path uses (lazy loading would otherwise
// load it, and may take device memory, on the first no-allocation call).
int lanczos_region_preload(mo_ed_ctx *ctx)
{
    cudaFuncAttributes a;
    MOED_CUDA(ctx, cudaFuncGetAttributes(&a, k_lz_reset));
    return MO_ED_OK;
}

size_t lanczos_region_bytes(const Sector &s, int prec, int nstep, int hv_rows)
{
    return lz_region(s, prec, nstep, hv_rows).end;
}

int lanczos_reference_in(mo_ed_ctx *ctx, const Sector &s, const double *h_vec, int nstep,
                         int *nstep_calc, double *a, double *b, void *scratch, size_t cap)
{
    const int prec = ctx->opt.precision;
    const int kind = prec == MO_ED_FP32 ? HV_F32 : HV_F64;
    LzBatch lb;
    lb.prec = prec;
    lb.nstep = nstep;
    lb.sec = {s};
    if (int rc = hv_lookup(ctx, s, kind, &lb.hv_variant, &lb.hv_rows)) return rc;
    const LzRegion g = lz_region(s, prec, nstep, lb.hv_rows);
    if (g.end > cap || ((size_t)scratch & 255)) return fail(ctx, MO_ED_ERR_CAPACITY, "Lanczos region too small");
    char *base = (char *)scratch;
    const size_t es = prec == MO_ED_FP32 ? sizeof(float) : sizeof(double);
    const long long Dp = s.Dpad();

    LzBatchDev d;
    memset(&d, 0, sizeof(d));
    d.nrun = 1;
    LzRunDev &R = d.run[0];
    R.u[0] = base + g.u0;
    R.u[1] = base + g.u12;
    R.u[2] = base + g.u12 + es * (size_t)Dp;
    R.w = base + g.w;
    R.D = Dp;
    R.upd_item0 = 0;
    R.chunk = vec_chunk(Dp);
    R.upd_nitems = (int)((Dp + R.chunk - 1) / R.chunk);
    R.hv_item0 = 0;
    R.hv_nitems = s.dn->nitems.at(lb.hv_rows);
    R.a = (double *)(base + g.coef);
    R.nrm = R.a + (nstep + 1);
    R.inv = R.nrm + (nstep + 1);
    R.cpl = R.inv + (nstep + 1);
    R.active = (int *)(base + g.flags);
    R.nstep_calc = R.active + 1;
    R.upd_part = (double *)(base + g.upd);
    R.hv_part = (double *)(base + g.hv);
    d.total_items = R.upd_nitems;

    k_lz_reset<<<1, kVecThreads, 0, ctx->stream>>>(d, nstep);
    MOED_CHECK_LAUNCH(ctx);
    if (prec == MO_ED_FP32) {
        double *stage = (double *)(base + g.u12);
        if (int rc = upload_padded(ctx, s, h_vec, stage, sizeof(double))) return rc;
        if (int rc = convert_f64_to_f32(ctx, stage, (float *)R.u[0], Dp)) return rc;
        if (int rc = lz_steps<float>(ctx, lb, d)) return rc;
    } else {
        if (int rc = upload_padded(ctx, s, h_vec, R.u[0], sizeof(double))) return rc;
        if (int rc = lz_steps<double>(ctx, lb, d)) return rc;
    }
    MOED_CUDA(ctx, cudaMemcpyAsync(a, R.a, sizeof(double) * (nstep + 1), cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaMemcpyAsync(b, R.nrm, sizeof(double) * (nstep + 1), cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaMemcpyAsync(nstep_calc, R.nstep_calc, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    b[0] = 0.0;
    return MO_ED_OK;
}

// ---------------------------------------------------------------------------
// thick-restart Lanczos with full reorthogonalisation (diag replacement)
// ---------------------------------------------------------------------------
constexpr int kTrlMaxNcv = 200;
constexpr size_t kTrlPoolBytes = (size_t)64 << 20;   // largest pooled Krylov vector

// column j of the projected matrix (the two CGS passes' coefficients h1 + h2),
// beta, 1/beta
__global__ void k_cgs_finish(const double *h1, const double *h2, int nv, const double *norm_part, int G,
                             double *Hcol, double *beta_out)
{
    __shared__ double sred[32];
    for (int l = threadIdx.x; l < nv; l += blockDim.x) Hcol[l] = h1[l] + h2[l];
    double acc = 0.0;
    for (int i = threadIdx.x; i < G; i += blockDim.x) acc += norm_part[i];
    double t = block_sum(acc, sred);
    if (threadIdx.x == 0) {
        double beta = sqrt(t);
        Hcol[nv] = beta;
        beta_out[0] = beta;
        beta_out[1] = beta > 0 ? 1.0 / beta : 0.0;
    }
}

template <typename T>
__global__ void k_scale_copy(const T *__restrict__ in, T *__restrict__ out, long long n,
                             const double *scale)
{
    const T s = (T)*scale;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = in[i] * s;
}

// Where the coefficients of the two CGS passes of an orthogonalize call are.
struct OrthoCoef {
    const double *p[2];
};

// part of orthogonalize: the dots' partials, their sums, and the two passes'
// coefficients
static size_t ortho_part_doubles(const mo_ed_ctx *ctx) { return dots_part_doubles(ctx) + 3 * (kMaxNcv + 2); }

// classical Gram-Schmidt, twice: w -= V (V^T w).  Each pass is a multi-dot
// and a multi-axpy; pass 1 leaves the axpys_blocks partials of ||w||^2 in norm_part.
template <typename T>
static int orthogonalize(mo_ed_ctx *ctx, const std::vector<DevBuf *> &basis, int nv, T *w,
                         long long D, double *part, double *norm_part, OrthoCoef *coef = nullptr)
{
    VPtrs<T> P = make_ptrs<T>(basis, nv);
    double *sums = part + dots_part_doubles(ctx);
    for (int pass = 0; pass < 2; ++pass) {
        double *hp = sums + (1 + pass) * (kMaxNcv + 2);
        const double *src;
        int rows;
        if (int rc = dots<T, 1>(ctx, P, nv, WPtrs<T>{{w, nullptr}}, D, part, sums, &src, &rows)) return rc;
        if (int rc = axpys<T, 1>(ctx, P, nv, src, rows, nullptr, WPtrs<T>{{w, nullptr}}, D,
                                 pass == 1 ? norm_part : nullptr, hp, 0))
            return rc;
        if (coef) coef->p[pass] = hp;
    }
    return MO_ED_OK;
}

// Steps k .. ncv - 1 of a cycle (H*v, two Gram-Schmidt passes against V_0 ..
// V_j, column j of the projected matrix, V_{j+1}) in one CTA, for sectors of
// up to kTsMaxDim elements: seven launches per step otherwise, 25 us of
// latency.  V_j and w are in shared memory (without row
// pads: jb.ld = nu), the earlier vectors in L1; a warp per dot.  start: w of
// the first vector, normalised here (else V_k is given).  A step of 70
// elements: 6 us.
constexpr int kTsThreads = 256;
constexpr long long kTsMaxDim = 1024;
template <typename T>
__global__ void __launch_bounds__(kTsThreads)
k_trl_steps(const __grid_constant__ HvJobT<T> jb, const ModelDev *__restrict__ mdl, const __grid_constant__ VPtrs<T> V,
            const T *start, int k, int ncv, int ld, double *__restrict__ Hp, int ldh)
{
    constexpr int NT = kTsThreads, NWARP = NT / 32;
    extern __shared__ double raw[];
    const int nimp = mdl->nimp, npair = mdl->npair, nu = jb.nu, nd = jb.nd, n = nu * nd;
    T *const xs = (T *)raw, *const ws = xs + n;
    int *const at = (int *)(ws + n);
    __shared__ T s_cross[kMaxImp * kMaxImp];
    __shared__ unsigned s_pmask[kMaxImp];
    __shared__ int s_t4[kMaxPair * kMaxImp];
    __shared__ double s_h[2][kTrlMaxNcv + 1], s_red[32], s_sc[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < npair * nimp; i += NT) s_t4[i] = mdl->t4[i];
    for (int i = tid; i < nimp; i += NT) s_pmask[i] = mdl->pairmask[i];
    for (int i = tid; i < nimp * nimp; i += NT) s_cross[i] = (T)mdl->cross[i];
    for (int d = wid; d < nd; d += NWARP)
        for (int u = lane; u < nu; u += 32) at[d * nu + u] = d * ld + u;
    const T Jc = (T)mdl->J;
    __syncthreads();
    // ||w|| and its inverse, fixed order
    const auto norm = [&] {
        double a = 0.0;
        for (int i = tid; i < n; i += NT) {
            const double v = widen(ws[i]);
            a = fma(v, v, a);
        }
        a = block_sum(a, s_red);
        if (tid == 0) {
            const double inv = a > 0.0 ? rsqrt_pos(a) : 0.0;
            s_sc[0] = a > 0.0 ? a * inv : a;
            s_sc[1] = inv;
        }
        __syncthreads();
    };
    // xs = w / ||w||, and to global memory with zero pads
    const auto put = [&](T *v) {
        const T s = (T)s_sc[1];
        for (int i = tid; i < n; i += NT) v[at[i]] = xs[i] = ws[i] * s;
        for (int d = wid; d < nd; d += NWARP)
            for (int u = nu + lane; u < ld; u += 32) v[d * ld + u] = T(0);
        __syncthreads();
    };
    if (start) {
        for (int i = tid; i < n; i += NT) ws[i] = start[at[i]];
        __syncthreads();
        norm();
        put(const_cast<T *>(V.p[k]));
    } else {
        for (int i = tid; i < n; i += NT) xs[i] = V.p[k][at[i]];
        __syncthreads();
    }
    for (int j = k; j < ncv; ++j) {
        for (int i = tid; i < n; i += NT) {
            const int d = i / nu, u = i - d * nu, inf = __ldg(jb.up_info + u), dinf = __ldg(jb.dn_info + d);
            const T diag = __ldg(jb.up_diag + u) + __ldg(jb.dn_diag + d) +
                           s_cross[((inf >> 8) & 0xff) * nimp + ((dinf >> 8) & 0xff)];
            ws[i] = hv_moves<T, T, false>(jb, mdl, xs, d, u, inf, dinf, s_pmask, s_t4, nimp, Jc, diag * xs[i]);
        }
        __syncthreads();
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            for (int l = wid; l <= j; l += NWARP) {
                const T *v = V.p[l];
                T s = T(0);
                for (int i = lane; i < n; i += 32) s += v[at[i]] * ws[i];
                s = warp_sum(s);
                if (lane == 0) s_h[pass][l] = widen(s);
            }
            __syncthreads();
            for (int i = tid; i < n; i += NT) {
                T w = ws[i];
#pragma unroll 4
                for (int l = 0; l <= j; ++l) w -= (T)s_h[pass][l] * V.p[l][at[i]];
                ws[i] = w;
            }
            __syncthreads();
        }
        norm();
        for (int l = tid; l <= j; l += NT) Hp[(size_t)j * ldh + l] = s_h[0][l] + s_h[1][l];
        if (tid == 0) Hp[(size_t)j * ldh + j + 1] = s_sc[0];
        if (j + 1 >= n) break;
        put(const_cast<T *>(V.p[j + 1]));
    }
}

template <typename T>
static int trl_solve(mo_ed_ctx *ctx, const Sector &s, int nev, std::vector<double> &vals,
                     std::vector<DevBuf> *vecs)
{
    const long long D = s.D();          // dimension
    const long long Dp = s.Dpad();      // device elements (row pads are zero)
    const int prec = sizeof(T) == 4 ? MO_ED_FP32 : MO_ED_FP64;
    const int kind = sizeof(T) == 4 ? HV_F32 : HV_F64;
    const int nwant = (int)std::min<long long>(nev, D);
    int ncv = ctx->opt.gs_ncv > 0 ? ctx->opt.gs_ncv : std::max(2 * nwant + 10, 40);
    ncv = (int)std::min<long long>(std::min(ncv, kTrlMaxNcv - 1), D);
    if (ncv < nwant) return fail(ctx, MO_ED_ERR_ARG, "gs_ncv smaller than nev");
    int kkeep = std::min(ncv - 1, nwant + (ncv - nwant) / 2);
    if (kkeep < nwant) kkeep = nwant;
    // Residual tolerance relative to ||H||.  FP32 vectors carry a noise floor
    // near eps_32*||H||; the stagnation test below accepts Ritz pairs that
    // stop improving there.
    const double tol = ctx->opt.gs_tol > 0 ? ctx->opt.gs_tol : (prec == MO_ED_FP32 ? 1e-7 : 1e-11);
    std::vector<double> res_hist;
    const size_t vb = sizeof(T) * (size_t)Dp;

    // Krylov vectors: sectors up to kTrlPoolBytes per vector reuse buffers kept
    // in the context (many small sectors: no allocation per sector)
    std::vector<DevBuf> local;
    std::vector<DevBuf> &store = vb <= kTrlPoolBytes ? ctx->trl_pool : local;
    if (store.size() < (size_t)(ncv + 2 + kkeep)) store.resize(ncv + 2 + kkeep);
    for (int i = 0; i < ncv + 2 + kkeep; ++i)
        if (int rc = ensure(ctx, store[i], vb)) return rc;
    std::vector<DevBuf *> V(ncv + 1);
    for (int i = 0; i <= ncv; ++i) V[i] = &store[i];
    DevBuf *W = &store[ncv + 1];
    std::vector<DevBuf *> spare(kkeep);
    for (int i = 0; i < kkeep; ++i) spare[i] = &store[ncv + 2 + i];

    const int G = (int)std::max(1LL, std::min((Dp + kVecThreads - 1) / kVecThreads, (long long)ctx->num_sms * 4));
    const int n2 = ncv + 2;
    std::vector<DevBuf> &sm = ctx->trl_small;   // projected-problem workspace, kept in the context
    if (sm.size() < 12) sm.resize(12);
    DevBuf &dHp = sm[0], &dh1 = sm[1], &dh2 = sm[2], &dpart = sm[3], &dnorm = sm[4], &dbeta = sm[5];
    DevBuf &devecs = sm[9], &dsc = sm[11];
    if (int rc = ensure(ctx, dHp, sizeof(double) * (size_t)n2 * n2)) return rc;
    if (int rc = ensure(ctx, dh1, sizeof(double) * n2)) return rc;
    if (int rc = ensure(ctx, dh2, sizeof(double) * n2)) return rc;
    if (int rc = ensure(ctx, dpart, sizeof(double) * ortho_part_doubles(ctx))) return rc;
    if (int rc = ensure(ctx, dnorm, sizeof(double) * axpys_blocks(ctx, Dp))) return rc;
    if (int rc = ensure(ctx, dbeta, sizeof(double) * 2)) return rc;
    if (int rc = ensure(ctx, devecs, sizeof(double) * (size_t)n2 * n2)) return rc;
    if (int rc = ensure(ctx, dsc, sizeof(double) * 4)) return rc;
    MOED_CUDA(ctx, cudaMemsetAsync(dHp.p, 0, dHp.bytes, ctx->stream));
    double *Hp = (double *)dHp.p;
    const int ldh = n2;

    long long matvecs = 0;
    auto hv = [&](const void *x, void *y) -> int {
        ++matvecs;
        return hv_single(ctx, s, kind, x, y);
    };
    auto normalize_into = [&](T *src, DevBuf *dst) -> int {
        // dst = src / ||src||
        if (int rc = dot_dev(ctx, prec, src, prec, src, Dp, (double *)dsc.p)) return rc;
        double nrm2;
        MOED_CUDA(ctx, cudaMemcpyAsync(&nrm2, dsc.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        double inv = nrm2 > 0 ? 1.0 / std::sqrt(nrm2) : 0.0;
        MOED_CUDA(ctx, cudaMemcpyAsync((double *)dsc.p + 1, &inv, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
        k_scale_copy<T><<<G, kVecThreads, 0, ctx->stream>>>(src, (T *)dst->p, Dp, (double *)dsc.p + 1);
        MOED_CHECK_LAUNCH(ctx);
        return MO_ED_OK;
    };

    // small sectors: a cycle's steps in one launch
    HvJobT<T> job;
    bool small = false;
    if (D <= kTsMaxDim) {
        if (int rc = hv_row_job<T>(ctx, s, kind, &job, &small)) return rc;
        job.ld = job.nu;
    }

    // start vector
    unsigned long long seed = 0x5eedULL + 977ULL * (unsigned)s.ne_up + 131ULL * (unsigned)s.ne_down;
    k_random<T><<<G, kVecThreads, 0, ctx->stream>>>((T *)W->p, Dp, s.ld(), s.up->n, seed);
    MOED_CHECK_LAUNCH(ctx);
    const T *start = small ? (const T *)W->p : nullptr;
    if (!small)
        if (int rc = normalize_into((T *)W->p, V[0])) return rc;

    int k = 0;           // kept Ritz vectors at the front of V
    int m = ncv;
    std::vector<double> theta(n2), ylast(n2), evecs_h;
    bool done = false;
    int cycle = 0;
    double anorm = 0.0;
    // A Krylov space holds one vector of each eigenspace.  Where the model can
    // have exactly degenerate levels, the converged vectors are
    // kept and a fresh random direction goes on from there, until one adds no
    // level to the lowest ones: the values before it, or empty
    std::vector<double> known;
    const bool search = ctx->degenerate && ncv >= nwant + 2;
    for (; cycle < ctx->opt.gs_maxcycles && !done; ++cycle) {
        m = ncv;
        // The steps of a cycle run without a host round trip; the diagonal and
        // the betas are read once at the end of the cycle.  A step whose beta
        // falls below the breakdown threshold ends the cycle there (its Krylov
        // space is invariant; later steps of the cycle are discarded).
        if (small) {
            m = (int)std::min<long long>(ncv, D);
            k_trl_steps<T><<<1, kTsThreads, (2 * sizeof(T) + sizeof(int)) * (size_t)D, ctx->stream>>>(
                job, ctx->d_mdl, make_ptrs<T>(V, ncv + 1), start, k, ncv, s.ld(), Hp, ldh);
            MOED_CHECK_LAUNCH(ctx);
            matvecs += m - k;
            start = nullptr;
        }
        for (int j = small ? ncv : k; j < ncv; ++j) {
            if (int rc = hv(V[j]->p, W->p)) return rc;
            const bool last = j + 1 >= D;   // Krylov space is the whole sector
            OrthoCoef oc;
            if (int rc = orthogonalize<T>(ctx, V, j + 1, (T *)W->p, Dp, (double *)dpart.p, (double *)dnorm.p, &oc))
                return rc;
            k_cgs_finish<<<1, 256, 0, ctx->stream>>>(oc.p[0], oc.p[1], j + 1, (const double *)dnorm.p, axpys_blocks(ctx, Dp),
                                                     Hp + (size_t)j * ldh, (double *)dbeta.p);
            MOED_CHECK_LAUNCH(ctx);
            if (!last) {
                k_scale_copy<T><<<G, kVecThreads, 0, ctx->stream>>>((const T *)W->p, (T *)V[j + 1]->p, Dp,
                                                                    (double *)dbeta.p + 1);
                MOED_CHECK_LAUNCH(ctx);
            }
            if (last) {
                m = j + 1;
                break;
            }
        }
        bool broke = false;
        std::vector<double> hc((size_t)ldh * m);
        {
            MOED_CUDA(ctx, cudaMemcpyAsync(hc.data(), Hp, sizeof(double) * hc.size(), cudaMemcpyDeviceToHost, ctx->stream));
            MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            for (int j = k; j < m; ++j) {
                const double diag = hc[(size_t)j * ldh + j], beta = hc[(size_t)j * ldh + j + 1];
                anorm = std::max(anorm, std::fabs(diag) + beta);
                if (j + 1 >= D) break;
                const double bd = (prec == MO_ED_FP32 ? 1e-5 : 1e-12) * std::max(anorm, 1.0);
                if (beta <= bd) {
                    m = j + 1;
                    broke = true;
                    break;
                }
            }
        }
        // Rayleigh-Ritz on span V[0..m-1], on the host as PARPACK does: the
        // projected matrix is diag(theta) on the kept block and the columns
        // of Hp after it (its entries are on the host already)
        evecs_h.resize((size_t)m * m);
        {
            std::vector<double> Am((size_t)m * m);
            for (int i = 0; i < m; ++i)
                for (int j = 0; j < m; ++j) {
                    const int r = std::min(i, j), c = std::max(i, j);
                    Am[(size_t)i * m + j] = c < k ? (r == c ? theta[r] : 0.0) : hc[(size_t)c * ldh + r];
                }
            if (!sym_eig(m, Am, theta.data(), evecs_h.data()))
                return fail(ctx, MO_ED_ERR_NOCONV, "projected eigenproblem did not converge");
            MOED_CUDA(ctx, cudaMemcpyAsync(devecs.p, evecs_h.data(), sizeof(double) * (size_t)m * m,
                                           cudaMemcpyHostToDevice, ctx->stream));
        }
        const double beta_m = m < D ? hc[(size_t)(m - 1) * ldh + m] : 0.0;
        int nconv = 0;
        double maxres = 0.0;
        for (int i = 0; i < std::min(nwant, m); ++i) {
            double res = std::fabs(beta_m * evecs_h[(size_t)i * m + (m - 1)]);
            maxres = std::max(maxres, res);
            if (res <= tol * std::max(anorm, 1.0) && nconv == i) ++nconv;
        }
        res_hist.push_back(maxres);
        ctx->diag_res_est = maxres;
        const size_t h = res_hist.size();
        const bool stalled = prec == MO_ED_FP32 && h >= 6 && maxres <= 1e-6 * std::max(anorm, 1.0) &&
                             maxres > 0.9 * res_hist[h - 6];
        const bool converged = nconv >= nwant || stalled;
        if (m >= D || (converged && (!search || cycle + 1 >= ctx->opt.gs_maxcycles))) {
            done = true;
            break;
        }
        // thick restart: keep kkeep lowest Ritz vectors, then the residual vector
        // after a breakdown every Ritz vector of the invariant subspace is kept
        bool fresh = broke;
        int kk = broke ? std::min(kkeep, m) : std::min(kkeep, m - 1);
        if (converged) {
            // the value after the wanted ones has to be known as well (1e-3 of
            // its distance from them: KryRun::go, eigs.cu; 1e-6 is where FP32
            // residuals stop falling)
            const double an = std::max(anorm, 1.0);
            bool settled = known.empty() || broke;
            if (!settled && m > nwant)
                settled = std::fabs(beta_m * evecs_h[(size_t)nwant * m + (m - 1)]) <=
                          std::max(1e-3 * (theta[nwant] - theta[nwant - 1]), (prec == MO_ED_FP32 ? 1e-6 : tol) * an);
            if (settled) {
                bool same = !known.empty();
                for (size_t i = 0; i < known.size(); ++i) same = same && known[i] - theta[i] <= 10 * tol * an;
                if (same) {
                    done = true;
                    break;
                }
                known.assign(theta.begin(), theta.begin() + nwant);
                res_hist.clear();
                fresh = true;
                kk = nwant;   // converged vectors only: the others leave a residual along V_m
            }
        }
        VPtrs<T> P = make_ptrs<T>(V, m);
        for (int c0 = 0; c0 < kk; c0 += 8) {
            const int nc = std::min(8, kk - c0);
            std::vector<DevBuf *> outs(spare.begin() + c0, spare.begin() + c0 + nc);
            VPtrs<T> X = make_ptrs<T>(outs, nc);
            if (int rc = rotate<T>(ctx, G, P, m, (const double *)devecs.p, m, c0, nc, X, Dp)) return rc;
        }
        for (int i = 0; i < kk; ++i) std::swap(V[i], spare[i]);
        if (fresh) {
            // invariant subspace, or a search: continue from a fresh random direction
            k_random<T><<<G, kVecThreads, 0, ctx->stream>>>((T *)W->p, Dp, s.ld(), s.up->n,
                                                            seed + 7919ULL * (cycle + 1) * kTrlMaxNcv);
            MOED_CHECK_LAUNCH(ctx);
            if (int rc = orthogonalize<T>(ctx, V, kk, (T *)W->p, Dp, (double *)dpart.p, (double *)dnorm.p))
                return rc;
            if (int rc = normalize_into((T *)W->p, V[kk])) return rc;
        } else {
            std::swap(V[kk], V[m]);
        }
        k = kk;
        MOED_CUDA(ctx, cudaMemsetAsync(dHp.p, 0, dHp.bytes, ctx->stream));
    }
    if (!done) return fail(ctx, MO_ED_ERR_NOCONV, "eigensolver did not converge");

    // Ritz vectors, then an FP64-accurate Rayleigh-Ritz on their span
    VPtrs<T> P = make_ptrs<T>(V, m);
    ctx->diag_cycles = cycle + 1;
    return ritz_pairs<T>(ctx, s, P, m, (const double *)devecs.p, nwant, nev, matvecs, vals, vecs);
}

// FP64 refinement of an FP32 eigenvector x (Dpad elements of sector s).
// The FP32 eigensolve leaves a residual near eps_32 * ||H|| in x, spread over
// the whole spectrum.  A Lanczos run of kRefineSteps FP64 steps from x (full
// CGS2 reorthogonalisation) and a Rayleigh-Ritz on its Krylov space damp every
// component away from the eigenvalue; the Ritz vector with the largest weight
// on x is the refined vector.  Rounds repeat from it until the Ritz residual
// is below 1e-9 * ||H|| or kRefineRounds have run: G(i w_n) inherits the
// vector's error to first order, and a residual 1e-9 * ||H|| leaves it near
// 1e-8 relative.  out receives the FP64 vector; res the last Ritz residual.
int refine_fp64(mo_ed_ctx *ctx, const Sector &s, const float *x, DevBuf &out, double *res)
{
    constexpr int kRefineSteps = 16, kRefineRounds = 3;
    const long long D = s.D(), Dp = s.Dpad();
    const int m0 = (int)std::min<long long>(kRefineSteps, D);
    const size_t vb = sizeof(double) * (size_t)Dp;
    std::vector<DevBuf> buf(m0 + 1);
    for (auto &b : buf)
        if (int rc = dev_alloc(ctx, b, vb)) return rc;
    std::vector<DevBuf *> V(m0);
    for (int i = 0; i < m0; ++i) V[i] = &buf[i];
    DevBuf *W = &buf[m0];
    const int G = (int)std::max(1LL, std::min((Dp + kVecThreads - 1) / kVecThreads, (long long)ctx->num_sms * 4));
    const int n2 = m0 + 2, ldh = n2;
    DevBuf dHp, dh1, dh2, dpart, dnorm, dbeta, devecs, dsc;
    if (int rc = dev_alloc(ctx, dHp, sizeof(double) * (size_t)n2 * n2)) return rc;
    if (int rc = dev_alloc(ctx, dh1, sizeof(double) * n2)) return rc;
    if (int rc = dev_alloc(ctx, dh2, sizeof(double) * n2)) return rc;
    if (int rc = dev_alloc(ctx, dpart, sizeof(double) * ortho_part_doubles(ctx))) return rc;
    if (int rc = dev_alloc(ctx, dnorm, sizeof(double) * axpys_blocks(ctx, Dp))) return rc;
    if (int rc = dev_alloc(ctx, dbeta, sizeof(double) * 2)) return rc;
    if (int rc = dev_alloc(ctx, devecs, sizeof(double) * (size_t)n2 * n2)) return rc;
    if (int rc = dev_alloc(ctx, dsc, sizeof(double) * 2)) return rc;
    if (int rc = dev_alloc(ctx, out, vb)) return rc;
    if (int rc = convert_f32_to_f64(ctx, x, (double *)out.p, Dp)) return rc;
    double *Hp = (double *)dHp.p;
    *res = -1.0;
    for (int round = 0; round < kRefineRounds; ++round) {
        // V[0] = out / ||out||
        if (int rc = dot_dev(ctx, MO_ED_FP64, out.p, MO_ED_FP64, out.p, Dp, (double *)dsc.p)) return rc;
        double nrm2 = 0.0;
        MOED_CUDA(ctx, cudaMemcpyAsync(&nrm2, dsc.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (!(nrm2 > 0)) return fail(ctx, MO_ED_ERR_NOCONV, "zero eigenvector in FP64 refinement");
        const double inv = 1.0 / std::sqrt(nrm2);
        MOED_CUDA(ctx, cudaMemcpyAsync((double *)dsc.p + 1, &inv, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
        k_scale_copy<double><<<G, kVecThreads, 0, ctx->stream>>>((const double *)out.p, (double *)V[0]->p, Dp,
                                                                 (double *)dsc.p + 1);
        MOED_CHECK_LAUNCH(ctx);
        MOED_CUDA(ctx, cudaMemsetAsync(dHp.p, 0, dHp.bytes, ctx->stream));
        // the steps run without a host round trip; a breakdown is found
        // afterwards and ends the Krylov space there (later steps are discarded)
        for (int j = 0; j < m0; ++j) {
            if (int rc = hv_single(ctx, s, HV_F64, V[j]->p, W->p)) return rc;
            OrthoCoef oc;
            if (int rc = orthogonalize<double>(ctx, V, j + 1, (double *)W->p, Dp, (double *)dpart.p,
                                               (double *)dnorm.p, &oc))
                return rc;
            k_cgs_finish<<<1, 256, 0, ctx->stream>>>(oc.p[0], oc.p[1], j + 1, (const double *)dnorm.p, axpys_blocks(ctx, Dp),
                                                     Hp + (size_t)j * ldh, (double *)dbeta.p);
            MOED_CHECK_LAUNCH(ctx);
            if (j + 1 < m0) {
                k_scale_copy<double><<<G, kVecThreads, 0, ctx->stream>>>((const double *)W->p, (double *)V[j + 1]->p,
                                                                         Dp, (double *)dbeta.p + 1);
                MOED_CHECK_LAUNCH(ctx);
            }
        }
        std::vector<double> hc((size_t)ldh * m0);
        MOED_CUDA(ctx, cudaMemcpyAsync(hc.data(), Hp, sizeof(double) * hc.size(), cudaMemcpyDeviceToHost, ctx->stream));
        MOED_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        int m = m0;
        double anorm = 0.0, beta_m = 0.0;
        for (int j = 0; j < m0; ++j) {
            const double diag = hc[(size_t)j * ldh + j], beta = hc[(size_t)j * ldh + j + 1];
            anorm = std::max(anorm, std::fabs(diag) + beta);
            beta_m = beta;
            if (j + 1 >= D || beta <= 1e-12 * std::max(anorm, 1.0)) {
                m = j + 1;
                beta_m = 0.0;   // invariant subspace: its Ritz pairs are exact
                break;
            }
        }
        // the projected tridiagonal problem on the host (symeig.h)
        std::vector<double> Am((size_t)m * m), w(m), ev((size_t)m * m);
        for (int i = 0; i < m; ++i)
            for (int j = 0; j < m; ++j) Am[(size_t)i * m + j] = hc[(size_t)std::max(i, j) * ldh + std::min(i, j)];
        if (!sym_eig(m, Am, w.data(), ev.data()))
            return fail(ctx, MO_ED_ERR_NOCONV, "projected eigenproblem did not converge");
        MOED_CUDA(ctx, cudaMemcpyAsync(devecs.p, ev.data(), sizeof(double) * ev.size(), cudaMemcpyHostToDevice,
                                       ctx->stream));
        int best = 0;
        for (int i = 1; i < m; ++i)
            if (std::fabs(ev[(size_t)i * m]) > std::fabs(ev[(size_t)best * m])) best = i;
        *res = std::fabs(beta_m * ev[(size_t)best * m + (m - 1)]);
        VPtrs<double> P = make_ptrs<double>(V, m);
        std::vector<DevBuf *> o(1, &out);
        VPtrs<double> X = make_ptrs<double>(o, 1);
        if (int rc = rotate<double>(ctx, G, P, m, (const double *)devecs.p, m, best, 1, X, Dp)) return rc;
        if (*res <= 1e-9 * std::max(anorm, 1.0)) break;
    }
    return MO_ED_OK;
}

int diag_sector(mo_ed_ctx *ctx, const Sector &s, int nev, std::vector<double> &vals,
                std::vector<DevBuf> *vecs)
{
    // the unrestarted solver where it applies (eigs.cu), else thick restarts
    bool done = false;
    const bool f32 = ctx->opt.precision == MO_ED_FP32;
    if (int rc = f32 ? plz_solve<float>(ctx, s, nev, vals, vecs, &done) : plz_solve<double>(ctx, s, nev, vals, vecs, &done))
        return rc;
    if (done) return MO_ED_OK;
    return f32 ? trl_solve<float>(ctx, s, nev, vals, vecs) : trl_solve<double>(ctx, s, nev, vals, vecs);
}

}  // namespace moed
