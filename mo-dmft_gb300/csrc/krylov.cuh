// krylov.cuh -- batched Lanczos state shared by krylov.cu and green.cu.
#pragma once

#include "internal.h"

namespace moed {

constexpr int kLzMaxRuns = 24;
// elements per item of the elementwise kernels: enough items to fill the chip
// first (0.73 million FP64 elements, k_lz_update: 16 us with 8,192 = 90 items,
// 12 us with 1,024), then few, so that the partials stay few
inline int vec_chunk(long long n) { return n < (1LL << 22) ? 1024 : 8192; }

// One run of the reference recurrence (ed_lanczos.F90:14-68) on the device.
// u[0..2] hold u_{j-2}, u_{j-1}, u_j (unnormalized, ring), w = H u_j.
struct LzRunDev {
    void *u[3];
    void *w;
    long long D;
    int chunk;                    // elements per item of the update kernel
    int upd_item0, upd_nitems;    // its items
    int hv_item0, hv_nitems;      // items of the H*v kernel
    double *a, *nrm;              // [nstep+1] device
    double *inv, *cpl;            // [nstep+1] device: 1 / sqrt(nrm[j]), sqrt(nrm[j] / nrm[j-1])
    int *active;                  // 1 while running
    int *nstep_calc;              // device
    double *upd_part, *hv_part;   // partial sums
};

struct LzBatchDev {
    int nrun, total_items;
    LzRunDev run[kLzMaxRuns];
};

// A batch of reference Lanczos runs sharing every launch.  Host-side owner of
// the device buffers; vectors are FP32 or FP64 per `prec`.
struct LzBatch {
    int prec = MO_ED_FP64;
    int nstep = 0;
    std::vector<Sector> sec;
    DevBuf own;                   // workspace of a large batch (small ones use the context's)
    std::vector<void *> vecs;     // 4 per run
    double *coef = nullptr;       // a, nrm, inv, cpl per run, nstep + 1 each
    int *flags = nullptr;         // active, nstep_calc per run
    double *upd_part = nullptr, *hv_part = nullptr;
    std::vector<int> upd_item0, upd_nitems, hv_item0, hv_nitems;
    int upd_total = 0, hv_total = 0;
    int hv_variant = 0, hv_rows = 0;   // H*v tile shape shared by all runs
};

// Allocate a batch for the given target sectors; start vectors are written
// by the caller into start_vector(b, r) (device, prec) before lz_run.
int lz_setup(mo_ed_ctx *ctx, LzBatch &b, const std::vector<Sector> &secs, int prec, int nstep);
void *lz_start_vector(LzBatch &b, int r);
// Run the recurrence for all runs; a, b (squared norms, b[0] = 0) and
// nstep_calc returned per run on the host.
int lz_run(mo_ed_ctx *ctx, LzBatch &b, std::vector<std::vector<double>> &a,
           std::vector<std::vector<double>> &bb, std::vector<int> &nstep_calc);

// FP64 sum of x*y over n elements (x, y of the given precisions), into *d_out.
int dot_dev(mo_ed_ctx *ctx, int prec_x, const void *x, int prec_y, const void *y, long long n,
            double *d_out);
// eigs.cu: the lowest eigenpairs by one long Lanczos run with periodic
// reorthogonalisation.  *done = false (and MO_ED_OK) when the sector or the
// options are not its case, or it gave up: the caller uses thick restarts.
template <typename T>
int plz_solve(mo_ed_ctx *ctx, const Sector &s, int nev, std::vector<double> &vals, std::vector<DevBuf> *vecs,
              bool *done);
template <typename T>
struct VPtrs;
// eigs.cu: Ritz vectors X_c = sum_l V_l Y[c * m + l] (c < nout, Y on the
// device), then the FP64 Rayleigh-Ritz on their span: vals[0 .. nout), and the
// vectors into *vecs if not null; entries nout .. nev of vals are DBL_MAX.
template <typename T>
int ritz_pairs(mo_ed_ctx *ctx, const Sector &s, const VPtrs<T> &V, int m, const double *d_Y, int nout, int nev,
               long long matvecs, std::vector<double> &vals, std::vector<DevBuf> *vecs);

int convert_f64_to_f32(mo_ed_ctx *ctx, const double *in, float *out, long long n);
int convert_f32_to_f64(mo_ed_ctx *ctx, const float *in, double *out, long long n);

}  // namespace moed
