// hv.cu -- matrix-free Kanamori H*v on a (Nup, Ndn) sector.
//
// Replaces multiply_H (ed_hamiltonian.F90:88-191).  For output element
// (d, u) (down rank d, up rank u, X[d][u]) the reference sums
//   diagonal       onsite + dens_dens                      (:112-141)
//   hybridisation  V c+_o c_k and V c+_k c_o, both spins     (:146-161)
//   spin-flip      -J c+_{i up} c_{i dn} c+_{j dn} c_{j up}  (:163-174)
//   pair hop       -J c+_{i up} c+_{i dn} c_{j up} c_{j dn}  (:176-187)
// gathering A at the state each operator maps row (d, u) to.  Here:
//   * diagonal = Dup[u] + Ddn[d] + Cross[imp(u)][imp(d)] (tables.cu);
//   * up-spin hops gather X[d][u'] for the precomputed moves (u', +-V) of u;
//   * down-spin hops are whole-row AXPYs from rows d';
//   * spin-flip / pair hop factor into an up-spin transfer T_{i<-j}(u) and a
//     down-spin transfer (T_{j<-i}(d) for spin-flip, T_{i<-j}(d) for pair
//     hopping) with coefficient +J t_up t_dn: reordering the four operators
//     of ed_operators.F90:183-213 / 236-266 gives a factor -1 that cancels
//     the -J.  Both transfers stay inside a bath group (rank offsets that
//     depend only on the impurity bits).
//
// Work decomposition (both kernels).  An item is up to R rows made of whole
// down-spin bath groups, so the partner rows of spin-flip / pair hopping are
// in the item.  Items are ordered by the bath occupations of the conserved
// subsystems, so the down-spin neighbours of the rows in flight stay
// L2-resident.  A kernel walks a batch of jobs (vectors of possibly different
// sectors) so that all excitation vectors of a Lanczos step share one launch;
// optionally each item writes the FP64 partial of x*y for the Lanczos alpha.
//
// k_hv (first design): a CTA stages its rows in shared memory transposed,
// S[u][r], by blocking loads; one shared load of S[u'] serves the up-spin move
// u -> u' for all rows of the item.  Each thread owns 4 consecutive columns:
// 16-byte global loads for the down-spin row AXPYs and 16-byte stores of y
// (rows are padded to a 128-byte stride); its column moves come from a
// chunk-major table, one contiguous block per slot.
//
// k_hv_async (below): double-buffered asynchronous stage, conflict-free
// scheduled up-spin gathers, precomputed item descriptors.  k_hv_wide: the
// FP32 successor of it for up to three orbitals.  k_hv_row: small sectors.
// k_hv_sorted: FP64 sums.
//
// Split (below): k_hv_down computes the down-spin hybridisation over
// down-spin blocks x column slices from shared memory, or k_hv_down_rows as
// row AXPYs from L2; then k_hv_async<SPLIT> adds the other terms.  The
// autotuner picks among all of them per (precision, sector).
#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <tuple>

#include "hvrow.cuh"
#include "internal.h"
#include "math64.cuh"

namespace moed {

constexpr int kMaxJobs = 24;

template <typename TA>
struct HvBatch {
    int njobs, total_items;
    HvJobT<TA> job[kMaxJobs];
};

template <typename T>
struct alignas(16) Vec4 {
    T v[4];
};

template <typename T, int R>
struct alignas(8) RowVec {
    T v[R];
};

// Spin-flip / pair-hop terms of one (row, column impurity pattern) pair: at
// most 2 for up to three orbitals.  Term t reads the staged partner row
// src[t] at column u + du[t] with coefficient c[t] (+-J with both transfer
// signs folded in).
template <typename TA>
struct alignas(16) Quad {
    int cnt;
    signed char du[2];
    unsigned char src[2];
    TA c[2];
};

template <typename T>
__device__ __forceinline__ Vec4<T> ldg4(const T *p)
{
    Vec4<T> r;
    if constexpr (sizeof(T) == 4) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
        r.v[0] = a.x;
        r.v[1] = a.y;
        r.v[2] = a.z;
        r.v[3] = a.w;
    } else {
        const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
        const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
        r.v[0] = a.x;
        r.v[1] = a.y;
        r.v[2] = b.x;
        r.v[3] = b.y;
    }
    return r;
}

__device__ __forceinline__ int4 ldg_i4(const int *p) { return __ldg(reinterpret_cast<const int4 *>(p)); }

template <typename T>
__device__ __forceinline__ void stg4(T *p, const T (&v)[4])
{
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
    }
}

// the 4 moves of slot s of one 4-column chunk
template <typename TA>
__device__ __forceinline__ void ld_moves(const HopEnt<TA> *p, HopEnt<TA> (&e)[4])
{
    if constexpr (sizeof(TA) == 4) {
        const int4 a = __ldg(reinterpret_cast<const int4 *>(p));
        const int4 b = __ldg(reinterpret_cast<const int4 *>(p) + 1);
        e[0].t = a.x;
        e[0].v = __int_as_float(a.y);
        e[1].t = a.z;
        e[1].v = __int_as_float(a.w);
        e[2].t = b.x;
        e[2].v = __int_as_float(b.y);
        e[3].t = b.z;
        e[3].v = __int_as_float(b.w);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int4 a = __ldg(reinterpret_cast<const int4 *>(p + k));
            e[k].t = a.x;
            e[k].v = __hiloint2double(a.w, a.z);
        }
    }
}

template <typename TX, typename TA, typename TY, int R, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
k_hv(const __grid_constant__ HvBatch<TA> batch, const ModelDev *__restrict__ mdl)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int npair = mdl->npair, nimp = mdl->nimp;
    int ldmax = 0;
    for (int i = 0; i < batch.njobs; ++i) ldmax = max(ldmax, batch.job[i].ld);
    // dynamic shared memory: staged rows transposed, S[u] = row values of
    // column u; then the interspecies diagonal and the 4-operator table
    RowVec<TX, R> *S = reinterpret_cast<RowVec<TX, R> *>(smem_raw);
    TA *s_cross = reinterpret_cast<TA *>(smem_raw + ((sizeof(RowVec<TX, R>) * (size_t)ldmax + 15) & ~(size_t)15));
    int *s_t4 = reinterpret_cast<int *>(s_cross + nimp * nimp);

    __shared__ unsigned s_pmask[kMaxImp];
    __shared__ RowVec<TA, R> s_crossT[kMaxImp];   // per item: cross[iu][id_r] for the R rows
    __shared__ int s_d[R], s_id[R], s_dcnt[R];
    __shared__ TA s_ddiag[R];
    __shared__ int s_dtgt[R][kMaxHop];
    __shared__ TA s_dval[R][kMaxHop];
    // per (row, pair): spin-flip / pair-hop partner as an item slot (>= 0) or
    // as -(1 + global row) when the partner row is not staged, and the
    // coefficient +-J; s_sfm[r] / s_phm[r]: pairs valid for row r
    __shared__ unsigned s_sfm[R], s_phm[R];
    __shared__ unsigned s_rowmask[kMaxPair];   // generic path: bit r spin-flip, bit 16+r pair hop
    __shared__ unsigned s_itemmask;
    __shared__ Quad<TA> s_q[R * kMaxImp];      // fast path table
    __shared__ int s_slow;                     // 1: an item needs the generic path
    __shared__ int s_sfsrc[R][kMaxPair], s_phsrc[R][kMaxPair];
    __shared__ TA s_sfc[R][kMaxPair], s_phc[R][kMaxPair];
    __shared__ double s_red[NT / 32];

    const int tid = threadIdx.x;
    for (int i = tid; i < npair * nimp; i += NT) s_t4[i] = mdl->t4[i];
    for (int i = tid; i < nimp; i += NT) s_pmask[i] = mdl->pairmask[i];
    for (int i = tid; i < nimp * nimp; i += NT) s_cross[i] = (TA)mdl->cross[i];
    const TA Jc = (TA)mdl->J;

    for (int item = blockIdx.x; item < batch.total_items; item += gridDim.x) {
        int j = 0;
        while (j + 1 < batch.njobs && item >= batch.job[j + 1].item0) ++j;
        const HvJobT<TA> &jb = batch.job[j];
        if (jb.active && *jb.active == 0) continue;
        const int it = item - jb.item0;
        const int nd = jb.nd, ld = jb.ld, nchunk = ld >> 2;
        const TX *__restrict__ x = (const TX *)jb.x;
        TY *__restrict__ y = (TY *)jb.y;

        __syncthreads();  // the previous item is done with S and the row tables
        if (tid < R) {
            const int r = tid;
            const int d = jb.items[it * R + r];
            if (d >= 0) {
                const int inf = jb.dn_info[d];
                s_d[r] = d;
                s_id[r] = (inf >> 8) & 0xff;
                s_dcnt[r] = inf & 0xff;
                s_ddiag[r] = jb.dn_diag[d];
            } else {
                s_d[r] = -1;
                s_id[r] = 0;
                s_dcnt[r] = 0;
                s_ddiag[r] = TA(0);
            }
            s_sfm[r] = 0u;
            s_phm[r] = 0u;
        }
        for (int p = tid; p < kMaxPair; p += NT) s_rowmask[p] = 0u;
        if (tid == 0) {
            s_itemmask = 0u;
            s_slow = 0;
        }
        __syncthreads();
        for (int i = tid; i < nimp * R; i += NT) {
            const int iu = i / R, r = i - iu * R;
            s_crossT[iu].v[r] = s_cross[iu * nimp + s_id[r]];
        }
        for (int i = tid; i < R * jb.dn_maxcnt; i += NT) {
            const int r = i / jb.dn_maxcnt, s = i - r * jb.dn_maxcnt;
            if (s < s_dcnt[r]) {
                s_dtgt[r][s] = jb.dn_tgt[(size_t)s * nd + s_d[r]];
                s_dval[r][s] = jb.dn_val[(size_t)s * nd + s_d[r]];
            }
        }
        if (tid < R * npair) {
            const int r = tid / npair, p = tid - r * npair;
            if (s_d[r] >= 0) {
                const int esf = s_t4[mdl->pair_rev[p] * nimp + s_id[r]];   // spin-flip: T_{j<-i}(d)
                const int eph = s_t4[p * nimp + s_id[r]];                  // pair hop:  T_{i<-j}(d)
                if (esf < 0) {
                    const int off = (int)(short)(esf & 0xffff), dp = s_d[r] + off, rp = r + off;
                    const bool local = rp >= 0 && rp < R && s_d[rp] == dp;
                    s_sfsrc[r][p] = local ? rp : -(1 + dp);
                    s_sfc[r][p] = (esf & 0x40000000) ? -Jc : Jc;
                    atomicOr(&s_sfm[r], 1u << p);
                    atomicOr(&s_rowmask[p], 1u << r);
                    atomicOr(&s_itemmask, 1u << p);
                    if (!local) s_slow = 1;
                }
                if (eph < 0) {
                    const int off = (int)(short)(eph & 0xffff), dp = s_d[r] + off, rp = r + off;
                    const bool local = rp >= 0 && rp < R && s_d[rp] == dp;
                    s_phsrc[r][p] = local ? rp : -(1 + dp);
                    s_phc[r][p] = (eph & 0x40000000) ? -Jc : Jc;
                    atomicOr(&s_phm[r], 1u << p);
                    atomicOr(&s_rowmask[p], 1u << (16 + r));
                    atomicOr(&s_itemmask, 1u << p);
                    if (!local) s_slow = 1;
                }
            }
        }
        __syncthreads();
        // fast-path table: terms of every (row, column impurity pattern)
        for (int i = tid; i < R * nimp; i += NT) {
            const int r = i / nimp, iu = i - r * nimp;
            Quad<TA> q;
            q.cnt = 0;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                q.du[t] = 0;
                q.src[t] = 0;
                q.c[t] = TA(0);
            }
            if (s_d[r] >= 0) {
                for (int p = 0; p < npair; ++p) {
                    const int e = s_t4[p * nimp + iu];
                    if (e >= 0) continue;
                    const int du = (int)(short)(e & 0xffff);
                    const TA tu = (e & 0x40000000) ? TA(-1) : TA(1);
                    if ((s_sfm[r] >> p) & 1u) {
                        if (q.cnt == 2) s_slow = 1;
                        else {
                            q.du[q.cnt] = (signed char)du;
                            q.src[q.cnt] = (unsigned char)max(s_sfsrc[r][p], 0);
                            q.c[q.cnt] = tu * s_sfc[r][p];
                            ++q.cnt;
                        }
                    }
                    if ((s_phm[r] >> p) & 1u) {
                        if (q.cnt == 2) s_slow = 1;
                        else {
                            q.du[q.cnt] = (signed char)du;
                            q.src[q.cnt] = (unsigned char)max(s_phsrc[r][p], 0);
                            q.c[q.cnt] = tu * s_phc[r][p];
                            ++q.cnt;
                        }
                    }
                }
            }
            s_q[i] = q;
        }
        // stage the rows, transposed (pad rows staged as zeros)
        for (int c = tid; c < nchunk; c += NT) {
            Vec4<TX> v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int d = jb.items[it * R + r];
                if (d >= 0) {
                    v[r] = ldg4(x + (size_t)d * ld + 4 * c);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[r].v[k] = TX(0);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                RowVec<TX, R> t;
#pragma unroll
                for (int r = 0; r < R; ++r) t.v[r] = v[r].v[k];
                S[4 * c + k] = t;
            }
        }
        __syncthreads();

        // item-uniform row data in registers
        TA ddiag[R];
        bool live[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            ddiag[r] = s_ddiag[r];
            live[r] = s_d[r] >= 0;
        }
        const bool slow = s_slow != 0;
        const bool want_dot = jb.dot_partial != nullptr;
        const unsigned imask = s_itemmask;
        double dacc = 0.0;
        int4 nx_inf = tid < nchunk ? ldg_i4(jb.up_info + 4 * tid) : make_int4(0, 0, 0, 0);
        Vec4<TA> nx_ud = tid < nchunk ? ldg4(jb.up_diag + 4 * tid) : Vec4<TA>{};
        for (int c = tid; c < nchunk; c += NT) {
            const int u0 = 4 * c;
            const int4 inf4 = nx_inf;
            const Vec4<TA> ud = nx_ud;
            if (c + NT < nchunk) {   // prefetch the next chunk's column data
                nx_inf = ldg_i4(jb.up_info + u0 + 4 * NT);
                nx_ud = ldg4(jb.up_diag + u0 + 4 * NT);
            }
            const int inf[4] = {inf4.x, inf4.y, inf4.z, inf4.w};
            TA acc[4][R];
            int cnt[4], iu[4];
            int maxc = 0;
            // diagonal
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                iu[k] = (inf[k] >> 8) & 0xff;
                cnt[k] = inf[k] & 0xff;
                maxc = max(maxc, cnt[k]);
                const RowVec<TX, R> sx = S[u0 + k];
                const RowVec<TA, R> cr = s_crossT[iu[k]];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[k][r] = (ud.v[k] + ddiag[r] + cr.v[r]) * (TA)sx.v[r];
            }
            // up-spin hybridisation: shared-memory gathers, all rows at once
            // The moves of SB slots are loaded together so that their L2
            // latencies overlap; a gather is issued only for a column's own
            // moves (no shared-memory traffic for padded slots).
            constexpr int SB = R > 4 ? 2 : 4;
            const HopEnt<TA> *tab = jb.up_tab + (size_t)c * jb.up_hw * 4;
            for (int s0 = 0; s0 < maxc; s0 += SB) {
                HopEnt<TA> e[SB][4];
#pragma unroll
                for (int t = 0; t < SB; ++t) {
                    if (s0 + t < maxc) ld_moves<TA>(tab + (size_t)(s0 + t) * 4, e[t]);
                }
#pragma unroll
                for (int t = 0; t < SB; ++t) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (s0 + t < cnt[k]) {
                            const RowVec<TX, R> g = S[e[t][k].t];
#pragma unroll
                            for (int r = 0; r < R; ++r) acc[k][r] += e[t][k].v * (TA)g.v[r];
                        }
                    }
                }
            }
            // down-spin hybridisation: row AXPYs (16-byte loads)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int n = s_dcnt[r];
#pragma unroll 4
                for (int s = 0; s < n; ++s) {
                    const TA v = s_dval[r][s];
                    const Vec4<TX> g = ldg4(x + (size_t)s_dtgt[r][s] * ld + u0);
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[k][r] += v * (TA)g.v[k];
                }
            }
            // spin-flip and pair hopping (partner rows are in the stage)
            if (!slow) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const Quad<TA> q = s_q[r * nimp + iu[k]];
#pragma unroll
                        for (int t = 0; t < 2; ++t)
                            if (t < q.cnt)
                                acc[k][r] += q.c[t] * (TA)reinterpret_cast<const TX *>(&S[u0 + k + q.du[t]])[q.src[t]];
                    }
                }
            } else {
                // generic: pairs valid for this column and for some row of the item
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    unsigned pm = s_pmask[iu[k]] & imask;
                    while (pm) {
                        const int p = __ffs(pm) - 1;
                        pm &= pm - 1;
                        const int e = s_t4[p * nimp + iu[k]];
                        const int uu = u0 + k + (int)(short)(e & 0xffff);
                        const bool neg = (e & 0x40000000) != 0;
                        const unsigned rm = s_rowmask[p];
                        const TX *su = reinterpret_cast<const TX *>(&S[uu]);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            if ((rm >> r) & 1u) {
                                const int src = s_sfsrc[r][p];
                                const TX xv = src >= 0 ? su[src] : __ldg(x + (size_t)(-1 - src) * ld + uu);
                                const TA cf = neg ? -s_sfc[r][p] : s_sfc[r][p];
                                acc[k][r] += cf * (TA)xv;
                            }
                            if ((rm >> (16 + r)) & 1u) {
                                const int src = s_phsrc[r][p];
                                const TX xv = src >= 0 ? su[src] : __ldg(x + (size_t)(-1 - src) * ld + uu);
                                const TA cf = neg ? -s_phc[r][p] : s_phc[r][p];
                                acc[k][r] += cf * (TA)xv;
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (live[r]) {
                    TY o[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) o[k] = (TY)acc[k][r];
                    stg4(y + (size_t)s_d[r] * ld + u0, o);
                }
            }
            if (want_dot) {   // x (re-read from the stage) . y of this chunk
                TA part = TA(0);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const RowVec<TX, R> sx = S[u0 + k];
#pragma unroll
                    for (int r = 0; r < R; ++r) part += (TA)sx.v[r] * (TA)(TY)acc[k][r];
                }
                dacc += (double)part;
            }
        }
        if (jb.dot_partial) {
            for (int off = 16; off > 0; off >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, off);
            if ((tid & 31) == 0) s_red[tid >> 5] = dacc;
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int w = 0; w < NT / 32; ++w) t += s_red[w];
                jb.dot_partial[it] = t;
            }
        }
    }
}

template <typename TX, typename TA, int R>
static size_t dyn_smem_bytes(int ld, const ModelDev &m)
{
    return ((sizeof(RowVec<TX, R>) * (size_t)ld + 15) & ~(size_t)15) + sizeof(TA) * (size_t)m.nimp * m.nimp +
           sizeof(int) * (size_t)m.npair * m.nimp;
}

// ---------------------------------------------------------------------------
// staged variant (k_hv_async)
// ---------------------------------------------------------------------------
// The same sum per element, organised for latency hiding and few instructions:
//   * stage layout [tile][r][32]: column u of staged row r sits at
//     ((u >> 5) * R + r) * 32 + (u & 31).  The R values of a column are 32
//     elements apart, so one address serves every row (immediate offsets),
//     and column u is in bank u mod 32 for every row;
//   * the rows of the next item and its descriptor (the row data k_hv
//     computes per item: row indices, down-spin moves, interspecies diagonal,
//     spin-flip / pair-hop terms; built once by k_item_desc) are copied
//     (cp.async, 16 bytes per thread, L2 only) into the second of two stage
//     buffers while the current item is computed: two barriers per item;
//   * warp w owns chunks c = w + NW * (kHvCh * i + q) (32 columns each, one
//     column per lane), so every global load and store of a warp covers one
//     128-byte line and the kHvCh chunks of an iteration share their address
//     arithmetic (immediate offsets);
//   * up-spin moves follow the conflict-free schedule (species_sched): the
//     entries hold the stage offset of the target, one bank-conflict-free
//     shared load per staged row and slot, no predication;
//   * down-spin row AXPYs: one row offset per move serves the kHvCh chunks.
constexpr int kHvCh = 4;

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all_but_newest() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

template <typename TA>
__device__ __forceinline__ int hv_find_job(const HvBatch<TA> &b, int item)
{
    int j = 0;
    while (j + 1 < b.njobs && item >= b.job[j + 1].item0) ++j;
    return j;
}

// next item of this CTA at or after `from` (stride gridDim.x) whose job is active
template <typename TA>
__device__ __forceinline__ int hv_next_item(const HvBatch<TA> &b, int from)
{
    for (int item = from; item < b.total_items; item += gridDim.x) {
        const HvJobT<TA> &jb = b.job[hv_find_job(b, item)];
        if (!jb.active || *jb.active != 0) return item;
    }
    return -1;
}

// Item descriptor: the per-item row data of k_hv (row indices, impurity
// patterns, down-spin moves, interspecies diagonal of the rows, spin-flip /
// pair-hop terms), computed once per (down species, R, precision) by
// k_item_desc and staged next to the rows.  Offsets are in 4-byte words.
struct DescGeom {
    int words, dm, nimp, npair;
    int o_d, o_id, o_dcnt, o_flags, o_ddiag, o_dtgt, o_dval, o_cross, o_quad;
    int o_sfsrc, o_phsrc, o_sfc, o_phc, o_rowmask;
};

template <typename TA, int R>
static DescGeom desc_geom(int dm, const ModelDev &m)
{
    const int ts = sizeof(TA) / 4;
    auto al = [](int w, int a) { return (w + a - 1) / a * a; };
    DescGeom g;
    g.dm = std::max(dm, 1);
    g.nimp = m.nimp;
    g.npair = std::max(m.npair, 1);
    int w = 0;
    g.o_d = w;       w += R;
    g.o_id = w;      w += R;
    g.o_dcnt = w;    w += R;
    g.o_flags = w;   w += 2;            // slow, item pair mask
    w = al(w, 2);
    g.o_ddiag = w;   w += R * ts;
    g.o_dtgt = w;    w += R * g.dm;
    w = al(w, 2);
    g.o_dval = w;    w += R * g.dm * ts;
    g.o_cross = w;   w += g.nimp * R * ts;
    w = al(w, 4);
    g.o_quad = w;    w += R * g.nimp * (int)(sizeof(Quad<TA>) / 4);
    g.o_sfsrc = w;   w += R * g.npair;
    g.o_phsrc = w;   w += R * g.npair;
    w = al(w, 2);
    g.o_sfc = w;     w += R * g.npair * ts;
    g.o_phc = w;     w += R * g.npair * ts;
    g.o_rowmask = w; w += g.npair;
    g.words = al(w, 4);
    return g;
}

// one thread per item: the row data the k_hv setup computes per item
template <typename TA, int R>
__global__ void k_item_desc(int nitems, const int *__restrict__ items, const int *__restrict__ dn_info,
                            const TA *__restrict__ dn_diag, const int *__restrict__ dn_tgt,
                            const TA *__restrict__ dn_val, int nd, const ModelDev *__restrict__ mdl, DescGeom g,
                            unsigned *__restrict__ out)
{
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    if (it >= nitems) return;
    unsigned *rec = out + (size_t)it * g.words;
    for (int i = 0; i < g.words; ++i) rec[i] = 0u;
    int *od = (int *)(rec + g.o_d), *oid = (int *)(rec + g.o_id), *ocnt = (int *)(rec + g.o_dcnt);
    int *oflags = (int *)(rec + g.o_flags);
    TA *oddiag = (TA *)(rec + g.o_ddiag);
    int *odtgt = (int *)(rec + g.o_dtgt);
    TA *odval = (TA *)(rec + g.o_dval);
    TA *ocross = (TA *)(rec + g.o_cross);
    Quad<TA> *oquad = (Quad<TA> *)(rec + g.o_quad);
    int *osfsrc = (int *)(rec + g.o_sfsrc), *ophsrc = (int *)(rec + g.o_phsrc);
    TA *osfc = (TA *)(rec + g.o_sfc), *ophc = (TA *)(rec + g.o_phc);
    unsigned *orowmask = rec + g.o_rowmask;
    const int nimp = mdl->nimp, npair = mdl->npair;
    const TA Jc = (TA)mdl->J;
    int d[R], id[R];
    unsigned sfm[R], phm[R];
    int slow = 0;
    unsigned itemmask = 0u;
    for (int r = 0; r < R; ++r) {
        d[r] = items[it * R + r];
        id[r] = 0;
        sfm[r] = phm[r] = 0u;
        int cnt = 0;
        TA dg = TA(0);
        if (d[r] >= 0) {
            const int inf = dn_info[d[r]];
            id[r] = (inf >> 8) & 0xff;
            cnt = inf & 0xff;
            dg = dn_diag[d[r]];
            for (int s = 0; s < cnt; ++s) {
                odtgt[r * g.dm + s] = dn_tgt[(size_t)s * nd + d[r]];
                odval[r * g.dm + s] = dn_val[(size_t)s * nd + d[r]];
            }
        }
        od[r] = d[r];
        oid[r] = id[r];
        ocnt[r] = cnt;
        oddiag[r] = dg;
    }
    for (int iu = 0; iu < nimp; ++iu)
        for (int r = 0; r < R; ++r) ocross[iu * R + r] = (TA)mdl->cross[iu * nimp + id[r]];
    for (int r = 0; r < R; ++r) {
        if (d[r] < 0) continue;
        for (int p = 0; p < npair; ++p) {
            const int esf = mdl->t4[mdl->pair_rev[p] * nimp + id[r]];   // spin-flip: T_{j<-i}(d)
            const int eph = mdl->t4[p * nimp + id[r]];                  // pair hop:  T_{i<-j}(d)
            if (esf < 0) {
                const int off = (int)(short)(esf & 0xffff), dp = d[r] + off, rp = r + off;
                const bool local = rp >= 0 && rp < R && d[rp] == dp;
                osfsrc[r * g.npair + p] = local ? rp : -(1 + dp);
                osfc[r * g.npair + p] = (esf & 0x40000000) ? -Jc : Jc;
                sfm[r] |= 1u << p;
                orowmask[p] |= 1u << r;
                itemmask |= 1u << p;
                if (!local) slow = 1;
            }
            if (eph < 0) {
                const int off = (int)(short)(eph & 0xffff), dp = d[r] + off, rp = r + off;
                const bool local = rp >= 0 && rp < R && d[rp] == dp;
                ophsrc[r * g.npair + p] = local ? rp : -(1 + dp);
                ophc[r * g.npair + p] = (eph & 0x40000000) ? -Jc : Jc;
                phm[r] |= 1u << p;
                orowmask[p] |= 1u << (16 + r);
                itemmask |= 1u << p;
                if (!local) slow = 1;
            }
        }
    }
    for (int r = 0; r < R; ++r)
        for (int iu = 0; iu < nimp; ++iu) {
            Quad<TA> q;
            q.cnt = 0;
            for (int t = 0; t < 2; ++t) {
                q.du[t] = 0;
                q.src[t] = 0;
                q.c[t] = TA(0);
            }
            if (d[r] >= 0) {
                for (int p = 0; p < npair; ++p) {
                    const int e = mdl->t4[p * nimp + iu];
                    if (e >= 0) continue;
                    const int du = (int)(short)(e & 0xffff);
                    const TA tu = (e & 0x40000000) ? TA(-1) : TA(1);
                    if ((sfm[r] >> p) & 1u) {
                        if (q.cnt == 2) slow = 1;
                        else {
                            q.du[q.cnt] = (signed char)du;
                            q.src[q.cnt] = (unsigned char)max(osfsrc[r * g.npair + p], 0);
                            q.c[q.cnt] = tu * osfc[r * g.npair + p];
                            ++q.cnt;
                        }
                    }
                    if ((phm[r] >> p) & 1u) {
                        if (q.cnt == 2) slow = 1;
                        else {
                            q.du[q.cnt] = (signed char)du;
                            q.src[q.cnt] = (unsigned char)max(ophsrc[r * g.npair + p], 0);
                            q.c[q.cnt] = tu * ophc[r * g.npair + p];
                            ++q.cnt;
                        }
                    }
                }
            }
            oquad[r * nimp + iu] = q;
        }
    oflags[0] = slow;
    oflags[1] = (int)itemmask;
}

// all threads: copy the rows and the descriptor of `item` into a stage
// buffer and its descriptor buffer, and commit the group
template <typename TX, typename TA, int R, int NT>
__device__ __forceinline__ void hv_stage_item(const HvBatch<TA> &b, int item, TX *stage, unsigned *desc,
                                              int dwords)
{
    const HvJobT<TA> &jb = b.job[hv_find_job(b, item)];
    const int it = item - jb.item0;
    const int ld = jb.ld;
    constexpr int EPV = 16 / sizeof(TX);   // elements per 16-byte copy
    const int nv = ld / EPV;
    const TX *x = (const TX *)jb.x;
    const unsigned *src_desc = jb.desc + (size_t)it * dwords;
    for (int q = threadIdx.x; q < dwords / 4; q += NT) cp_async16(desc + 4 * q, src_desc + 4 * q);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int d = jb.items[it * R + r];
        if (d < 0) continue;
        const TX *src = x + (size_t)d * ld;
        for (int q = threadIdx.x; q < nv; q += NT) {
            const int u = q * EPV;
            cp_async16(stage + ((u >> 5) * R + r) * 32 + (u & 31), src + u);
        }
    }
    cp_async_commit();
}

// SPLIT: k_hv_down has already written the down-spin hybridisation into y;
// this kernel adds the other terms to it instead of computing the row AXPYs.
template <typename TX, typename TA, typename TY, int R, int NT, int MINB, bool SPLIT>
__global__ void __launch_bounds__(NT, MINB)
k_hv_async(const __grid_constant__ HvBatch<TA> batch, const ModelDev *__restrict__ mdl, const DescGeom g)
{
    extern __shared__ __align__(16) unsigned char smem_async[];
    const int nimp = mdl->nimp;
    int ldmax = 0;
    for (int i = 0; i < batch.njobs; ++i) ldmax = max(ldmax, batch.job[i].ld);
    const int stage_elems = R * ldmax;
    TX *stage0 = reinterpret_cast<TX *>(smem_async);
    TX *stage1 = stage0 + stage_elems;
    unsigned *desc0 = reinterpret_cast<unsigned *>(smem_async + ((2 * (size_t)stage_elems * sizeof(TX) + 15) & ~(size_t)15));
    unsigned *desc1 = desc0 + g.words;
    int *s_t4 = reinterpret_cast<int *>(desc1 + g.words);
    __shared__ unsigned s_pmask[kMaxImp];
    __shared__ double s_red[NT / 32];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    for (int i = tid; i < mdl->npair * nimp; i += NT) s_t4[i] = mdl->t4[i];
    for (int i = tid; i < nimp; i += NT) s_pmask[i] = mdl->pairmask[i];
    __syncthreads();

    int cur = hv_next_item(batch, (int)blockIdx.x);
    if (cur >= 0) hv_stage_item<TX, TA, R, NT>(batch, cur, stage0, desc0, g.words);
    int k = 0;
    while (cur >= 0) {
        const int buf = k & 1;
        const int nxt = hv_next_item(batch, cur + (int)gridDim.x);
        // buffers (k+1)&1 were released by the barrier that ended item k-1;
        // one commit group per iteration either way
        if (nxt >= 0) hv_stage_item<TX, TA, R, NT>(batch, nxt, buf ? stage0 : stage1, buf ? desc0 : desc1, g.words);
        else cp_async_commit();

        const HvJobT<TA> &jb = batch.job[hv_find_job(batch, cur)];
        const int it = cur - jb.item0;
        const int ld = jb.ld, nch = ld >> 5;
        const TX *__restrict__ x = (const TX *)jb.x;
        TY *__restrict__ y = (TY *)jb.y;
        cp_async_wait_all_but_newest();   // this thread's copies of the current item
        __syncthreads();                  // everyone's
        const TX *S = buf ? stage1 : stage0;
        const unsigned *dsc = buf ? desc1 : desc0;
        const int *s_d = (const int *)(dsc + g.o_d);
        const int *s_dcnt = (const int *)(dsc + g.o_dcnt);
        const int *s_dtgt = (const int *)(dsc + g.o_dtgt);
        const TA *s_dval = (const TA *)(dsc + g.o_dval);
        const TA *s_crossT = (const TA *)(dsc + g.o_cross);
        const Quad<TA> *s_q = (const Quad<TA> *)(dsc + g.o_quad);
        const int *s_sfsrc = (const int *)(dsc + g.o_sfsrc), *s_phsrc = (const int *)(dsc + g.o_phsrc);
        const TA *s_sfc = (const TA *)(dsc + g.o_sfc), *s_phc = (const TA *)(dsc + g.o_phc);
        const unsigned *s_rowmask = dsc + g.o_rowmask;
        const bool slow = ((const int *)(dsc + g.o_flags))[0] != 0;
        const unsigned imask = (unsigned)((const int *)(dsc + g.o_flags))[1];
        const int dm = g.dm, npr = g.npair;

        TA ddiag[R];
        bool live[R];
        int dcnt[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            ddiag[r] = ((const TA *)(dsc + g.o_ddiag))[r];
            live[r] = s_d[r] >= 0;
            dcnt[r] = s_dcnt[r];
        }
        const bool want_dot = jb.dot_partial != nullptr;
        double dacc = 0.0;
        constexpr int SB = 4;
        constexpr int DB = 2;
        for (int cb = warp; cb < nch; cb += NW * kHvCh) {
            // chunks cb + NW*q, q < kHvCh; column of this lane in chunk q: ub + 32*NW*q
            const int ub = 32 * cb + lane;
            bool has[kHvCh];
            int iu[kHvCh];
            int2 h[kHvCh];
            TA acc[kHvCh][R];
#pragma unroll
            for (int q = 0; q < kHvCh; ++q) {
                has[q] = cb + NW * q < nch;
                h[q] = has[q] ? __ldg(jb.up_sched_hdr + cb + NW * q) : make_int2(0, 0);
            }
            // the first DB down-spin moves of every row (SPLIT: the down-spin
            // part already in y): loads in flight early
            TX gd[R][DB][kHvCh];
            TY yp[R][kHvCh];
            if constexpr (SPLIT) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const TY *yr = y + (size_t)(live[r] ? s_d[r] : 0) * ld + ub;
#pragma unroll
                    for (int q = 0; q < kHvCh; ++q) yp[r][q] = (live[r] && has[q]) ? yr[32 * NW * q] : TY(0);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int t = 0; t < DB; ++t) {
                        const bool mv = t < dcnt[r];
                        const TX *xr = x + (size_t)s_dtgt[r * dm + (mv ? t : 0)] * ld + ub;
#pragma unroll
                        for (int q = 0; q < kHvCh; ++q)
                            gd[r][t][q] = (mv && has[q]) ? __ldg(xr + 32 * NW * q) : TX(0);
                    }
            }
            // first SB schedule entries of every chunk
            HopEnt<TA> e0[kHvCh][SB];
#pragma unroll
            for (int q = 0; q < kHvCh; ++q)
#pragma unroll
                for (int t = 0; t < SB; ++t)
                    e0[q][t] = (t < h[q].y) ? jb.up_sched[h[q].x + 32 * t + lane] : HopEnt<TA>{};
            // diagonal
#pragma unroll
            for (int q = 0; q < kHvCh; ++q) {
                const int u = ub + 32 * NW * q;
                int inf = 0;
                TA ud = TA(0);
                if (has[q]) {
                    inf = __ldg(jb.up_info + u);
                    ud = __ldg(jb.up_diag + u);
                }
                iu[q] = (inf >> 8) & 0xff;
#pragma unroll
                for (int r = 0; r < R; ++r) acc[q][r] = TA(0);
                if (has[q]) {
                    const TX *so = S + ((u >> 5) * R) * 32 + (u & 31);
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        acc[q][r] = (ud + ddiag[r] + s_crossT[iu[q] * R + r]) * (TA)so[32 * r];
                }
            }
            // up-spin hybridisation: scheduled conflict-free gathers
#pragma unroll
            for (int q = 0; q < kHvCh; ++q) {
                const int ns = h[q].y;
                const HopEnt<TA> *tab = jb.up_sched + h[q].x + lane;
                HopEnt<TA> e[SB];
#pragma unroll
                for (int t = 0; t < SB; ++t) e[t] = e0[q][t];
                for (int s0 = 0; s0 < ns; s0 += SB) {
                    HopEnt<TA> f[SB];
#pragma unroll
                    for (int t = 0; t < SB; ++t) f[t] = (s0 + SB + t < ns) ? tab[32 * (s0 + SB + t)] : HopEnt<TA>{};
#pragma unroll
                    for (int t = 0; t < SB; ++t) {
                        if (s0 + t < ns) {
                            const TX *st = S + e[t].t;
#pragma unroll
                            for (int r = 0; r < R; ++r) acc[q][r] += e[t].v * (TA)st[32 * r];
                        }
                    }
#pragma unroll
                    for (int t = 0; t < SB; ++t) e[t] = f[t];
                }
            }
            // spin-flip and pair hopping (partner rows staged)
#pragma unroll
            for (int q = 0; q < kHvCh; ++q) {
                if (!has[q]) continue;
                const int u = ub + 32 * NW * q;
                if (!slow) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const Quad<TA> qd = s_q[r * nimp + iu[q]];
                        if (qd.cnt > 0) {
#pragma unroll
                            for (int t = 0; t < 2; ++t) {
                                if (t < qd.cnt) {
                                    const int w = u + qd.du[t];
                                    acc[q][r] += qd.c[t] * (TA)S[((w >> 5) * R + qd.src[t]) * 32 + (w & 31)];
                                }
                            }
                        }
                    }
                } else {
                    unsigned pm = s_pmask[iu[q]] & imask;
                    while (pm) {
                        const int p = __ffs(pm) - 1;
                        pm &= pm - 1;
                        const int e = s_t4[p * nimp + iu[q]];
                        const int w = u + (int)(short)(e & 0xffff);
                        const bool neg = (e & 0x40000000) != 0;
                        const unsigned rm = s_rowmask[p];
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            if ((rm >> r) & 1u) {
                                const int src = s_sfsrc[r * npr + p];
                                const TX xv = src >= 0 ? S[((w >> 5) * R + src) * 32 + (w & 31)]
                                                       : __ldg(x + (size_t)(-1 - src) * ld + w);
                                const TA cf = neg ? -s_sfc[r * npr + p] : s_sfc[r * npr + p];
                                acc[q][r] += cf * (TA)xv;
                            }
                            if ((rm >> (16 + r)) & 1u) {
                                const int src = s_phsrc[r * npr + p];
                                const TX xv = src >= 0 ? S[((w >> 5) * R + src) * 32 + (w & 31)]
                                                       : __ldg(x + (size_t)(-1 - src) * ld + w);
                                const TA cf = neg ? -s_phc[r * npr + p] : s_phc[r * npr + p];
                                acc[q][r] += cf * (TA)xv;
                            }
                        }
                    }
                }
            }
            // down-spin hybridisation: the early loads, then the remaining moves
            if constexpr (SPLIT) {
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int q = 0; q < kHvCh; ++q) acc[q][r] += (TA)yp[r][q];
            } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int t = 0; t < DB; ++t) {
                    if (t < dcnt[r]) {
                        const TA v = s_dval[r * dm + t];
#pragma unroll
                        for (int q = 0; q < kHvCh; ++q) acc[q][r] += v * (TA)gd[r][t][q];
                    }
                }
                for (int t0 = DB; t0 < dcnt[r]; t0 += DB) {
                    TX g2[DB][kHvCh];
#pragma unroll
                    for (int t = 0; t < DB; ++t) {
                        const bool mv = t0 + t < dcnt[r];
                        const TX *xr = x + (size_t)s_dtgt[r * dm + (mv ? t0 + t : t0)] * ld + ub;
#pragma unroll
                        for (int q = 0; q < kHvCh; ++q) g2[t][q] = (mv && has[q]) ? __ldg(xr + 32 * NW * q) : TX(0);
                    }
#pragma unroll
                    for (int t = 0; t < DB; ++t) {
                        if (t0 + t < dcnt[r]) {
                            const TA v = s_dval[r * dm + t0 + t];
#pragma unroll
                            for (int q = 0; q < kHvCh; ++q) acc[q][r] += v * (TA)g2[t][q];
                        }
                    }
                }
            }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!live[r]) continue;
                TY *yr = y + (size_t)s_d[r] * ld + ub;
#pragma unroll
                for (int q = 0; q < kHvCh; ++q)
                    if (has[q]) yr[32 * NW * q] = (TY)acc[q][r];
            }
            if (want_dot) {
                TA part = TA(0);
#pragma unroll
                for (int q = 0; q < kHvCh; ++q) {
                    if (!has[q]) continue;
                    const int u = ub + 32 * NW * q;
                    const TX *so = S + ((u >> 5) * R) * 32 + (u & 31);
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (live[r]) part += (TA)so[32 * r] * (TA)(TY)acc[q][r];
                }
                dacc += (double)part;
            }
        }
        if (want_dot) {
            for (int off = 16; off > 0; off >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, off);
            if (lane == 0) s_red[warp] = dacc;
        }
        __syncthreads();   // item done: its buffers are free
        if (want_dot && tid == 0) {
            double t = 0.0;
            for (int w = 0; w < NW; ++w) t += s_red[w];
            jb.dot_partial[it] = t;
        }
        cur = nxt;
        ++k;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---------------------------------------------------------------------------
// k_hv_down: the down-spin hybridisation of the split H*v,
//   y[d][u] = sum over moves (d -> d', t) of t * x[d'][u],
// for every row d, written (not accumulated) into y; k_hv_async<SPLIT> then
// adds the other terms.  The rows of a down-spin block (equal electron counts
// in every conserved subsystem) are closed under the moves, so a chunk = one
// block x a range of columns is independent of all others.  A CTA stages the
// block's move list once ({target index within the block, signed coupling})
// and then walks the chunk's column slices, staged by cp.async and double-
// buffered when two slices fit.  A slice is kb groups of WB bytes (one 64- or
// 128-byte line segment) of every row of the block, kb as large as the buffer
// allows, so small blocks take wide slices.  Every element of x is read from
// memory once per H*v and the moves read shared memory only.  CTAs take
// contiguous chunk ranges, so consecutive chunks usually share the block and
// its move list.
// ---------------------------------------------------------------------------
template <typename TA>
__device__ __forceinline__ int hv_tile_job(const HvBatch<TA> &b, int tile)
{
    int j = 0;
    while (j + 1 < b.njobs && tile >= b.job[j + 1].tile0) ++j;
    return j;
}

struct DownLayout {        // shared-memory layout of k_hv_down, in bytes
    int ptr, rows, mv, x0, x1;
};

// stage columns [col, col + kw * W) of the block's rows: row i at buf + i * kw * W
template <typename TX, int NT, int WB>
__device__ __forceinline__ void hv_down_slice(const TX *__restrict__ x, const int *s_rows, int nr, int ld,
                                              int col, int kw, TX *buf)
{
    constexpr int CPG = WB / 16;                // 16-byte copies per group of a row
    constexpr int EPV = 16 / (int)sizeof(TX);
    const int cpr = kw * CPG;
    for (int q = threadIdx.x; q < nr * cpr; q += NT) {
        const int i = q / cpr, c = q - i * cpr;
        cp_async16(buf + (size_t)i * cpr * EPV + c * EPV, x + (size_t)s_rows[i] * ld + col + c * EPV);
    }
}

template <typename TX, typename TA, typename TY, int NT, int WB>
__global__ void __launch_bounds__(NT, 1)
k_hv_down(const __grid_constant__ HvBatch<TA> batch, int total, const DownLayout L, int cap_rows, int dbuf)
{
    extern __shared__ __align__(16) unsigned char smem_down[];
    constexpr int W = WB / (int)sizeof(TX);   // columns per group (one WB-byte segment of a row)
    constexpr int RPW = 32 / W;               // groups per warp pass
    constexpr int NW = NT / 32;
    int *s_ptr = reinterpret_cast<int *>(smem_down + L.ptr);
    int *s_rows = reinterpret_cast<int *>(smem_down + L.rows);
    HopEnt<TA> *s_mv = reinterpret_cast<HopEnt<TA> *>(smem_down + L.mv);
    TX *const xb0 = reinterpret_cast<TX *>(smem_down + L.x0);
    TX *const xb1 = reinterpret_cast<TX *>(smem_down + L.x1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane / W, c = lane - sub * W;
    const int c_begin = (int)((long long)total * blockIdx.x / gridDim.x);
    const int c_end = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
    int have_job = -1, have_blk = -1;
    for (int ch = c_begin; ch < c_end; ++ch) {
        const int jid = hv_tile_job(batch, ch);
        const HvJobT<TA> &jb = batch.job[jid];
        if (jb.active && *jb.active == 0) continue;
        const int lc = ch - jb.tile0;
        // block of this chunk: last b with chunks[b].x <= lc
        int lo = 0, hi = jb.dblk_n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(&jb.dblk_chunks[mid].x) <= lc) lo = mid;
            else hi = mid - 1;
        }
        const int blk = lo;
        const int2 cinfo = jb.dblk_chunks[blk];
        const int ld = jb.ld;
        const int col0 = (lc - cinfo.x) * cinfo.y * 32;
        const int col1 = min(ld, col0 + cinfo.y * 32);
        const int p0 = __ldg(jb.dblk_off + blk), nr = __ldg(jb.dblk_off + blk + 1) - p0;
        const TX *x = (const TX *)jb.x;
        TY *y = (TY *)jb.y;
        __syncthreads();   // the previous chunk is done with shared memory
        if (jid != have_job || blk != have_blk) {
            const int m0 = __ldg(jb.dblk_ptr + p0), nm = __ldg(jb.dblk_ptr + p0 + nr) - m0;
            for (int i = tid; i <= nr; i += NT) s_ptr[i] = __ldg(jb.dblk_ptr + p0 + i) - m0;
            for (int i = tid; i < nr; i += NT) s_rows[i] = __ldg(jb.dblk_rows + p0 + i);
            for (int i = tid; i < nm; i += NT) s_mv[i] = jb.dblk_mv[m0 + i];
            have_job = jid;
            have_blk = blk;
            __syncthreads();
        }
        // a slice = kb groups of W columns of every row (small blocks: wide slices)
        const int ngr = (col1 - col0) / W;
        const int kb = max(1, min(cap_rows / nr, ngr));
        const int ns = (ngr + kb - 1) / kb;
        hv_down_slice<TX, NT, WB>(x, s_rows, nr, ld, col0, min(kb, ngr), xb0);
        cp_async_commit();
        for (int sl = 0; sl < ns; ++sl) {
            const TX *S = (dbuf && (sl & 1)) ? xb1 : xb0;
            const int kw = min(kb, ngr - sl * kb);   // groups in this slice
            if (dbuf && sl + 1 < ns) {
                hv_down_slice<TX, NT, WB>(x, s_rows, nr, ld, col0 + (sl + 1) * kb * W, min(kb, ngr - (sl + 1) * kb),
                                          (sl & 1) ? xb0 : xb1);
                cp_async_commit();
                cp_async_wait_all_but_newest();
            } else {
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
            __syncthreads();
            const int ws = kw * W;               // row stride of the staged slice
            TY *ys = y + col0 + sl * kb * W + c;
            if (kw == 1) {
                // one group per row (large blocks): 4 moves in flight
                for (int i = warp * RPW + sub; i < nr; i += NW * RPW) {
                    const int b1 = s_ptr[i], e1 = s_ptr[i + 1];
                    const TX *Sc = S + c;
                    TA a = TA(0);
                    int e = b1;
                    for (; e + 4 <= e1; e += 4) {
                        const HopEnt<TA> m0 = s_mv[e], m1 = s_mv[e + 1], m2 = s_mv[e + 2], m3 = s_mv[e + 3];
                        const TX x0 = Sc[m0.t * W], x1 = Sc[m1.t * W], x2 = Sc[m2.t * W], x3 = Sc[m3.t * W];
                        a += m0.v * (TA)x0;
                        a += m1.v * (TA)x1;
                        a += m2.v * (TA)x2;
                        a += m3.v * (TA)x3;
                    }
                    for (; e < e1; ++e) {
                        const HopEnt<TA> m = s_mv[e];
                        a += m.v * (TA)Sc[m.t * W];
                    }
                    ys[(size_t)s_rows[i] * ld] = (TY)a;
                }
            } else {
                // several groups per row (small blocks, wide slices): each move
                // serves up to KQ groups
                constexpr int KQ = 4;
                const int npass = (kw + KQ - 1) / KQ;
                for (int it = warp * RPW + sub; it < nr * npass; it += NW * RPW) {
                    const int i = it / npass, g0 = (it - i * npass) * KQ;
                    const int b1 = s_ptr[i], e1 = s_ptr[i + 1];
                    const TX *Sc = S + g0 * W + c;
                    TA a[KQ];
#pragma unroll
                    for (int q = 0; q < KQ; ++q) a[q] = TA(0);
                    for (int e = b1; e < e1; ++e) {
                        const HopEnt<TA> m = s_mv[e];
                        const TX *Sm = Sc + m.t * ws;
#pragma unroll
                        for (int q = 0; q < KQ; ++q)
                            if (g0 + q < kw) a[q] += m.v * (TA)Sm[q * W];
                    }
                    TY *yr = ys + (size_t)s_rows[i] * ld + g0 * W;
#pragma unroll
                    for (int q = 0; q < KQ; ++q)
                        if (g0 + q < kw) yr[q * W] = (TY)a[q];
                }
            }
            __syncthreads();   // slice done: its buffer is free
            if (!dbuf && sl + 1 < ns) {
                hv_down_slice<TX, NT, WB>(x, s_rows, nr, ld, col0 + (sl + 1) * kb * W, min(kb, ngr - (sl + 1) * kb),
                                          xb0);
                cp_async_commit();
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---------------------------------------------------------------------------
// k_hv_down_rows: the same down-spin term as k_hv_down, as row AXPYs,
//   y[d][c] = sum over moves (d -> d', t) of t * x[d'][c],
// straight from the species' per-row move tables (dn_info / dn_tgt /
// dn_val), with no staging.  A tile is one row d times 4 NT CPT columns,
// each thread CPT chunks of four consecutive columns, 4 NT apart (16-byte
// loads and stores; rows are padded to a multiple of 32 elements).  The
// row's move targets and couplings are staged in shared memory first, one
// per thread, so the x loads of all its moves can be in flight at once.
// Tiles run
// column-tile-major: the CTAs in flight share one column tile of x (C4 with
// CPT = 2: 6,435 rows x 1,024 columns, 26 MB), which stays in L2 while each
// source segment is read by the rows that move to it, so x comes from memory
// about once per H*v.
// ---------------------------------------------------------------------------
// The host guarantees dn_maxcnt <= NT (launch_batch_rows).
template <typename TX, typename TA, typename TY, int NT, int CPT>
__global__ void __launch_bounds__(NT)
k_hv_down_rows(const __grid_constant__ HvBatch<TA> batch, int total)
{
    __shared__ int s_tgt[NT];
    __shared__ TA s_val[NT];
    for (int t = blockIdx.x; t < total; t += gridDim.x) {   // t is uniform over the CTA
        const int jid = hv_tile_job(batch, t);
        const HvJobT<TA> &jb = batch.job[jid];
        if (jb.active && *jb.active == 0) continue;
        const int lt = t - jb.tile0;
        const int ct = lt / jb.nd, d = lt - ct * jb.nd;
        const int cnt = min(__ldg(&jb.dn_info[d]) & 0xff, NT);
        __syncthreads();   // the previous tile is done with s_tgt / s_val
        if ((int)threadIdx.x < cnt) {
            s_tgt[threadIdx.x] = __ldg(&jb.dn_tgt[(size_t)threadIdx.x * jb.nd + d]);
            s_val[threadIdx.x] = __ldg(&jb.dn_val[(size_t)threadIdx.x * jb.nd + d]);
        }
        __syncthreads();
        const int c0 = ct * 4 * NT * CPT + 4 * (int)threadIdx.x;
        if (c0 >= jb.ld) continue;   // ld is a multiple of 4: a chunk at c < ld ends before ld
        const TX *x = (const TX *)jb.x;
        TA a[CPT][4];
#pragma unroll
        for (int k = 0; k < CPT; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) a[k][q] = TA(0);
#pragma unroll 4
        for (int h = 0; h < cnt; ++h) {
            const TA v = s_val[h];
            const TX *xr = x + (size_t)s_tgt[h] * jb.ld;
#pragma unroll
            for (int k = 0; k < CPT; ++k)
                if (k == 0 || c0 + k * 4 * NT < jb.ld) {   // chunk 0 is in range (checked above)
                    const Vec4<TX> xv = ldg4(xr + c0 + k * 4 * NT);
#pragma unroll
                    for (int q = 0; q < 4; ++q) a[k][q] += v * (TA)xv.v[q];
                }
        }
        TY *yr = (TY *)jb.y + (size_t)d * jb.ld;
#pragma unroll
        for (int k = 0; k < CPT; ++k)
            if (k == 0 || c0 + k * 4 * NT < jb.ld) {
                TY o[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) o[q] = (TY)a[k][q];
                stg4(yr + c0 + k * 4 * NT, o);
            }
    }
}

// ---------------------------------------------------------------------------
// k_hv_row: one thread per element, one CTA per row (items of R = 1).
// For small sectors the kernels above are bound by their set-up (barriers,
// staging, tables of the item) and leave most threads without a column: a
// sector of 4,900 elements took 10 us in FP32 and 12 us in FP64 on 18 of 256
// or 512 threads per CTA.  Here the only barriers load the row's interspecies
// diagonal; every term reads its operands directly (L1 / L2), the row's
// down-spin moves as uniform loads, so a launch costs a few dependent loads.
// ---------------------------------------------------------------------------
template <typename TX, typename TA, typename TY, int NT>
__global__ void __launch_bounds__(NT)
k_hv_row(const __grid_constant__ HvBatch<TA> batch, const ModelDev *__restrict__ mdl)
{
    __shared__ TA s_cross[kMaxImp];
    __shared__ unsigned s_pmask[kMaxImp];
    __shared__ int s_t4[kMaxPair * kMaxImp];
    __shared__ double s_red[NT / 32];
    const int tid = threadIdx.x, nimp = mdl->nimp, npair = mdl->npair;
    for (int i = tid; i < npair * nimp; i += NT) s_t4[i] = mdl->t4[i];
    for (int i = tid; i < nimp; i += NT) s_pmask[i] = mdl->pairmask[i];
    const TA Jc = (TA)mdl->J;
    for (int item = blockIdx.x; item < batch.total_items; item += gridDim.x) {
        int j = 0;
        while (j + 1 < batch.njobs && item >= batch.job[j + 1].item0) ++j;
        const HvJobT<TA> &jb = batch.job[j];
        if (jb.active && *jb.active == 0) continue;
        const int it = item - jb.item0, d = jb.items[it], ld = jb.ld;
        const TX *__restrict__ x = (const TX *)jb.x;
        const TX *__restrict__ xd = x + (size_t)d * ld;
        TY *__restrict__ y = (TY *)jb.y + (size_t)d * ld;
        const int dinf = __ldg(jb.dn_info + d), id = (dinf >> 8) & 0xff;
        const TA ddiag = __ldg(jb.dn_diag + d);
        __syncthreads();   // the previous row is done with s_cross and s_red
        for (int i = tid; i < nimp; i += NT) s_cross[i] = (TA)mdl->cross[i * nimp + id];
        __syncthreads();
        double dacc = 0.0;
        for (int u = tid; u < ld; u += NT) {
            const int inf = __ldg(jb.up_info + u), iu = (inf >> 8) & 0xff;
            const TX xv = __ldg(xd + u);
            const TA acc = hv_moves<TX, TA, true>(jb, mdl, x, d, u, inf, dinf, s_pmask, s_t4, nimp, Jc,
                                                  (__ldg(jb.up_diag + u) + ddiag + s_cross[iu]) * (TA)xv);
            y[u] = (TY)acc;
            if (jb.dot_partial) dacc += (double)((TA)xv * (TA)(TY)acc);
        }
        if (jb.dot_partial) {
            for (int off = 16; off > 0; off >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, off);
            if ((tid & 31) == 0) s_red[tid >> 5] = dacc;
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int w = 0; w < NT / 32; ++w) t += s_red[w];
                jb.dot_partial[it] = t;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// k_hv_wide: FP32, up to three orbitals, R = 4 or 8 rows per item.
// The same fused sum as k_hv_async, arranged so that one schedule entry and
// one down-spin address serve more elements:
//   * the staged rows lie in planes of 16 bytes per column (4 rows each): a
//     move of a column reads 4 rows with one 16-byte load, where k_hv_async
//     took one 4-byte load per row;
//   * a lane owns two neighbouring columns: 8-byte loads of the down-spin
//     rows and stores of y, one row address for both, one 16-byte load for the
//     schedule entries of both;
//   * the quarter warps' targets of a slot fall in 8 different bank groups
//     (species_wide), so the 16-byte loads have no conflicts;
//   * a bath group of 2 or 3 rows sits in rows 0-2 of a plane; T_{i<-j} of the
//     up spin couples its rows pairwise (spin-flip one way, pair hopping the
//     other, the same sign), so the 4-operator terms are, per transition of
//     the column, one 16-byte load of the partner column and 6 FMAs with three
//     coefficients from a table of the model, without branches.
// Bound by shared-memory wavefronts and their latency (ncu, 15 million
// elements: 55 % of the LSU pipe, DRAM at 19 %): a slot serves the lanes that
// have a move in it, 58 % of them.  Ground sector of 3 orbitals x 4 levels, 41
// million elements: R = 8 after k_hv_down_rows 322 us (320, of it k_hv_wide 216,
// with x . y in FP32 over the row: 12 bytes of spills now, 4 then),
// two CTAs of R = 4 fused 345 us, R = 4 split 335 us; k_hv_async<SPLIT, 4> 463.
// Tried and not kept: more slots or moves in flight at fewer warps (350-550
// us, registers), skipping the lanes without a move by predicate (the same).
// ---------------------------------------------------------------------------
struct WideLayout {        // dynamic shared memory, in bytes
    int plane, cross, mv, jtab, dm;
};

__device__ __forceinline__ float4 wide_ld(const unsigned char *p) { return *reinterpret_cast<const float4 *>(p); }

// SPLIT: k_hv_down_rows has written the down-spin hybridisation into y; this
// kernel adds the other terms.  SB: schedule slots in flight; DB: down-spin
// moves of 4 rows in flight.
template <int R, int NT, int MINB, bool SPLIT, int SB, int DB>
__global__ void __launch_bounds__(NT, MINB)
k_hv_wide(const __grid_constant__ HvBatch<float> batch, const ModelDev *__restrict__ mdl, const WideLayout L)
{
    constexpr int NW = NT / 32, NP = R / 4;
    extern __shared__ __align__(16) unsigned char smem_wide[];
    float *const s_cross = reinterpret_cast<float *>(smem_wide + L.cross);   // [nimp][R]: interspecies + row diagonal
    HopEnt<float> *const s_mv = reinterpret_cast<HopEnt<float> *>(smem_wide + L.mv);   // [R][dm]: {row offset, coupling}
    const float4 *const s_j = reinterpret_cast<const float4 *>(smem_wide + L.jtab);    // [2][nimp][2]
    __shared__ int s_d[R], s_cnt[R], s_type[NP], s_most[NP];   // s_most: largest count of a plane's rows
    __shared__ double s_red[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nimp = mdl->nimp, npair = mdl->npair, norb = mdl->norb;

    // 4-operator table: for a group with ty + 1 impurity electrons and column
    // pattern iu, transition t: coefficients of the row pairs (0,1), (0,2),
    // (1,2) and the byte offset of the partner column
    if (tid < 2 * nimp) {
        const int ty = tid / nimp, iu = tid - ty * nimp;
        int nt = 0;
        float4 e[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        for (int p = 0; p < npair && nt < 2; ++p) {
            const int tu = mdl->t4[p * nimp + iu];   // T_{i<-j} of the up spin
            if (tu >= 0) continue;
            float c[3] = {0.f, 0.f, 0.f};
            if (ty + 1 < norb) {
                int idx = 0;
                for (int a = 0; a < nimp; ++a) {     // patterns of the group, in rank order
                    if (__popc(a) != ty + 1) continue;
                    const int td = mdl->t4[p * nimp + a];   // T_{i<-j} of the down spin on pattern a
                    if (td < 0) {
                        const int b = idx + (int)(short)(td & 0xffff);
                        const float v = (float)mdl->J * ((((tu ^ td) & 0x40000000) != 0) ? -1.f : 1.f);
                        c[min(idx, b) + max(idx, b) - 1] = v;   // (0,1) 0, (0,2) 1, (1,2) 2
                    }
                    ++idx;
                }
            }
            e[nt] = make_float4(c[0], c[1], c[2], __int_as_float((int)(short)(tu & 0xffff) * 16));
            ++nt;
        }
        float4 *o = const_cast<float4 *>(s_j) + 2 * tid;
        o[0] = e[0];
        o[1] = e[1];
    }

    int cur = hv_next_item(batch, (int)blockIdx.x);
    while (cur >= 0) {
        const HvJobT<float> &jb = batch.job[hv_find_job(batch, cur)];
        const int it = cur - jb.item0, ld = jb.ld, nd = jb.nd;
        const float *__restrict__ x = (const float *)jb.x;
        float *__restrict__ y = (float *)jb.y;
        const int *const rows = jb.items + (size_t)it * R;
        __syncthreads();   // the previous item is done with shared memory
        if (tid < R) {
            const int d = __ldg(rows + tid);
            const int inf = d >= 0 ? __ldg(jb.dn_info + d) : 0;
            s_d[tid] = d;
            s_cnt[tid] = inf & 0xff;
            if ((tid & 3) == 0) {
                const int pc = __popc((inf >> 8) & 0xff);
                s_type[tid >> 2] = (d >= 0 && pc > 0 && pc < norb) ? pc : 0;
            }
            int most = inf & 0xff;
            most = max(most, __shfl_xor_sync((1u << R) - 1u, most, 1));
            most = max(most, __shfl_xor_sync((1u << R) - 1u, most, 2));
            if ((tid & 3) == 0) s_most[tid >> 2] = most;
        }
        for (int i = tid; i < nimp * R; i += NT) {
            const int iu = i / R, d = __ldg(rows + (i - iu * R));
            const int id = d >= 0 ? (__ldg(jb.dn_info + d) >> 8) & 0xff : 0;
            s_cross[i] = d >= 0 ? (float)mdl->cross[iu * nimp + id] + __ldg(jb.dn_diag + d) : 0.f;
        }
        if (!SPLIT)
            for (int i = tid; i < R * jb.dn_maxcnt; i += NT) {
                const int s = i / R, r = i - s * R, d = __ldg(rows + r);
                if (d >= 0 && s < (__ldg(jb.dn_info + d) & 0xff)) {
                    HopEnt<float> e;
                    e.t = __ldg(jb.dn_tgt + (size_t)s * nd + d) * ld;
                    e.v = __ldg(jb.dn_val + (size_t)s * nd + d);
                    s_mv[r * L.dm + s] = e;
                }
            }
        {   // stage: two neighbouring columns of R rows per thread
            int dr[R];
#pragma unroll
            for (int r = 0; r < R; ++r) dr[r] = __ldg(rows + r);
            for (int u = 2 * tid; u < ld; u += 2 * NT) {
                float2 v[R];
#pragma unroll
                for (int r = 0; r < R; ++r)
                    v[r] = dr[r] >= 0 ? __ldg(reinterpret_cast<const float2 *>(x + (size_t)dr[r] * ld + u))
                                      : make_float2(0.f, 0.f);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    unsigned char *o = smem_wide + p * L.plane + 16 * u;
                    *reinterpret_cast<float4 *>(o) = make_float4(v[4 * p].x, v[4 * p + 1].x, v[4 * p + 2].x, v[4 * p + 3].x);
                    *reinterpret_cast<float4 *>(o + 16) = make_float4(v[4 * p].y, v[4 * p + 1].y, v[4 * p + 2].y, v[4 * p + 3].y);
                }
            }
        }
        const int nxt = hv_next_item(batch, cur + (int)gridDim.x);
        if (nxt >= 0) {   // the next item's rows into L2, one 128-byte line per thread and turn
            const HvJobT<float> &jn = batch.job[hv_find_job(batch, nxt)];
            const int *const rn = jn.items + (size_t)(nxt - jn.item0) * R;
            const int lines = jn.ld >> 5;
            for (int i = tid; i < R * lines; i += NT) {
                const int r = i / lines, d = __ldg(rn + r);
                if (d >= 0)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"((const float *)jn.x + (size_t)d * jn.ld +
                                                                  32 * (i - r * lines)));
            }
        }
        __syncthreads();
        const bool want_dot = jb.dot_partial != nullptr;
        double dacc = 0.0;
        const int nunit = (ld + 63) >> 6;
        for (int c = warp; c < nunit; c += NW) {
            const int u = 64 * c + 2 * lane;
            const bool has = u < ld;             // ld is a multiple of 32: both columns or none
            const int uc = has ? u : 0;
            const int2 h = __ldg(jb.up_sched_hdr + c);
            const float4 *ent = reinterpret_cast<const float4 *>(jb.up_sched + h.x) + lane;   // two entries per lane
            float4 e[SB];
#pragma unroll
            for (int t = 0; t < SB; ++t) e[t] = t < h.y ? __ldg(ent + 32 * t) : make_float4(0.f, 0.f, 0.f, 0.f);
            const int2 inf = __ldg(reinterpret_cast<const int2 *>(jb.up_info + uc));
            const float2 ud = __ldg(reinterpret_cast<const float2 *>(jb.up_diag + uc));
            const float *xu = x + uc;
            float acc[2][R];
            // down-spin rows, DB moves of 4 rows at a time; the first batch is in
            // flight during the diagonal
            float2 g[4][DB];
            auto load_moves = [&](int r0, int s0) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int t = 0; t < DB; ++t) {
                        g[q][t] = make_float2(0.f, 0.f);
                        if (s0 + t < s_cnt[r0 + q])
                            g[q][t] = __ldg(reinterpret_cast<const float2 *>(xu + (unsigned)s_mv[(r0 + q) * L.dm + s0 + t].t));
                    }
            };
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 yp = make_float2(0.f, 0.f);
                if constexpr (SPLIT) {
                    const int d = s_d[r];
                    if (has && d >= 0) yp = *reinterpret_cast<const float2 *>(y + (size_t)d * ld + u);
                }
                acc[0][r] = yp.x;
                acc[1][r] = yp.y;
            }
            if constexpr (!SPLIT) load_moves(0, 0);
            // diagonal and 4-operator terms
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int iu = ((k ? inf.y : inf.x) >> 8) & 0xff;
                const float udk = k ? ud.y : ud.x;
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const unsigned char *S = smem_wide + p * L.plane + 16 * (uc + k);
                    float *a = acc[k] + 4 * p;
                    const float4 xa = wide_ld(S);
                    const float4 ca = *reinterpret_cast<const float4 *>(s_cross + iu * R + 4 * p);
                    a[0] += (udk + ca.x) * xa.x;
                    a[1] += (udk + ca.y) * xa.y;
                    a[2] += (udk + ca.z) * xa.z;
                    a[3] += (udk + ca.w) * xa.w;
                    const int ty = s_type[p];
                    if (ty) {
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            const float4 j = s_j[((ty - 1) * nimp + iu) * 2 + t];
                            const float4 v = wide_ld(S + __float_as_int(j.w));
                            a[0] += j.x * v.y + j.y * v.z;
                            a[1] += j.x * v.x + j.z * v.z;
                            a[2] += j.y * v.x + j.z * v.y;
                        }
                    }
                }
            }
            if constexpr (!SPLIT) {
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const int n = s_most[p];
                    for (int s0 = 0; s0 < n; s0 += DB) {
                        if (p > 0 || s0 > 0) load_moves(4 * p, s0);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
#pragma unroll
                            for (int t = 0; t < DB; ++t)
                                if (s0 + t < s_cnt[4 * p + q]) {
                                    const float v = s_mv[(4 * p + q) * L.dm + s0 + t].v;
                                    acc[0][4 * p + q] += v * g[q][t].x;
                                    acc[1][4 * p + q] += v * g[q][t].y;
                                }
                    }
                }
            }
            // up-spin moves: SB slots ahead
            for (int s0 = 0; s0 < h.y; s0 += SB) {
                float4 f[SB];
#pragma unroll
                for (int t = 0; t < SB; ++t)
                    f[t] = s0 + SB + t < h.y ? __ldg(ent + 32 * (s0 + SB + t)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int t = 0; t < SB; ++t) {
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const unsigned char *S = smem_wide + __float_as_int(k ? e[t].z : e[t].x);
                        const float v = k ? e[t].w : e[t].y;
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const float4 ga = wide_ld(S + p * L.plane);
                            float *a = acc[k] + 4 * p;
                            a[0] += v * ga.x;
                            a[1] += v * ga.y;
                            a[2] += v * ga.z;
                            a[3] += v * ga.w;
                        }
                    }
                }
#pragma unroll
                for (int t = 0; t < SB; ++t) e[t] = f[t];
            }
            if (has) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int d = s_d[r];
                    if (d >= 0) *reinterpret_cast<float2 *>(y + (size_t)d * ld + u) = make_float2(acc[0][r], acc[1][r]);
                }
                if (want_dot) {   // rows that are not there are staged as zeros
                    // 2 R products in FP32, then FP64, as k_hv_async
                    float part = 0.f;
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const float4 xa = wide_ld(smem_wide + p * L.plane + 16 * (u + k));
                            const float *a = acc[k] + 4 * p;
                            part += (xa.x * a[0] + xa.y * a[1]) + (xa.z * a[2] + xa.w * a[3]);
                        }
                    dacc += widen(part);
                }
            }
        }
        if (want_dot) {
            for (int off = 16; off > 0; off >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, off);
            if (lane == 0) s_red[warp] = dacc;
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int w = 0; w < NW; ++w) t += s_red[w];
                jb.dot_partial[it] = t;
            }
        }
        cur = nxt;
    }
}

// ---------------------------------------------------------------------------
// k_hv_sorted: FP64 sums (FP64 or FP32 x), one row per CTA.
// Bound by the FP64 pipe, which a warp instruction holds for 64 cycles
// whatever its active lanes: k_hv issues a chunk's largest move count for
// every column of it (57 % of the lanes of 3 orbitals x 4 levels have a move)
// and FP32 x takes conversions on the same pipe.  Here
//   * the up-spin moves, the diagonal and the 4-operator terms run over
//     columns sorted by impurity pattern and move count (species_sorted): the
//     lanes of a warp have the same number of moves and the same 4-operator
//     terms;
//   * their sums go to a second shared-memory row; after one barrier the
//     down-spin AXPYs, uniform over the row, run in column order and write y;
//   * FP32 x is widened with integer operations, once per staged element and
//     per AXPY operand.
// One row and its sums are 104 KB at most, so two CTAs per SM overlap their
// loads.  FP64, us: 32 million elements of 3 orbitals x 4 levels 1,646 (k_hv)
// -> 1,012 (15 FP64 instructions per element take 830 at the pipe's rate),
// 0.85 million of 3 x 3 61 -> 33, dense V of 2 x 11 (2.9 million) 214 -> 163.
// ---------------------------------------------------------------------------
constexpr int kSortTerms = 6;   // 4-operator terms of a (row, pattern): at most (norb / 2)^2

template <typename TX, typename TY, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
k_hv_sorted(const __grid_constant__ HvBatch<double> batch, const ModelDev *__restrict__ mdl, int ldmax)
{
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) double smem_sorted[];
    double *const S = smem_sorted, *const A = S + ldmax;
    __shared__ double s_coef[2 * kMaxHop + 1], s_c[kMaxImp], s_jc[kMaxImp][kSortTerms], s_v[kMaxHop], s_red[NW];
    __shared__ int s_jn[kMaxImp], s_jo[kMaxImp][kSortTerms], s_off[kMaxHop];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nimp = mdl->nimp, npair = mdl->npair, ncpl = mdl->ncpl;
    for (int i = tid; i <= 2 * ncpl; i += NT)
        s_coef[i] = i == 2 * ncpl ? 0.0 : (i & 1) ? -mdl->cval[i >> 1] : mdl->cval[i >> 1];

    for (int cur = hv_next_item(batch, (int)blockIdx.x); cur >= 0; cur = hv_next_item(batch, cur + (int)gridDim.x)) {
        const HvJobT<double> &jb = batch.job[hv_find_job(batch, cur)];
        const int it = cur - jb.item0, ld = jb.ld, nd = jb.nd, d = __ldg(jb.items + it);
        const TX *__restrict__ x = (const TX *)jb.x;
        const TX *__restrict__ xd = x + (size_t)d * ld;
        TY *__restrict__ y = (TY *)jb.y + (size_t)d * ld;
        const int dinf = __ldg(jb.dn_info + d), id = (dinf >> 8) & 0xff, cnt = dinf & 0xff;
        __syncthreads();   // the previous row is done with shared memory
        for (int i = tid; i < cnt; i += NT) {
            s_off[i] = __ldg(jb.dn_tgt + (size_t)i * nd + d) * ld;
            s_v[i] = __ldg(jb.dn_val + (size_t)i * nd + d);
        }
        for (int iu = tid; iu < nimp; iu += NT) {
            s_c[iu] = mdl->cross[iu * nimp + id] + __ldg(jb.dn_diag + d);
            // spin-flip and pair-hop terms of this row for columns of pattern iu
            int n = 0;
            for (int p = 0; p < npair; ++p) {
                const int e = mdl->t4[p * nimp + iu];
                if (e >= 0) continue;
                const int esf = mdl->t4[mdl->pair_rev[p] * nimp + id], eph = mdl->t4[p * nimp + id];
                const int f = esf < 0 ? esf : eph;   // T_{j<-i}(d) or T_{i<-j}(d): never both
                if (f < 0 && n < kSortTerms) {
                    s_jo[iu][n] = (d + (int)(short)(f & 0xffff)) * ld + (int)(short)(e & 0xffff);
                    s_jc[iu][n] = ((e ^ f) & 0x40000000) ? -mdl->J : mdl->J;
                    ++n;
                }
            }
            s_jn[iu] = n;
        }
        for (int u = tid; u < ld; u += NT) {
            S[u] = widen(__ldg(xd + u));
            if (u >= jb.nu) A[u] = 0.0;
        }
        __syncthreads();
        for (int c = warp; c < jb.srt_n; c += NW) {
            const int2 h = __ldg(jb.srt_hdr + c);
            // a lane without a column reads as lane 0 does: the 4-operator
            // terms' partner columns exist for every column of the pattern, and
            // not for any other
            const int uc = __ldg(jb.srt_col + 32 * c + lane), u0 = __shfl_sync(0xffffffffu, uc, 0), u = uc >= 0 ? uc : u0;
            const int ns = h.y & 0xffff, iu = h.y >> 16;
            const unsigned *ent = jb.srt_ent + h.x + lane;
            // the loops below end by a branch: a predicated-off FP64 instruction
            // would hold the pipe as long as one that counts.  The operands
            // of the next QE / QD turns are in flight in a queue.
            constexpr int QE = 4;
            unsigned e[QE];
#pragma unroll
            for (int t = 0; t < QE; ++t) e[t] = t < ns ? __ldg(ent + 32 * t) : 0u;
            const int nj = s_jn[iu];
            double acc = (__ldg(jb.up_diag + u) + s_c[iu]) * S[u];
            if (nj > 0) {
                TX g = __ldg(x + (s_jo[iu][0] + u));
#pragma unroll 1
                for (int t = 0; t < nj; ++t) {
                    const TX h2 = t + 1 < nj ? __ldg(x + (s_jo[iu][t + 1] + u)) : TX(0);
                    acc = fma(s_jc[iu][t], widen(g), acc);
                    g = h2;
                }
            }
#pragma unroll 1
            for (int s = 0; s < ns; ++s) {
                const unsigned m = e[0];
#pragma unroll
                for (int t = 0; t + 1 < QE; ++t) e[t] = e[t + 1];
                e[QE - 1] = s + QE < ns ? __ldg(ent + 32 * (s + QE)) : 0u;
                acc = fma(s_coef[m >> 16], S[m & 0xffffu], acc);
            }
            if (uc >= 0) A[u] = acc;
        }
        __syncthreads();
        const bool want_dot = jb.dot_partial != nullptr;
        double dacc = 0.0;
        for (int u = tid; u < ld; u += NT) {   // ld is a multiple of 32: whole warps
            double acc = A[u];
            constexpr int QD = 6;
            TX g[QD];
#pragma unroll
            for (int t = 0; t < QD; ++t) g[t] = t < cnt ? __ldg(x + (s_off[t] + u)) : TX(0);
#pragma unroll 1
            for (int s = 0; s < cnt; ++s) {
                const TX h2 = g[0];
#pragma unroll
                for (int t = 0; t + 1 < QD; ++t) g[t] = g[t + 1];
                g[QD - 1] = s + QD < cnt ? __ldg(x + (s_off[s + QD] + u)) : TX(0);
                acc = fma(s_v[s], widen(h2), acc);
            }
            y[u] = (TY)acc;
            if (want_dot) dacc = fma(S[u], acc, dacc);
        }
        if (want_dot) {
            for (int off = 16; off > 0; off >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, off);
            if (lane == 0) s_red[warp] = dacc;
            __syncthreads();
            if (tid == 0) {
                double t = 0.0;
                for (int w = 0; w < NW; ++w) t += s_red[w];
                jb.dot_partial[it] = t;
            }
        }
    }
}

template <typename TX, typename TA, int R>
static size_t dyn_smem_bytes_async(int ld, const ModelDev &m, const DescGeom &g)
{
    return ((2 * (size_t)R * ld * sizeof(TX) + 15) & ~(size_t)15) + sizeof(unsigned) * 2 * (size_t)g.words +
           sizeof(int) * (size_t)m.npair * m.nimp;
}

// ---------------------------------------------------------------------------
// tile-shape variants and the autotuner
// ---------------------------------------------------------------------------
// A variant fixes the kernel, the rows per item R, the CTA size NT and the CTAs
// per SM the register budget is cut for (MINB).  The kernels add the terms of an
// element in different orders (k_hv and k_hv_row by column and move, k_hv_async
// and k_hv_wide as their gather schedules have them, k_hv_sorted the down-spin
// moves last), so their outputs agree to rounding.  The first H*v of a (kind,
// Nup, Ndn) shape of kTuneMinElems elements or more times each variant on that
// sector (scratch vectors, CUDA events on the context stream) and keeps the
// fastest.  A variant number belongs to these tables, not to the interface:
// programs that pin one take it from the list of hv_tuning.
// k_hv_wide<8> has 26 warps: they take the 101 units of 64 columns of a row of
// 6,435 in four turns, and their 72 registers a thread are 91 % of an SM's.
struct HvVariant {
    int R, NT, MINB;
    // 0: k_hv, or k_hv_row when R = 1; 1: k_hv_async (double-buffered asynchronous stage);
    // 2 / 3: split, k_hv_down on 128- / 64-byte row slices + k_hv_async<SPLIT>;
    // 4: split, k_hv_down_rows (row AXPYs from L2) + k_hv_async<SPLIT>
    int staged;
    bool wide = false;   // k_hv_wide in the place of k_hv_async
    bool sorted = false; // k_hv_sorted (one row per item)
    int key() const { return wide ? kWideKey + R : R; }   // of the item table
};
static const HvVariant kVarF32[] = {{4, 512, 2, 1, true}, {4, 256, 2, 0}, {6, 512, 1, 0}, {3, 256, 3, 0},
                                    {8, 832, 1, 4, true}, {4, 512, 1, 1}, {3, 512, 1, 1}, {4, 512, 2, 4, true},
                                    {2, 256, 2, 1}, {3, 512, 1, 2}, {4, 512, 1, 2}, {3, 512, 1, 3},
                                    {3, 512, 1, 4}, {4, 512, 1, 4}, {4, 512, 1, 4}, {1, 128, 8, 0}};
static const HvVariant kVarF64[] = {{2, 512, 1, 1}, {2, 512, 1, 2}, {2, 512, 1, 4}, {1, 128, 8, 0},
                                    {1, 512, 2, 0, false, true}, {1, 256, 4, 0, false, true}, {1, 128, 6, 0, false, true}};
// the small sectors' shapes (hv_prepare)
static const int kRowVarF32 = 15, kRowVarF64 = 3;       // k_hv_row
static const int kSmallVarF32 = 8, kSmallVarF64 = 5;    // k_hv_async<2, 256>, k_hv_sorted<256>
static const int kNVarF32 = sizeof(kVarF32) / sizeof(kVarF32[0]);
static const int kNVarF64 = sizeof(kVarF64) / sizeof(kVarF64[0]);

static const HvVariant &variant(int kind, int v) { return kind == HV_F32 ? kVarF32[v] : kVarF64[v]; }
static int nvariants(int kind) { return kind == HV_F32 ? kNVarF32 : kNVarF64; }

constexpr long long kTuneMinElems = 1ll << 18;   // smaller sectors take a shape by rule (hv_prepare)

static long long shape_key(int kind, const Sector &s) { return ((long long)kind << 32) | (s.ne_up << 16) | s.ne_down; }

template <typename TA>
void hv_fill_job(const mo_ed_ctx *ctx, const Sector &s, int R, const void *x, void *y, HvJobT<TA> &j)
{
    const bool f32 = sizeof(TA) == 4;
    (void)ctx;
    j.x = x;
    j.y = y;
    j.dot_partial = nullptr;
    j.active = nullptr;
    j.nu = s.up->n;
    j.nd = s.dn->n;
    j.ld = s.ld();
    auto it = s.dn->items.find(R);
    j.items = it != s.dn->items.end() ? it->second : nullptr;
    j.nitems = it != s.dn->items.end() ? s.dn->nitems.at(R) : 0;
    j.item0 = 0;
    j.up_info = s.up->info;
    j.up_tab = f32 ? (const HopEnt<TA> *)s.up->tab_f : (const HopEnt<TA> *)s.up->tab_d;
    j.up_diag = f32 ? (const TA *)s.up->diag_f : (const TA *)s.up->diag_d;
    j.up_hw = s.up->hw;
    j.up_maxcnt = s.up->max_cnt;
    j.dn_info = s.dn->info;
    j.dn_tgt = s.dn->hop_tgt;
    j.dn_val = f32 ? (const TA *)s.dn->hop_val_f : (const TA *)s.dn->hop_val_d;
    j.dn_diag = f32 ? (const TA *)s.dn->diag_f : (const TA *)s.dn->diag_d;
    j.dn_maxcnt = s.dn->max_cnt;
    j.pad = 0;
    j.up_sched_hdr = s.up->sched_hdr;
    j.up_sched_ent = s.up->sched_ent;
    {
        auto dsc = s.dn->desc.find(R * 2 + (f32 ? 0 : 1));
        j.desc = dsc != s.dn->desc.end() ? dsc->second : nullptr;
    }
    j.srt_hdr = s.up->srt_hdr;
    j.srt_col = s.up->srt_col;
    j.srt_ent = s.up->srt_ent;
    j.srt_n = s.up->srt_n;
    j.dblk_off = s.dn->dblk_off;
    j.dblk_rows = s.dn->dblk_rows;
    j.dblk_ptr = s.dn->dblk_ptr;
    j.dblk_mv = f32 ? (const HopEnt<TA> *)s.dn->dblk_mv_f : (const HopEnt<TA> *)s.dn->dblk_mv_d;
    {
        auto ch = s.dn->dblk_chunks.find(s.ld());
        j.dblk_chunks = ch != s.dn->dblk_chunks.end() ? ch->second : nullptr;
        j.ntiles = ch != s.dn->dblk_chunks.end() ? s.dn->dblk_nchunks.at(s.ld()) : 0;
    }
    j.dblk_n = s.dn->dblk_n;
    j.dblk_max = s.dn->dblk_max;
    j.dblk_mvmax = s.dn->dblk_mvmax;
    j.tile0 = 0;
    if (f32 && R >= kWideKey) {
        j.up_sched_hdr = s.up->wide_hdr;
        j.up_sched = (const HopEnt<TA> *)s.up->wide_ent;
    } else if (f32) {
        auto sf = s.up->sched_rf.find(R);
        j.up_sched = sf != s.up->sched_rf.end() ? (const HopEnt<TA> *)sf->second : nullptr;
    } else {
        auto sd = s.up->sched_rd.find(R);
        j.up_sched = sd != s.up->sched_rd.end() ? (const HopEnt<TA> *)sd->second : nullptr;
    }
}
template void hv_fill_job<float>(const mo_ed_ctx *, const Sector &, int, const void *, void *, HvJobT<float> &);
template void hv_fill_job<double>(const mo_ed_ctx *, const Sector &, int, const void *, void *, HvJobT<double> &);

// Makes kernel k launchable with smem bytes of dynamic shared memory (and the
// full carveout) and returns its resident CTAs per SM at nt threads.  The
// runtime calls cost more than the launch of a small sector's H*v, so they
// are made once per (device, kernel): the shared-memory limit only ever
// rises, and the occupancy is kept per (device, kernel, size, threads).
// Process-wide, under a lock, so contexts on one device agree.
static std::mutex g_kfit_mu;
static std::map<std::pair<int, const void *>, size_t> g_kfit_smem;
static std::map<std::tuple<int, const void *, size_t, int>, int> g_kfit_occ;

template <typename K>
static int kernel_fit(mo_ed_ctx *ctx, K k, int nt, size_t smem, int *per_sm)
{
    std::lock_guard<std::mutex> lock(g_kfit_mu);
    const void *kp = (const void *)k;
    auto ins = g_kfit_smem.emplace(std::make_pair(ctx->device, kp), (size_t)0);
    size_t &set = ins.first->second;
    if (ins.second)
        MOED_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    if (smem > set) {
        MOED_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        set = smem;
    }
    const auto key = std::make_tuple(ctx->device, kp, smem, nt);
    auto it = g_kfit_occ.find(key);
    if (it == g_kfit_occ.end()) {
        int n = 0;
        MOED_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, nt, smem));
        it = g_kfit_occ.emplace(key, n).first;
    }
    *per_sm = it->second;
    return MO_ED_OK;
}

template <typename TX, typename TA, typename TY, int R, int NT, int MINB>
static int launch_batch(mo_ed_ctx *ctx, const HvBatch<TA> &b)
{
    if (b.total_items <= 0) return MO_ED_OK;
    int ldmax = 0;
    for (int i = 0; i < b.njobs; ++i) {
        ldmax = std::max(ldmax, b.job[i].ld);
        if (!b.job[i].items) return fail(ctx, MO_ED_ERR_STATE, "H*v item table missing");
    }
    const size_t smem = dyn_smem_bytes<TX, TA, R>(ldmax, ctx->mdl);
    auto kern = k_hv<TX, TA, TY, R, NT, MINB>;
    int per_sm = 0;
    if (int rc = kernel_fit(ctx, kern, NT, smem, &per_sm)) return rc;
    if (per_sm < 1) return fail(ctx, MO_ED_ERR_ARG, "sector rows too long for the shared-memory stage");
    const int grid = std::min(b.total_items, ctx->num_sms * per_sm);
    kern<<<grid, NT, smem, ctx->stream>>>(b, ctx->d_mdl);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

template <typename TX, typename TA, typename TY, int R, int NT, int MINB = 1, bool SPLIT = false>
static int launch_batch_async(mo_ed_ctx *ctx, const HvBatch<TA> &b)
{
    if (b.total_items <= 0) return MO_ED_OK;
    int ldmax = 0;
    for (int i = 0; i < b.njobs; ++i) {
        ldmax = std::max(ldmax, b.job[i].ld);
        if (!b.job[i].items || !b.job[i].up_sched_hdr || !b.job[i].up_sched || !b.job[i].desc)
            return fail(ctx, MO_ED_ERR_STATE, "H*v tables missing");
    }
    const DescGeom g = desc_geom<TA, R>(ctx->mdl.ncpl, ctx->mdl);
    const size_t smem = dyn_smem_bytes_async<TX, TA, R>(ldmax, ctx->mdl, g);
    auto kern = k_hv_async<TX, TA, TY, R, NT, MINB, SPLIT>;
    int per_sm = 0;
    if (int rc = kernel_fit(ctx, kern, NT, smem, &per_sm)) return rc;
    if (per_sm < 1) return fail(ctx, MO_ED_ERR_ARG, "sector rows too long for the shared-memory stage");
    const int grid = std::min(b.total_items, ctx->num_sms * per_sm);
    kern<<<grid, NT, smem, ctx->stream>>>(b, ctx->d_mdl, g);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

constexpr int kDownNT = 1024;
constexpr size_t kDownSmemMax = 220 * 1024;   // dynamic shared memory of one k_hv_down CTA

static size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }

// shared-memory layout of k_hv_down for blocks of up to `rows` rows and `mv`
// moves and slices of wb bytes per row; nbuf = 1 or 2 slice buffers
static DownLayout down_layout(int rows, int mv, size_t wb, int nbuf, size_t ent_bytes, size_t *total)
{
    DownLayout L;
    size_t o = 0;
    L.ptr = (int)o;
    o = align16(o + sizeof(int) * ((size_t)rows + 1));
    L.rows = (int)o;
    o = align16(o + sizeof(int) * (size_t)rows);
    L.mv = (int)o;
    o = align16(o + ent_bytes * (size_t)std::max(mv, 1));
    L.x0 = (int)o;
    o += (size_t)rows * wb;
    L.x1 = (int)o;
    if (nbuf == 2) o += (size_t)rows * wb;
    *total = o;
    return L;
}

// Split H*v: k_hv_down writes the down-spin hybridisation into y, then
// k_hv_async<SPLIT> adds the other terms (both on the context stream).
template <typename TX, typename TA, typename TY, int R, int NT, int MINB, int WB>
static int launch_batch_split(mo_ed_ctx *ctx, const HvBatch<TA> &b0)
{
    if (b0.total_items <= 0) return MO_ED_OK;
    HvBatch<TA> b = b0;
    int tiles = 0, maxrows = 0, maxmv = 0;
    for (int i = 0; i < b.njobs; ++i) {
        HvJobT<TA> &j = b.job[i];
        if (!j.dblk_ptr || !j.dblk_chunks || j.dblk_n < 1 || j.ld % 32 != 0)
            return fail(ctx, MO_ED_ERR_STATE, "H*v down-spin block tables missing");
        j.tile0 = tiles;
        tiles += j.ntiles;
        maxrows = std::max(maxrows, j.dblk_max);
        maxmv = std::max(maxmv, j.dblk_mvmax);
    }
    size_t smem = 0;
    int dbuf = 1;
    DownLayout L = down_layout(maxrows, maxmv, WB, 2, sizeof(HopEnt<TA>), &smem);
    if (smem > kDownSmemMax) {
        dbuf = 0;
        L = down_layout(maxrows, maxmv, WB, 1, sizeof(HopEnt<TA>), &smem);
    }
    if (smem > kDownSmemMax) return fail(ctx, MO_ED_ERR_ARG, "down-spin blocks too large for the split H*v");
    auto kd = k_hv_down<TX, TA, TY, kDownNT, WB>;
    int per_sm = 0;
    if (int rc = kernel_fit(ctx, kd, kDownNT, smem, &per_sm)) return rc;
    if (per_sm < 1) return fail(ctx, MO_ED_ERR_ARG, "down-spin blocks too large for the split H*v");
    const int grid = std::min(tiles, ctx->num_sms * per_sm);
    kd<<<grid, kDownNT, smem, ctx->stream>>>(b, tiles, L, maxrows, dbuf);
    MOED_CHECK_LAUNCH(ctx);
    return launch_batch_async<TX, TA, TY, R, NT, MINB, true>(ctx, b);
}

// Split H*v with the row-AXPY down pass: k_hv_down_rows writes the
// down-spin hybridisation into y, then k_hv_async<SPLIT> adds the rest.
constexpr int kRowsNT = 128;   // 512 CPT columns per tile
template <typename TX, typename TA, typename TY, int CPT>
static int launch_rows_pass(mo_ed_ctx *ctx, HvBatch<TA> &b)
{
    long long tiles = 0;
    for (int i = 0; i < b.njobs; ++i) {
        HvJobT<TA> &j = b.job[i];
        if (!j.dn_info || !j.dn_tgt || !j.dn_val || j.ld % 4 != 0)
            return fail(ctx, MO_ED_ERR_STATE, "H*v down-spin move tables missing");
        if (j.dn_maxcnt > kRowsNT) return fail(ctx, MO_ED_ERR_ARG, "more down-spin moves per row than the row-AXPY CTA stages");
        j.tile0 = (int)tiles;
        j.ntiles = j.nd * ((j.ld + 4 * kRowsNT * CPT - 1) / (4 * kRowsNT * CPT));
        tiles += j.ntiles;
    }
    if (tiles > INT_MAX) return fail(ctx, MO_ED_ERR_ARG, "too many row tiles for the row-AXPY H*v");
    auto kd = k_hv_down_rows<TX, TA, TY, kRowsNT, CPT>;
    int per_sm = 0;
    if (int rc = kernel_fit(ctx, kd, kRowsNT, 0, &per_sm)) return rc;
    const int grid = (int)std::min<long long>(tiles, (long long)ctx->num_sms * std::max(per_sm, 1));
    if (grid > 0) {
        kd<<<grid, kRowsNT, 0, ctx->stream>>>(b, (int)tiles);
        MOED_CHECK_LAUNCH(ctx);
    }
    return MO_ED_OK;
}

template <typename TX, typename TA, typename TY, int R, int NT, int MINB, int CPT = 2>
static int launch_batch_rows(mo_ed_ctx *ctx, const HvBatch<TA> &b0)
{
    if (b0.total_items <= 0) return MO_ED_OK;
    HvBatch<TA> b = b0;
    if (int rc = launch_rows_pass<TX, TA, TY, CPT>(ctx, b)) return rc;
    return launch_batch_async<TX, TA, TY, R, NT, MINB, true>(ctx, b);
}

// One element per thread (k_hv_row), one CTA per row.
constexpr int kRowNT = 128;
template <typename TX, typename TA, typename TY>
static int launch_batch_row(mo_ed_ctx *ctx, const HvBatch<TA> &b)
{
    if (b.total_items <= 0) return MO_ED_OK;
    for (int i = 0; i < b.njobs; ++i)
        if (!b.job[i].items) return fail(ctx, MO_ED_ERR_STATE, "H*v item table missing");
    const int grid = std::min(b.total_items, ctx->num_sms * 16);   // 16 CTAs of 128 threads fill an SM
    k_hv_row<TX, TA, TY, kRowNT><<<grid, kRowNT, 0, ctx->stream>>>(b, ctx->d_mdl);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

template <typename TX, typename TY, int NT, int MINB>
static int launch_batch_sorted(mo_ed_ctx *ctx, const HvBatch<double> &b)
{
    if (b.total_items <= 0) return MO_ED_OK;
    int ldmax = 0;
    for (int i = 0; i < b.njobs; ++i) {
        ldmax = std::max(ldmax, b.job[i].ld);
        if (!b.job[i].items || !b.job[i].srt_ent) return fail(ctx, MO_ED_ERR_STATE, "H*v tables missing");
    }
    const size_t smem = 2 * sizeof(double) * (size_t)ldmax;
    auto kern = k_hv_sorted<TX, TY, NT, MINB>;
    int per_sm = 0;
    if (int rc = kernel_fit(ctx, kern, NT, smem, &per_sm)) return rc;
    if (per_sm < 1) return fail(ctx, MO_ED_ERR_ARG, "sector rows too long for the shared-memory stage");
    kern<<<std::min(b.total_items, ctx->num_sms * per_sm), NT, smem, ctx->stream>>>(b, ctx->d_mdl, ldmax);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

// shared memory of k_hv_wide for rows of up to ldmax columns
static WideLayout wide_layout(int ldmax, int rows, const ModelDev &m, size_t *total)
{
    WideLayout L;
    L.plane = 16 * ldmax;
    L.dm = std::max(m.ncpl, 1);
    L.cross = rows / 4 * L.plane;
    L.mv = L.cross + (int)sizeof(float) * m.nimp * rows;
    L.jtab = (int)align16((size_t)L.mv + sizeof(HopEnt<float>) * rows * (size_t)L.dm);
    *total = (size_t)L.jtab + sizeof(float4) * 4 * (size_t)m.nimp;
    return L;
}

template <int R, int NT, int MINB, bool SPLIT, int SB, int DB>
static int launch_batch_wide(mo_ed_ctx *ctx, const HvBatch<float> &b0)
{
    if (b0.total_items <= 0) return MO_ED_OK;
    if (ctx->mdl.norb > 3) return fail(ctx, MO_ED_ERR_ARG, "more orbitals than this H*v tile shape takes");
    HvBatch<float> b = b0;
    int ldmax = 0;
    for (int i = 0; i < b.njobs; ++i) {
        ldmax = std::max(ldmax, b.job[i].ld);
        if (!b.job[i].items || !b.job[i].up_sched_hdr || !b.job[i].up_sched)
            return fail(ctx, MO_ED_ERR_STATE, "H*v tables missing");
    }
    size_t smem = 0;
    const WideLayout L = wide_layout(ldmax, R, ctx->mdl, &smem);
    auto kern = k_hv_wide<R, NT, MINB, SPLIT, SB, DB>;
    int per_sm = 0;
    if (int rc = kernel_fit(ctx, kern, NT, smem, &per_sm)) return rc;
    if (per_sm < 1) return fail(ctx, MO_ED_ERR_ARG, "sector rows too long for the shared-memory stage");
    if (SPLIT)
        if (int rc = launch_rows_pass<float, float, float, 2>(ctx, b)) return rc;
    const int grid = std::min(b.total_items, ctx->num_sms * per_sm);
    kern<<<grid, NT, smem, ctx->stream>>>(b, ctx->d_mdl, L);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

// Whether the split kernel fits every down-spin block of the model (any
// electron count: at most dblk_bound rows and dblk_mv_bound moves).
static bool split_fits(const mo_ed_ctx *ctx, size_t wb, size_t ent_bytes)
{
    size_t smem = 0;
    down_layout(ctx->dblk_bound, ctx->dblk_mv_bound, wb, 1, ent_bytes, &smem);
    return smem <= kDownSmemMax;
}

template <typename TA, int R>
static int build_desc_r(mo_ed_ctx *ctx, Species *dn, unsigned **out)
{
    const DescGeom g = desc_geom<TA, R>(ctx->mdl.ncpl, ctx->mdl);
    const int n = dn->nitems.at(R);
    unsigned *p = nullptr;
    MOED_CUDA(ctx, cudaMalloc(&p, sizeof(unsigned) * (size_t)g.words * std::max(n, 1)));
    *out = p;
    const bool f32 = sizeof(TA) == 4;
    k_item_desc<TA, R><<<(n + 127) / 128, 128, 0, ctx->stream>>>(
        n, dn->items.at(R), dn->info, f32 ? (const TA *)dn->diag_f : (const TA *)dn->diag_d, dn->hop_tgt,
        f32 ? (const TA *)dn->hop_val_f : (const TA *)dn->hop_val_d, dn->n, ctx->d_mdl, g, p);
    MOED_CHECK_LAUNCH(ctx);
    return MO_ED_OK;
}

// item descriptors of the down species for R rows per item (k_hv_async)
static int species_desc(mo_ed_ctx *ctx, Species *dn, int R, bool f32)
{
    const int key = R * 2 + (f32 ? 0 : 1);
    if (dn->desc.count(key)) return MO_ED_OK;
    unsigned *p = nullptr;
    int rc;
    switch (R) {
    case 2: rc = f32 ? build_desc_r<float, 2>(ctx, dn, &p) : build_desc_r<double, 2>(ctx, dn, &p); break;
    case 3: rc = f32 ? build_desc_r<float, 3>(ctx, dn, &p) : build_desc_r<double, 3>(ctx, dn, &p); break;
    case 4: rc = f32 ? build_desc_r<float, 4>(ctx, dn, &p) : build_desc_r<double, 4>(ctx, dn, &p); break;
    default: return fail(ctx, MO_ED_ERR_ARG, "no item descriptors for this rows-per-item");
    }
    if (p) dn->desc[key] = p;
    return rc;
}

template <typename TA>
static int launch_variant(mo_ed_ctx *ctx, int kind, int v, const HvBatch<TA> &b)
{
    if constexpr (sizeof(TA) == 4) {
        (void)kind;
        switch (v) {
        case 0: return launch_batch_wide<4, 512, 2, false, 2, 2>(ctx, b);
        case 1: return launch_batch<float, float, float, 4, 256, 2>(ctx, b);
        case 2: return launch_batch<float, float, float, 6, 512, 1>(ctx, b);
        case 3: return launch_batch<float, float, float, 3, 256, 3>(ctx, b);
        case 4: return launch_batch_wide<8, 832, 1, true, 2, 1>(ctx, b);
        case 5: return launch_batch_async<float, float, float, 4, 512>(ctx, b);
        case 6: return launch_batch_async<float, float, float, 3, 512>(ctx, b);
        case 7: return launch_batch_wide<4, 512, 2, true, 2, 1>(ctx, b);
        case 8: return launch_batch_async<float, float, float, 2, 256, 2>(ctx, b);
        case 9: return launch_batch_split<float, float, float, 3, 512, 1, 128>(ctx, b);
        case 10: return launch_batch_split<float, float, float, 4, 512, 1, 128>(ctx, b);
        case 11: return launch_batch_split<float, float, float, 3, 512, 1, 64>(ctx, b);
        case 12: return launch_batch_rows<float, float, float, 3, 512, 1>(ctx, b);
        case 13: return launch_batch_rows<float, float, float, 4, 512, 1>(ctx, b);
        case 14: return launch_batch_rows<float, float, float, 4, 512, 1, 4>(ctx, b);   // 2,048-column tiles
        default: return launch_batch_row<float, float, float>(ctx, b);
        }
    } else if (kind == HV_F64) {
        switch (v) {
        case 0: return launch_batch_async<double, double, double, 2, 512>(ctx, b);
        case 1: return launch_batch_split<double, double, double, 2, 512, 1, 128>(ctx, b);
        case 2: return launch_batch_rows<double, double, double, 2, 512, 1>(ctx, b);
        case 3: return launch_batch_row<double, double, double>(ctx, b);
        case 4: return launch_batch_sorted<double, double, 512, 2>(ctx, b);
        case 5: return launch_batch_sorted<double, double, 256, 4>(ctx, b);
        default: return launch_batch_sorted<double, double, 128, 6>(ctx, b);
        }
    } else {
        switch (v) {
        case 0: return launch_batch_async<float, double, double, 2, 512>(ctx, b);
        case 1: return launch_batch_split<float, double, double, 2, 512, 1, 128>(ctx, b);
        case 2: return launch_batch_rows<float, double, double, 2, 512, 1>(ctx, b);
        case 3: return launch_batch_row<float, double, double>(ctx, b);
        case 4: return launch_batch_sorted<float, double, 512, 2>(ctx, b);
        case 5: return launch_batch_sorted<float, double, 256, 4>(ctx, b);
        default: return launch_batch_sorted<float, double, 128, 6>(ctx, b);
        }
    }
}

template <typename TA>
static int hv_run_jobs(mo_ed_ctx *ctx, int kind, int v, const HvJobT<TA> *jobs, int njobs)
{
    HvBatch<TA> b;
    b.njobs = 0;
    b.total_items = 0;
    for (int i = 0; i < njobs; ++i) {
        if (b.njobs == kMaxJobs) {
            if (int rc = launch_variant<TA>(ctx, kind, v, b)) return rc;
            b.njobs = 0;
            b.total_items = 0;
        }
        b.job[b.njobs] = jobs[i];
        b.job[b.njobs].item0 = b.total_items;
        b.total_items += jobs[i].nitems;
        b.njobs++;
    }
    if (b.njobs == 0) return MO_ED_OK;
    return launch_variant<TA>(ctx, kind, v, b);
}

int hv_launch_f32(mo_ed_ctx *ctx, int v, const HvJobT<float> *jobs, int njobs)
{
    return hv_run_jobs<float>(ctx, HV_F32, v, jobs, njobs);
}
int hv_launch_f64(mo_ed_ctx *ctx, int kind, int v, const HvJobT<double> *jobs, int njobs)
{
    return hv_run_jobs<double>(ctx, kind, v, jobs, njobs);
}

static int launch_one(mo_ed_ctx *ctx, const Sector &s, int kind, int v, const void *x, void *y)
{
    const int R = variant(kind, v).key();
    if (kind == HV_F32) {
        HvJobT<float> j;
        hv_fill_job<float>(ctx, s, R, x, y, j);
        return hv_launch_f32(ctx, v, &j, 1);
    }
    HvJobT<double> j;
    hv_fill_job<double>(ctx, s, R, x, y, j);
    return hv_launch_f64(ctx, kind, v, &j, 1);
}

// tables variant v of `kind` reads for sector s: the item table of its R,
// and for the staged kernel the up-spin schedule and the item descriptors
static int prepare_variant(mo_ed_ctx *ctx, const Sector &s, int kind, int v)
{
    const HvVariant &h = variant(kind, v);
    const int *items;
    int n;
    if (int rc = species_items(ctx, s.dn, h.key(), &items, &n)) return rc;
    if (h.sorted) return species_sorted(ctx, s.up);
    if (!h.staged) return MO_ED_OK;
    if (h.wide) return species_wide(ctx, s.up);
    if (h.staged == 2 || h.staged == 3) {
        // the split kernel stages whole down-spin blocks: the largest block of
        // the model (any electron count) must fit one CTA's shared memory
        const size_t wb = h.staged == 2 ? 128 : 64;
        if (!split_fits(ctx, wb, kind == HV_F32 ? sizeof(HopEnt<float>) : sizeof(HopEnt<double>)))
            return fail(ctx, MO_ED_ERR_ARG, "down-spin blocks too large for the split H*v");
        if (int rc = species_dblocks(ctx, s.dn, s.ld())) return rc;
    }
    if (int rc = species_sched(ctx, s.up, h.R)) return rc;
    return species_desc(ctx, s.dn, h.R, kind == HV_F32);
}

// Time every variant once on sector s and keep the fastest.
static int tune(mo_ed_ctx *ctx, const Sector &s, int kind, int *best)
{
    const size_t ex = kind == HV_F64 ? sizeof(double) : sizeof(float);
    const size_t ey = kind == HV_F32 ? sizeof(float) : sizeof(double);
    DevBuf dx, dy;
    if (int rc = dev_alloc(ctx, dx, ex * (size_t)s.Dpad())) return rc;
    if (int rc = dev_alloc(ctx, dy, ey * (size_t)s.Dpad())) return rc;
    MOED_CUDA(ctx, cudaMemsetAsync(dx.p, 0, dx.bytes, ctx->stream));
    cudaEvent_t e0, e1;
    MOED_CUDA(ctx, cudaEventCreate(&e0));
    MOED_CUDA(ctx, cudaEventCreate(&e1));
    float tbest = 1e30f;
    *best = -1;
    std::vector<float> &times = ctx->hv_times[shape_key(kind, s)];
    times.assign(nvariants(kind), -1.0f);
    for (int v = 0; v < nvariants(kind); ++v) {
        if (int rc = prepare_variant(ctx, s, kind, v)) {
            if (rc == MO_ED_ERR_ARG) continue;   // variant not applicable to this model
            return rc;
        }
        if (launch_one(ctx, s, kind, v, dx.p, dy.p) != MO_ED_OK) {   // variant does not fit this sector
            cudaGetLastError();
            continue;
        }
        float tv = 1e30f;
        for (int rep = 0; rep < 3; ++rep) {
            MOED_CUDA(ctx, cudaEventRecord(e0, ctx->stream));
            if (int rc = launch_one(ctx, s, kind, v, dx.p, dy.p)) return rc;
            MOED_CUDA(ctx, cudaEventRecord(e1, ctx->stream));
            MOED_CUDA(ctx, cudaEventSynchronize(e1));
            float ms = 0.f;
            MOED_CUDA(ctx, cudaEventElapsedTime(&ms, e0, e1));
            tv = std::min(tv, ms);
        }
        times[v] = tv;
        if (tv < tbest) {
            tbest = tv;
            *best = v;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (*best < 0) return fail(ctx, MO_ED_ERR_ARG, "no H*v tile shape fits this sector");
    ctx->err.clear();
    return MO_ED_OK;
}

int hv_prepare(mo_ed_ctx *ctx, const Sector &s, int kind, int *v_out, int *R_out)
{
    const long long key = shape_key(kind, s);
    auto it = ctx->hv_choice.find(key);
    int v;
    if (it != ctx->hv_choice.end()) {
        v = it->second;
    } else if (s.Dpad() < kTuneMinElems) {
        // small sector: timing the variants would cost more than it saves.
        // k_hv_row against the best other shape, us: FP32 (k_hv_async<2, 256>)
        // 8.3 : 8.3 at 15,876 elements, 10.3 : 8.3 at 63,504, 22.9 : 14.5 at
        // 213,444; FP64 (k_hv_sorted<256>) 12.4 : 8.3 at 63,504, 34.9 : 24.8 at
        // 213,444; at 4,900 both are the launch.
        const bool tiny = s.D() < (1 << 15);
        v = kind == HV_F32 ? (tiny ? kRowVarF32 : kSmallVarF32) : (tiny ? kRowVarF64 : kSmallVarF64);
        ctx->hv_choice[key] = v;
        ctx->hv_times[key].assign(nvariants(kind), -1.0f);
    } else {
        if (int rc = tune(ctx, s, kind, &v)) return rc;
        ctx->hv_choice[key] = v;
    }
    if (int rc = prepare_variant(ctx, s, kind, v)) return rc;
    if (v_out) *v_out = v;
    if (R_out) *R_out = variant(kind, v).key();
    return MO_ED_OK;
}

int hv_tuning(mo_ed_ctx *ctx, const Sector &s, int kind, int cap, int *nvar, int *shape, float *ms, int *chosen)
{
    int v;
    if (int rc = hv_prepare(ctx, s, kind, &v, nullptr)) return rc;
    const std::vector<float> &t = ctx->hv_times[shape_key(kind, s)];
    *nvar = nvariants(kind);
    *chosen = v;
    for (int i = 0; i < *nvar && i < cap; ++i) {
        const HvVariant &h = variant(kind, i);
        if (shape) {
            shape[4 * i] = h.R;
            shape[4 * i + 1] = h.NT;
            shape[4 * i + 2] = h.MINB;
            shape[4 * i + 3] = h.staged;
        }
        if (ms) ms[i] = i < (int)t.size() ? t[i] : -1.0f;
    }
    return MO_ED_OK;
}

int hv_prepare_rows(mo_ed_ctx *ctx, const Sector &s, int kind, int v)
{
    return prepare_variant(ctx, s, kind, v);
}

int hv_lookup(mo_ed_ctx *ctx, const Sector &s, int kind, int *v_out, int *R_out)
{
    auto it = ctx->hv_choice.find(shape_key(kind, s));
    if (it == ctx->hv_choice.end())
        return fail(ctx, MO_ED_ERR_STATE, "H*v tile shape of this sector not chosen yet");
    const HvVariant &h = variant(kind, it->second);
    const int R = h.key();
    bool ready = s.dn->items.count(R) != 0;
    if (h.sorted)
        ready = ready && s.up->srt_ent != nullptr;
    else if (h.wide)
        ready = ready && s.up->wide_ent != nullptr;
    else if (h.staged)
        ready = ready && s.up->sched_rf.count(R) && s.dn->desc.count(R * 2 + (kind == HV_F32 ? 0 : 1));
    if (h.staged == 2 || h.staged == 3)
        ready = ready && s.dn->dblk_ptr != nullptr && s.dn->dblk_chunks.count(s.ld());
    if (!ready) return fail(ctx, MO_ED_ERR_STATE, "H*v item table of this sector not built yet");
    if (v_out) *v_out = it->second;
    if (R_out) *R_out = R;
    return MO_ED_OK;
}

int hv_set_variant(mo_ed_ctx *ctx, const Sector &s, int kind, int v)
{
    if (v < 0 || v >= nvariants(kind)) return fail(ctx, MO_ED_ERR_ARG, "H*v variant out of range");
    if (int rc = prepare_variant(ctx, s, kind, v)) return rc;
    ctx->hv_choice[shape_key(kind, s)] = v;
    return MO_ED_OK;
}

int hv_single(mo_ed_ctx *ctx, const Sector &s, int kind, const void *x, void *y)
{
    int v;
    if (int rc = hv_prepare(ctx, s, kind, &v, nullptr)) return rc;
    return launch_one(ctx, s, kind, v, x, y);
}

template <typename TA>
static int multi_jobs(mo_ed_ctx *ctx, const Sector &s, int kind, int v, int n, const void *const *x, void *const *y)
{
    std::vector<HvJobT<TA>> jobs(n);
    for (int i = 0; i < n; ++i) hv_fill_job<TA>(ctx, s, variant(kind, v).key(), x[i], y[i], jobs[i]);
    return hv_run_jobs<TA>(ctx, kind, v, jobs.data(), n);
}

int hv_multi(mo_ed_ctx *ctx, const Sector &s, int kind, int n, const void *const *x, void *const *y)
{
    int v;
    if (int rc = hv_prepare(ctx, s, kind, &v, nullptr)) return rc;
    return kind == HV_F32 ? multi_jobs<float>(ctx, s, kind, v, n, x, y) : multi_jobs<double>(ctx, s, kind, v, n, x, y);
}

int hv_dot_parts(mo_ed_ctx *ctx, const Sector &s, int kind, int *nparts)
{
    int v, R;
    if (int rc = hv_prepare(ctx, s, kind, &v, &R)) return rc;
    *nparts = s.dn->nitems.at(R);
    return MO_ED_OK;
}

// The tables of a sector whose H*v is k_hv_row (*row), for kernels that apply
// H to their own vectors.
template <typename TA>
int hv_row_job(mo_ed_ctx *ctx, const Sector &s, int kind, HvJobT<TA> *job, bool *row)
{
    int v;
    if (int rc = hv_prepare(ctx, s, kind, &v, nullptr)) return rc;
    *row = v == (kind == HV_F32 ? kRowVarF32 : kRowVarF64);
    if (*row) hv_fill_job<TA>(ctx, s, variant(kind, v).key(), nullptr, nullptr, *job);
    return MO_ED_OK;
}
template int hv_row_job<float>(mo_ed_ctx *, const Sector &, int, HvJobT<float> *, bool *);
template int hv_row_job<double>(mo_ed_ctx *, const Sector &, int, HvJobT<double> *, bool *);

int hv_single_dot(mo_ed_ctx *ctx, const Sector &s, int kind, const void *x, void *y, double *dot)
{
    int v;
    if (int rc = hv_prepare(ctx, s, kind, &v, nullptr)) return rc;
    if (kind == HV_F32) {
        HvJobT<float> j;
        hv_fill_job<float>(ctx, s, variant(kind, v).key(), x, y, j);
        j.dot_partial = dot;
        return hv_launch_f32(ctx, v, &j, 1);
    }
    HvJobT<double> j;
    hv_fill_job<double>(ctx, s, variant(kind, v).key(), x, y, j);
    j.dot_partial = dot;
    return hv_launch_f64(ctx, kind, v, &j, 1);
}

}  // namespace moed
