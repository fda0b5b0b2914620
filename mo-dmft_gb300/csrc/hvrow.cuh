// hvrow.cuh -- one element of H*v from the species tables, every operand read
// where it lies: the body of k_hv_row (hv.cu) and of the small sectors'
// Lanczos kernels (eigs.cu).
#pragma once

#include "internal.h"

namespace moed {

__device__ __forceinline__ HopEnt<float> ldg_ent(const HopEnt<float> *p)
{
    const int2 v = __ldg((const int2 *)p);
    HopEnt<float> e;
    e.t = v.x;
    e.v = __int_as_float(v.y);
    return e;
}
__device__ __forceinline__ HopEnt<double> ldg_ent(const HopEnt<double> *p)
{
    const int4 v = __ldg((const int4 *)p);
    HopEnt<double> e;
    e.t = v.x;
    e.v = __hiloint2double(v.w, v.z);
    return e;
}

// (H x)(d, u) without the diagonal term.  NC: x is constant for the launch
// (read through the non-coherent path); otherwise plain loads (x may be in
// shared memory).  inf, dinf: up_info[u], dn_info[d]; pmask, t4: the model's
// tables in shared memory.
template <typename TX, typename TA, bool NC>
__device__ __forceinline__ TA hv_moves(const HvJobT<TA> &jb, const ModelDev *__restrict__ mdl, const TX *x, int d, int u,
                                       int inf, int dinf, const unsigned *pmask, const int *t4, int nimp, TA Jc, TA acc)
{
    const auto ld_x = [](const TX *p) { return NC ? __ldg(p) : *p; };
    const int ld = jb.ld, iu = (inf >> 8) & 0xff, cnt = inf & 0xff, id = (dinf >> 8) & 0xff, dcnt = dinf & 0xff;
    const TX *xd = x + (size_t)d * ld;
    // up-spin moves of the column, 4 at a time
    const HopEnt<TA> *tab = jb.up_tab + (size_t)(u >> 2) * jb.up_hw * 4 + (u & 3);
    for (int s0 = 0; s0 < cnt; s0 += 4) {
        HopEnt<TA> e[4];
        TX g[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) e[t] = ldg_ent(tab + 4 * min(s0 + t, cnt - 1));
#pragma unroll
        for (int t = 0; t < 4; ++t) g[t] = ld_x(xd + e[t].t);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (s0 + t < cnt) acc += e[t].v * (TA)g[t];
    }
    // down-spin moves of the row
    for (int s0 = 0; s0 < dcnt; s0 += 4) {
        TA v[4];
        TX g[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int s = min(s0 + t, dcnt - 1);
            v[t] = __ldg(jb.dn_val + (size_t)s * jb.nd + d);
            g[t] = ld_x(x + (size_t)__ldg(jb.dn_tgt + (size_t)s * jb.nd + d) * ld + u);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (s0 + t < dcnt) acc += v[t] * (TA)g[t];
    }
    // spin-flip and pair hopping
    unsigned pm = pmask[iu];
    while (pm) {
        const int p = __ffs(pm) - 1;
        pm &= pm - 1;
        const int e = t4[p * nimp + iu];
        const TX *xu = x + u + (int)(short)(e & 0xffff);
        const TA c = (e & 0x40000000) ? -Jc : Jc;
        const int esf = t4[__ldg(mdl->pair_rev + p) * nimp + id];   // spin-flip: T_{j<-i}(d)
        const int eph = t4[p * nimp + id];                          // pair hop:  T_{i<-j}(d)
        if (esf < 0) {
            const TX g = ld_x(xu + (long long)(d + (int)(short)(esf & 0xffff)) * ld);
            acc += ((esf & 0x40000000) ? -c : c) * (TA)g;
        }
        if (eph < 0) {
            const TX g = ld_x(xu + (long long)(d + (int)(short)(eph & 0xffff)) * ld);
            acc += ((eph & 0x40000000) ? -c : c) * (TA)g;
        }
    }
    return acc;
}

}  // namespace moed
