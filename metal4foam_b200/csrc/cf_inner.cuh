// cf_inner.cuh -- what the kernels that run a whole inner solve share
// (cf_clupcg.cu, cf_resident.cu, cf_clubicg.cu, cf_resbicg.cu): the solver state
// every CTA keeps, and a row of A x with its entries in registers.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include "cf_internal.cuh"
#include "cf_kernels.cuh"

namespace cf {

// k_inner_setup's state
__device__ __forceinline__ void inner_state_init(InnerState& S, double target, int maxIter, int ips,
                                                 int stagLimit)
{
    S.stagLimit = stagLimit > 0 ? stagLimit : STAG_LIMIT;
    S.wArA = S.wArAold = S.wApA = S.alpha = S.beta = S.res = 0.0;
    S.rA0rA = S.rA0rAold = S.rA0AyA = S.omega = S.tAtA = S.tAsA = S.resS = 0.0;
    S.bestRes = 1.0e300;
    S.target = target;
    S.finalResSum = 0.0;
    S.it = 0;
    S.maxIter = maxIter;
    S.ips = ips < 1 ? 1 : ips;
    S.lastSync = 0;
    S.noProgress = 0;
    S.cur = S.best = 0;
    S.nxt = 1;
    S.converged = S.singular = S.stagnated = S.done = S.early = 0;
    S.sel = 0;
    S.ticket = 0u;
    S.waitErr = 0;
}

// The bookkeeping of k_pcg_update (for every iteration but the first) and of
// the last Chebyshev step, once {sum|r| of the last update, z.r} are known.
// One thread does it; the others form beta themselves and learn of the end
// of the solve at the next reduction.
__device__ __forceinline__ void inner_after_apply(InnerState& S, bool first, double res,
                                                  double wArA)
{
    if (!first)
    {
        S.res = res;
        S.cur = S.nxt;
        S.it = S.it + 1;
        inner_sync_point(&S, true);
    }
    if (!S.done)
    {
        S.wArAold = S.wArA;
        S.wArA = wArA;
    }
}

// k_inner_final's choice; `store`: the state goes back to global memory,
// without its error word, which another CTA may set at any time.
__device__ __forceinline__ void inner_finish(InnerState& S, InnerState* st, bool store)
{
    if (S.early)   // BiCGStab's |s| exit returns its last iterate
    {
        S.sel = S.cur;
    }
    else if (S.bestRes < S.finalResSum)
    {
        S.sel = S.best;
        S.finalResSum = S.bestRes;
    }
    else
    {
        S.sel = S.cur;
    }
    if (store)
    {
        InnerState t = S;
        t.cur = t.best = t.sel;   // (a later choice between them changes nothing)
        memcpy((void*)st, (const void*)&t, offsetof(InnerState, waitErr));
    }
}

template <int W>
__device__ __forceinline__ float row_apply(const unsigned int (&ix)[(W + 1) / 2],
                                           const float (&v)[W], const float* x, float acc)
{
    float t[W];
#pragma unroll
    for (int k = 0; k < W; ++k)
        t[k] = x[(k & 1) ? (ix[k >> 1] >> 16) : (ix[k >> 1] & 0xffffu)];
#pragma unroll
    for (int k = 0; k < W; ++k) acc = __fadd_rn(acc, __fmul_rn(v[k], t[k]));
    return acc;
}

// entries of local row l (paired order), base = (rowBase + slice start) W
template <int W>
__device__ __forceinline__ void row_index(const unsigned short* idx, long long sb, int lane,
                                          unsigned int (&ix)[(W + 1) / 2])
{
#pragma unroll
    for (int g = 0; g < W / 2; ++g)
        ix[g] = *reinterpret_cast<const unsigned int*>(idx + sb + 64 * g + 2 * lane);
    if constexpr (W & 1) ix[W / 2] = idx[sb + 32 * (W - 1) + lane];
}

}  // namespace cf
