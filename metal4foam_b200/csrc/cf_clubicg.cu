// cf_clubicg.cu -- the inner BiCGStab of a small mesh inside ONE thread-block
// cluster of up to 16 CTAs.
//
// The graph loop's three launches per iteration cost 7-8 us each on small
// meshes (23 us per iteration at 12K cells): every gathered entry waits for
// four vectors and every launch ends in a grid-wide sum.  Here the vectors and
// matrix rows stay in registers, y and z are formed once and gathered from
// shared memory, boundary rows are pushed into the reader's shared memory as
// {value, epoch} words (cf_cluster_ll.cuh), and there are two such exchanges
// and three reductions per iteration, none with a cluster barrier.
//
// Measured on one box, us per inner iteration, graph loop / this kernel: 240
// cells 2-D 19.8 / 2.9, 1,000 3-D 23.0 / 3.4, 12K 3-D 21.9 / 7.2, 22K 3-D 23.2 /
// 13.1, 36K 2-D 23.3 / 16.6, 39K 3-D 23.6 / 21.4 (10 rows per thread: no room
// in the registers for more).
//
// BiCGStab amplifies the last bit of its scalars, so the FP64 sums fold in
// the graph loop's order: its kernels run one row per thread on ceil(n / 256)
// blocks at these sizes; a CTA owns whole 256-row blocks, thread t of it the
// rows t of each, the block sums and the sum over the blocks are block_sum's
// trees, and the results are the graph loop's bit for bit.
#include "cudafoam.h"
#include "cf_cluster_ll.cuh"
#include "cf_host.hpp"
#include "cf_inner.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <string>
#include <vector>

using namespace cf;
namespace cg = cooperative_groups;

#define CLB_CUDA(call)                                                          \
    do                                                                          \
    {                                                                           \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess)                                                  \
            return fail(CF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace cf {

namespace {

constexpr int CLB_MAX_R = 10;                              // 256-row blocks of a CTA at most
constexpr int CLB_BLOCKS = CLU_MAX_CTAS * CLB_MAX_R;       // of the mesh
constexpr int CLB_FIRST_ROWS = 32768;                      // for a first solve
constexpr int CLB_FIRST_HALO = 2560;
// reduction values: rA0.AyA | sum|s|, s.t, t.t | sum|r|, rA0.r
constexpr int CLB_VALUES = 6;

struct CluBicgArgs
{
    CluSplit split;
    InnerRun run;
    int blocks;     // 256-row blocks of the mesh
    int perCta;     // of a CTA
};

struct ClbShared
{
    double ws[3][CLB_MAX_R][NT / 32];
    double fs[3][NT / 32];
    u64 words[CLB_VALUES][CLB_BLOCKS][2];
    int stop, bad;
    InnerState S;
};

// block_sum's fold of eight warp sums (the lanes past them add zeros)
__device__ __forceinline__ double fold8(const double* w)
{
    return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// The block sums of v[r][i] (row i of every thread: one 256-row block) to
// every CTA, as words of value v0 + r.
template <int NR, int R>
__device__ __forceinline__ void clb_send(double (&v)[NR][R], int v0, const CluBicgArgs& a, int rank,
                                         int ctas, unsigned int epoch, ClbShared& sh)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int wid = tid >> 5;
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const double t = warp_sum(v[r][i]);
            if (lane == 0) sh.ws[r][i][wid] = t;
        }
    __syncthreads();
    for (int k = tid; k < NR * R * ctas; k += NT)
    {
        const int to = k % ctas;
        const int q = k / ctas;
        const int r = q / R;
        const int i = q - r * R;
        const int blk = rank * a.perCta + i;
        if (i >= a.perCta || blk >= a.blocks) continue;
        const u64 b = (u64)__double_as_longlong(fold8(sh.ws[r][i]));
        const unsigned int at = remote_addr(smem_addr(&sh.words[v0 + r][blk][0]), to);
        st_remote(at, (unsigned int)b, epoch);
        st_remote(at + 8, (unsigned int)(b >> 32), epoch);
    }
}

// Warp r gathers value v0 + r; the totals are fold8(sh.fs[r]) after the next
// barrier (one block per thread of the last block's fold: at most 256 blocks).
template <int NR>
__device__ __forceinline__ void clb_recv(int v0, const CluBicgArgs& a, unsigned int epoch,
                                         ClbShared& sh, long long polls)
{
    const int lane = threadIdx.x & 31;
    const int r = threadIdx.x >> 5;
    if (r >= NR) return;
    for (int k = 0; k < (a.blocks + 31) / 32; ++k)
    {
        double t = 0.0;
        if (32 * k + lane < a.blocks)
        {
            const unsigned int at = smem_addr(&sh.words[v0 + r][32 * k + lane][0]);
            const u64 lo = wait_local(at, epoch, &sh.bad, polls);
            const u64 hi = wait_local(at + 8, epoch, &sh.bad, polls);
            t = __longlong_as_double((long long)((hi << 32) | lo));
        }
        t = warp_sum(t);
        if (lane == 0) sh.fs[r][k] = t;
    }
}

template <int W, int R>
__global__ void __launch_bounds__(NT, 1) k_clu_bicg(const __grid_constant__ CluBicgArgs a)
{
    extern __shared__ float zmem[];
    __shared__ ClbShared sh;
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x;
    const int ctas = (int)cl.num_blocks();
    const int rank = (int)cl.block_rank();
    const InnerRun& N = a.run;
    const CluSplit& C = a.split;
    const ResPart P = C.parts[rank];
    const int locP = C.locP;
    const int zs = locP + 2 * C.halo + 2;
    float* yb = zmem;
    float* zb = zmem + zs;
    const double mean = N.mean ? *N.mean : 0.0;
    if (tid == 0)
    {
        inner_state_init(sh.S, N.target, N.maxIter, N.ips, N.stagLimit);
        sh.stop = sh.bad = 0;
    }
    for (int i = tid; i < CLB_VALUES * CLB_BLOCKS * 2; i += NT) (&sh.words[0][0][0])[i] = 0;
    if (tid < 3 * (NT / 32)) (&sh.fs[0][0])[tid] = 0.0;
    for (int i = P.nloc + tid; i < zs; i += NT) yb[i] = zb[i] = 0.0f;
    unsigned int ix[R][(W + 1) / 2];
    unsigned int dst[R][2];
    float v[R][W], dg[R], rd[R], r[R], r0[R], p[R], A[R], d[R];
    unsigned int ep = 1;
#pragma unroll
    for (int i = 0; i < R; ++i)
    {
        const int l = tid + i * NT;
        dg[i] = rd[i] = r[i] = r0[i] = p[i] = A[i] = d[i] = 0.0f;
        dst[i][0] = dst[i][1] = CLU_NONE;
#pragma unroll
        for (int k = 0; k < (W + 1) / 2; ++k) ix[i][k] = (unsigned)(zs - 2) * 0x10001u;
#pragma unroll
        for (int k = 0; k < W; ++k) v[i][k] = 0.0f;
        if (l >= P.nloc) continue;
        const int g = P.rowBase + l;
        const long long sb = ((long long)P.rowBase + (l & ~31)) * W;
        row_index<W>(C.idx, sb, l & 31, ix[i]);
#pragma unroll
        for (int k = 0; k < W; ++k)
        {
            const int e = C.emap[pair_index(sb, W, k, l & 31)];
            v[i][k] = e >= 0 ? N.val32[e] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (q < C.ndest) dst[i][q] = C.dest[(size_t)q * C.rowsP + g];
        dg[i] = N.diag32[g];
        rd[i] = N.rD32[g];
        r[i] = r0[i] = (float)(N.r64[g] - mean);
    }
    auto push = [&](int i, unsigned int buf, float x) {
        if (dst[i][0] == CLU_NONE) return;
        st_remote(remote_addr(buf + 8 * (dst[i][0] & 0xffffu), dst[i][0] >> 16),
                  __float_as_uint(x), ep);
        if (dst[i][1] == CLU_NONE) return;
        st_remote(remote_addr(buf + 8 * (dst[i][1] & 0xffffu), dst[i][1] >> 16),
                  __float_as_uint(x), ep);
        for (int q = 2; q < C.ndest; ++q)
        {
            const unsigned int t =
                __ldg(C.dest + (size_t)q * C.rowsP + P.rowBase + tid + i * NT);
            if (t == CLU_NONE) break;
            st_remote(remote_addr(buf + 8 * (t & 0xffffu), t >> 16), __float_as_uint(x), ep);
        }
    };
    auto halo_wait = [&](const float* x) {
        const unsigned int at = smem_addr(x + locP);
        for (int h = tid; h < P.nh; h += NT) wait_local(at + 8 * h, ep, &sh.bad, N.polls);
    };
    cl.sync();
    double rA0rA;
    {
        double acc[1][R];
#pragma unroll
        for (int i = 0; i < R; ++i) acc[0][i] = (double)r[i] * (double)r[i];
        clb_send<1, R>(acc, 5, a, rank, ctas, ep, sh);
        clb_recv<1>(5, a, ep, sh, N.polls);
        __syncthreads();
        rA0rA = fold8(sh.fs[0]);
    }
    double beta = 0.0, omega = 0.0, res = 0.0;
    bool first = true;
    for (;;)
    {
        ++ep;
        const float bf = (float)beta;
        const float of = (float)omega;
        // p, y = rD p (k_bicg_ab forms them at every gathered column)
        {
            const unsigned int buf = smem_addr(yb + locP);
#pragma unroll
            for (int i = 0; i < R; ++i)
            {
                p[i] = __fadd_rn(r[i], __fmul_rn(bf, __fsub_rn(p[i], __fmul_rn(of, A[i]))));
                const float y = __fmul_rn(rd[i], p[i]);
                push(i, buf, y);
                if (tid + i * NT < P.nloc) yb[tid + i * NT] = y;
            }
        }
        halo_wait(yb);
        __syncthreads();
        {
            double acc[1][R];
#pragma unroll
            for (int i = 0; i < R; ++i)
            {
                const float y = yb[min(tid + i * NT, zs - 2)];
                A[i] = row_apply<W>(ix[i], v[i], yb, __fmul_rn(dg[i], y));
                acc[0][i] = (double)r0[i] * (double)A[i];
            }
            clb_send<1, R>(acc, 0, a, rank, ctas, ep, sh);
        }
        // the checks of the iteration before, while the sum is on its way
        if (tid == NT - 1)
        {
            InnerState& S = sh.S;
            if (!first)
            {
                S.res = res;
                S.omega = omega;
                S.cur = S.nxt;
                S.it = S.it + 1;
                inner_sync_point(&S, false);
            }
            sh.stop = S.done || sh.bad;
        }
        clb_recv<1>(0, a, ep, sh, N.polls);
        __syncthreads();
        first = false;
        if (sh.stop) break;
        const double alpha = rA0rA / fold8(sh.fs[0]);
        const float af = (float)alpha;
        ++ep;
        double acc3[3][R];
        {
            const unsigned int buf = smem_addr(zb + locP);
#pragma unroll
            for (int i = 0; i < R; ++i)
            {
                r[i] = __fsub_rn(r[i], __fmul_rn(af, A[i]));   // s
                const float z = __fmul_rn(rd[i], r[i]);
                push(i, buf, z);
                if (tid + i * NT < P.nloc) zb[tid + i * NT] = z;
                acc3[0][i] = (double)fabsf(r[i]);
            }
        }
        halo_wait(zb);
        __syncthreads();
        float t[R];
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const float z = zb[min(tid + i * NT, zs - 2)];
            t[i] = row_apply<W>(ix[i], v[i], zb, __fmul_rn(dg[i], z));
            acc3[1][i] = (double)r[i] * (double)t[i];
            acc3[2][i] = (double)t[i] * (double)t[i];
        }
        clb_send<3, R>(acc3, 1, a, rank, ctas, ep, sh);
        clb_recv<3>(1, a, ep, sh, N.polls);
        __syncthreads();
        const double resS = fold8(sh.fs[0]);
        // k_bicg_cd's checks: breakdown, the |s| exit, and only then omega
        const bool broken = !isfinite(rA0rA) || !isfinite(alpha) || !isfinite(resS);
        const bool early = !broken && resS <= N.target;
        omega = fold8(sh.fs[1]) / fold8(sh.fs[2]);
        float* dn = N.D + (size_t)sh.S.nxt * N.dStride + P.rowBase;
        if (broken || early)
        {
            if (early)
            {
#pragma unroll
                for (int i = 0; i < R; ++i)
                {
                    const int l = tid + i * NT;
                    if (l < P.nloc) dn[l] = __fadd_rn(d[i], __fmul_rn(af, yb[l]));
                }
            }
            __syncthreads();
            if (tid == NT - 1)
            {
                InnerState& S = sh.S;
                S.resS = resS;
                S.done = 1;
                if (broken)
                {
                    S.singular = 1;
                }
                else
                {
                    S.early = 1;
                    S.cur = S.nxt;
                    S.it = S.it + 1;
                    S.finalResSum = resS;
                    S.converged = 1;
                }
            }
            break;
        }
        const float wf = (float)omega;
        ++ep;
        double acc2[2][R];
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const int l = min(tid + i * NT, zs - 2);
            d[i] = __fadd_rn(d[i], __fadd_rn(__fmul_rn(af, yb[l]), __fmul_rn(wf, zb[l])));
            if (l < P.nloc) dn[l] = d[i];
            r[i] = __fsub_rn(r[i], __fmul_rn(wf, t[i]));
            acc2[0][i] = (double)fabsf(r[i]);
            acc2[1][i] = (double)r0[i] * (double)r[i];
        }
        clb_send<2, R>(acc2, 4, a, rank, ctas, ep, sh);
        clb_recv<2>(4, a, ep, sh, N.polls);
        __syncthreads();
        res = fold8(sh.fs[0]);
        const double next = fold8(sh.fs[1]);
        beta = (next / rA0rA) * (alpha / omega);
        rA0rA = next;
    }
    __syncthreads();
    if (tid == NT - 1)
    {
        if (sh.bad) atomicExch(&N.st->waitErr, 1);
        inner_finish(sh.S, N.st, rank == 0);
    }
    // (before the first update no correction has been written: 0)
    if (sh.S.it == 0)
    {
        for (int l = tid; l < P.nloc; l += NT) N.D[P.rowBase + l] = 0.0f;
    }
    cl.sync();   // no CTA leaves while another may still store into it
}

template <int W>
const void* kernel_r(int R)
{
    switch (R)
    {
        case 1: return (const void*)k_clu_bicg<W, 1>;
        case 2: return (const void*)k_clu_bicg<W, 2>;
        case 3: return (const void*)k_clu_bicg<W, 3>;
        case 4: return (const void*)k_clu_bicg<W, 4>;
        case 6: return (const void*)k_clu_bicg<W, 6>;
        case 8: return (const void*)k_clu_bicg<W, 8>;
        case 10: return (const void*)k_clu_bicg<W, 10>;
    }
    return nullptr;
}

const void* kernel_of(int W, int R)
{
    return W == 4 ? kernel_r<4>(R) : W == 5 ? kernel_r<5>(R) : kernel_r<6>(R);
}

int per_cta(int n)
{
    const int blocks = (n + NT - 1) / NT;
    return (blocks + CLU_MAX_CTAS - 1) / CLU_MAX_CTAS;
}

}  // namespace

void clu_bicg_release(cf_context* c)
{
    if (!c->cluBicgShared) clu_plan_free(static_cast<CluPlan*>(c->cluBicg));
    c->cluBicg = nullptr;
    c->cluBicgTried = c->cluBicgShared = false;
}

void clu_bicg_prepare(cf_context* c, bool first)
{
    if (c->cluBicgTried) return;
    // A mesh of more than 32,768 cells, or one numbered so that the blocks read
    // most of the others, gains little next to the 2 to 3 ms that its split takes
    // the host (39K cells in natural order, first solve: 5.1 ms without, 6.8
    // with; 22K scattered 4.9 and 7, 12K 4.4 and 4.4).  Others gain more at once
    // than it takes (12K in natural order 4.0 and 2.2, 22K 5.0 and 3.3).
    if (first && c->n > CLB_FIRST_ROWS) return;
    c->cluBicgTried = true;
    if (c->hostSliceOff.empty() || c->maxRowLen > 6 || c->n > NT * CLB_BLOCKS) return;
    // the graph loop's kernels run one row per thread on these blocks
    const int need = (c->n + NT - 1) / NT;
    const DevSell S = sell_of(c);
    const void* fns[] = {(const void*)k_bicg_init, (const void*)bicg_ab_kernel(S),
                         (const void*)bicg_cd_kernel(S), (const void*)k_bicg_e};
    for (const void* f : fns)
        if (grid_for(c, f, c->n) != need) return;
    const int per = per_cta(c->n);
    int rows = 1;
    for (int R : {1, 2, 3, 4, 6, 8, 10})
    {
        rows = R;
        if (per <= R) break;
    }
    CluPlan* p = nullptr;
    ResHost H;
    try
    {
        const LentLayout lent(c);
        if (!res_blocks(c->n, lent.L, per * NT, H, 4,
                        first ? CLB_FIRST_HALO : CLU_MAX_HALO))
        {
            c->cluBicgTried = !first;
            return;
        }
    }
    catch (...)
    {
        return;   // no memory for the split
    }
    if (clu_plan_upload(H, (int)H.parts.size(), 2, 0, 0, 0, kernel_of(H.W, rows), rows, NT,
                        c->stream, &p) != CF_OK)
        cudaGetLastError();
    c->cluBicg = p;
}

int clu_bicg_inner(cf_context* c, double target, int maxIter, int ips, int stagLimit, bool* ran)
{
    *ran = false;
    if (maxIter <= 0) return CF_OK;
    clu_bicg_prepare(c, c->bicgSolves == 0);
    const CluPlan* p = static_cast<const CluPlan*>(c->cluBicg);
    if (!p) return CF_OK;
    cudaStream_t s = c->stream;
    CluBicgArgs a;
    a.split = p->split;
    a.run = inner_run(c, nullptr, target, maxIter, ips, 1, stagLimit);
    a.blocks = (c->n + NT - 1) / NT;
    a.perCta = per_cta(c->n);
    void* args[] = {(void*)&a};
    const int rc = clu_launch_fn(p->fn, p->split.ctas, p->threads, p->smem, args, 1, s);
    if (rc != CF_OK) return rc;
    c->launches++;
    CLB_CUDA(cudaEventRecord(c->ev1, s));
    CLB_CUDA(cudaMemcpyAsync(c->h_st, c->d_st, sizeof(InnerState), cudaMemcpyDeviceToHost, s));
    CLB_CUDA(cudaStreamSynchronize(s));
    if (c->h_st->waitErr)
    {
        // a wait gave up: this solve goes through the graph path
        CLB_CUDA(cudaMemsetAsync(&c->d_st->waitErr, 0, sizeof(int), s));
        c->backoff.gaveUp();
        return CF_OK;
    }
    c->backoff.worked();
    *ran = true;
    return CF_OK;
}

}  // namespace cf
