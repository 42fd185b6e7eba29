// cf_resbicg.cu -- the inner BiCGStab of one system as ONE cooperative launch
// with one CTA per SM.
//
// The graph loop gathers four vectors (rA, p, AyA, rD) for every matrix entry
// of the first SpMV and three for the second, and reads the matrix twice per
// iteration from L2 or HBM: 31 us per iteration at 64^3, 46 at 96^3.  Here
// the matrix sits in shared memory and r, r0, p, AyA and t of a row in
// registers; y and z are formed once per iteration, stored, and gathered after
// a grid barrier (a flag per CTA).
//
// BiCGStab amplifies the last bit of its scalars, so the FP64 sums fold in
// the graph loop's order.  Its kernels run on G = SMs x m blocks (m = 8, 6 or
// 5 by their registers), block b taking the 256-row groups b, b + G, ...;
// here CTA c takes the groups c, c + SMs, c + 2 SMs, ..., which holds whole
// blocks for every m: thread t of it adds row t of the groups of one block in
// that block's order, the block sums are block_sum's trees, and one CTA per
// value folds them as the last block of grid_sum does.  Every result is the
// graph loop's bit for bit.
//
// Per iteration (graph loop, here): 36^3 21.6, 11.9 us; 64^3 30.7, 16.3;
// 96^3 47.5, 26.1.  What is left is latency: two grid barriers and three
// folds, about 1.2 and 2.7 us each, and at 96^3 the gathers of y and z from L2
// and the correction's round trip.  The block sums sit densely: 128 bytes
// apart they cost the folding CTA more lines (96^3 27.8 us).
//
// Every wait is bounded; one that gives up sets waitErr and the solve runs
// through the graph loop.
#include "cudafoam.h"
#include "cf_host.hpp"
#include "cf_inner.cuh"
#include "cf_resident.cuh"

#include <algorithm>
#include <condition_variable>
#include <mutex>
#include <new>
#include <string>

using namespace cf;

#define RSB_CUDA(call)                                                          \
    do                                                                          \
    {                                                                           \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess)                                                  \
            return fail(CF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace cf {

namespace {

typedef unsigned long long u64;

constexpr int RSB_MAX_R = 24;        // 256-row groups per CTA at most
constexpr int RSB_MAX_CTAS = 256;
constexpr int RSB_ABOVE = NT * 160;  // rows that fit one cluster (cf_clubicg.cu)
constexpr int RSB_COPIES = 8;        // copies of words every CTA polls
// A flag has a 128-byte line of its own (in lines of 8 or 32 flags, whose
// writers and pollers meet in L2, a barrier takes 3 to 7 us instead of about
// 1: 64^3 19.9 and 17.4 us per iteration, 16.3 so), in two copies: one and
// eight are 0 to 4 % slower.
constexpr int RSB_FLAG_STRIDE = 32;   // 4-byte words between flags
constexpr int RSB_FLAG_COPIES = 2;
constexpr int RSB_TOT_STRIDE = 16;    // 8-byte words between totals
constexpr int RSB_MAX_BLOCKS = 8 * RSB_MAX_CTAS;
// reduction values: rA0.AyA | sum|s|, s.t, t.t | sum|r|, rA0.r
constexpr int RSB_VALUES = 6;

// blocks per SM of the graph loop's kernels (their registers), by slice width
__host__ __device__ constexpr int rsb_ab(int W) { return W == 4 ? 8 : 6; }
__host__ __device__ constexpr int rsb_cd(int W) { return W == 4 ? 5 : 6; }
constexpr int RSB_MAX_K = 3;         // systems on one matrix that a launch can carry
constexpr int RSB_E = 8;             // k_bicg_e and k_bicg_init

// one system of a launch
struct ResBicgSystem
{
    InnerRun run;
    float* y;
    float* z;
};

struct ResBicgArgs
{
    DevSell A;
    ResBicgSystem sys[RSB_MAX_K];
    int count;              // systems of this launch
    u64* part;              // [RSB_MAX_K][values][RSB_MAX_BLOCKS][2 words]
    u64* tot;               // [copies][RSB_MAX_K][values], RSB_TOT_STRIDE apart
    unsigned int* flags;    // [copies][RSB_MAX_CTAS], RSB_FLAG_STRIDE apart
    unsigned int* epoch;    // last epoch used by the launches before
    int groups;             // 256-row groups of the mesh
};

template <int K>
struct RsbShared
{
    double ws[K][3][8][NT / 32];
    double fs[NT / 32];
    double tot[K][3];
    int stop[K];
    int bad;
    InnerState S[K];
};

__device__ __forceinline__ void ld2(const u64* p, u64& x, u64& y)
{
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p));
}

__device__ __forceinline__ void st_dbl(u64* p, double x, unsigned int epoch)
{
    const u64 b = (u64)__double_as_longlong(x);
    const u64 lo = ((u64)epoch << 32) | (b & 0xffffffffu);
    const u64 hi = ((u64)epoch << 32) | (b >> 32);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi));
}

// whether a bounded wait goes on
__device__ __forceinline__ bool rsb_more(long long& spins, int* bad, InnerState* st,
                                         long long polls)
{
    if ((++spins & 1023) != 0 && spins <= polls) return true;
    if (*(volatile int*)bad) return false;
    if (spins > polls || *(volatile int*)&st->waitErr)
    {
        atomicExch(&st->waitErr, 1);
        *(volatile int*)bad = 1;
        return false;
    }
    return true;
}

__device__ __forceinline__ double rsb_wait(const u64* p, unsigned int epoch, int* bad,
                                           InnerState* st, long long polls)
{
    u64 lo, hi;
    long long spins = 0;
    ld2(p, lo, hi);
    while ((unsigned int)(lo >> 32) != epoch || (unsigned int)(hi >> 32) != epoch)
    {
        if (!rsb_more(spins, bad, st, polls)) return 0.0;
        ld2(p, lo, hi);
    }
    return __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffu)));
}

__device__ __forceinline__ double fold8(const double* w)
{
    return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// The butterfly sums of K values at once: at every step half of the lanes
// go on with one value of a pair and half with the other, so a value costs
// about one exchange instead of five.  A sum is the one warp_sum forms (its
// additions commute).  Lane l ends with the sum of value K_index(l).
template <int K, int O>
__device__ __forceinline__ void warp_sums(double (&v)[K])
{
    if constexpr (O > 0)
    {
        constexpr int H = (K + 1) / 2;
        const bool hi = (threadIdx.x & O) != 0;
        double w[H];
#pragma unroll
        for (int i = 0; i < H; ++i)
        {
            if (2 * i + 1 < K)
            {
                const double keep = hi ? v[2 * i + 1] : v[2 * i];
                const double send = hi ? v[2 * i] : v[2 * i + 1];
                w[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
            }
            else
            {
                w[i] = v[2 * i] + __shfl_xor_sync(0xffffffffu, v[2 * i], O);
            }
        }
        warp_sums<H, O / 2>(w);
        v[0] = w[0];
    }
}

__device__ __forceinline__ int warp_sums_index(int lane) { return (int)(__brev((unsigned)lane) >> 27); }

__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Everything stored before is visible to every CTA after.
__device__ __forceinline__ void rsb_barrier(const ResBicgArgs& a, unsigned int epoch, int* bad)
{
    const int tid = threadIdx.x;
    __syncthreads();
    if (tid < RSB_FLAG_COPIES)
    {
        fence_acq_rel();
        unsigned int* f = a.flags + (size_t)(tid * RSB_MAX_CTAS + blockIdx.x) * RSB_FLAG_STRIDE;
        asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(f), "r"(epoch));
    }
    if (tid < (int)gridDim.x)
    {
        const unsigned int* f =
            a.flags + (size_t)((blockIdx.x % RSB_FLAG_COPIES) * RSB_MAX_CTAS + tid) * RSB_FLAG_STRIDE;
        long long spins = 0;
        for (;;)
        {
            unsigned int v;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f));
            if (v == epoch || !rsb_more(spins, bad, a.sys[0].run.st, a.sys[0].run.polls))
                break;
        }
        fence_acq_rel();
    }
    __syncthreads();
}

// acc[r][x]: this thread's sum of value r of system k over the groups of its
// block x (block x SMs + CTA of the value's G blocks); the sums of its warp.
template <int K, int NR, int M>
__device__ __forceinline__ void rsb_warps(double (&acc)[NR][M], int k, RsbShared<K>& sh)
{
    const int lane = threadIdx.x & 31;
    double v[NR * M];
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int x = 0; x < M; ++x) v[r * M + x] = acc[r][x];
    warp_sums<NR * M, 16>(v);
    const int i = warp_sums_index(lane);
    if (i < NR * M) sh.ws[k][i / M][i % M][threadIdx.x >> 5] = v[0];
}

// The totals of values v0 .. v0 + NR of the systems in `act` over all blocks,
// in sh.tot after the call.
template <int K, int NR, int M>
__device__ __forceinline__ void rsb_reduce(const ResBicgArgs& a, int act, int v0, int G,
                                           unsigned int epoch, RsbShared<K>& sh, bool book,
                                           bool first, const double (&res)[K],
                                           const double (&omega)[K])
{
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int wid = tid >> 5;
    const int P = (int)gridDim.x;
    InnerState* st = a.sys[0].run.st;
    const long long polls = a.sys[0].run.polls;
    if (K == 1) act = 1;
    __syncthreads();
    if (tid < K * NR * M)
    {
        const int k = tid / (NR * M);
        const int r = tid / M - k * NR;
        const int x = tid % M;
        const int b = x * P + (int)blockIdx.x;
        if (b < G && (act >> k & 1))
            st_dbl(a.part + ((size_t)(k * RSB_VALUES + v0 + r) * RSB_MAX_BLOCKS + b) * 2,
                   fold8(sh.ws[k][r][x]), epoch);
    }
    // the checks of the iteration before, while the sums are on their way
    if (book)
    {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((act >> k & 1) && tid == NT - 1 - 32 * k)
            {
                InnerState& S = sh.S[k];
                if (!first)
                {
                    S.res = res[k];
                    S.omega = omega[k];
                    S.cur = S.nxt;
                    S.it = S.it + 1;
                    inner_sync_point(&S, false);
                }
                sh.stop[k] = S.done;
            }
    }
    // one of the last CTAs (they have the fewest rows) folds a value as
    // grid_sum's last block does
    const int mine = P - 1 - (int)blockIdx.x;
    if (mine < K * NR && (act >> (mine / NR) & 1))
    {
        const int v = (mine / NR) * RSB_VALUES + v0 + mine % NR;
        const u64* w = a.part + (size_t)v * RSB_MAX_BLOCKS * 2;
        double t = 0.0;
        for (int b = tid; b < G; b += NT) t += rsb_wait(w + (size_t)b * 2, epoch, &sh.bad, st, polls);
        t = warp_sum(t);
        if (lane == 0) sh.fs[wid] = t;
        __syncthreads();
        if (tid < RSB_COPIES)
            st_dbl(a.tot + ((size_t)tid * RSB_MAX_K * RSB_VALUES + v) * RSB_TOT_STRIDE,
                   fold8(sh.fs), epoch);
    }
    if (tid < K * NR && (act >> (tid / NR) & 1))
    {
        const int v = (tid / NR) * RSB_VALUES + v0 + tid % NR;
        sh.tot[tid / NR][tid % NR] =
            rsb_wait(a.tot + ((size_t)(blockIdx.x % RSB_COPIES) * RSB_MAX_K * RSB_VALUES + v) *
                                 RSB_TOT_STRIDE,
                     epoch, &sh.bad, st, polls);
    }
    __syncthreads();
}

template <int W, int R, int K>
__global__ void __launch_bounds__(NT, 1) k_res_bicg(const __grid_constant__ ResBicgArgs a)
{
    extern __shared__ float smem[];
    __shared__ RsbShared<K> sh;
    constexpr int MA = rsb_ab(W) < R ? rsb_ab(W) : R;
    constexpr int MC = rsb_cd(W) < R ? rsb_cd(W) : R;
    constexpr int ME = RSB_E < R ? RSB_E : R;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int wid = tid >> 5;
    const int P = (int)gridDim.x;
    const int c = (int)blockIdx.x;
    const int n = a.A.n;
    const float* rD32 = a.sys[0].run.rD32;
    const float* diag32 = a.sys[0].run.diag32;
    const int gA = min(P * rsb_ab(W), a.groups);
    const int gC = min(P * rsb_cd(W), a.groups);
    const int gE = min(P * RSB_E, a.groups);
    float* sval = smem;
    short* sidx = reinterpret_cast<short*>(smem + R * NT * W);
    unsigned int ep = *(volatile unsigned int*)a.epoch;
    const int all = K == 1 ? 1 : (1 << a.count) - 1;
    if (tid < K && (all >> tid & 1))
    {
        const InnerRun& N = a.sys[tid].run;
        inner_state_init(sh.S[tid], N.target, N.maxIter, N.ips, N.stagLimit);
    }
    if (tid < K) sh.stop[tid] = 0;
    if (tid == 0) sh.bad = 0;
    float r[K][R], r0[K][R], p[K][R], A[K][R], t[K][R];
    auto row_of = [&](int q) { return (P * q + c) * NT + tid; };
#pragma unroll
    for (int q = 0; q < R; ++q)
    {
        // this warp's slice of the paired stream; padding becomes an entry 0
        // of the row itself
        const int slice = (P * q + c) * (NT / 32) + wid;
        const int at = (q * (NT / 32) + wid) * 32 * W;
#pragma unroll
        for (int k = 0; k < W; ++k)
        {
            const int o = (int)pair_index(0, W, k, lane);
            short x = COL16_PAD;
            float u = 0.0f;
            if (slice < a.A.nslices)
            {
                x = a.A.pcol16[(size_t)slice * 32 * W + o];
                u = a.A.pval[(size_t)slice * 32 * W + o];
            }
            sidx[at + o] = x == COL16_PAD ? (short)0 : x;
            sval[at + o] = x == COL16_PAD ? 0.0f : u;
        }
        const int row = row_of(q);
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            r[k][q] = r0[k][q] = row < n && (all >> k & 1) ? (float)a.sys[k].run.r64[row] : 0.0f;
            p[k][q] = A[k][q] = t[k][q] = 0.0f;
        }
    }
    __syncthreads();
    // entry products of row q of this thread on x, added to acc
    auto spmv = [&](int q, const float* x, float acc) -> float {
        const int at = (q * (NT / 32) + wid) * 32 * W;
        const int row = min(row_of(q), n - 1);
        short o[W];
        float u[W];
#pragma unroll
        for (int g = 0; g < W / 2; ++g)
        {
            const short2 oo = *reinterpret_cast<const short2*>(sidx + at + 64 * g + 2 * lane);
            const float2 uu = *reinterpret_cast<const float2*>(sval + at + 64 * g + 2 * lane);
            o[2 * g] = oo.x;
            o[2 * g + 1] = oo.y;
            u[2 * g] = uu.x;
            u[2 * g + 1] = uu.y;
        }
        if constexpr (W & 1)
        {
            o[W - 1] = sidx[at + 32 * (W - 1) + lane];
            u[W - 1] = sval[at + 32 * (W - 1) + lane];
        }
        float xv[W];
#pragma unroll
        for (int k = 0; k < W; ++k) xv[k] = x[row + o[k]];
#pragma unroll
        for (int k = 0; k < W; ++k) acc = __fadd_rn(acc, __fmul_rn(u[k], xv[k]));
        return acc;
    };
    double rA0rA[K], beta[K], omega[K], res[K], alpha[K];
#pragma unroll
    for (int k = 0; k < K; ++k) rA0rA[k] = beta[k] = omega[k] = res[k] = alpha[k] = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        double acc[1][ME];
#pragma unroll
        for (int x = 0; x < ME; ++x) acc[0][x] = 0.0;
#pragma unroll
        for (int q = 0; q < R; ++q) acc[0][q % RSB_E] += (double)r[k][q] * (double)r[k][q];
        rsb_warps<K, 1, ME>(acc, k, sh);
    }
    ++ep;
    rsb_reduce<K, 1, ME>(a, all, 5, gE, ep, sh, false, true, res, omega);
#pragma unroll
    for (int k = 0; k < K; ++k) rA0rA[k] = sh.tot[k][0];
    int act = all;        // systems that go on
    bool first = true;
    for (;;)
    {
        // p, y = rD p (k_bicg_ab forms them at every gathered column)
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (K > 1 && !(act >> k & 1)) continue;
            const float bf = (float)beta[k];
            const float of = (float)omega[k];
            float* y = a.sys[k].y;
#pragma unroll
            for (int q = 0; q < R; ++q)
            {
                const int row = row_of(q);
                p[k][q] = __fadd_rn(r[k][q],
                                    __fmul_rn(bf, __fsub_rn(p[k][q], __fmul_rn(of, A[k][q]))));
                if (row < n) y[row] = __fmul_rn(__ldg(rD32 + row), p[k][q]);
            }
        }
        ++ep;
        rsb_barrier(a, ep, &sh.bad);
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (K > 1 && !(act >> k & 1)) continue;
            const float* y = a.sys[k].y;
            double acc[1][MA];
#pragma unroll
            for (int x = 0; x < MA; ++x) acc[0][x] = 0.0;
#pragma unroll
            for (int q = 0; q < R; ++q)
            {
                const int row = row_of(q);
                const float d = row < n ? __fmul_rn(__ldg(diag32 + row), y[row]) : 0.0f;
                A[k][q] = spmv(q, y, d);
                acc[0][q % rsb_ab(W)] += (double)r0[k][q] * (double)A[k][q];
            }
            rsb_warps<K, 1, MA>(acc, k, sh);
        }
        rsb_reduce<K, 1, MA>(a, act, 0, gA, ep, sh, true, first, res, omega);
        first = false;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (sh.stop[k]) act &= ~(1 << k);
        if (act == 0 || sh.bad) break;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (K > 1 && !(act >> k & 1)) continue;
            alpha[k] = rA0rA[k] / sh.tot[k][0];
            const float af = (float)alpha[k];
            float* z = a.sys[k].z;
#pragma unroll
            for (int q = 0; q < R; ++q)
            {
                const int row = row_of(q);
                r[k][q] = __fsub_rn(r[k][q], __fmul_rn(af, A[k][q]));   // s
                if (row < n) z[row] = __fmul_rn(__ldg(rD32 + row), r[k][q]);
            }
        }
        ++ep;
        rsb_barrier(a, ep, &sh.bad);
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (K > 1 && !(act >> k & 1)) continue;
            const float* z = a.sys[k].z;
            double acc[3][MC];
#pragma unroll
            for (int x = 0; x < MC; ++x) acc[0][x] = acc[1][x] = acc[2][x] = 0.0;
#pragma unroll
            for (int q = 0; q < R; ++q)
            {
                const int row = row_of(q);
                const float d = row < n ? __fmul_rn(__ldg(diag32 + row), z[row]) : 0.0f;
                t[k][q] = spmv(q, z, d);
                acc[0][q % rsb_cd(W)] += (double)fabsf(r[k][q]);
                acc[1][q % rsb_cd(W)] += (double)r[k][q] * (double)t[k][q];
                acc[2][q % rsb_cd(W)] += (double)t[k][q] * (double)t[k][q];
            }
            rsb_warps<K, 3, MC>(acc, k, sh);
        }
        rsb_reduce<K, 3, MC>(a, act, 1, gC, ep, sh, false, false, res, omega);
        int now = act;
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (K > 1 && !(act >> k & 1)) continue;
            const InnerRun& N = a.sys[k].run;
            const float* y = a.sys[k].y;
            const float* z = a.sys[k].z;
            const float af = (float)alpha[k];
            const double resS = sh.tot[k][0];
            // k_bicg_cd's checks: breakdown, the |s| exit, and only then omega
            const bool broken = !isfinite(rA0rA[k]) || !isfinite(alpha[k]) || !isfinite(resS);
            const bool early = !broken && resS <= N.target;
            omega[k] = sh.tot[k][1] / sh.tot[k][2];
            const float* dc = N.D + (size_t)sh.S[k].cur * N.dStride;
            float* dn = N.D + (size_t)sh.S[k].nxt * N.dStride;
            const bool start = sh.S[k].it == 0;   // (no correction yet: 0)
            if (broken || early)
            {
                now &= ~(1 << k);
                if (early)
                {
#pragma unroll
                    for (int q = 0; q < R; ++q)
                    {
                        const int row = row_of(q);
                        if (row < n)
                            dn[row] = __fadd_rn(start ? 0.0f : dc[row], __fmul_rn(af, y[row]));
                    }
                }
                __syncthreads();
                if (tid == NT - 1)
                {
                    InnerState& S = sh.S[k];
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
                continue;
            }
            const float wf = (float)omega[k];
            double acc[2][ME];
#pragma unroll
            for (int x = 0; x < ME; ++x) acc[0][x] = acc[1][x] = 0.0;
            // (the loads of a few rows before their stores: the compiler cannot
            // tell dn from the vectors it reads)
            constexpr int U = R < 8 ? R : 8;
#pragma unroll
            for (int q0 = 0; q0 < R; q0 += U)
            {
                float dd[U], yy[U], zz[U];
#pragma unroll
                for (int q = q0; q < q0 + U && q < R; ++q)
                {
                    const int row = min(row_of(q), n - 1);
                    dd[q - q0] = start ? 0.0f : dc[row];
                    yy[q - q0] = y[row];
                    zz[q - q0] = z[row];
                }
#pragma unroll
                for (int q = q0; q < q0 + U && q < R; ++q)
                {
                    const int row = row_of(q);
                    if (row < n)
                        dn[row] = __fadd_rn(dd[q - q0], __fadd_rn(__fmul_rn(af, yy[q - q0]),
                                                                  __fmul_rn(wf, zz[q - q0])));
                    r[k][q] = __fsub_rn(r[k][q], __fmul_rn(wf, t[k][q]));
                    acc[0][q % RSB_E] += (double)fabsf(r[k][q]);
                    acc[1][q % RSB_E] += (double)r0[k][q] * (double)r[k][q];
                }
            }
            rsb_warps<K, 2, ME>(acc, k, sh);
        }
        act = now;
        if (act == 0) break;
        ++ep;
        rsb_reduce<K, 2, ME>(a, act, 4, gE, ep, sh, false, false, res, omega);
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            if (K > 1 && !(act >> k & 1)) continue;
            res[k] = sh.tot[k][0];
            const double next = sh.tot[k][1];
            beta[k] = (next / rA0rA[k]) * (alpha[k] / omega[k]);
            rA0rA[k] = next;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        if (!(all >> k & 1)) continue;
        if (tid == NT - 1) inner_finish(sh.S[k], a.sys[k].run.st, c == 0);
        // (before the first update no correction has been written: 0)
        if (sh.S[k].it == 0)
        {
            for (int q = 0; q < R; ++q)
                if (row_of(q) < n) a.sys[k].run.D[row_of(q)] = 0.0f;
        }
    }
    if (c == 0 && tid == 0) *a.epoch = ep;
}

// groups per CTA the kernels are compiled for
const int RSB_ROWS[] = {2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16, 18, 20, 22, 24};
constexpr int RSB_TURNS_ABOVE = 2560; // rows per SM from which solves side by side take turns
constexpr int RSB_TEAM_R = 10;        // for several systems (15 registers per group of rows)

template <int W>
const void* kernel_r(int R)
{
    switch (R)
    {
        case 2: return (const void*)k_res_bicg<W, 2, 1>;
        case 3: return (const void*)k_res_bicg<W, 3, 1>;
        case 4: return (const void*)k_res_bicg<W, 4, 1>;
        case 5: return (const void*)k_res_bicg<W, 5, 1>;
        case 6: return (const void*)k_res_bicg<W, 6, 1>;
        case 7: return (const void*)k_res_bicg<W, 7, 1>;
        case 8: return (const void*)k_res_bicg<W, 8, 1>;
        case 10: return (const void*)k_res_bicg<W, 10, 1>;
        case 12: return (const void*)k_res_bicg<W, 12, 1>;
        case 14: return (const void*)k_res_bicg<W, 14, 1>;
        case 16: return (const void*)k_res_bicg<W, 16, 1>;
        case 18: return (const void*)k_res_bicg<W, 18, 1>;
        case 20: return (const void*)k_res_bicg<W, 20, 1>;
        case 22: return (const void*)k_res_bicg<W, 22, 1>;
        case 24: return (const void*)k_res_bicg<W, 24, 1>;
    }
    return nullptr;
}

template <int W>
const void* team_kernel_r(int R)
{
    switch (R)
    {
        case 2: return (const void*)k_res_bicg<W, 2, RSB_MAX_K>;
        case 3: return (const void*)k_res_bicg<W, 3, RSB_MAX_K>;
        case 4: return (const void*)k_res_bicg<W, 4, RSB_MAX_K>;
        case 5: return (const void*)k_res_bicg<W, 5, RSB_MAX_K>;
        case 6: return (const void*)k_res_bicg<W, 6, RSB_MAX_K>;
        case 7: return (const void*)k_res_bicg<W, 7, RSB_MAX_K>;
        case 8: return (const void*)k_res_bicg<W, 8, RSB_MAX_K>;
        case 10: return (const void*)k_res_bicg<W, 10, RSB_MAX_K>;
    }
    return nullptr;
}

const void* kernel_of(int W, int R, int systems)
{
    if (systems > 1)
        return W == 4 ? team_kernel_r<4>(R) : W == 5 ? team_kernel_r<5>(R) : team_kernel_r<6>(R);
    return W == 4 ? kernel_r<4>(R) : W == 5 ? kernel_r<5>(R) : kernel_r<6>(R);
}

// what the launches on one topology share: the device words, the kernels
struct Plan
{
    int groups = 0;
    size_t smem = 0;
    const void* fn = nullptr;       // one system
    const void* team = nullptr;     // up to RSB_MAX_K (null: one at a time)
    u64* part = nullptr;
    u64* tot = nullptr;
    unsigned int* flags = nullptr;
    unsigned int* epoch = nullptr;
    size_t bytes = 0;
    char* base = nullptr;
};

bool usable(int device, const void* fn, size_t smem)
{
    cudaFuncAttributes fa;
    int maxSmem = 0;
    int occ = 0;
    const bool ok =
        cudaFuncGetAttributes(&fa, fn) == cudaSuccess &&
        cudaDeviceGetAttribute(&maxSmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) ==
            cudaSuccess &&
        smem + fa.sharedSizeBytes <= (size_t)maxSmem &&
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(maxSmem - fa.sharedSizeBytes)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, NT, smem) == cudaSuccess &&
        occ >= 1;
    if (!ok) cudaGetLastError();
    return ok;
}

// The inner solves of `count` contexts on one matrix as one launch on the
// first one's stream, whose end the host waits for.  *ran stays false when
// they are to go through the graph loop.
int launch(cf_context* const* ctx, const InnerRun* runs, int count, bool* ran)
{
    cf_context* c = ctx[0];
    const Plan* w = static_cast<const Plan*>(c->resBicg);
    cudaStream_t s = c->stream;
    RSB_CUDA(cudaSetDevice(c->device));
    ResBicgArgs a = {};
    a.A = sell_of(c);
    a.count = count;
    a.part = w->part;
    a.tot = w->tot;
    a.flags = w->flags;
    a.epoch = w->epoch;
    a.groups = w->groups;
    for (int k = 0; k < count; ++k)
    {
        a.sys[k].run = runs[k];
        a.sys[k].run.polls = std::min(a.sys[k].run.polls, 1LL << 22);
        a.sys[k].y = ctx[k]->d_W1;
        a.sys[k].z = ctx[k]->d_Z1;
        RSB_CUDA(cudaEventRecord(ctx[k]->ev0, ctx[k]->stream));
        if (k) RSB_CUDA(cudaStreamWaitEvent(s, ctx[k]->ev0, 0));
    }
    void* args[] = {(void*)&a};
    if (cudaLaunchCooperativeKernel(count > 1 ? w->team : w->fn, dim3(c->numSMs), dim3(NT), args,
                                    w->smem, s) != cudaSuccess)
    {
        cudaGetLastError();   // (the graph loop then)
        return CF_OK;
    }
    c->launches++;
    for (int k = 0; k < count; ++k)
    {
        RSB_CUDA(cudaEventRecord(ctx[k]->ev1, s));
        RSB_CUDA(cudaMemcpyAsync(ctx[k]->h_st, ctx[k]->d_st, sizeof(InnerState),
                                 cudaMemcpyDeviceToHost, s));
    }
    RSB_CUDA(cudaStreamSynchronize(s));
    if (c->h_st->waitErr)
    {
        RSB_CUDA(cudaMemsetAsync(w->base, 0, w->bytes, s));
        RSB_CUDA(cudaMemsetAsync(&c->d_st->waitErr, 0, sizeof(int), s));
        RSB_CUDA(cudaStreamSynchronize(s));
        for (int k = 0; k < count; ++k) ctx[k]->backoff.gaveUp();
        return CF_OK;
    }
    for (int k = 0; k < count; ++k) ctx[k]->backoff.worked();
    *ran = true;
    return CF_OK;
}

}  // namespace

// The components of a multi-RHS solve run the FP64 driver on host threads of
// their own and meet for their inner solves: whoever comes last launches the
// kernel for those that wait.  A component that has ended leaves.
struct ResBicgTeam
{
    std::mutex mutex;
    std::condition_variable changed;
    int members = 0;
    int count = 0;                       // waiting
    cf_context* ctx[RSB_MAX_K];
    InnerRun run[RSB_MAX_K];
    unsigned long long round = 0;        // launches made
    bool ran = false;                    // the last one
    int rc = CF_OK;
    std::string msg;

    // (with the mutex held)
    void go()
    {
        ran = false;
        rc = CF_OK;
        {
            std::unique_lock<std::mutex> turn(res_device_lock(ctx[0]->device));
            rc = launch(ctx, run, count, &ran);
        }
        if (rc != CF_OK) msg = cf_last_error();
        count = 0;
        ++round;
        changed.notify_all();
    }
    int solve(cf_context* c, const InnerRun& r, bool* result)
    {
        std::unique_lock<std::mutex> lock(mutex);
        ctx[count] = c;
        run[count] = r;
        ++count;
        const unsigned long long mine = round;
        if (count == members)
            go();
        else
            changed.wait(lock, [&] { return round != mine; });
        // (the next round needs every waiter of this one)
        *result = ran;
        return rc == CF_OK ? CF_OK : fail(rc, msg);
    }
    void leave()
    {
        std::lock_guard<std::mutex> lock(mutex);
        --members;
        if (count > 0 && count == members) go();
    }
};

ResBicgTeam* res_bicg_team(cf_context* c, int members)
{
    const Plan* w = static_cast<const Plan*>(c->resBicg);
    if (!w || !w->team || members < 2 || members > RSB_MAX_K) return nullptr;
    ResBicgTeam* t = new (std::nothrow) ResBicgTeam();
    if (t) t->members = members;
    return t;
}

void res_bicg_leave(ResBicgTeam* t) { t->leave(); }

void res_bicg_team_free(ResBicgTeam* t) { delete t; }

void res_bicg_release(cf_context* c)
{
    Plan* w = static_cast<Plan*>(c->resBicg);
    if (w && !c->resBicgShared)
    {
        if (w->base) cudaFree(w->base);
        delete w;
    }
    c->resBicg = nullptr;
    c->resBicgTried = false;
    c->resBicgShared = false;
}

void res_bicg_prepare(cf_context* c)
{
    if (c->resBicgTried) return;
    const DevSell A = sell_of(c);
    const int P = c->numSMs;
    const int groups = (c->n + NT - 1) / NT;
    const int W = A.ellW;
    // smaller meshes run in a cluster, or through the graph loop
    if (c->n <= RSB_ABOVE || !c->coopLaunch || !A.pval || P > RSB_MAX_CTAS ||
        groups > P * RSB_MAX_R || c->device >= 64 || W < 4 || W > 6 || !spmv_default(c))
        return;
    c->resBicgTried = true;
    int R = 0;
    for (int k : RSB_ROWS)
        if (R == 0 && (long long)k * P >= groups) R = k;
    // the graph loop's grids must be the ones whose order is kept
    if (grid_for(c, (const void*)k_bicg_init, c->n) != std::min(P * RSB_E, groups) ||
        grid_for(c, (const void*)k_bicg_e, c->n) != std::min(P * RSB_E, groups) ||
        grid_for(c, (const void*)bicg_ab_kernel(A), c->n) != std::min(P * rsb_ab(W), groups) ||
        grid_for(c, (const void*)bicg_cd_kernel(A), c->n) != std::min(P * rsb_cd(W), groups))
        return;
    Plan* w = new (std::nothrow) Plan();
    if (!w) return;
    w->groups = groups;
    w->smem = (size_t)R * NT * W * (sizeof(float) + sizeof(short));
    w->fn = kernel_of(W, R, 1);
    if (R <= RSB_TEAM_R) w->team = kernel_of(W, R, RSB_MAX_K);
    if (w->team && !usable(c->device, w->team, w->smem)) w->team = nullptr;
    const size_t part = sizeof(u64) * 2 * RSB_MAX_K * RSB_VALUES * RSB_MAX_BLOCKS;
    const size_t tot = sizeof(u64) * RSB_TOT_STRIDE * RSB_MAX_K * RSB_VALUES * RSB_COPIES;
    const size_t flags = sizeof(unsigned int) * RSB_FLAG_COPIES * RSB_MAX_CTAS * RSB_FLAG_STRIDE;
    w->bytes = part + tot + flags + 256;
    if (!usable(c->device, w->fn, w->smem) ||
        cudaMalloc((void**)&w->base, w->bytes) != cudaSuccess ||
        cudaMemsetAsync(w->base, 0, w->bytes, c->stream) != cudaSuccess)
    {
        cudaGetLastError();
        if (w->base) cudaFree(w->base);
        delete w;
        return;
    }
    w->part = reinterpret_cast<u64*>(w->base);
    w->tot = reinterpret_cast<u64*>(w->base + part);
    w->flags = reinterpret_cast<unsigned int*>(w->base + part + tot);
    w->epoch = reinterpret_cast<unsigned int*>(w->base + part + tot + flags);
    c->resBicg = w;
}

int res_bicg_inner(cf_context* c, double target, int maxIter, int ips, int stagLimit, bool* ran)
{
    *ran = false;
    res_bicg_prepare(c);
    // (the plan may be older than a switch to the 32-bit column stream)
    if (maxIter <= 0 || !c->resBicg || !sell_of(c).pval) return CF_OK;
    const InnerRun run = inner_run(c, nullptr, target, maxIter, ips, 1, stagLimit);
    if (c->resBicgTeam) return c->resBicgTeam->solve(c, run, ran);
    // One resident launch at a time on the device; the others wait or go
    // through the graph loop, which gives the same bits.  A launch of two
    // groups of rows per SM leaves room for graph loops beside it; of the
    // larger meshes, which do not, two take turns and more keep the graph loop
    // each, until it needs HBM.  ms, in turns / a launch beside graph loops /
    // graph loops only: 50K cells 3 at once 10.3 / 6.9 / 8.8, 8 at once 31 / 19 /
    // 24; 110K 2: 7.1 / 9.6 / 8.2, 3: 11.8 / 13.6 / 10.9, 8: 36 / 30 / 24; 262K 2:
    // 12.1 / 13.0 / 15.1, 3: 18.1 / 18.9 / 17.0, 8: 55 / 56 / 53; 405K 3: 22 / 26 /
    // 22, 8: 69 / 70 / 66; 593K 3: 26 / 33 / 31, 8: 76 / 83 / 85; 885K 2: 23 / 31 / 33,
    // 8: 105 / 115 / 135.
    const int rows = c->n / c->numSMs;
    const int beside = std::max(c->concurrent, res_in_flight(c->device).load());
    std::unique_lock<std::mutex> turn(res_device_lock(c->device), std::defer_lock);
    if (beside <= 2 || rows > RSB_TURNS_ABOVE)
        turn.lock();
    else if (rows > 2 * NT || !turn.try_lock())
        return CF_OK;
    return launch(&c, &run, 1, ran);
}

}  // namespace cf
