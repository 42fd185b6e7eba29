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
#include <mutex>
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
constexpr int RSB_E = 8;             // k_bicg_e and k_bicg_init

struct ResBicgArgs
{
    DevSell A;
    InnerRun run;
    float* y;
    float* z;
    u64* part;              // [values][RSB_MAX_BLOCKS][2 words]
    u64* tot;               // [copies][values], RSB_TOT_STRIDE apart
    unsigned int* flags;    // [copies][RSB_MAX_CTAS], RSB_FLAG_STRIDE apart
    unsigned int* epoch;    // last epoch used by the launches before
    int groups;             // 256-row groups of the mesh
};

struct RsbShared
{
    double ws[3][8][NT / 32];
    double fs[NT / 32];
    double tot[3];
    int stop, bad;
    InnerState S;
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
__device__ __forceinline__ bool rsb_more(long long& spins, RsbShared& sh, InnerState* st,
                                         long long polls)
{
    if ((++spins & 1023) != 0 && spins <= polls) return true;
    if (*(volatile int*)&sh.bad) return false;
    if (spins > polls || *(volatile int*)&st->waitErr)
    {
        atomicExch(&st->waitErr, 1);
        *(volatile int*)&sh.bad = 1;
        return false;
    }
    return true;
}

__device__ __forceinline__ double rsb_wait(const u64* p, unsigned int epoch, RsbShared& sh,
                                           InnerState* st, long long polls)
{
    u64 lo, hi;
    long long spins = 0;
    ld2(p, lo, hi);
    while ((unsigned int)(lo >> 32) != epoch || (unsigned int)(hi >> 32) != epoch)
    {
        if (!rsb_more(spins, sh, st, polls)) return 0.0;
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
__device__ __forceinline__ void rsb_barrier(const ResBicgArgs& a, unsigned int epoch, RsbShared& sh)
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
            if (v == epoch || !rsb_more(spins, sh, a.run.st, a.run.polls)) break;
        }
        fence_acq_rel();
    }
    __syncthreads();
}

// acc[r][x]: this thread's sum of value v0 + r over the groups of its block x
// (block x SMs + CTA of the value's G blocks).  The totals are in sh.tot after
// the call.
template <int NR, int M>
__device__ __forceinline__ void rsb_reduce(const ResBicgArgs& a, double (&acc)[NR][M], int v0, int G,
                                           unsigned int epoch, RsbShared& sh, bool book, bool first,
                                           double res, double omega)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int wid = tid >> 5;
    const int P = (int)gridDim.x;
    {
        double v[NR * M];
#pragma unroll
        for (int r = 0; r < NR; ++r)
#pragma unroll
            for (int x = 0; x < M; ++x) v[r * M + x] = acc[r][x];
        warp_sums<NR * M, 16>(v);
        const int k = warp_sums_index(lane);
        if (k < NR * M) sh.ws[k / M][k % M][wid] = v[0];
    }
    __syncthreads();
    if (tid < NR * M)
    {
        const int r = tid / M;
        const int x = tid - r * M;
        const int b = x * P + (int)blockIdx.x;
        if (b < G) st_dbl(a.part + ((size_t)(v0 + r) * RSB_MAX_BLOCKS + b) * 2, fold8(sh.ws[r][x]), epoch);
    }
    // the checks of the iteration before, while the sums are on their way
    if (book && tid == NT - 1)
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
    // one of the last CTAs (they have the fewest rows) folds a value as
    // grid_sum's last block does
    const int mine = P - 1 - (int)blockIdx.x;
    if (mine < NR)
    {
        const u64* w = a.part + (size_t)(v0 + mine) * RSB_MAX_BLOCKS * 2;
        double t = 0.0;
        for (int b = tid; b < G; b += NT)
            t += rsb_wait(w + (size_t)b * 2, epoch, sh, a.run.st, a.run.polls);
        t = warp_sum(t);
        if (lane == 0) sh.fs[wid] = t;
        __syncthreads();
        if (tid < RSB_COPIES)
            st_dbl(a.tot + ((size_t)tid * RSB_VALUES + v0 + mine) * RSB_TOT_STRIDE, fold8(sh.fs), epoch);
    }
    if (tid < NR)
        sh.tot[tid] = rsb_wait(a.tot + ((size_t)(blockIdx.x % RSB_COPIES) * RSB_VALUES + v0 + tid) * RSB_TOT_STRIDE,
                               epoch, sh, a.run.st, a.run.polls);
    __syncthreads();
}

template <int W, int R>
__global__ void __launch_bounds__(NT, 1) k_res_bicg(const __grid_constant__ ResBicgArgs a)
{
    extern __shared__ float smem[];
    __shared__ RsbShared sh;
    constexpr int MA = rsb_ab(W) < R ? rsb_ab(W) : R;
    constexpr int MC = rsb_cd(W) < R ? rsb_cd(W) : R;
    constexpr int ME = RSB_E < R ? RSB_E : R;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int wid = tid >> 5;
    const int P = (int)gridDim.x;
    const int c = (int)blockIdx.x;
    const int n = a.A.n;
    const InnerRun& N = a.run;
    const int gA = min(P * rsb_ab(W), a.groups);
    const int gC = min(P * rsb_cd(W), a.groups);
    const int gE = min(P * RSB_E, a.groups);
    float* sval = smem;
    short* sidx = reinterpret_cast<short*>(smem + R * NT * W);
    unsigned int ep = *(volatile unsigned int*)a.epoch;
    if (tid == 0)
    {
        inner_state_init(sh.S, N.target, N.maxIter, N.ips, N.stagLimit);
        sh.stop = sh.bad = 0;
    }
    float r[R], r0[R], p[R], A[R], t[R];
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
        r[q] = r0[q] = row < n ? (float)N.r64[row] : 0.0f;
        p[q] = A[q] = t[q] = 0.0f;
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
    double rA0rA;
    {
        double acc[1][ME];
#pragma unroll
        for (int x = 0; x < ME; ++x) acc[0][x] = 0.0;
#pragma unroll
        for (int q = 0; q < R; ++q) acc[0][q % RSB_E] += (double)r[q] * (double)r[q];
        ++ep;
        rsb_reduce<1, ME>(a, acc, 5, gE, ep, sh, false, true, 0.0, 0.0);
        rA0rA = sh.tot[0];
    }
    double beta = 0.0, omega = 0.0, res = 0.0;
    bool first = true;
    for (;;)
    {
        const float bf = (float)beta;
        const float of = (float)omega;
        // p, y = rD p (k_bicg_ab forms them at every gathered column)
#pragma unroll
        for (int q = 0; q < R; ++q)
        {
            const int row = row_of(q);
            p[q] = __fadd_rn(r[q], __fmul_rn(bf, __fsub_rn(p[q], __fmul_rn(of, A[q]))));
            if (row < n) a.y[row] = __fmul_rn(__ldg(N.rD32 + row), p[q]);
        }
        ++ep;
        rsb_barrier(a, ep, sh);
        {
            double acc[1][MA];
#pragma unroll
            for (int x = 0; x < MA; ++x) acc[0][x] = 0.0;
#pragma unroll
            for (int q = 0; q < R; ++q)
            {
                const int row = row_of(q);
                const float d = row < n ? __fmul_rn(__ldg(N.diag32 + row), a.y[row]) : 0.0f;
                A[q] = spmv(q, a.y, d);
                acc[0][q % rsb_ab(W)] += (double)r0[q] * (double)A[q];
            }
            rsb_reduce<1, MA>(a, acc, 0, gA, ep, sh, true, first, res, omega);
        }
        first = false;
        if (sh.stop) break;
        const double alpha = rA0rA / sh.tot[0];
        const float af = (float)alpha;
        double acc3[3][MC];
#pragma unroll
        for (int x = 0; x < MC; ++x) acc3[0][x] = acc3[1][x] = acc3[2][x] = 0.0;
#pragma unroll
        for (int q = 0; q < R; ++q)
        {
            const int row = row_of(q);
            r[q] = __fsub_rn(r[q], __fmul_rn(af, A[q]));   // s
            if (row < n) a.z[row] = __fmul_rn(__ldg(N.rD32 + row), r[q]);
            acc3[0][q % rsb_cd(W)] += (double)fabsf(r[q]);
        }
        ++ep;
        rsb_barrier(a, ep, sh);
#pragma unroll
        for (int q = 0; q < R; ++q)
        {
            const int row = row_of(q);
            const float d = row < n ? __fmul_rn(__ldg(N.diag32 + row), a.z[row]) : 0.0f;
            t[q] = spmv(q, a.z, d);
            acc3[1][q % rsb_cd(W)] += (double)r[q] * (double)t[q];
            acc3[2][q % rsb_cd(W)] += (double)t[q] * (double)t[q];
        }
        rsb_reduce<3, MC>(a, acc3, 1, gC, ep, sh, false, false, 0.0, 0.0);
        const double resS = sh.tot[0];
        // k_bicg_cd's checks: breakdown, the |s| exit, and only then omega
        const bool broken = !isfinite(rA0rA) || !isfinite(alpha) || !isfinite(resS);
        const bool early = !broken && resS <= N.target;
        omega = sh.tot[1] / sh.tot[2];
        const int cur = sh.S.cur;
        const float* dc = N.D + (size_t)cur * N.dStride;
        float* dn = N.D + (size_t)sh.S.nxt * N.dStride;
        const bool start = sh.S.it == 0;   // (no correction yet: 0)
        if (broken || early)
        {
            if (early)
            {
#pragma unroll
                for (int q = 0; q < R; ++q)
                {
                    const int row = row_of(q);
                    if (row < n)
                        dn[row] = __fadd_rn(start ? 0.0f : dc[row], __fmul_rn(af, a.y[row]));
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
        double acc2[2][ME];
#pragma unroll
        for (int x = 0; x < ME; ++x) acc2[0][x] = acc2[1][x] = 0.0;
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
                yy[q - q0] = a.y[row];
                zz[q - q0] = a.z[row];
            }
#pragma unroll
            for (int q = q0; q < q0 + U && q < R; ++q)
            {
                const int row = row_of(q);
                if (row < n)
                    dn[row] = __fadd_rn(dd[q - q0], __fadd_rn(__fmul_rn(af, yy[q - q0]),
                                                              __fmul_rn(wf, zz[q - q0])));
                r[q] = __fsub_rn(r[q], __fmul_rn(wf, t[q]));
                acc2[0][q % RSB_E] += (double)fabsf(r[q]);
                acc2[1][q % RSB_E] += (double)r0[q] * (double)r[q];
            }
        }
        ++ep;
        rsb_reduce<2, ME>(a, acc2, 4, gE, ep, sh, false, false, 0.0, 0.0);
        res = sh.tot[0];
        const double next = sh.tot[1];
        beta = (next / rA0rA) * (alpha / omega);
        rA0rA = next;
    }
    __syncthreads();
    if (tid == NT - 1) inner_finish(sh.S, N.st, c == 0);
    // (before the first update no correction has been written: 0)
    if (sh.S.it == 0)
    {
        for (int q = 0; q < R; ++q)
            if (row_of(q) < n) N.D[row_of(q)] = 0.0f;
    }
    if (c == 0 && tid == 0) *a.epoch = ep;
}

const int RSB_ROWS[] = {2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16, 18, 20, 22, 24};

template <int W>
const void* kernel_r(int R)
{
    switch (R)
    {
        case 2: return (const void*)k_res_bicg<W, 2>;
        case 3: return (const void*)k_res_bicg<W, 3>;
        case 4: return (const void*)k_res_bicg<W, 4>;
        case 5: return (const void*)k_res_bicg<W, 5>;
        case 6: return (const void*)k_res_bicg<W, 6>;
        case 7: return (const void*)k_res_bicg<W, 7>;
        case 8: return (const void*)k_res_bicg<W, 8>;
        case 10: return (const void*)k_res_bicg<W, 10>;
        case 12: return (const void*)k_res_bicg<W, 12>;
        case 14: return (const void*)k_res_bicg<W, 14>;
        case 16: return (const void*)k_res_bicg<W, 16>;
        case 18: return (const void*)k_res_bicg<W, 18>;
        case 20: return (const void*)k_res_bicg<W, 20>;
        case 22: return (const void*)k_res_bicg<W, 22>;
        case 24: return (const void*)k_res_bicg<W, 24>;
    }
    return nullptr;
}

const void* kernel_of(int W, int R)
{
    return W == 4 ? kernel_r<4>(R) : W == 5 ? kernel_r<5>(R) : kernel_r<6>(R);
}

// the device words of a context's launches
struct Words
{
    u64* part = nullptr;
    u64* tot = nullptr;
    unsigned int* flags = nullptr;
    unsigned int* epoch = nullptr;
    size_t bytes = 0;
    char* base = nullptr;
};

}  // namespace

void res_bicg_release(cf_context* c)
{
    Words* w = static_cast<Words*>(c->resBicg);
    if (w)
    {
        if (w->base) cudaFree(w->base);
        delete w;
    }
    c->resBicg = nullptr;
    c->resBicgTried = false;
}

int res_bicg_inner(cf_context* c, double target, int maxIter, int ips, int stagLimit, bool* ran)
{
    *ran = false;
    const DevSell A = sell_of(c);
    const int P = c->numSMs;
    const int groups = (c->n + NT - 1) / NT;
    if (maxIter <= 0 || !c->coopLaunch || !A.pval || P > RSB_MAX_CTAS ||
        groups > P * RSB_MAX_R || c->device >= 64)
        return CF_OK;
    const int W = A.ellW;
    if (W < 4 || W > 6) return CF_OK;
    int R = 0;
    for (int k : RSB_ROWS)
        if (R == 0 && (long long)k * P >= groups) R = k;
    const void* fn = kernel_of(W, R);
    const size_t smem = (size_t)R * NT * W * (sizeof(float) + sizeof(short));
    if (!c->resBicgTried)
    {
        c->resBicgTried = true;
        // the graph loop's grids must be the ones whose order is kept
        const bool grids =
            grid_for(c, (const void*)k_bicg_init, c->n) == std::min(P * RSB_E, groups) &&
            grid_for(c, (const void*)k_bicg_e, c->n) == std::min(P * RSB_E, groups) &&
            grid_for(c, (const void*)bicg_ab_kernel(A), c->n) == std::min(P * rsb_ab(W), groups) &&
            grid_for(c, (const void*)bicg_cd_kernel(A), c->n) == std::min(P * rsb_cd(W), groups);
        int maxSmem = 0;
        int occ = 0;
        if (!grids ||
            cudaDeviceGetAttribute(&maxSmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device) !=
                cudaSuccess ||
            smem + 2048 > (size_t)maxSmem ||
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 maxSmem - 2048) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, NT, smem) != cudaSuccess ||
            occ < 1)
        {
            cudaGetLastError();
            return CF_OK;
        }
        Words* w = new Words();
        const size_t part = sizeof(u64) * 2 * RSB_VALUES * RSB_MAX_BLOCKS;
        const size_t tot = sizeof(u64) * RSB_TOT_STRIDE * RSB_VALUES * RSB_COPIES;
        const size_t flags = sizeof(unsigned int) * RSB_FLAG_COPIES * RSB_MAX_CTAS * RSB_FLAG_STRIDE;
        w->bytes = part + tot + flags + 256;
        if (cudaMalloc((void**)&w->base, w->bytes) != cudaSuccess ||
            cudaMemsetAsync(w->base, 0, w->bytes, c->stream) != cudaSuccess)
        {
            cudaGetLastError();
            if (w->base) cudaFree(w->base);
            delete w;
            return CF_OK;
        }
        w->part = reinterpret_cast<u64*>(w->base);
        w->tot = reinterpret_cast<u64*>(w->base + part);
        w->flags = reinterpret_cast<unsigned int*>(w->base + part + tot);
        w->epoch = reinterpret_cast<unsigned int*>(w->base + part + tot + flags);
        c->resBicg = w;
    }
    Words* w = static_cast<Words*>(c->resBicg);
    if (!w) return CF_OK;
    // one resident launch at a time on the device: the components of a
    // multi-RHS solve take turns, other solves go through the graph loop
    std::unique_lock<std::mutex> turn(res_device_lock(c->device), std::defer_lock);
    if (c->waitTurn)
        turn.lock();
    else if (!turn.try_lock())
        return CF_OK;
    cudaStream_t s = c->stream;
    ResBicgArgs a;
    a.A = A;
    a.run = inner_run(c, nullptr, target, maxIter, ips, 1, stagLimit);
    a.run.polls = std::min(a.run.polls, 1LL << 22);
    a.y = c->d_W1;
    a.z = c->d_Z1;
    a.part = w->part;
    a.tot = w->tot;
    a.flags = w->flags;
    a.epoch = w->epoch;
    a.groups = groups;
    void* args[] = {(void*)&a};
    RSB_CUDA(cudaEventRecord(c->ev0, s));
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(P), dim3(NT), args, smem, s);
    if (e != cudaSuccess)
    {
        cudaGetLastError();   // (the graph loop then)
        return CF_OK;
    }
    c->launches++;
    RSB_CUDA(cudaEventRecord(c->ev1, s));
    RSB_CUDA(cudaMemcpyAsync(c->h_st, c->d_st, sizeof(InnerState), cudaMemcpyDeviceToHost, s));
    RSB_CUDA(cudaStreamSynchronize(s));
    if (c->h_st->waitErr)
    {
        RSB_CUDA(cudaMemsetAsync(w->base, 0, w->bytes, s));
        RSB_CUDA(cudaMemsetAsync(&c->d_st->waitErr, 0, sizeof(int), s));
        return CF_OK;
    }
    *ran = true;
    return CF_OK;
}

}  // namespace cf
