// cf_resident.cu -- the inner PCG of one system as ONE launch in which every
// CTA keeps one compact part of the mesh (cf_partition.cu) on its SM.
//
// What bounds the graph-driven loop (cf_solve.cu) below about a million
// cells is not bytes: its nine launches per iteration cost 3.4-5 us each
// (24K-300K cells: 30-43 us per iteration) whatever the mesh.  Here an
// iteration has no launch and no grid barrier:
//
//  * z and p of a part live in shared memory, the part's rows with a
//    neighbour elsewhere are published to L2 as 8-byte words {value, epoch}
//    and read by polling the word itself, so a Chebyshev step waits for its
//    neighbours' boundary values only (one store-to-load trip through L2),
//    with no fence, no flag and no barrier across CTAs;
//  * p of the halo rows is advanced locally from the received z (the same
//    operations as its owner's), so the p-update SpMV needs no exchange of
//    its own;
//  * the two reductions per iteration (p.q, and z.r together with the
//    previous update's sum|r|) are all-gathers of one FP64 partial per CTA
//    through the same {value, epoch} words; every CTA folds them in the same
//    order and keeps its own copy of the solver state.  The stopping tests
//    of an update are therefore made one Chebyshev apply later; nothing of
//    that apply is kept when they end the solve;
//  * the matrix entries and the row-private vectors stay in registers (256
//    threads of up to 10 rows), in larger parts the entries of some rows in
//    shared memory (512 threads of up to 12 rows).
//
// Measured on one box, us per inner iteration, graph loop / this kernel
// (Chebyshev 8): 24K cells 3-D 28.7 / 15.7, 200K prisms 43.7 / 18.0, 262K
// 3-D 45.7 / 17.4, 307K 2-D 44.2 / 15.0, 448K 3-D 56.0 / 29.6; Jacobi, 262K:
// 17.5 / 8.4.  What is left at 24K-300K cells is
// the trip of a word from SM to SM through L2, 1,750 cycles there and back in
// the median pair (measured with two CTAs bouncing one word), ten times per
// iteration.  128^3 does not fit on the SMs: with the rest of the matrix
// streamed through the same kernel it took 193 us against 173 of the graph
// loop, so larger meshes keep that.  512 or 1,024 threads with fewer rows
// each were slower (262K: 20.7 and 26.5 us): the rows of a thread are
// independent, so few threads lose nothing and their barriers cost less.
//
// Per row the arithmetic is the graph path's (row_f32's entries in stored
// order, separately rounded), so every vector is the same given the same
// scalars; the FP64 sums fold in an order of their own.
//
// Buffers: exchange words have two parities.  The owner of a word writes
// exchange e + 2 only after it has received exchange e + 1 from every part
// it borders, and they sent e + 1 after reading e (the matrix pattern is
// symmetric, so every reader of a part is also read by it).  The same holds
// for the reductions over all parts.  Every wait is bounded; a wait that
// gives up sets the state's waitErr and the kernel ends at the next
// reduction, after which the caller runs the graph path instead.
#include "cudafoam.h"
#include "cf_host.hpp"
#include "cf_inner.cuh"
#include "cf_cluster_ll.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

using namespace cf;

#define RES_CUDA(call)                                                          \
    do                                                                          \
    {                                                                           \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess)                                                  \
            return fail(CF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace cf {

struct ResPlan
{
    int nparts = 0, W = 0, slots = 0, rowsP = 0, maxHalo = 0;
    int R = 0;                    // rows per thread
    int TB = 0, threads = 0;
    size_t smem = 0;
    const void* fn = nullptr;
    std::vector<void*> allocs;
    ResPart* parts = nullptr;
    int* rowMap = nullptr;
    unsigned short* idx = nullptr;
    int* emap = nullptr;
    int* haloSlot = nullptr;
    u64* ll = nullptr;
    u64* red = nullptr;
    unsigned int* epoch = nullptr;
    float* dw = nullptr;
    float* dc = nullptr;
};

namespace {

constexpr int RES_MAX_PARTS = 256;   // CTAs of one system at most
constexpr int RES_MAX_ROWS = 6144;   // rows of a part at most (the last entry of CHIP)
constexpr int RES_COPIES = 8;        // copies of every reduction word
// A part's words have a 128-byte line of their own (with four parts to a line,
// whose writers and pollers meet in L2: 64^3 Jacobi 8.66 us per iteration, 8.29
// so; prism 200K order 8 18.1 and 17.9).
constexpr int RES_STRIDE = 16;       // 8-byte words
constexpr size_t RES_RED_WORDS = (size_t)RES_COPIES * RES_MAX_PARTS * RES_STRIDE;
constexpr int RES_HQ = 4;            // halo slots a thread keeps in registers

struct ResArgs
{
    const ResPart* parts;
    int nparts;
    const int* rowMap;
    const unsigned short* idx;
    const int* emap;
    const int* haloSlot;
    u64* ll;                 // [2][slots]
    int slots;
    u64* red;                // [2][copy][part][2 values x 2 words]
    unsigned int* epoch;     // last epoch used by the launches before
    float* dw;               // [3 rowsP] corrections (part order)
    float* dc;               // [rowsP] current correction of the lean kernels
    int rowsP;
    InnerRun run;
};

__device__ __forceinline__ u64 ld_word(const u64* p)
{
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ void st_word(u64* p, unsigned int lo, unsigned int epoch)
{
    const u64 v = ((u64)epoch << 32) | lo;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v));
}

template <class P>
__device__ __forceinline__ void swap_ptr(P*& x, P*& y)
{
    P* t = x;
    x = y;
    y = t;
}

__device__ __forceinline__ void st_double(u64* p, double x, unsigned int epoch)
{
    const u64 b = (u64)__double_as_longlong(x);
    const u64 lo = ((u64)epoch << 32) | (b & 0xffffffffu);
    const u64 hi = ((u64)epoch << 32) | (b >> 32);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi));
}

__device__ __forceinline__ void ld_words(const u64* p, u64& x, u64& y)
{
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p));
}

struct ResShared
{
    double red[2][32];
    double cross[2][32];
    int stop, bad;
    InnerState S;
};

// Waits until the word carries `epoch`; gives up after `polls` reads or when
// another wait of the grid has given up.
__device__ __forceinline__ unsigned int wait_word(const u64* p, u64 first, unsigned int epoch,
                                                  ResShared& sh, InnerState* st, long long polls)
{
    u64 v = first;
    if ((unsigned int)(v >> 32) == epoch) return (unsigned int)v;
    long long spins = 0;
    for (;;)
    {
        v = ld_word(p);
        if ((unsigned int)(v >> 32) == epoch) return (unsigned int)v;
        if ((++spins & 1023) == 0 || spins > polls)
        {
            if (*(volatile int*)&sh.bad) return 0u;
            if (spins > polls || *(volatile int*)&st->waitErr)
            {
                atomicExch(&st->waitErr, 1);
                *(volatile int*)&sh.bad = 1;
                return 0u;
            }
        }
    }
}

// The same for a double split over two neighbouring words.
__device__ __forceinline__ double wait_double(const u64* p, u64 lo, u64 hi, unsigned int epoch,
                                              ResShared& sh, InnerState* st, long long polls)
{
    long long spins = 0;
    while ((unsigned int)(lo >> 32) != epoch || (unsigned int)(hi >> 32) != epoch)
    {
        ld_words(p, lo, hi);
        if ((++spins & 1023) == 0 || spins > polls)
        {
            if (*(volatile int*)&sh.bad) return 0.0;
            if (spins > polls || *(volatile int*)&st->waitErr)
            {
                atomicExch(&st->waitErr, 1);
                *(volatile int*)&sh.bad = 1;
                return 0.0;
            }
        }
    }
    return __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffu)));
}

// This part's halo values of exchange `epoch` into x[nlocP ..].
__device__ __forceinline__ void halo_recv(const ResArgs& a, const ResPart& P, const int (&hs)[RES_HQ],
                                          const u64* ll, unsigned int epoch, float* x,
                                          ResShared& sh, int tid, int T)
{
    u64 v[RES_HQ];
#pragma unroll
    for (int q = 0; q < RES_HQ; ++q)
        if (hs[q] >= 0) v[q] = ld_word(ll + hs[q]);
#pragma unroll
    for (int q = 0; q < RES_HQ; ++q)
        if (hs[q] >= 0)
            x[P.nlocP + tid + q * T] =
                __uint_as_float(wait_word(ll + hs[q], v[q], epoch, sh, a.run.st, a.run.polls));
    for (int h = tid + RES_HQ * T; h < P.nh; h += T)
    {
        const u64* p = ll + __ldg(a.haloSlot + P.haloBase + h);
        x[P.nlocP + h] = __uint_as_float(wait_word(p, ld_word(p), epoch, sh, a.run.st, a.run.polls));
    }
}

// Sums of v[0..NR) over the CTA, published under `epoch` in RES_COPIES
// copies, each polled by every RES_COPIES-th part: with one copy every CTA's
// reads queue on the same few L2 lines ahead of the stores they wait for
// (15.6 us per Jacobi iteration at 148 parts), with a copy for every part
// the scattered stores take as long (11.1 us).
template <int NR>
__device__ __forceinline__ void red_send(double (&v)[NR], u64* red, int rank, unsigned int epoch,
                                         ResShared& sh, int tid, int T)
{
    const int lane = tid & 31;
    const int wid = tid >> 5;
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = warp_sum(v[r]);
    if (lane == 0)
    {
#pragma unroll
        for (int r = 0; r < NR; ++r) sh.red[r][wid] = v[r];
    }
    __syncthreads();
    if (wid == 0)
    {
        double t[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) t[r] = warp_sum(lane < (T >> 5) ? sh.red[r][lane] : 0.0);
        if (lane < RES_COPIES)
        {
            u64* w = red + ((size_t)lane * RES_MAX_PARTS + rank) * RES_STRIDE;
#pragma unroll
            for (int r = 0; r < NR; ++r) st_double(w + 2 * r, t[r], epoch);
        }
    }
}

// Gathers the partials of every part; sh.cross[r][0 .. warps) then holds the
// warps' sums (valid after the next barrier).
template <int NR>
__device__ __forceinline__ void red_recv(const ResArgs& a, const u64* red, int rank,
                                         unsigned int epoch, ResShared& sh, int tid, int T)
{
    const int lane = tid & 31;
    const int wid = tid >> 5;
    if (wid * 32 >= a.nparts) return;
    double acc[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = 0.0;
    for (int p = tid; p < a.nparts; p += T)
    {
        const u64* w = red + ((size_t)(rank % RES_COPIES) * RES_MAX_PARTS + p) * RES_STRIDE;
        u64 f[NR][2];
#pragma unroll
        for (int r = 0; r < NR; ++r) ld_words(w + 2 * r, f[r][0], f[r][1]);
#pragma unroll
        for (int r = 0; r < NR; ++r)
        {
            acc[r] += wait_double(w + 2 * r, f[r][0], f[r][1], epoch, sh, a.run.st, a.run.polls);
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
    {
        const double t = warp_sum(acc[r]);
        if (lane == 0) sh.cross[r][wid] = t;
    }
}

__device__ __forceinline__ double red_total(const ResArgs& a, const ResShared& sh, int r, int T)
{
    const int nw = min((a.nparts + 31) >> 5, T >> 5);
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += sh.cross[r][w];
    return t;
}

__device__ __forceinline__ void state_init(const ResArgs& a, ResShared& sh)
{
    const InnerState* s = a.run.st;
    if (a.run.fromState)
        inner_state_init(sh.S, s->target, s->maxIter, s->ips, s->stagLimit);
    else
        inner_state_init(sh.S, a.run.target, a.run.maxIter, a.run.ips, a.run.stagLimit);
    sh.stop = 0;
    sh.bad = 0;
}

// ------------------------------------------------- parts that fit on the SM

// R rows per thread (row i of a thread: local row tid + i T).  The matrix
// entries of the first RM of them stay in registers, those of the others in
// shared memory; diag, 1/diag, r and w always stay in registers.  Results go
// to the next z only after the gathers from the current one (the compiler
// cannot tell the two buffers apart).
template <int W, int R, int RM, int TB>
__global__ void __launch_bounds__(TB, 1) k_res_chip(const __grid_constant__ ResArgs a)
{
    extern __shared__ float zmem[];
    __shared__ ResShared sh;
    if (a.run.fromState && a.run.st->done) return;   // (the whole grid)
    constexpr bool LEAN = R * TB > 2560;   // z, delta and q of a row are not kept in registers
    // Rows of the first RB thread rows are finished and published one after
    // the other, the rest (rows no other part reads, mostly) in whatever
    // order keeps most gathers in flight: a part's boundary is 6% of its rows
    // on 2-D meshes and up to half on 3-D ones.  us per iteration with RB 0 /
    // 1 / 2 / 4: 262K 3-D 19.7 / 18.6 / 17.1 / 17.4, 200K prisms 19.3 / 19.1 /
    // 18.7 / 18.0, 307K 2-D 15.0 / 14.9 / 15.1 / 15.0.
    constexpr int RB = W == 4 ? 1 : 4;
    const int tid = threadIdx.x;
    const int T = blockDim.x;
    const int rank = blockIdx.x;
    const ResPart P = a.parts[rank];
    const int zs = P.nlocP + P.nh + 1;
    float* zc = zmem;          // current z
    float* zn = zmem + zs;     // the next
    float* pb = zmem + 2 * zs;
    // matrix rows from RM T on: values, then columns
    const int m0 = RM * T;
    const int mRows = max(0, P.nlocP - m0);
    float* sval = zmem + ((3 * zs + 1) & ~1);
    unsigned short* sidx = reinterpret_cast<unsigned short*>(sval + (size_t)mRows * W);
    const bool cheb = a.run.order > 1;
    const float c1 = cheb ? __ldg(a.run.chebC) : 1.0f;
    const double mean =
        a.run.mean && (!a.run.useMean || *a.run.useMean) ? *a.run.mean : 0.0;
    unsigned int ep = *(volatile unsigned int*)a.epoch;
    if (tid == 0)
    {
        state_init(a, sh);
        zc[zs - 1] = zn[zs - 1] = pb[zs - 1] = 0.0f;
    }
    int hs[RES_HQ];
#pragma unroll
    for (int q = 0; q < RES_HQ; ++q)
        hs[q] = tid + q * T < P.nh ? a.haloSlot[P.haloBase + tid + q * T] : -1;
    for (int h = tid; h < P.nh; h += T) pb[P.nlocP + h] = 0.0f;
    for (int l = P.nloc + tid; l < P.nlocP; l += T) zc[l] = zn[l] = pb[l] = 0.0f;

    constexpr int RMA = RM > 0 ? RM : 1;
    constexpr int RK = LEAN ? 1 : R;
    unsigned int ix[RMA][(W + 1) / 2];
    float v[RMA][W];
    float dg[R], rd[R], r[R], w[R];
    float z[RK], d[RK];
    double accR = 0.0;
    double accZ = 0.0;
    u64* lw = a.ll;               // words of the next exchange
    u64* lr = a.ll + a.slots;     // words of the last one
    u64* redA = a.red;            // {sum|r|, z.r}
    u64* redB = a.red + RES_RED_WORDS;   // p.q
    float* dcur = a.dc + P.rowBase;      // delta of a row when it is not in a register
    ++ep;
#pragma unroll
    for (int i = 0; i < R; ++i)
    {
        const int l = tid + i * T;
        const int g = l < P.nlocP ? a.rowMap[P.rowBase + l] : -1;
        dg[i] = rd[i] = r[i] = w[i] = 0.0f;
        if (!LEAN) z[LEAN ? 0 : i] = d[LEAN ? 0 : i] = 0.0f;
        const long long sb = ((long long)P.rowBase + (l & ~31)) * W;
        if (i < RM)
        {
#pragma unroll
            for (int k = 0; k < (W + 1) / 2; ++k)
                ix[i < RM ? i : 0][k] = (unsigned)(zs - 1) * 0x10001u;
#pragma unroll
            for (int k = 0; k < W; ++k) v[i < RM ? i : 0][k] = 0.0f;
            if (g >= 0)
            {
                row_index<W>(a.idx, sb, l & 31, ix[i < RM ? i : 0]);
#pragma unroll
                for (int k = 0; k < W; ++k)
                {
                    const int e = a.emap[pair_index(sb, W, k, l & 31)];
                    v[i < RM ? i : 0][k] = e >= 0 ? a.run.val32[e] : 0.0f;
                }
            }
        }
        else if (l < P.nlocP)
        {
            const int at0 = ((l - m0) & ~31) * W;
#pragma unroll
            for (int k = 0; k < W; ++k)
            {
                const int o = (int)pair_index(0, W, k, l & 31);
                const int e = a.emap[sb + o];
                sval[at0 + o] = e >= 0 ? a.run.val32[e] : 0.0f;
                sidx[at0 + o] = a.idx[sb + o];
            }
        }
        if (g < 0) continue;
        dg[i] = a.run.diag32[g];
        rd[i] = a.run.rD32[g];
        const float ra = (float)(a.run.r64[g] - mean);
        r[i] = ra;
        const float z0 = cheb ? __fmul_rn(__fmul_rn(c1, rd[i]), ra) : __fmul_rn(ra, rd[i]);
        w[i] = z0;
        if (LEAN)
            dcur[l] = 0.0f;
        else
            z[LEAN ? 0 : i] = z0;
        if (!cheb) accZ += (double)z0 * (double)ra;
        zc[l] = z0;
        pb[l] = 0.0f;
        if (l < P.nb) st_word(lw + P.llBase + l, __float_as_uint(z0), ep);
    }
    __syncthreads();
    swap_ptr(lw, lr);
    // one row of A x plus acc
    auto row = [&](int i, int l, const float* x, float acc) -> float {
        if (i < RM) return row_apply<W>(ix[i < RM ? i : 0], v[i < RM ? i : 0], x, acc);
        unsigned int jx[(W + 1) / 2];
        float u[W];
        const int sb = ((l - m0) & ~31) * W;
        const int lane = l & 31;
#pragma unroll
        for (int g = 0; g < W / 2; ++g)
        {
            jx[g] = *reinterpret_cast<const unsigned int*>(sidx + sb + 64 * g + 2 * lane);
            const float2 t = *reinterpret_cast<const float2*>(sval + sb + 64 * g + 2 * lane);
            u[2 * g] = t.x;
            u[2 * g + 1] = t.y;
        }
        if constexpr (W & 1)
        {
            jx[W / 2] = sidx[sb + 32 * (W - 1) + lane];
            u[W - 1] = sval[sb + 32 * (W - 1) + lane];
        }
        return row_apply<W>(jx, u, x, acc);
    };
    // from here on exchange `ep` (words lr) carries the current z
    bool first = true;
    double wArA = 0.0;
    for (;;)
    {
        if (cheb) accZ = 0.0;
        for (int j = 1; j < a.run.order; ++j)
        {
            const float c2 = __ldg(a.run.chebC + 2 * j - 1);
            const float c3 = __ldg(a.run.chebC + 2 * j);
            halo_recv(a, P, hs, lr, ep, zc, sh, tid, T);
            __syncthreads();
            ++ep;
            const bool last = j == a.run.order - 1;
            if constexpr (!LEAN)
            {
                // (rows past the part's end hold zeros and need no test)
#pragma unroll
                for (int i = 0; i < R; ++i)
                {
                    const float av = row(i, tid + i * T, zc, __fmul_rn(dg[i], z[i]));
                    w[i] = __fadd_rn(__fmul_rn(c2, w[i]),
                                     __fmul_rn(__fmul_rn(c3, rd[i]), __fsub_rn(r[i], av)));
                    z[i] = __fadd_rn(z[i], w[i]);
                    if (tid + i * T < P.nb)
                        st_word(lw + P.llBase + tid + i * T, __float_as_uint(z[i]), ep);
                    if (i < RB) __syncwarp();
                }
#pragma unroll
                for (int i = 0; i < R; ++i)
                {
                    if (tid + i * T < P.nloc) zn[tid + i * T] = z[i];
                    if (last) accZ += (double)z[i] * (double)r[i];
                }
            }
            else
            {
#pragma unroll
                for (int i0 = 0; i0 < R; i0 += 4)
                {
                    float zv[4];
#pragma unroll
                    for (int i = i0; i < i0 + 4 && i < R; ++i)
                    {
                        const int l = tid + i * T;
                        if (l >= P.nloc) continue;
                        const float zl = zc[l];
                        const float av = row(i, l, zc, __fmul_rn(dg[i], zl));
                        const float wn = __fadd_rn(
                            __fmul_rn(c2, w[i]), __fmul_rn(__fmul_rn(c3, rd[i]), __fsub_rn(r[i], av)));
                        zv[i - i0] = __fadd_rn(zl, wn);
                        w[i] = wn;
                        if (l < P.nb) st_word(lw + P.llBase + l, __float_as_uint(zv[i - i0]), ep);
                        if (last) accZ += (double)zv[i - i0] * (double)r[i];
                    }
#pragma unroll
                    for (int i = i0; i < i0 + 4 && i < R; ++i)
                        if (tid + i * T < P.nloc) zn[tid + i * T] = zv[i - i0];
                }
            }
            swap_ptr(lw, lr);
            swap_ptr(zc, zn);
        }
        // all-gather of {sum|r|, z.r}; the halo of z meanwhile
        {
            double acc[2] = {accR, accZ};
            red_send<2>(acc, redA, rank, ep, sh, tid, T);
            halo_recv(a, P, hs, lr, ep, zc, sh, tid, T);
            red_recv<2>(a, redA, rank, ep, sh, tid, T);
            __syncthreads();
        }
        const double zr = red_total(a, sh, 1, T);
        const float beta = first ? 0.0f : (float)(zr / wArA);
        wArA = zr;
        const double rsum = red_total(a, sh, 0, T);
        // p = z + beta p (own rows and halo), q = A p (kept in the free z
        // buffer when it is not kept in a register)
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const int l = tid + i * T;
            if (l >= P.nloc) continue;
            pb[l] = __fadd_rn(LEAN ? zc[l] : z[LEAN ? 0 : i], __fmul_rn(beta, pb[l]));
        }
        for (int h = P.nlocP + tid; h < P.nlocP + P.nh; h += T)
            pb[h] = __fadd_rn(zc[h], __fmul_rn(beta, pb[h]));
        __syncthreads();
        ++ep;
        double acc[1] = {0.0};
        float q[RK];
        if constexpr (!LEAN)
        {
#pragma unroll
            for (int i = 0; i < R; ++i)
            {
                const float pr = pb[min(tid + i * T, zs - 1)];
                q[i] = row(i, tid + i * T, pb, __fmul_rn(dg[i], pr));
                acc[0] += (double)pr * (double)q[i];
            }
        }
        else
        {
#pragma unroll
            for (int i0 = 0; i0 < R; i0 += 4)
            {
                float qv[4];
#pragma unroll
                for (int i = i0; i < i0 + 4 && i < R; ++i)
                {
                    const int l = tid + i * T;
                    if (l >= P.nloc) continue;
                    const float pr = pb[l];
                    qv[i - i0] = row(i, l, pb, __fmul_rn(dg[i], pr));
                    acc[0] += (double)pr * (double)qv[i - i0];
                }
#pragma unroll
                for (int i = i0; i < i0 + 4 && i < R; ++i)
                    if (tid + i * T < P.nloc) zn[tid + i * T] = qv[i - i0];
            }
        }
        {
            red_send<1>(acc, redB, rank, ep, sh, tid, T);
            // the bookkeeping of the update before, while p.q is on its way
            if (tid == T - 1) 
            {
                inner_after_apply(sh.S, first, rsum, wArA);
                sh.stop = sh.S.done || sh.bad;
            }
            red_recv<1>(a, redB, rank, ep, sh, tid, T);
            __syncthreads();
            first = false;
        }
        if (sh.stop) break;
        const double pq = red_total(a, sh, 0, T);
        const float alpha = (float)(wArA / pq);
        if (tid == T - 1) sh.S.wApA = pq;
        const int nxt = sh.S.nxt;
        ++ep;
        accR = accZ = 0.0;
        float* dn = a.dw + (size_t)nxt * a.rowsP + P.rowBase;
#pragma unroll
        for (int i0 = 0; i0 < R; i0 += 4)
        {
            float dd[4];
            if (LEAN)
            {
#pragma unroll
                for (int i = i0; i < i0 + 4 && i < R; ++i)
                    dd[i - i0] = tid + i * T < P.nloc ? dcur[tid + i * T] : 0.0f;
            }
#pragma unroll
            for (int i = i0; i < i0 + 4 && i < R; ++i)
            {
                const int l = tid + i * T;
                if (l >= P.nloc) continue;
                const float rn = __fsub_rn(r[i], __fmul_rn(alpha, LEAN ? zn[l] : q[LEAN ? 0 : i]));
                const float z0 = cheb ? __fmul_rn(__fmul_rn(c1, rd[i]), rn) : __fmul_rn(rn, rd[i]);
                if (l < P.nb) st_word(lw + P.llBase + l, __float_as_uint(z0), ep);
                zc[l] = z0;
                const float dv = __fadd_rn(LEAN ? dd[i - i0] : d[LEAN ? 0 : i],
                                           __fmul_rn(alpha, pb[l]));
                dn[l] = dv;
                if (LEAN)
                    dcur[l] = dv;
                else
                    d[LEAN ? 0 : i] = dv;
                r[i] = rn;
                w[i] = z0;
                if (!LEAN) z[LEAN ? 0 : i] = z0;
                accR += (double)fabsf(rn);
                if (!cheb) accZ += (double)z0 * (double)rn;
            }
        }
        swap_ptr(lw, lr);
    }
    if (tid == T - 1) inner_finish(sh.S, a.run.st, rank == 0);
    __syncthreads();
    const int sel = sh.S.sel;
    const float* ds = a.dw + (size_t)sel * a.rowsP + P.rowBase;
    float* out = a.run.D + (size_t)sel * a.run.dStride;
#pragma unroll
    for (int i = 0; i < R; ++i)
    {
        const int l = tid + i * T;
        // (before the first update no correction has been written: 0)
        if (l < P.nloc) out[a.rowMap[P.rowBase + l]] = sh.S.it > 0 ? ds[l] : 0.0f;
    }
    if (rank == 0 && tid == 0) *a.epoch = ep;
}

// ------------------------------------------------------------------- host

std::mutex g_resident[64];
std::atomic<int> g_inFlight[64];

// The kernels: R rows per thread, RM of them with their matrix entries in
// registers, at most TB threads.  In order of preference; the first whose
// rows and shared memory suffice is taken.
struct ChipKernel
{
    int R, RM, TB;
    const void* fn[3];   // W = 4, 5, 6
};
#define RES_CHIP(R, RM, TB)                                                              \
    {                                                                                    \
        R, RM, TB,                                                                       \
        {                                                                                \
            (const void*)k_res_chip<4, R, RM, TB>, (const void*)k_res_chip<5, R, RM, TB>, \
                (const void*)k_res_chip<6, R, RM, TB>                                    \
        }                                                                                \
    }
const ChipKernel CHIP[] = {
    RES_CHIP(1, 1, 256),  RES_CHIP(2, 2, 256),  RES_CHIP(3, 3, 256), RES_CHIP(4, 4, 256),
    RES_CHIP(5, 5, 256),  RES_CHIP(6, 6, 256),  RES_CHIP(7, 7, 256), RES_CHIP(8, 8, 256),
    RES_CHIP(9, 9, 256),  RES_CHIP(10, 10, 256), RES_CHIP(6, 4, 512), RES_CHIP(8, 4, 512),
    RES_CHIP(10, 5, 512), RES_CHIP(12, 5, 512)};

template <class T>
int up(ResPlan* p, T** d, const T* h, size_t count, cudaStream_t s)
{
    RES_CUDA(cudaMalloc((void**)d, std::max<size_t>(count, 1) * sizeof(T)));
    p->allocs.push_back((void*)*d);
    if (h && count)
        RES_CUDA(cudaMemcpyAsync(*d, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
    return CF_OK;
}

}  // namespace

std::mutex& res_device_lock(int device) { return g_resident[device & 63]; }
std::atomic<int>& res_in_flight(int device) { return g_inFlight[device & 63]; }

void res_plan_free(ResPlan* p)
{
    if (!p) return;
    for (void* q : p->allocs) cudaFree(q);
    delete p;
}

int res_reset(const ResPlan* p, cudaStream_t s)
{
    RES_CUDA(cudaMemsetAsync(p->ll, 0, sizeof(u64) * 2 * (size_t)std::max(p->slots, 1), s));
    RES_CUDA(cudaMemsetAsync(p->red, 0, sizeof(u64) * 2 * RES_RED_WORDS, s));
    RES_CUDA(cudaMemsetAsync(p->epoch, 0, sizeof(unsigned int), s));
    return CF_OK;
}

int res_plan_build(int device, int n, const HostLayout& L, bool ordered, int nparts,
                   long long entOff, int rowOff, cudaStream_t s, ResPlan** plan)
{
    *plan = nullptr;
    if (L.maxw > 6 || nparts < 1 || nparts > RES_MAX_PARTS ||
        n > (long long)nparts * RES_MAX_ROWS)
        return CF_OK;
    ResHost H;
    ResPlan* p = nullptr;
    try
    {
        if (!res_partition(n, L, ordered, nparts, H, 4)) return CF_OK;
        if (entOff)
            for (int32_t& e : H.emap)
                if (e >= 0) e += (int32_t)entOff;
        if (rowOff)
            for (int32_t& r : H.rowMap)
                if (r >= 0) r += rowOff;
        p = new ResPlan();
        p->allocs.reserve(16);
    }
    catch (...)
    {
        res_plan_free(p);
        return CF_OK;   // no memory for the split
    }
    p->nparts = nparts;
    p->W = H.W;
    p->slots = H.slots;
    p->rowsP = H.rowsP;
    p->maxHalo = H.maxHalo;
    int maxSmem = 0;
    if (cudaDeviceGetAttribute(&maxSmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) !=
        cudaSuccess)
        maxSmem = 0;
    // z (two buffers) and p; the parts differ in their halo, so the largest
    size_t zf = 0;
    for (const ResPart& q : H.parts) zf = std::max(zf, (size_t)3 * (q.nlocP + q.nh + 1) + 1);
    const size_t zbytes = sizeof(float) * ((zf + 1) & ~(size_t)1);
    const size_t avail = (size_t)std::max(maxSmem - 2048, 0);   // static shared state
    for (const ChipKernel& k : CHIP)
    {
        if (H.maxLocP > k.R * k.TB) continue;
        const int threads = ((H.maxLocP + k.R - 1) / k.R + 31) / 32 * 32;
        const size_t mrows = (size_t)std::max(0, H.maxLocP - k.RM * threads);
        const size_t smem = zbytes + mrows * H.W * 6;
        if (smem > avail) continue;
        p->R = k.R;
        p->TB = k.TB;
        p->threads = threads;
        p->smem = smem;
        p->fn = k.fn[H.W - 4];
        break;
    }
    // (the attribute: one value for every context of the process, so a solve
    // on another thread never lowers it under a launch)
    int occ = 0;
    if (!p->fn ||
        cudaFuncSetAttribute(p->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)avail) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, p->fn, p->threads, p->smem) !=
            cudaSuccess ||
        occ < 1)
    {
        cudaGetLastError();
        res_plan_free(p);
        return CF_OK;
    }
    int rc = up(p, &p->parts, H.parts.data(), H.parts.size(), s);
    if (rc == CF_OK) rc = up(p, &p->rowMap, H.rowMap.data(), H.rowMap.size(), s);
    if (rc == CF_OK) rc = up(p, &p->idx, (const unsigned short*)H.idx.data(), H.idx.size(), s);
    if (rc == CF_OK) rc = up(p, &p->emap, H.emap.data(), H.emap.size(), s);
    if (rc == CF_OK) rc = up(p, &p->haloSlot, H.haloSlot.data(), H.haloSlot.size(), s);
    if (rc == CF_OK) rc = up<u64>(p, &p->ll, nullptr, 2 * (size_t)H.slots, s);
    if (rc == CF_OK) rc = up<u64>(p, &p->red, nullptr, 2 * RES_RED_WORDS, s);
    if (rc == CF_OK) rc = up<unsigned int>(p, &p->epoch, nullptr, 1, s);
    if (rc == CF_OK) rc = up<float>(p, &p->dw, nullptr, 3 * (size_t)H.rowsP, s);
    if (rc == CF_OK && p->R * p->TB > 2560)
        rc = up<float>(p, &p->dc, nullptr, (size_t)H.rowsP, s);
    if (rc == CF_OK) rc = res_reset(p, s);
    if (rc == CF_OK && cudaStreamSynchronize(s) != cudaSuccess)   // the host arrays end here
        rc = fail(CF_ERR_CUDA, "split over the SMs: upload");
    if (rc != CF_OK)
    {
        res_plan_free(p);
        return rc;
    }
    *plan = p;
    return CF_OK;
}

int res_launch(const ResPlan* p, const InnerRun& run, cudaStream_t s)
{
    ResArgs a;
    a.parts = p->parts;
    a.nparts = p->nparts;
    a.rowMap = p->rowMap;
    a.idx = p->idx;
    a.emap = p->emap;
    a.haloSlot = p->haloSlot;
    a.ll = p->ll;
    a.slots = p->slots;
    a.red = p->red;
    a.epoch = p->epoch;
    a.dw = p->dw;
    a.dc = p->dc;
    a.rowsP = p->rowsP;
    a.run = run;
    a.run.polls = std::min(run.polls, 1LL << 22);
    void* args[] = {(void*)&a};
    const cudaError_t e = cudaLaunchCooperativeKernel(p->fn, dim3(p->nparts), dim3(p->threads),
                                                      args, p->smem, s);
    if (e != cudaSuccess)
        return fail(CF_ERR_CUDA, std::string("cudaLaunchCooperativeKernel: ") + cudaGetErrorString(e));
    return CF_OK;
}

InnerRun inner_run(const cf_context* c, const double* mean, double target, int maxIter, int ips,
                   int order, int stagLimit)
{
    InnerRun r;
    r.val32 = c->d_val32;
    r.diag32 = c->d_diag32;
    r.rD32 = c->d_rD32;
    r.chebC = c->d_chebC;
    r.r64 = c->d_r64;
    r.mean = mean;
    r.useMean = nullptr;
    r.D = c->d_D;
    r.dStride = c->n;
    r.st = c->d_st;
    r.fromState = 0;
    r.order = order;
    r.target = target;
    r.maxIter = maxIter;
    r.ips = ips;
    r.stagLimit = stagLimit;
    r.polls = c->waitPolls;
    return r;
}

void resident_release(cf_context* c)
{
    res_plan_free(static_cast<ResPlan*>(c->resident));
    c->resident = nullptr;
    c->residentTried = false;
}

namespace {

void resident_build(cf_context* c)
{
    const int nparts = std::min(c->numSMs, RES_MAX_PARTS);
    if (!c->coopLaunch || c->n > (long long)nparts * RES_MAX_ROWS || c->hostSliceOff.empty()) return;
    ResPlan* p = nullptr;
    {
        const LentLayout lent(c);
        if (res_plan_build(c->device, c->n, lent.L, !c->identityPerm, nparts, 0, 0, c->stream,
                           &p) != CF_OK)
            cudaGetLastError();   // no memory for the split: the graph path
    }
    if (p && p->maxHalo > SPLIT_MAX_HALO)
    {
        res_plan_free(p);
        p = nullptr;
    }
    c->resident = p;
}

}  // namespace

int resident_inner(cf_context* c, const double* mean, double target, int maxIter, int ips,
                   int order, int stagLimit, bool* ran)
{
    *ran = false;
    if (maxIter <= 0 || c->solves < RESIDENT_AFTER_SOLVES ||
        c->n < RESIDENT_MIN_ROWS_PER_SM * c->numSMs || c->maxRowLen < 4)
        return CF_OK;
    if (c->concurrent >= RESIDENT_BESIDE && c->n > RESIDENT_BESIDE_MIN * c->numSMs &&
        c->n <= RESIDENT_BESIDE_MAX * c->numSMs)
        return CF_OK;
    if (!c->residentTried)
    {
        c->residentTried = true;
        resident_build(c);
    }
    const ResPlan* p = static_cast<const ResPlan*>(c->resident);
    if (!p) return CF_OK;
    std::lock_guard<std::mutex> turn(res_device_lock(c->device));
    cudaStream_t s = c->stream;
    const int rc = res_launch(p, inner_run(c, mean, target, maxIter, ips, order, stagLimit), s);
    if (rc != CF_OK) return rc;
    c->launches++;
    // the device is taken until the launch has ended
    RES_CUDA(cudaEventRecord(c->ev1, s));
    RES_CUDA(cudaMemcpyAsync(c->h_st, c->d_st, sizeof(InnerState), cudaMemcpyDeviceToHost, s));
    RES_CUDA(cudaStreamSynchronize(s));
    if (c->h_st->waitErr)
    {
        // a wait gave up: this solve goes through the graph path
        const int rr = res_reset(p, s);
        if (rr != CF_OK) return rr;
        RES_CUDA(cudaMemsetAsync(&c->d_st->waitErr, 0, sizeof(int), s));
        c->backoff.gaveUp();
        return CF_OK;
    }
    c->backoff.worked();
    *ran = true;
    return CF_OK;
}

}  // namespace cf
