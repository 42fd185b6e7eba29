// cf_clupcg.cu -- the inner PCG of a small mesh inside ONE thread-block
// cluster of up to 16 CTAs.
//
// Every CTA owns one part of the mesh (cf_partition.cu); its matrix entries
// and row-private vectors stay in registers (256 threads of up to 10 rows), z
// and p in shared memory.  A row that other CTAs read is stored into their
// shared memory as a {value, epoch} word (cf_cluster_ll.cuh) and they poll
// their own memory for it, so a Chebyshev step has no cluster barrier and no
// global access.  p of the halo rows is advanced locally; each of the two
// reductions per iteration pushes one FP64 partial per CTA to every CTA, and
// all fold them in rank order.  The structure and the arithmetic per row are
// cf_resident.cu's, with the trip through L2 replaced; several systems run as
// several clusters of one launch.
//
// Measured on one box, us per inner iteration, graph loop / the cluster
// kernel before it (cf_cluster.cu, distributed shared memory read in place
// and a cluster barrier per phase) / this one: 128^2 Poisson, Chebyshev 4,
// 22.2 / 14.7 / 4.7; 3,000 cells 2-D 27.5 / - / 5.9; 12K 3-D 30.6 / - / 8.5;
// 24K 3-D 31.2 / - / 12.1 (15.7 split over all SMs); 32K 2-D 31.9 / - / 9.3;
// Jacobi, 9,000 cells 13.1 / - / 2.4.  39K 3-D takes 19.4 (split over all
// SMs: 16), so the mesh may have up to CLU_MAX_ENTRIES entries.
//
// A word of an exchange may be overwritten by the exchange after next: its
// owner has then received the exchange in between from every row that reads
// it (the matrix pattern is symmetric), and those rows sent it after reading.
#include "cudafoam.h"
#include "cf_cluster_ll.cuh"
#include "cf_host.hpp"
#include "cf_inner.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

using namespace cf;
namespace cg = cooperative_groups;

#define CLU_CUDA(call)                                                          \
    do                                                                          \
    {                                                                           \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess)                                                  \
            return fail(CF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

namespace cf {

namespace {

constexpr int CLU_T = 256;          // threads per CTA at most
constexpr int CLU_MAX_ENTRIES = 163840;   // rows x entries per row at most
constexpr int CLU_MAX_R = 10;       // rows per thread at most
constexpr int RB = 4;               // rows of a thread finished and pushed one after the other
constexpr int CLU_SMEM = 200 * 1024;   // dynamic shared memory at most

struct CluShared
{
    double red[2][CLU_T / 32];
    u64 words[2][CLU_MAX_CTAS][4];   // [A / B][sender][2 values x 2 words]
    double tot[2];
    int stop, bad;
    InnerState S;
};

struct CluArgs
{
    const CluSys* list;   // the systems of the launch, or null: `one`
    CluSys one;
};

// Sums of v[0..NR) over the CTA, pushed to every CTA of the cluster.
template <int NR>
__device__ __forceinline__ void clu_send(double (&v)[NR], int which, int rank, int ctas,
                                         unsigned int epoch, CluShared& sh, int tid, int T)
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
    if (wid == 0 && lane < ctas)
    {
        const unsigned int at = remote_addr(smem_addr(&sh.words[which][rank][0]), lane);
#pragma unroll
        for (int r = 0; r < NR; ++r)
        {
            double p[CLU_T / 32];
#pragma unroll
            for (int w = 0; w < CLU_T / 32; ++w) p[w] = w < (T >> 5) ? sh.red[r][w] : 0.0;
            const double t = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
            const u64 b = (u64)__double_as_longlong(t);
            st_remote(at + 16 * r, (unsigned int)b, epoch);
            st_remote(at + 16 * r + 8, (unsigned int)(b >> 32), epoch);
        }
    }
}

// One warp gathers the partials (polled by all warps, the shared-memory
// traffic of the polls kept the words they wait for out for thousands of
// cycles); the totals are in sh.tot after the next barrier.
template <int NR>
__device__ __forceinline__ void clu_recv(int which, int ctas, unsigned int epoch, CluShared& sh,
                                         int tid, long long polls)
{
    if (tid >= 32) return;
    const int lane = tid;
    double tot[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) tot[r] = 0.0;
    if (lane < ctas)
    {
        const unsigned int at = smem_addr(&sh.words[which][lane][0]);
#pragma unroll
        for (int r = 0; r < NR; ++r)
        {
            const u64 lo = wait_local(at + 16 * r, epoch, &sh.bad, polls);
            const u64 hi = wait_local(at + 16 * r + 8, epoch, &sh.bad, polls);
            tot[r] = __longlong_as_double((long long)((hi << 32) | lo));
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
    {
#pragma unroll
        for (int o = CLU_MAX_CTAS / 2; o > 0; o >>= 1)
            tot[r] += __shfl_xor_sync(0xffffffffu, tot[r], o);
        if (lane == 0) sh.tot[r] = tot[r];
    }
}

template <int W, int R>
__global__ void __launch_bounds__(CLU_T, 1) k_clu_pcg(const __grid_constant__ CluArgs a)
{
    extern __shared__ float zmem[];
    __shared__ CluShared sh;
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x;
    const int T = blockDim.x;
    const int ctas = (int)cl.num_blocks();
    const int rank = (int)cl.block_rank();
    const CluSys& Y = a.list ? a.list[blockIdx.x / ctas] : a.one;
    const InnerRun& N = Y.run;
    if (N.fromState && N.st->done) return;   // (the whole cluster)
    const CluSplit& C = Y.split;
    const ResPart P = C.parts[rank];
    const int locP = C.locP;
    const int zs = locP + 2 * C.halo + 2;    // floats of one buffer (even)
    float* zc = zmem;          // current z
    float* zn = zmem + zs;     // the next
    float* pb = zmem + 2 * zs;
    const bool cheb = N.order > 1;
    const float c1 = cheb ? __ldg(N.chebC) : 1.0f;
    const double mean = N.mean && (!N.useMean || *N.useMean) ? *N.mean : 0.0;
    if (tid == 0)
    {
        if (N.fromState)
            inner_state_init(sh.S, N.st->target, N.st->maxIter, N.st->ips, N.st->stagLimit);
        else
            inner_state_init(sh.S, N.target, N.maxIter, N.ips, N.stagLimit);
        sh.stop = sh.bad = 0;
    }
    for (int i = tid; i < 2 * CLU_MAX_CTAS * 4; i += T) (&sh.words[0][0][0])[i] = 0;
    // rows past the part's end, halo words (epoch 0), the slots that hold 0
    for (int i = P.nloc + tid; i < zs; i += T) zc[i] = zn[i] = pb[i] = 0.0f;
    unsigned int ix[R][(W + 1) / 2];
    unsigned int dst[R][2];
    float v[R][W], dg[R], rd[R], r[R], w[R], z[R], d[R];
    double accR = 0.0;
    double accZ = 0.0;
    unsigned int ep = 1;
#pragma unroll
    for (int i = 0; i < R; ++i)
    {
        const int l = tid + i * T;
        const int g = l < P.nlocP ? C.rowMap[P.rowBase + l] : -1;
        dg[i] = rd[i] = r[i] = w[i] = z[i] = d[i] = 0.0f;
        dst[i][0] = dst[i][1] = CLU_NONE;
#pragma unroll
        for (int k = 0; k < (W + 1) / 2; ++k) ix[i][k] = (unsigned)(zs - 2) * 0x10001u;
#pragma unroll
        for (int k = 0; k < W; ++k) v[i][k] = 0.0f;
        if (g < 0) continue;
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
            if (q < C.ndest) dst[i][q] = C.dest[(size_t)q * C.rowsP + P.rowBase + l];
        dg[i] = N.diag32[g];
        rd[i] = N.rD32[g];
        const float ra = (float)(N.r64[g] - mean);
        r[i] = ra;
        z[i] = w[i] = cheb ? __fmul_rn(__fmul_rn(c1, rd[i]), ra) : __fmul_rn(ra, rd[i]);
        if (!cheb) accZ += (double)z[i] * (double)ra;
        zc[l] = z[i];
        pb[l] = 0.0f;
    }
    // x of row i (local row l) to the CTAs that read it, into their words of
    // the buffer at `buf`
    auto push = [&](int i, int l, unsigned int buf, float x) {
        if (dst[i][0] == CLU_NONE) return;
        st_remote(remote_addr(buf + 8 * (dst[i][0] & 0xffffu), dst[i][0] >> 16),
                  __float_as_uint(x), ep);
        if (dst[i][1] == CLU_NONE) return;
        st_remote(remote_addr(buf + 8 * (dst[i][1] & 0xffffu), dst[i][1] >> 16),
                  __float_as_uint(x), ep);
        for (int q = 2; q < C.ndest; ++q)
        {
            const unsigned int t = __ldg(C.dest + (size_t)q * C.rowsP + P.rowBase + l);
            if (t == CLU_NONE) break;
            st_remote(remote_addr(buf + 8 * (t & 0xffffu), t >> 16), __float_as_uint(x), ep);
        }
    };
    auto halo_wait = [&]() {
        const unsigned int at = smem_addr(zc + locP);
        for (int h = tid; h < P.nh; h += T) wait_local(at + 8 * h, ep, &sh.bad, N.polls);
    };
    cl.sync();
#pragma unroll
    for (int i = 0; i < R; ++i) push(i, tid + i * T, smem_addr(zc + locP), z[i]);
    // from here on exchange `ep` carries the current z
    bool first = true;
    double wArA = 0.0;
    for (;;)
    {
        if (cheb) accZ = 0.0;
        for (int j = 1; j < N.order; ++j)
        {
            const float c2 = __ldg(N.chebC + 2 * j - 1);
            const float c3 = __ldg(N.chebC + 2 * j);
            halo_wait();
            __syncthreads();
            ++ep;
            const bool last = j == N.order - 1;
            const unsigned int buf = smem_addr(zn + locP);
            // (rows past the part's end hold zeros and need no test)
#pragma unroll
            for (int i = 0; i < R; ++i)
            {
                const float av = row_apply<W>(ix[i], v[i], zc, __fmul_rn(dg[i], z[i]));
                w[i] = __fadd_rn(__fmul_rn(c2, w[i]),
                                 __fmul_rn(__fmul_rn(c3, rd[i]), __fsub_rn(r[i], av)));
                z[i] = __fadd_rn(z[i], w[i]);
                if (i < RB)
                {
                    push(i, tid + i * T, buf, z[i]);
                    __syncwarp();
                }
            }
#pragma unroll
            for (int i = RB; i < R; ++i) push(i, tid + i * T, buf, z[i]);
#pragma unroll
            for (int i = 0; i < R; ++i)
            {
                if (tid + i * T < P.nloc) zn[tid + i * T] = z[i];
                if (last) accZ += (double)z[i] * (double)r[i];
            }
            float* t = zc;
            zc = zn;
            zn = t;
        }
        // all-gather of {sum|r|, z.r}; the halo of z meanwhile
        {
            double acc[2] = {accR, accZ};
            clu_send<2>(acc, 0, rank, ctas, ep, sh, tid, T);
            halo_wait();
            clu_recv<2>(0, ctas, ep, sh, tid, N.polls);
            __syncthreads();
        }
        const double zr = sh.tot[1];
        const double rsum = sh.tot[0];
        const float beta = first ? 0.0f : (float)(zr / wArA);
        wArA = zr;
        // p = z + beta p (own rows, and the halo values this thread has waited
        // for), q = A p
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const int l = tid + i * T;
            if (l < P.nloc) pb[l] = __fadd_rn(z[i], __fmul_rn(beta, pb[l]));
        }
        for (int h = tid; h < P.nh; h += T)
            pb[locP + 2 * h] = __fadd_rn(zc[locP + 2 * h], __fmul_rn(beta, pb[locP + 2 * h]));
        __syncthreads();
        ++ep;
        double acc[1] = {0.0};
        float q[R];
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const float pr = pb[min(tid + i * T, zs - 2)];
            q[i] = row_apply<W>(ix[i], v[i], pb, __fmul_rn(dg[i], pr));
            acc[0] += (double)pr * (double)q[i];
        }
        clu_send<1>(acc, 1, rank, ctas, ep, sh, tid, T);
        // the bookkeeping of the update before, while p.q is on its way
        if (tid == T - 1)
        {
            inner_after_apply(sh.S, first, rsum, wArA);
            sh.stop = sh.S.done || sh.bad;
        }
        clu_recv<1>(1, ctas, ep, sh, tid, N.polls);
        __syncthreads();
        first = false;
        if (sh.stop) break;
        const double pq = sh.tot[0];
        const float alpha = (float)(wArA / pq);
        if (tid == T - 1) sh.S.wApA = pq;
        float* dn = Y.dw + (size_t)sh.S.nxt * C.rowsP + P.rowBase;
        ++ep;
        accR = accZ = 0.0;
        const unsigned int buf = smem_addr(zc + locP);
#pragma unroll
        for (int i = 0; i < R; ++i)
        {
            const int l = tid + i * T;
            if (l >= P.nloc) continue;
            r[i] = __fsub_rn(r[i], __fmul_rn(alpha, q[i]));
            z[i] = w[i] =
                cheb ? __fmul_rn(__fmul_rn(c1, rd[i]), r[i]) : __fmul_rn(r[i], rd[i]);
            push(i, l, buf, z[i]);
            zc[l] = z[i];
            d[i] = __fadd_rn(d[i], __fmul_rn(alpha, pb[l]));
            dn[l] = d[i];
            accR += (double)fabsf(r[i]);
            if (!cheb) accZ += (double)z[i] * (double)r[i];
        }
    }
    if (tid == T - 1)
    {
        if (sh.bad) atomicExch(&N.st->waitErr, 1);
        inner_finish(sh.S, N.st, rank == 0);
    }
    __syncthreads();
    const int sel = sh.S.sel;
    const float* ds = Y.dw + (size_t)sel * C.rowsP + P.rowBase;
    float* out = N.D + (size_t)sel * N.dStride;
#pragma unroll
    for (int i = 0; i < R; ++i)
    {
        const int l = tid + i * T;
        // (before the first update no correction has been written: 0)
        if (l < P.nloc) out[C.rowMap[P.rowBase + l]] = sh.S.it > 0 ? ds[l] : 0.0f;
    }
    cl.sync();   // no CTA leaves while another may still store into it
}

template <int W>
const void* kernel_r(int R)
{
    switch (R)
    {
        case 1: return (const void*)k_clu_pcg<W, 1>;
        case 2: return (const void*)k_clu_pcg<W, 2>;
        case 3: return (const void*)k_clu_pcg<W, 3>;
        case 4: return (const void*)k_clu_pcg<W, 4>;
        case 6: return (const void*)k_clu_pcg<W, 6>;
        case 8: return (const void*)k_clu_pcg<W, 8>;
        case 10: return (const void*)k_clu_pcg<W, 10>;
    }
    return nullptr;
}

const void* kernel_of(int W, int R)
{
    return W == 4 ? kernel_r<4>(R) : W == 5 ? kernel_r<5>(R) : kernel_r<6>(R);
}

// Arrays packed into one device allocation and one copy (a split is made by
// the first solve that uses it).
struct Pack
{
    std::vector<char> host;
    template <class T>
    size_t add(const T* h, size_t count)
    {
        const size_t at = (host.size() + 255) & ~(size_t)255;
        host.resize(at + count * sizeof(T));
        if (h && count) memcpy(host.data() + at, h, count * sizeof(T));
        return at;
    }
};

void config(int ctas, int threads, size_t smem, int count, cudaStream_t s, cudaLaunchConfig_t* cfg,
            cudaLaunchAttribute* attr)
{
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)ctas;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    *cfg = {};
    cfg->gridDim = dim3((unsigned)(ctas * count));
    cfg->blockDim = dim3((unsigned)threads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = s;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

}  // namespace

void clu_plan_free(CluPlan* p)
{
    if (!p) return;
    for (void* q : p->allocs) cudaFree(q);
    delete p;
}

int clu_plan_build(int n, const HostLayout& L, bool ordered, int ctas, long long entOff,
                   int rowOff, cudaStream_t s, CluPlan** plan)
{
    *plan = nullptr;
    if (L.maxw > 6 || n < 1) return CF_OK;
    ctas = std::max(1, std::min({ctas, CLU_MAX_CTAS, n}));
    if (n > (long long)ctas * CLU_T * CLU_MAX_R ||
        (long long)n * std::max(4, (int)L.maxw) > CLU_MAX_ENTRIES)
        return CF_OK;
    ResHost H;
    try
    {
        if (!res_partition(n, L, ordered, ctas, H, 4)) return CF_OK;
    }
    catch (...)
    {
        return CF_OK;   // no memory for the split
    }
    int rows = 1;
    for (int R : {1, 2, 3, 4, 6, 8, 10})
    {
        rows = R;
        if (H.maxLocP <= R * CLU_T) break;
    }
    const int threads = ((H.maxLocP + rows - 1) / rows + 31) / 32 * 32;
    return clu_plan_upload(H, ctas, 3, 3, entOff, rowOff, kernel_of(H.W, rows), rows, threads, s,
                           plan);
}

int clu_plan_upload(ResHost& H, int ctas, int buffers, int nd, long long entOff, int rowOff,
                    const void* fn, int R, int threads, cudaStream_t s, CluPlan** plan)
{
    *plan = nullptr;
    const int W = H.W;
    const int halo = std::max(H.maxHalo, 1);
    std::vector<unsigned int> dest;
    CluPlan* p = nullptr;
    int ndest = 0;
    try
    {
        // readers of every row that has some
        std::vector<int> slotRow(H.slots), count(H.slots, 0);
        for (const ResPart& q : H.parts)
            for (int l = 0; l < q.nb; ++l) slotRow[q.llBase + l] = q.rowBase + l;
        for (int t : H.haloSlot) ndest = std::max(ndest, ++count[t]);
        dest.assign((size_t)ndest * H.rowsP, CLU_NONE);
        std::fill(count.begin(), count.end(), 0);
        for (int c = 0; c < ctas; ++c)
            for (int h = 0; h < H.parts[c].nh; ++h)
            {
                const int t = H.haloSlot[H.parts[c].haloBase + h];
                dest[(size_t)count[t]++ * H.rowsP + slotRow[t]] = ((unsigned)c << 16) | (unsigned)h;
            }
        // columns in the common layout
        const int zero = H.maxLocP + 2 * halo;
        if (zero > 65535 || halo > CLU_MAX_HALO) return CF_OK;
        for (const ResPart& q : H.parts)
            for (long long e = (long long)q.rowBase * W; e < ((long long)q.rowBase + q.nlocP) * W; ++e)
            {
                const int x = H.idx[e];
                if (x >= q.nlocP + q.nh)
                    H.idx[e] = (uint16_t)zero;
                else if (x >= q.nlocP)
                    H.idx[e] = (uint16_t)(H.maxLocP + 2 * (x - q.nlocP));
            }
        for (int32_t& e : H.emap)
            if (e >= 0) e += (int32_t)entOff;
        for (int32_t& r : H.rowMap)
            if (r >= 0) r += rowOff;
        p = new CluPlan();
        p->allocs.reserve(1);
    }
    catch (...)
    {
        clu_plan_free(p);
        return CF_OK;   // no memory for the split
    }
    p->W = W;
    p->R = R;
    p->fn = fn;
    p->threads = threads;
    p->smem = sizeof(float) * buffers * (size_t)(H.maxLocP + 2 * halo + 2);
    p->split.rowsP = H.rowsP;
    p->split.ndest = ndest;
    p->split.ctas = ctas;
    p->split.locP = H.maxLocP;
    p->split.halo = halo;
    // the attributes are the function's, shared by every context of the
    // process: one value, so no solve lowers it under another's launch
    int clusters = 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(ctas, p->threads, p->smem, 1, s, &cfg, &attr);
    if (p->smem > (size_t)CLU_SMEM ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, CLU_SMEM) !=
            cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess || clusters < 1)
    {
        cudaGetLastError();
        clu_plan_free(p);
        return CF_OK;
    }
    Pack k;
    size_t at[5] = {};
    try
    {
        at[0] = k.add(H.parts.data(), H.parts.size());
        at[1] = k.add(H.rowMap.data(), H.rowMap.size());
        at[2] = k.add(H.idx.data(), H.idx.size());
        at[3] = k.add(H.emap.data(), H.emap.size());
        at[4] = k.add(dest.data(), dest.size());
    }
    catch (...)
    {
        clu_plan_free(p);
        return CF_OK;
    }
    const size_t dwAt = (k.host.size() + 255) & ~(size_t)255;
    char* base = nullptr;
    int rc = CF_OK;
    if (cudaMalloc((void**)&base, dwAt + sizeof(float) * nd * (size_t)H.rowsP) != cudaSuccess)
        rc = fail(CF_ERR_CUDA, "cluster split: cudaMalloc");
    if (rc == CF_OK) p->allocs.push_back(base);
    if (rc == CF_OK &&
        (cudaMemcpyAsync(base, k.host.data(), k.host.size(), cudaMemcpyHostToDevice, s) !=
             cudaSuccess ||
         cudaStreamSynchronize(s) != cudaSuccess))   // the host arrays end here
        rc = fail(CF_ERR_CUDA, "cluster split: upload");
    p->split.parts = reinterpret_cast<const ResPart*>(base + at[0]);
    p->split.rowMap = reinterpret_cast<const int*>(base + at[1]);
    p->split.idx = reinterpret_cast<const unsigned short*>(base + at[2]);
    p->split.emap = reinterpret_cast<const int*>(base + at[3]);
    p->split.dest = reinterpret_cast<const unsigned int*>(base + at[4]);
    p->dw = reinterpret_cast<float*>(base + dwAt);
    if (rc != CF_OK)
    {
        clu_plan_free(p);
        return rc;
    }
    *plan = p;
    return CF_OK;
}

int clu_launch_fn(const void* fn, int ctas, int threads, size_t smem, void** args, int count,
                  cudaStream_t s)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(ctas, threads, smem, count, s, &cfg, &attr);
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess)
        return fail(CF_ERR_CUDA, std::string("cluster launch: ") + cudaGetErrorString(e));
    return CF_OK;
}

int clu_launch(int W, int R, int ctas, int threads, size_t smem, const CluSys* one,
               const CluSys* d_list, int count, cudaStream_t s)
{
    CluArgs a;
    a.list = d_list;
    if (one) a.one = *one;
    else std::memset((void*)&a.one, 0, sizeof(a.one));
    void* args[] = {(void*)&a};
    return clu_launch_fn(kernel_of(W, R), ctas, threads, smem, args, count, s);
}

void clu_release(cf_context* c)
{
    clu_plan_free(static_cast<CluPlan*>(c->clu));
    c->clu = nullptr;
    c->cluTried = false;
}

int clu_inner(cf_context* c, const double* mean, double target, int maxIter, int ips, int order,
              int stagLimit, bool* ran)
{
    *ran = false;
    if (maxIter <= 0) return CF_OK;
    if (!c->cluTried)
    {
        c->cluTried = true;
        if (c->hostSliceOff.empty()) return CF_OK;
        CluPlan* plan = nullptr;
        const int ctas = std::min(CLU_MAX_CTAS, (c->n + CLU_T - 1) / CLU_T);
        {
            const LentLayout lent(c);
            if (clu_plan_build(c->n, lent.L, !c->identityPerm, ctas, 0, 0, c->stream, &plan) !=
                CF_OK)
                cudaGetLastError();   // no memory for the split: another path
        }
        if (plan && plan->split.halo > SPLIT_MAX_HALO)
        {
            clu_plan_free(plan);
            plan = nullptr;
        }
        c->clu = plan;
    }
    CluPlan* p = static_cast<CluPlan*>(c->clu);
    if (!p) return CF_OK;
    cudaStream_t s = c->stream;
    CluSys Y;
    Y.split = p->split;
    Y.run = inner_run(c, mean, target, maxIter, ips, order, stagLimit);
    Y.dw = p->dw;
    const int rc = clu_launch(p->W, p->R, p->split.ctas, p->threads, p->smem, &Y, nullptr, 1, s);
    if (rc != CF_OK) return rc;
    c->launches++;
    CLU_CUDA(cudaEventRecord(c->ev1, s));
    CLU_CUDA(cudaMemcpyAsync(c->h_st, c->d_st, sizeof(InnerState), cudaMemcpyDeviceToHost, s));
    CLU_CUDA(cudaStreamSynchronize(s));
    if (c->h_st->waitErr)
    {
        // a wait gave up: this solve goes through the graph path
        CLU_CUDA(cudaMemsetAsync(&c->d_st->waitErr, 0, sizeof(int), s));
        c->backoff.gaveUp();
        return CF_OK;
    }
    c->backoff.worked();
    *ran = true;
    return CF_OK;
}

}  // namespace cf
