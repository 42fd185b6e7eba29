// cf_cluster_ll.cuh -- words between the CTAs of one thread-block cluster:
// 8-byte {value, epoch} words stored straight into the reader's shared
// memory and polled there (300 cycles one way measured, against 875 through
// L2), and the split of a mesh over the CTAs that the cluster kernels read.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "cf_internal.cuh"
#include "cf_resident.cuh"

struct cf_context;

namespace cf {

typedef unsigned long long u64;

constexpr int CLU_MAX_CTAS = 16;
constexpr int CLU_MAX_HALO = 8191;   // halo values of a part at most
constexpr unsigned int CLU_NONE = 0xffffffffu;

// Every part has the same shared-memory layout of a gathered vector, in
// floats: own rows [0, locP), halo words [locP, locP + 2 halo) (the value is
// the low half of its word), then the slot that holds 0; idx counts in it.
struct CluSplit
{
    const ResPart* parts;
    const int* rowMap;            // [rowsP] internal row, -1 padding
    const unsigned short* idx;    // [rowsP W] paired order per slice
    const int* emap;              // [rowsP W]
    const unsigned int* dest;     // [ndest][rowsP] readers of a row: CTA << 16 | halo value
    int rowsP, ndest, ctas, locP, halo;
};

// One system of a cluster launch.
struct CluSys
{
    CluSplit split;
    InnerRun run;
    float* dw;                    // [3][rowsP] corrections (part order)
};

// The device copy of a split and the kernel that runs it.
struct CluPlan
{
    int W = 0, R = 0, threads = 0;
    size_t smem = 0;
    const void* fn = nullptr;
    CluSplit split = {};
    float* dw = nullptr;
    std::vector<void*> allocs;
};

struct HostLayout;

// Splits a mesh over at most `ctas` CTAs for the cluster PCG (entOff, rowOff
// as for res_plan_build); leaves plan null when the kernel does not take it.
int clu_plan_build(int n, const HostLayout& L, bool ordered, int ctas, long long entOff,
                   int rowOff, cudaStream_t s, CluPlan** plan);
void clu_plan_free(CluPlan* plan);
// Parts of the above for other cluster kernels: a split (of `ctas` parts) in
// the common layout onto the device, with room for nd corrections, for a
// kernel that keeps `buffers` gathered vectors in shared memory.
int clu_plan_upload(ResHost& H, int ctas, int buffers, int nd, long long entOff, int rowOff,
                    const void* fn, int R, int threads, cudaStream_t s, CluPlan** plan);
int clu_launch_fn(const void* fn, int ctas, int threads, size_t smem, void** args, int count,
                  cudaStream_t s);
// One launch: the system `one`, or the `count` systems of d_list, whose plans
// share W, R and the number of CTAs (threads, smem: the largest of theirs).
int clu_launch(int W, int R, int ctas, int threads, size_t smem, const CluSys* one,
               const CluSys* d_list, int count, cudaStream_t s);

__device__ __forceinline__ unsigned int smem_addr(const void* p)
{
    return (unsigned int)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned int remote_addr(unsigned int addr, unsigned int rank)
{
    unsigned int r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void st_remote(unsigned int addr, unsigned int lo, unsigned int epoch)
{
    const u64 v = ((u64)epoch << 32) | lo;
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v));
}

__device__ __forceinline__ u64 ld_local(unsigned int addr)
{
    u64 v;
    asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}

// Waits for the word at addr to carry `epoch`; gives up after `polls` reads
// (*bad is then set and every later wait of the CTA gives up soon).
__device__ __forceinline__ unsigned int wait_local(unsigned int addr, unsigned int epoch,
                                                   volatile int* bad, long long polls)
{
    u64 v = ld_local(addr);
    long long spins = 0;
    while ((unsigned int)(v >> 32) != epoch)
    {
        if (++spins > polls || ((spins & 255) == 0 && *bad))
        {
            *bad = 1;
            return 0u;
        }
        v = ld_local(addr);
    }
    return (unsigned int)v;
}

}  // namespace cf
