// cf_resident.cuh -- the mesh split behind the resident inner PCG
// (cf_resident.cu): host-side partition of one matrix into parts, one per
// CTA, and the device layout the kernel reads.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <vector>

#include "cf_internal.cuh"

namespace cf {

struct HostLayout;

// One part = the rows of one CTA.  Local rows 0 .. nb-1 have a neighbour in
// another part (their values are published), nb .. nloc-1 do not.  Local
// indices of a gathered vector: own rows, then (from nlocP, nloc rounded up
// to whole slices) the nh halo values, then one slot that holds 0 and that
// padding entries name.
struct ResPart
{
    int nloc, nlocP, nb, nh;
    int rowBase;      // first padded row of the part in the part-ordered arrays
    int haloBase;     // first halo entry in haloSlot
    int llBase;       // slot of local row 0 in the exchange buffer
    int pad_;
};

struct ResHost
{
    int W = 0;                        // entries per row (padded)
    int slots = 0;                    // exchange slots (boundary rows of all parts)
    int rowsP = 0;                    // padded rows of all parts
    int maxLocP = 0, maxHalo = 0;
    std::vector<ResPart> parts;
    std::vector<int32_t> rowMap;      // [rowsP] internal row, -1 padding
    std::vector<uint16_t> idx;        // [rowsP * W] local column, paired order per slice
    std::vector<int32_t> emap;        // [rowsP * W] entry of the SELL arrays, -1 padding
    std::vector<int32_t> haloSlot;    // exchange slot of every halo value
};

// One inner PCG on the staged FP32 operator, as the kernels that run it whole
// take it (everything in the internal row order).
struct InnerRun
{
    const float* val32;
    const float* diag32;
    const float* rD32;
    const float* chebC;
    const double* r64;
    const double* mean;           // subtracted from r64 (null: 0) ...
    const int* useMean;           // ... when this is null or points to != 0
    float* D;                     // [3][dStride] corrections
    long long dStride;
    InnerState* st;
    int fromState;                // target, maxIter, ips, stagLimit (and done) as *st has them
    int order;
    double target;
    int maxIter, ips, stagLimit;
    long long polls;              // reads a bounded wait makes before it gives up
};

// The mesh split over the CTAs of one cooperative launch (cf_resident.cu).
// entOff, rowOff: where the entries and rows of L start when its arrays are
// part of a larger concatenation.  *plan stays null when no kernel takes the
// mesh.
struct ResPlan;
int res_plan_build(int device, int n, const HostLayout& L, bool ordered, int nparts,
                   long long entOff, int rowOff, cudaStream_t s, ResPlan** plan);
void res_plan_free(ResPlan* plan);
// The waits of a resident launch need all its CTAs on the device: launches
// run under this lock until they have ended, with at most one CTA per SM in
// all.
std::mutex& res_device_lock(int device);
int res_launch(const ResPlan* plan, const InnerRun& run, cudaStream_t s);
// fresh exchange words after a wait has given up
int res_reset(const ResPlan* plan, cudaStream_t s);

// Halo values of a part from which cudaPCG does not use a split: every part
// then reads most of the others, and the exchanges cost more than the launches
// they replace.  Meshes stay far below (2,000 at 900K cells); random links of
// six per row, ms per solve graph loop / split: 20K in one cluster (6,900 halo
// values) 0.47 / 0.70, 60K over the SMs (2,300) 0.55 / 0.49, 200K (7,500) 0.77 /
// 0.89.
constexpr int SPLIT_MAX_HALO = 4096;

// Splits the rows of L (its internal order; `ordered`: reverse
// Cuthill-McKee) into nparts parts of equal size (within one row).  Returns
// false when a part would need more than 65,535 local indices or the rows
// are wider than 8.  Rows are padded to `width` entries at least.
bool res_partition(int n, const HostLayout& L, bool ordered, int nparts, ResHost& R,
                   int width = 0);
// The same with consecutive ranges of rowsPerPart rows (whole slices) in the
// internal order; every row counts as read elsewhere.  False also when a part
// would have more than maxHalo halo values.
bool res_blocks(int n, const HostLayout& L, int rowsPerPart, ResHost& R, int width, int maxHalo);

}  // namespace cf
