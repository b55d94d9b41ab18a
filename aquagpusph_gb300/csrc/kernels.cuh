// Kernel-side helpers and launcher declarations shared by the .cu files.
#pragma once

#include "aqua_internal.cuh"
#include "arith.cuh"

namespace aqua {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;   // keys per block
// sweep variants: threads per block x queued neighbours per thread (the
// staging depth) x queue entry x candidate staging: 0 = (128, 128, 16-bit,
// loads), 1 = (64, 128, 16-bit, loads), 2 = (64, 64, 32-bit, loads),
// 3 = (64, 128, 16-bit, bulk copies), 4 = (64, 64, 32-bit, bulk copies);
// direct sweep (no queue, each candidate group summed as it is loaded):
// 5 = 64 threads, 6 = 128 threads, and with the next group's records
// prefetched by asynchronous copies: 7 = 64 threads, 8 = 128 threads;
// those with the register budget of 28 resident warps per SM (9 = 64,
// 10 = 128 threads), 32 (11, 12) or 36 (13, 14)
// 15 to 17, alike: the clustered sweep of the fast 3-D build (BIe walls,
// midpoint scheme; 8 warps per block, 2,048 neighbour records staged per pass),
// the quad sweep everywhere else
constexpr int kSweepClustered = 15;
constexpr int kSweepVariants = 18;
constexpr int kSweepClusteredDefault = 16;
constexpr unsigned kSweepClusteredBlocks = 3;
// Steps of more particles than this look whether the particles lie on a lattice
// (k_octants) and are then swept by octant.  A step on a lattice with h = 2
// spacings, by octant and by box: 316,544 particles 433 and 413 us, 5.88M 5.76
// and 6.27 ms; the look and the kernel that returns at once take 8 and 3 us
// (serialised), 1 to 2% of a step of 400,000.
constexpr uint32_t kOctantMin = 600000;
// Wendland C2 (Wendland{2D,3D}.hcl:44-66): the constant factors of W and F;
// float products folded at compile time, as the OpenCL compiler folds them
template<int D>
struct WendlandC;
template<>
struct WendlandC<3>
{
    static constexpr float W = 0.08203125f * 0.318309886f;
    static constexpr float F = 0.8203125f * 0.318309886f;
};
template<>
struct WendlandC<2>
{
    static constexpr float W = 0.109375f * 0.318309886f;
    static constexpr float F = 1.09375f * 0.318309886f;
};

// The reference's vec type: float4 in 3-D, float2 in 2-D
template<int D>
struct Vec;
template<>
struct Vec<3>
{
    static constexpr int VS = 4;
    __device__ __forceinline__ static void load(const float* p, uint32_t i, float x[4])
    {
        const float4 v = reinterpret_cast<const float4*>(p)[i];
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        x[3] = v.w;
    }
    __device__ __forceinline__ static void store(float* p, uint32_t i, const float x[4])
    {
        reinterpret_cast<float4*>(p)[i] = make_float4(x[0], x[1], x[2], x[3]);
    }
};
template<>
struct Vec<2>
{
    static constexpr int VS = 2;
    __device__ __forceinline__ static void load(const float* p, uint32_t i, float x[4])
    {
        const float2 v = reinterpret_cast<const float2*>(p)[i];
        x[0] = v.x;
        x[1] = v.y;
        x[2] = 0.f;
        x[3] = 0.f;
    }
    __device__ __forceinline__ static void store(float* p, uint32_t i, const float x[4])
    {
        reinterpret_cast<float2*>(p)[i] = make_float2(x[0], x[1]);
    }
};

// link-list / sort launchers (linklist.cu).  `cid` (case of each particle)
// may be NULL: every particle then belongs to case 0.
cudaError_t launch_begin(DevScalars* sc, CaseScalars* cs, uint32_t n_cases,
                         uint2* cells, uint2* wall_range, uint8_t* cell_mark,
                         uint32_t ncap, uint32_t N, uint32_t* sort_scratch,
                         cudaStream_t s);
// all of it in one launch, for at most kSmallMax particles and kSmallCases
// cases: keys and permutation in keys / vals[passes & 1].  Whole steps with
// it and with the separate kernels: 42 against 55 us for 8,206 particles, 147
// against 161 for 15,640 and 98 against 104 for 46,600 in 5 cases; at 57,600
// they are equal (558 and 555), so the line lies between.
constexpr uint32_t kSmallMax = 49152;
constexpr uint32_t kSmallCases = 32;   // one lane each
template<int D>
cudaError_t prepare_small_linklist();
template<int D>
cudaError_t launch_small_linklist(const Consts& c, const float* r,
                                  const int32_t* imove, const uint32_t* cid,
                                  uint32_t N, uint32_t n_cases, CaseScalars* cs,
                                  DevScalars* sc, const StepBufs& b,
                                  uint8_t* cell_mark, uint32_t ncap,
                                  uint32_t passes, cudaStream_t s);
template<int D>
cudaError_t launch_minmax(const Consts& c, const float* r, const int32_t* imove,
                          const uint32_t* cid, uint32_t N, CaseScalars* cs,
                          DevScalars* sc, cudaStream_t s);
template<int D>
cudaError_t launch_ncells(const Consts& c, CaseScalars* cs, uint32_t n_cases,
                          DevScalars* sc, uint32_t ncap, cudaStream_t s);
// icell keys of the positions and the digit histograms (launch_begin() has
// reset the sort scratch); then launch_radix_passes(..., hist_ready = true)
template<int D>
cudaError_t launch_icell_hist(const Consts& c, const float* r,
                              const int32_t* imove, const uint32_t* cid,
                              uint32_t N, const CaseScalars* cs, DevScalars* sc,
                              uint32_t* keys, uint32_t* scratch,
                              uint32_t passes, cudaStream_t s);
cudaError_t launch_radix_passes(uint32_t* keys[2], uint32_t* vals[2],
                                uint32_t n, uint32_t passes, uint32_t* scratch,
                                bool hist_ready, DevScalars* sc,
                                cudaStream_t s, uint32_t* last_keys = nullptr,
                                uint32_t* last_vals = nullptr,
                                uint32_t* inverse = nullptr);
size_t sort_scratch_words(uint32_t n);
cudaError_t launch_inverse_perm(const uint32_t* perm, uint32_t* inv,
                                uint32_t n, const DevScalars* sc,
                                cudaStream_t s);
cudaError_t launch_ihoc(const uint32_t* keys, uint32_t n, uint32_t* ihoc,
                        uint32_t ncap, const DevScalars* sc, cudaStream_t s);
cudaError_t launch_iota(uint32_t* p, uint32_t n, cudaStream_t s);
uint32_t sort_blocks(uint32_t n);
uint32_t sort_passes(uint32_t key_bits);

// step launchers (step.cu)
struct StepArgs
{
    uint32_t N;
    uint32_t ncap;
    VarSet src;        // previous step's Variables (previous order)
    VarSet dst;        // this step's Variables (new order)
    StepBufs b;
    const uint32_t* skeys;  // sorted cell keys
    const uint32_t* perm;   // sorted -> previous index
    DevScalars* sc;
    CaseScalars* cs;        // per-case scalars (n_cases)
    const CaseMotion* cm;   // per-case prescribed motion (n_cases)
    uint32_t n_cases;
    int extras;        // write the intermediate operators
    int clustered;     // the gather writes rec0/rec1 and the cell list for
                       // the clustered sweep instead of posq/velq/pmq
    uint32_t cluster;  // particles per cluster of the quad sweep (4 or 8)
};
// Whether the clustered sweep of this step goes by octant: on a lattice the
// sampled cells make at most 1.06 times the clusters (1.89M particles, h = 1.6
// spacings: 2.18 ms, by box 2.60), sheared by less than a spacing 1.18 times and
// more (5.88M, h = 2: 1.67 times; by octant 8.83, by box 7.87)
__device__ __forceinline__ bool
sweep_by_octant(const DevScalars* sc)
{
    return sc->by_cut > 0 && sc->by_octant * 8u <= sc->by_cut * 9u;
}
// gather / sweep of the step in the exact (IEEE, no FMA) or fast
// (-use_fast_math) compilation
template<int D>
cudaError_t launch_gather(bool fast, const Consts& c, const StepArgs& a,
                          cudaStream_t s);
template<int D>
cudaError_t launch_sweep(bool fast, const Consts& c, const StepArgs& a,
                         unsigned grid, int variant, cudaStream_t s);
cudaError_t launch_finalize(DevScalars* sc, CaseScalars* cs,
                            const CaseMotion* cm, uint32_t n_cases,
                            cudaStream_t s);
template<int D>
cudaError_t launch_motion(const StepArgs& a, cudaStream_t s);
// Copies between device arrays, all in one launch: `n` spans of `words` 32-bit
// words; with `cid`, cid[0 .. N) = 0 and the records of a state of one case
// are written as well (aqua_set_state).
constexpr int kMaxSpans = 14;
struct CopySpans
{
    uint32_t* dst[kMaxSpans];
    const uint32_t* src[kMaxSpans];
    uint64_t words[kMaxSpans];
    int n;
};
struct StateRecords
{
    DevScalars* sc;
    CaseScalars* cs;
    CaseMotion* cm;
    uint32_t* offsets;
    uint32_t* cid;
    uint32_t N;
    DevScalars sc0;
    CaseScalars cs0;
    CaseMotion cm0;
};
cudaError_t launch_copy_spans(const CopySpans& spans, const StateRecords& rec,
                              cudaStream_t s);
cudaError_t launch_set_case_ids(uint32_t* cid, const uint32_t* offsets,
                                uint32_t n_cases, uint32_t N, cudaStream_t s);
cudaError_t launch_export_ihoc(const uint2* cells, uint32_t* ihoc,
                               uint32_t ncap, const DevScalars* sc,
                               cudaStream_t s);

// output.cu: report values in original particle order, free-surface sensors
constexpr uint32_t kMaxFsSensors = 64;
constexpr uint32_t kReportValues = AQUA_REPORT_MAX_VALUES;  // report staging
struct FreeSurfaceSensors
{
    float xy[kMaxFsSensors][2];
};
cudaError_t launch_unsorted(const uint32_t* id, const float* src, uint32_t nc,
                            uint32_t N, uint32_t first, uint32_t n, float* out,
                            cudaStream_t s);
cudaError_t launch_unsorted_int(const uint32_t* id, const int32_t* src,
                                uint32_t N, uint32_t first, uint32_t n,
                                float* out, cudaStream_t s);
cudaError_t launch_free_surface(int dims, const float* r, const int32_t* imove,
                                const uint32_t* cid, int32_t case_index,
                                uint32_t N, const FreeSurfaceSensors& sensors,
                                uint32_t n_sensors, float dr, int* keys,
                                float* out, cudaStream_t s);

template<int D>
cudaError_t launch_bi_walls(bool fast, const Consts& c, const StepArgs& a,
                            unsigned sms, cudaStream_t s);
// clusters of at most 8 particles of one cell (clu, cperm) and the sweep
// over them
template<int D>
cudaError_t launch_clusters(const Consts& c, const StepArgs& a, cudaStream_t s);
template<int D>
cudaError_t launch_sweep_quad(bool fast, const Consts& c, const StepArgs& a,
                              unsigned sms, cudaStream_t s);

namespace exact {
template<int D>
cudaError_t launch_bi_walls_impl(const Consts& c, const StepArgs& a, unsigned sms,
                                 cudaStream_t s);
template<int D>
cudaError_t launch_sweep_quad_impl(const Consts& c, const StepArgs& a,
                                   unsigned sms, cudaStream_t s);
template<int D>
cudaError_t launch_gather_impl(const Consts& c, const StepArgs& a, cudaStream_t s);
template<int D>
cudaError_t launch_sweep_impl(const Consts& c, const StepArgs& a, unsigned grid,
                              int variant, cudaStream_t s);
}  // namespace exact
namespace fast {
// the clustered sweep over the cells of launch_clusters()
cudaError_t launch_sweep_cl(const Consts& c, const StepArgs& a, unsigned grid,
                            cudaStream_t s);
// sets the kernels' dynamic shared memory limit (once, before any capture)
cudaError_t prepare_sweep_cl();
template<int D>
cudaError_t launch_bi_walls_impl(const Consts& c, const StepArgs& a, unsigned sms,
                                 cudaStream_t s);
template<int D>
cudaError_t launch_sweep_quad_impl(const Consts& c, const StepArgs& a,
                                   unsigned sms, cudaStream_t s);
template<int D>
cudaError_t launch_gather_impl(const Consts& c, const StepArgs& a, cudaStream_t s);
template<int D>
cudaError_t launch_sweep_impl(const Consts& c, const StepArgs& a, unsigned grid,
                              int variant, cudaStream_t s);
}  // namespace fast

}  // namespace aqua
