// bsj_kernels.h -- launch interface between the host engine and the level kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "bsj_device.cuh"

namespace bsj {

// Everything a level kernel needs, passed by value (fits the kernel parameter space).
struct StepArgs {
    const SegDesc* segs;
    SegState* st;
    const int32_t* rank_prefix;   // [nseg+1] prefix sums of K (flattened rank space)
    const int32_t* chunk_prefix;  // [nseg+1] prefix sums of ceil(K/chunk)
    int32_t* kcnt;                // candidate keys per chunk of the current level
    uint2* kmm;                   // per chunk of the current level: min / max score bits of
                                  // its keys ({~0, 0} when it has none)
    int32_t nseg;
    int32_t total_ranks;
    int32_t total_chunks;
    int32_t sb_max;               // per-warp state buffer bytes (max sbytes)
    int32_t max_n;                // largest n of the batch (k_step key staging)
    // the beams this launch works on: [seg_lo, seg_hi) and their chunk / rank ranges
    // (several ranges run as independent branches of one graph)
    int32_t seg_lo, seg_hi;
    int32_t chunk_lo, chunk_hi;
    int32_t rank_lo, rank_hi;
    int32_t chunk;                // ranks per k_step CTA (one of kChunkSizes)
    int32_t select_force;         // kSel* route flags for k_select (0 = by level size)
    int32_t group_step;           // k_step form: 0 warp per survivor; 1-4 a lane group per
                                  // survivor (k_step_g: 4 lanes copy / bulk, 8 lanes copy / bulk)
    int32_t select_cluster;       // CTAs per beam of k_select: 1, or 2 / 4 (cluster launch)
    uint8_t* beam_pool;
    uint8_t* slot_pool;
    unsigned long long* keys;
    uint32_t* sel;
    uint32_t* masks;
    uint32_t* hist;
    uint8_t* aux_pool;
    const uint32_t* ops;          // (duration << 8) | machine per op, per instance
    int32_t* group_best;
    int32_t* seq_pool;
    uint8_t* pos_pool;            // branch -> ready position tables (SegDesc::pos_off)
    const float* noise;           // [1000]: (float)k / 1e9f, IEEE round-to-nearest
    const double* dnoise;         // [1000]: (double)k / 1e6 (BS-PMS noise), IEEE round-to-nearest
};

// k_step variants (the autotuner's candidates besides the default rule): a warp per
// survivor with 8, 16 or 32 survivors per CTA; a group of 4 lanes per survivor (32 per
// CTA) or of 8 lanes (16 per CTA), the parent snapshots staged by the group's 16-byte
// copies or by one bulk copy.  Group variants apply to beam groups whose beams are all
// gpu-v2 / clean; other groups run the warp kernel with the same chunk size.  Public
// codes (bsj_plan_set_chunk): 8, 16, 32 (warp), 1, 2, 3, 4 (group).
constexpr int kNumStepVariants = 7;
constexpr int kStepVariantChunk[kNumStepVariants] = {8, 16, 32, 32, 32, 16, 16};
constexpr int kStepVariantGroup[kNumStepVariants] = {0, 0, 0, 1, 2, 3, 4};
constexpr int kStepVariantCode[kNumStepVariants] = {8, 16, 32, 1, 2, 3, 4};

// k_heap launch configuration: the largest K, child-table row (bytes) and n of the
// launch's ICH/PMS beams, and the parents prepared per chunk.
struct HeapCfg {
    int32_t kmax, chunk, ab, nmax;
};

// ---- resident search (bsj_search.cu): all levels of a gpu-mode beam in one kernel ----
constexpr int kSearchThreads = 512;
constexpr int kSearchBinBits = 9;
constexpr int kSearchBins = 1 << kSearchBinBits;   // score bins of the selection
constexpr int kSearchMaxCluster = 16;
constexpr int kSearchNarrow = 4;       // blocks per beam of the narrow form, but for search_shares' 8
constexpr int kSearchMinBuf = 2048;    // keys the sort's buffer holds at least
constexpr int kSearchMinList = 1024;   // candidate keys the list holds at least

// Snapshot by ready position (bytes): i32 tr[m] | i32 jr[n] | u16 op[n] | u8 mc[n] |
// u16 r, u16 ns, i32 cmax, u32 lineage, u32 stamp (16-byte aligned).
struct SearchLay {
    int off_jr, off_op, off_mc, off_hdr, bytes;
    __host__ __device__ __forceinline__ SearchLay(int n, int m)
    {
        off_jr = 4 * m;
        off_op = off_jr + 4 * n;
        off_mc = (off_op + 2 * n + 3) & ~3;
        off_hdr = (off_mc + n + 15) & ~15;
        bytes = off_hdr + 16;
    }
};

// A survivor's entry (filler flag | parent rank << 7 | ready position or branch) names one of the
// P parents and a place in a list of n: only then are its copies inside the beam's buffers.
__host__ __device__ __forceinline__ bool search_entry_ok(uint32_t e, int P, int n)
{
    return ((e & ~kFillerFlag) >> 7) < (uint32_t)P && (e & 127u) < (uint32_t)n;
}

// Position i is one of the ready list's (first header word: list length | operations done << 16).
// Applied past its end, an operation would shorten an empty list to 65 535 entries.
__host__ __device__ __forceinline__ bool search_position_ok(int i, uint32_t header)
{
    return i >= 0 && i < (int)(header & 0xFFFFu);
}

// One launch: its beams, blocks per beam, lanes per survivor and shared-memory layout.
struct SearchCfg {
    const int32_t* list;        // the launch's beams
    unsigned long long* spill;  // candidate keys past list_cap (offsets as StepArgs::keys; null: lists fit)
    int32_t cluster, lanes, rs, stage_stride;
    uint32_t c_magic;
    uint32_t paths;             // kPath* bits of the launch itself
    int32_t list_cap, buf_cap;
    int32_t wide;               // report the cluster route
    int32_t ahead;              // the staging area holds a block's whole share
    int32_t off_mask, off_sel, off_info, off_list, off_stage;
    size_t smem;
};

bool search_layout(SearchCfg& cf, int cluster, int lanes, int kmax, int nmax, int opsmax, int smax, size_t limit);
// The current device's limits: dynamic shared memory of a block, clusters of each size that
// run at once.
struct SearchDevice {
    size_t smem = 0;
    int clusters[kSearchMaxCluster + 1] = {};
};
constexpr int kSearchSizes[] = {1, 2, 4, 8, 12, 16};   // blocks per beam
cudaError_t search_device(SearchDevice& out);
// Estimated microseconds per level with C blocks (for choosing C only).
double search_level_us(int n, int K, bool v1, int C);
// Blocks per beam with the smallest estimate among sizes up to cmax that the device runs and
// whose layout fits, or the smallest size above where there is none; 0 if nothing fits.
int search_blocks(const SearchDevice& dev, int n, int m, int K, bool v1, int cmax);
// Lanes per survivor for C blocks.
int search_lanes(int n, int K, int C);
cudaError_t launch_search(const StepArgs& a, const SearchCfg& cf, int nbeams, bool v1, cudaStream_t stream);

// Grid / shared-memory sizing helpers.
size_t step_smem_bytes(int sb_max, int max_n, int chunk);
size_t select_smem_bytes(int sort_cap);
size_t heap_smem_bytes(const HeapCfg& c);
// Largest chunk in [1, kHeapMaxChunk] whose k_heap shared memory fits `budget`; 0 if none.
int heap_pick_chunk(HeapCfg c, size_t budget);

// Launchers (asynchronous on `stream`).
// k_step is instantiated per NQ = ceil(n/32) in {1, 2, 4} and chunk size (a.chunk);
// nq_mask has bit NQ set for each class present in the batch (one launch per class).
cudaError_t launch_step(const StepArgs& a, int s, int grid, int nq_mask, cudaStream_t stream);
int nq_class(int n);
cudaError_t launch_gather_v1(const StepArgs& a, int s, int grid, cudaStream_t stream);
cudaError_t launch_select(const StepArgs& a, int s, int sort_cap, cudaStream_t stream);
cudaError_t launch_heap(const StepArgs& a, int s, const HeapCfg& hc, cudaStream_t stream);
// Fills noise[0..1000) with (float)k / 1e9f (once per plan; k_step copies it per CTA).
cudaError_t launch_noise_table(float* noise, double* dnoise, cudaStream_t stream);
// `max_levels`, `kmax_gpu`: largest N, and largest K of the gpu-mode beams (0: none).
cudaError_t launch_finalize(const StepArgs& a, int max_levels, int kmax_gpu, cudaStream_t stream);
cudaError_t configure_kernels(int sort_cap, const HeapCfg* hc, int sb_max, int max_n);
// Raise (never lower) the dynamic shared-memory limits of k_select and k_step to what
// a launch with `sort_cap` / `sb_max` needs.
cudaError_t raise_kernel_smem(int sort_cap, int sb_max, int max_n);

}  // namespace bsj
