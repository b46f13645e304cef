// engine_internal.h -- declarations shared between the host engine
// (crp_engine.cu) and the kernel translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "device_plan.cuh"

namespace crp {

// Field signature the stepping kernels are specialised for.
enum FieldSig {
    FS_GENERIC = 0,    // any sum of (possibly periodic) components
    FS_GRID = 1,       // one MagneticFieldGrid, not wrapped
    FS_PLANE_WAVE = 2, // one PlaneWaveTurbulence, not wrapped
    FS_GALACTIC = 5,   // one galactic field class (JF12, UF23, PT11, TF17, KST24), not wrapped
    FS_PLANE_WAVE_BLOCK = 4,  // FS_PLANE_WAVE, the mode sums shared by a block (chosen per launch)
    FS_GRID_PERIODIC = 3  // FS_GRID with a periodic grid of power-of-two dimensions, no
                          // clipVolume and with pair records: no runtime checks
};

// Persistent stepping launch (chain.cuh persistent_body): `grid` CTAs of 128
// threads take work from the virtual queue described by *q -- its pending
// list (list_a or list_b, by q->cur) followed by its main range -- until it
// is empty or budget_ns of device time have passed; unfinished candidates
// go to the other list.  Kernel parameters are fixed for a whole run, so
// the launches can be captured in a CUDA graph.
struct PersistentArgs {
    const DevQueue *q;
    uint32_t *list_a;
    uint32_t *list_b;
    int burst;
    int refill;
    unsigned long long budget_ns;
    uint64_t step_cap;
};

// Candidates per warp of a chunked launch of n candidates.  A launch that
// cannot give every scheduler of the GPU a full warp (four per SM) spreads its
// candidates over one warp per scheduler instead: its run time is the slowest
// warp's chain of dependent instructions, and a warp with fewer candidates
// makes fewer passes for lanes that diverge (retries, cell changes, early ends).
// More warps than that share a scheduler and lose again (10^4 Cash-Karp
// candidates, FP64, 64^3 grid: 7.8 ms at 32 per warp, 6.9 ms at 4 warps per SM,
// 7.2 ms at 8; 10^5 nuclei: 71.3 ms at 4, 73.1 ms at 8).
constexpr int kSpreadWarpsPerSm = 4;
inline int lanes_per_warp(uint64_t n, int num_sms, int warps_per_sm) {
    const uint64_t warps = (uint64_t)num_sms * (uint64_t)warps_per_sm;
    const uint64_t l = (n + warps - 1) / warps;
    return l < 1 ? 1 : l > 32 ? 32 : (int)l;
}

// Runs up to this size ask for the next grid cell ahead (step_*_bp.cu).
constexpr uint64_t kAskAheadCandidates = 592 * 40;

// Warps of candidates per block of a chunked launch over a PlaneWaveTurbulence
// field evaluated by the block: the fewest whose blocks are resident at once (592:
// four per SM), so that a small run has the most warps per candidate.  0: each
// thread sums for itself, for fewer modes than pay for the barriers, for tables
// that leave room for one block per SM only, and in the FP64 form for runs that
// fill the GPU thread by thread (its terms are added by three warps of four:
// 10^5 candidates, 100 modes: 1.50 ms thread by thread, 2.07 ms by blocks;
// 20 000 candidates, 200 modes: 5.16 and 4.06 ms; the mixed form 4 x 10^5
// candidates, 300 modes: 7.08 and 3.92 ms, 20 modes: 0.86 and 0.82 ms).
constexpr int kWaveMaxModes = 1365;
inline int wave_block_warps(uint64_t n, int n_modes, bool fp64) {
    if (n_modes < (fp64 ? 32 : 8) || n_modes > kWaveMaxModes) return 0;
    if (n <= 592u * 32u) return 1;
    if (n <= 592u * 64u) return 2;
    return fp64 ? 0 : 4;
}

// Dynamic shared memory a kernel may be launched with: MOST, the largest that
// any plan asks of it.  The limit belongs to the kernel, not to a launch: setting
// it to one plan's table would lower it under another thread's launch.
template <size_t MOST, class Kernel>
inline cudaError_t allow_shared(Kernel kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST);
}

// step_fp64.cu
// One launch of the chunked stepping kernel: slots t < n (`lanes` of them per
// warp) advance candidate perm[t] (t without perm) by at most max_steps chain
// iterations; candidates still active afterwards are appended to perm_out
// (may be null) and counted in cnt->active_left.
cudaError_t launch_fp64_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                              uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                              const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                              cudaStream_t st);
cudaError_t launch_fp64_field(const DevPlan &P, uint64_t n, const double *pos, double *out,
                              cudaStream_t st);
cudaError_t launch_fp64_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                   DevCounters *cnt, const DevRecords &rec, int fs, int grid,
                                   cudaStream_t st);

// step_mixed.cu
cudaError_t launch_mixed_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                               uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                               const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                               cudaStream_t st);
// step_fp64_bp.cu, step_fp64_ck.cu, step_mixed_bp.cu, step_mixed_ck.cu: the
// Boris-push and Cash-Karp parts of the launchers above and below
cudaError_t launch_fp64_bp_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                                  uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                                  const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                                  cudaStream_t st);
cudaError_t launch_fp64_bp_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                DevCounters *cnt, const DevRecords &rec, int fs, int grid, cudaStream_t st);
cudaError_t launch_fp64_ck_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                                  uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                                  const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                                  cudaStream_t st);
cudaError_t launch_fp64_ck_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                DevCounters *cnt, const DevRecords &rec, int fs, int grid, cudaStream_t st);
cudaError_t launch_mixed_bp_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                                  uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                                  const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                                  cudaStream_t st);
cudaError_t launch_mixed_bp_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                DevCounters *cnt, const DevRecords &rec, int fs, int grid, cudaStream_t st);
cudaError_t launch_mixed_ck_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                                  uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                                  const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                                  cudaStream_t st);
cudaError_t launch_mixed_ck_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                DevCounters *cnt, const DevRecords &rec, int fs, int grid, cudaStream_t st);
cudaError_t launch_mixed_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                    DevCounters *cnt, const DevRecords &rec, int fs, int grid,
                                    cudaStream_t st);
cudaError_t launch_mixed_field(const DevPlan &P, uint64_t n, const double *pos, double *out,
                               cudaStream_t st);

}  // namespace crp
