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

// Runs up to 40 candidates per scheduler ask for the next grid cell ahead
// (step_*_bp.cu).
inline bool ask_ahead(uint64_t n, int num_sms) { return n <= 160 * (uint64_t)num_sms; }

// Chunked launches over a PlaneWaveTurbulence field summed by the block
// (FS_PLANE_WAVE_BLOCK).  The largest tables taken are the ones of which two blocks
// fit on an SM beside the kernel's own arrays: 98 KB (FP64, 11 KB beside it) and
// 102 KB (mixed, 9 KB).
constexpr int kWaveMaxModesFp64 = 1365, kWaveMaxModesMixed = 2600;
// Blocks per SM that the kernels' registers are held to.  FP64 Cash-Karp spills 300 B
// at 4 (14 000 candidates x 200 modes: 1.45 ms, 1.23 at 3); the FP64 push loses at 3.
// The mixed adaptive push is faster at 3 below 37 888 candidates (3000 x 200 modes:
// 0.177 and 0.117 ms) and slower above (75 000: 0.48 and 0.50).
constexpr int wave_blocks(bool fp64, bool ck) { return fp64 && ck ? 3 : 4; }
// Blocks per SM of one launch: those, or as many as fit in 228 KB of shared memory
// (the table, the kernel's own arrays and 1 KB of the system's each).
inline uint64_t wave_blocks_per_sm(int n_modes, bool fp64, bool ck) {
    const size_t block = (fp64 ? 11 * 1024 + (size_t)n_modes * 72 : 9 * 1024 + (size_t)((n_modes + 1) / 2) * 80) + 1024;
    const uint64_t room = 228 * 1024 / block, most = (uint64_t)wave_blocks(fp64, ck);
    return room < most ? room : most;
}

// Warps of candidates per block of such a launch; 0: each thread sums for itself.
// A block of four warps sums the modes for 32 candidates (or 64, 128: fewer
// blocks, more candidates per table read).
//
// FP64 (its terms are added by three warps of four): the sums by the block pay
// while all blocks are resident at once, else a run that fills the GPU thread by
// thread is faster (fixed push: 18 900 candidates x 500 modes 1.05 ms with
// blocks left over, 0.93 thread by thread, 0.73 by 64; 28 000 x 1000 modes 2.82
// and 1.94 ms).  64 per block at four blocks per SM pay for long sums only (37 800
// candidates: 40 modes 1.07, 100 modes 0.94 of the time thread by thread).
//
// Mixed: 32 while those blocks are resident at once, then 64, then 128 (fixed push,
// 4 x 10^5 candidates x 300 modes: 7.08 ms thread by thread, 3.92 here).  Cash-Karp
// holds its stages meanwhile, and more candidates per block wait longer: sums of
// 100 modes stay at 32 per block up to 20 blocks per SM, of 200 always (28 000 x 200
// modes: 0.26 ms, 0.41 at 64, 0.45 thread by thread; 150 000 x 100: 0.89, 0.82 at
// 128).  Where two full warps per scheduler sum for themselves and no observer or
// boundary divides them (pm: the chain ends with MaximumTrajectoryLength), that is
// the faster up to 500 modes (37 800 x 100 modes: 0.25 ms, 0.29 at 32, 0.32 at 64; x
// 500: 1.06 and 0.98; with an observer 37 000 x 40 modes: 1.04 and 0.80 at 64).
inline int wave_block_warps(uint64_t n, int n_modes, int num_sms, bool fp64, bool ck, bool pm) {
    if (n_modes < (fp64 ? 32 : 8) || n_modes > (fp64 ? kWaveMaxModesFp64 : kWaveMaxModesMixed)) return 0;
    const uint64_t sms = (uint64_t)num_sms, per_sm = wave_blocks_per_sm(n_modes, fp64, ck);
    auto blocks = [n](int warps) { return (n + 32 * (uint64_t)warps - 1) / (32 * (uint64_t)warps); };
    if (blocks(1) <= per_sm * sms) return 1;
    if (fp64) return blocks(2) <= (per_sm == 4 && n_modes < 100 ? 3 : per_sm) * sms ? 2 : 0;
    if (ck) {
        if (pm && n_modes < 500 && blocks(1) > 6 * sms && blocks(1) <= 8 * sms) return 0;
        if (n_modes >= 200 || (n_modes >= 100 && blocks(1) <= 20 * sms)) return 1;
    }
    return blocks(2) <= 4 * sms ? 2 : 4;
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
