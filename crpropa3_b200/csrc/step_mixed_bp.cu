// step_mixed_bp.cu -- the mixed-precision Boris push (PropagationBP) kernels: chunked
// and persistent launches of the fixed-step and adaptive forms for every field
// signature (the device code is in mixed_device.cuh).
#include "mixed_device.cuh"

namespace crp {

cudaError_t launch_mixed_bp_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                                  uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                                  const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                                  cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const DevModule &pm = P.modules[P.prop_index];
    const bool fixed = pm.min_step == pm.max_step;
    if (fixed && fs == FS_GRID_PERIODIC && P.shape == CS_PM) {
        const uint64_t slots = (uint64_t)(block / 32) * (uint64_t)lanes;
        const unsigned grid = (unsigned)((n + slots - 1) / slots);
        // about one warp per scheduler or less (40 candidates for each): nothing else
        // hides the gathers' latency (256^3 grid, 1000 steps, mixed: 2000 candidates
        // 0.81 -> 0.68 ms, 20 011 0.79 -> 0.76 ms; 50 000 lose, 1.02 -> 1.19 ms)
        if (ask_ahead(n, P.num_sms))
            mixed_boris_kernel<BorisPush<true>><<<grid, block, 0, st>>>(
                P, s, n, lanes, max_steps, step_cap, cnt, rec, perm, perm_out);
        else
            mixed_boris_kernel<BorisPush<false>><<<grid, block, 0, st>>>(
                P, s, n, lanes, max_steps, step_cap, cnt, rec, perm, perm_out);
        return cudaGetLastError();
    }
    return fixed ? launch_prop<BPFixed>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st)
                 : launch_prop<BPAdaptive>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st);
}

cudaError_t launch_mixed_bp_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                       DevCounters *cnt, const DevRecords &rec, int fs, int grid, cudaStream_t st) {
    const DevModule &pm = P.modules[P.prop_index];
    const bool fixed = pm.min_step == pm.max_step;
    return fixed ? launch_persistent_prop<BPFixedPersistent>(P, s, a, cnt, rec, fs, grid, st)
                 : launch_persistent_prop<BPAdaptive>(P, s, a, cnt, rec, fs, grid, st);
}

}  // namespace crp
