// step_fp64_ck.cu -- the FP64 Cash-Karp (PropagationCK) kernels: chunked
// and persistent launches of the fixed-step and adaptive forms for every field
// signature (the device code is in fp64_device.cuh).
#include "fp64_device.cuh"

namespace crp {

cudaError_t launch_fp64_ck_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                                  uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                                  const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                                  cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const DevModule &pm = P.modules[P.prop_index];
    const bool fixed = pm.min_step == pm.max_step;
    if (fixed && fs == FS_GENERIC && lanes == 32) {  // every warp full: field_sum_call
        fp64_chunk_kernel<CKFixedInlined, FS_GENERIC, CS_GENERIC><<<(unsigned)((n + block - 1) / block), block, 0, st>>>(
            P, s, n, lanes, max_steps, step_cap, cnt, rec, perm, perm_out);
        return cudaGetLastError();
    }
    return fixed ? launch_prop<CKFixed>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st)
                 : launch_prop<CKAdaptive>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st);
}

cudaError_t launch_fp64_ck_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                       DevCounters *cnt, const DevRecords &rec, int fs, int grid, cudaStream_t st) {
    const DevModule &pm = P.modules[P.prop_index];
    const bool fixed = pm.min_step == pm.max_step;
    return fixed ? launch_persistent_prop<CKFixed>(P, s, a, cnt, rec, fs, grid, st)
                 : launch_persistent_prop<CKAdaptive>(P, s, a, cnt, rec, fs, grid, st);
}

}  // namespace crp
