// step_fp64.cu -- the FP64 form of the stepping path (device code:
// fp64_device.cuh): the DiffusionSDE kernels, the field kernel and the
// launchers.  The Boris and Cash-Karp kernels are in step_fp64_bp.cu and
// step_fp64_ck.cu.  Every FP64 unit is compiled with -fmad=false.
#include "fp64_device.cuh"

namespace crp {
namespace {

__global__ void fp64_field_kernel(const __grid_constant__ DevPlan P, uint64_t n, const double *pos, double *out) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    d3 b = field_at<FS_GENERIC>(P, mk(pos[i], pos[n + i], pos[2 * n + i]));
    out[i] = b.x; out[n + i] = b.y; out[2 * n + i] = b.z;
}

}  // namespace

cudaError_t launch_fp64_chunk(const DevPlan &P, const DevState &s, uint64_t n, int max_steps,
                              uint64_t step_cap, DevCounters *cnt, const DevRecords &rec,
                              const uint32_t *perm, uint32_t *perm_out, int fs, int block, int lanes,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    int prop = P.modules[P.prop_index].propagator;
    if (prop == CRP_PROP_BP)
        return launch_fp64_bp_chunk(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st);
    if (prop == CRP_PROP_CK)
        return launch_fp64_ck_chunk(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st);
    return launch_prop<SDE>(P, s, n, max_steps, step_cap, cnt, rec, perm, perm_out, fs, block, lanes, st);
}

cudaError_t launch_fp64_persistent(const DevPlan &P, const DevState &s, const PersistentArgs &a,
                                   DevCounters *cnt, const DevRecords &rec, int fs, int grid,
                                   cudaStream_t st) {
    const int prop = P.modules[P.prop_index].propagator;
    if (prop == CRP_PROP_BP) return launch_fp64_bp_persistent(P, s, a, cnt, rec, fs, grid, st);
    if (prop == CRP_PROP_CK) return launch_fp64_ck_persistent(P, s, a, cnt, rec, fs, grid, st);
    return launch_persistent_prop<SDE>(P, s, a, cnt, rec, fs, grid, st);
}

cudaError_t launch_fp64_field(const DevPlan &P, uint64_t n, const double *pos, double *out,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    fp64_field_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(P, n, pos, out);
    return cudaGetLastError();
}

}  // namespace crp
