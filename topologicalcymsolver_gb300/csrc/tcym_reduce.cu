// Sums of reduction records in launches of their own: one lattice's (the restore on
// caller-owned memory) and every ensemble member's, each in a fixed order, with the
// Kahan-compensated N_CS accumulator (FP64, on the device).
#include "tcym_batch.cuh"

namespace tcym {

__global__ void __launch_bounds__(kRedThreads) k_finalize(const double *partial, int blocks, Finish fin) {
    __shared__ double sh[used_count(kUsedAll) * kRedThreads], t[P_WIDTH];
    sum_records<kUsedAll, kRedThreads, false>(partial, blocks, sh, t);
    finish_record(t, fin);
}

cudaError_t preload_finalize() {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, k_finalize);
}

cudaError_t finalize_obs(const double *partial, int blocks, int na, int64_t V, double ncs_dt, double *result,
                         cudaStream_t st) {
    k_finalize<<<1, kRedThreads, 0, st>>>(partial, blocks, make_finish(result, na, V, ncs_dt));
    return cudaGetLastError();
}

// One block per member; out[2i] = E.B, out[2i+1] = N_CS of member i.
__global__ void __launch_bounds__(kRedThreads) k_finalize_members(const MemberReduce *items, double *out) {
    __shared__ double sh[used_count(kUsedSample) * kRedThreads], t[P_WIDTH];
    const MemberReduce it = items[blockIdx.x];
    sum_records<kUsedSample, kRedThreads, false>(it.partial + (int64_t)it.red_begin * P_WIDTH, it.red_blocks, sh, t);
    const double v = (double)it.V;
    finish_record(t, Finish{it.result, nullptr, 1.0 / v, (double)it.na * v, 3.0 * v, it.ncs_dt, 0.0, 0, 0},
                  out ? out + 2 * blockIdx.x : nullptr, out ? out + 2 * blockIdx.x + 1 : nullptr);
}

cudaError_t finalize_members(const MemberReduce *items, int n, double *out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_finalize_members<<<n, kRedThreads, 0, st>>>(items, out);
    return cudaGetLastError();
}

}  // namespace tcym
