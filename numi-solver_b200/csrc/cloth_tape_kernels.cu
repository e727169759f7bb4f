// The frame and batch kernels of rollout gradients: the default kernels with
// the adjoint tape and the record of fruit contact.  A translation unit of
// their own, like the edge/edge kernels, so that the kernels that step
// cloths carry neither (cloth_kernels.cuh, kTaped).
#define NC_TAPE_KERNELS
#define NC_EDGE_KERNELS
#include "cloth_frame.cuh"

__global__ void __launch_bounds__(NC_BLOCK_MAX, 1) numi_cloth_frame_tape_kernel(DeviceCloth d, Schedule s) {
    extern __shared__ __align__(16) unsigned char nc_dynamic_smem[];
    run_frame<false, false, false>(d, s, blockIdx.x, gridDim.x, nc_dynamic_smem);
}

__global__ void __launch_bounds__(NC_BLOCK_MAX, 1) numi_cloth_batch_tape_kernel(const DeviceCloth* cloths,
                                                                              uint32_t count, Schedule s,
                                                                              unsigned int* queue) {
    NC_BATCH_BODY(false)
}

__global__ void __launch_bounds__(NC_BLOCK_MAX, 1)
    numi_cloth_batch_cluster_tape_kernel(const DeviceCloth* cloths, uint32_t count, Schedule s, unsigned int* queue,
                                         uint32_t ranks) {
    NC_BATCH_CLUSTER_BODY
}
