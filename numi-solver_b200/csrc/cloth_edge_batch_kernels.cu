// The batch kernel with the edge/edge yarn self-collision phases, whose box
// tree may keep its lists in global memory (Schedule::tree_lists): a call
// that the frame kernel, compiled apart in cloth_edge_kernels.cu, does not pay
// for in registers.
#define NC_EDGE_KERNELS
#define NC_EDGE_BATCH_KERNELS
#include "cloth_frame.cuh"

__global__ void __launch_bounds__(NC_BLOCK_MAX, 1) numi_cloth_batch_edge_kernel(const DeviceCloth* cloths, uint32_t count,
                                                                              Schedule s, unsigned int* queue) {
    NC_BATCH_BODY(true)
}
