// Persistent batched form of the row-vector forward projector (see fpr_kernel.cuh).
#include "fpr_kernel.cuh"

namespace tomo {
namespace fpr {

__global__ void __launch_bounds__(kThreads, 1)
    fpr_kernel_persist(const FpLaunch* __restrict__ descs, const int4* __restrict__ items, int n_items,
                       int* __restrict__ cursor) {
    int& s_item = *reinterpret_cast<int*>(fsm + 16);  // between the barrier and the block infos
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(cursor, 1);
        __syncthreads();
        const int i = s_item;
        if (i >= n_items) return;
        const int4 it = items[i];
        const FpLaunch* a = descs + it.x;
        const int zc = a->rv.zc;
        const bool f32 = a->vtype == kVolF32;
        const bool ok = zc == 8   ? (f32 ? fpr_item<8, 4>(a, it) : fpr_item<8, 2>(a, it))
                        : zc == 6 ? (f32 ? fpr_item<6, 4>(a, it) : fpr_item<6, 2>(a, it))
                                  : (f32 ? fpr_item<4, 4>(a, it) : fpr_item<4, 2>(a, it));
        if (!ok) return;
        __syncthreads();  // shared memory (and s_item) are free for the next item
    }
}

}  // namespace fpr

cudaError_t fpr_persist_attr() {
    return cudaFuncSetAttribute(fpr::fpr_kernel_persist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kFprSmemMax);
}

cudaError_t launch_fpr_persist(const FpLaunch* descs, const int4* items, int n_items, int* cursor, int grid,
                               size_t smem, cudaStream_t s) {
    if (n_items <= 0) return cudaSuccess;
    if (grid <= 0 || smem > kFprSmemMax) return cudaErrorInvalidValue;
    fpr::fpr_kernel_persist<<<grid, fpr::kThreads, smem, s>>>(descs, items, n_items, cursor);
    count_launch();
    return cudaGetLastError();
}

}  // namespace tomo
