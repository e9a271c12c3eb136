// Row-vector forward projector, chunks of 4 planes.
#include "fpr_kernel.cuh"

TOMO_FPR_INSTANTIATE(4)
