// Row-vector forward projector, chunks of 8 planes.
#include "fpr_kernel.cuh"

TOMO_FPR_INSTANTIATE(8)
