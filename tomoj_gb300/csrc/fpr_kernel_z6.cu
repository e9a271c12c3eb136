// Row-vector forward projector, chunks of 6 planes.
#include "fpr_kernel.cuh"

TOMO_FPR_INSTANTIATE(6)
