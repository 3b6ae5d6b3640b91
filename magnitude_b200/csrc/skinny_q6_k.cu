// Small-batch kernels for Q6_K weights.
#include "skinny_kernel.cuh"

SK_INSTANTIATE(q6_k, QT_Q6_K)
