// Small-batch kernels for Q4_K weights.
#include "skinny_kernel.cuh"

SK_INSTANTIATE(q4_k, QT_Q4_K)
