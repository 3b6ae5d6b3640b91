// Small-batch kernels for Q5_K weights.
#include "skinny_kernel.cuh"

SK_INSTANTIATE(q5_k, QT_Q5_K)
