// Small-batch kernels for Q4_0 weights.
#include "skinny_kernel.cuh"

SK_INSTANTIATE(q4_0, QT_Q4_0)
