// Small-batch kernels for Q8_0 weights.
#include "skinny_kernel.cuh"

SK_INSTANTIATE(q8_0, QT_Q8_0)
