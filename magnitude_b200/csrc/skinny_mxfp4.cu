// Small-batch kernels for MXFP4 weights.
#include "skinny_kernel.cuh"

SK_INSTANTIATE(mxfp4, QT_MXFP4)
