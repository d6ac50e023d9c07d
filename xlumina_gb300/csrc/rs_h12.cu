// RS / VRS passes of 6144-point transforms as two halves (one translation unit of
// rs_half.cuh).
#include "rs_half.cuh"

XL_RS_HALF_INSTANTIATE(12)
