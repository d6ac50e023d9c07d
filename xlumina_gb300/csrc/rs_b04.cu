// RS / VRS passes of 1024-point transforms on the block FFT engine (one
// translation unit of rs_blk.cuh).
#include "rs_blk.cuh"

XL_RS_BLK_INSTANTIATE(4)
