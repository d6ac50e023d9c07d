// Chirp-z kernels of 3072-point transforms on the block FFT engine (one
// translation unit of czt_blk.cuh).
#include "czt_blk.cuh"

XL_CZT_BLK_INSTANTIATE(12)
