// Chain kernels: products with NVFP4 weights.
#include "chain_mv.cuh"

MK_CHAIN_TABLE(mk_chain_fp4, 2, MK_CHAIN_KERNEL(8, 2, 2, true, 8))
