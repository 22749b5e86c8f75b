// Chain kernels: products with NVFP4 weights.
#include "chain_mv.cuh"

MK_CHAIN_TABLE(mk_chain_fp4, 2)
