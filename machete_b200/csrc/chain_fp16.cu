// Chain kernels: products with fp16 weights.
#include "chain_mv.cuh"

MK_CHAIN_TABLE(mk_chain_fp16, 1)
