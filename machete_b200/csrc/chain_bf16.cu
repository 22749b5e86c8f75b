// Chain kernels: products with bf16 weights.
#include "chain_mv.cuh"

MK_CHAIN_TABLE(mk_chain_bf16, 0)
