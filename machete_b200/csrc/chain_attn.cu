// Chain kernels: split-KV attention, head dim 64 / 128, with and without the fused q/k norm, seven participants and four.
#include "chain_attn.cuh"

using namespace mk;

static const mk_chain_attn_variant kVariants[] = {
    {64, 0, 7, 2, mk::at_chain_kernel<64, false, 7, 2>},
    {64, 0, 4, 3, mk::at_chain_kernel<64, false, 4, 3>},
    {64, 0, 4, 4, mk::at_chain_kernel<64, false, 4, 4>},
    {64, 1, 7, 2, mk::at_chain_kernel<64, true, 7, 2>},
    {64, 1, 4, 3, mk::at_chain_kernel<64, true, 4, 3>},
    {64, 1, 4, 4, mk::at_chain_kernel<64, true, 4, 4>},
    {128, 0, 7, 2, mk::at_chain_kernel<128, false, 7, 2>},
    {128, 0, 4, 3, mk::at_chain_kernel<128, false, 4, 3>},
    {128, 1, 7, 2, mk::at_chain_kernel<128, true, 7, 2>},
    {128, 1, 4, 3, mk::at_chain_kernel<128, true, 4, 3>},
};

extern "C" const mk_chain_attn_variant* mk_chain_attn(int* n) {
  *n = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
  return kVariants;
}
