// Chain kernels: split-KV attention, head dim 64 / 128, with and without the fused q/k norm.
#include "chain_attn.cuh"

using namespace mk;

static const mk_chain_attn_variant kVariants[] = {
    {64, 0, mk::at_chain_kernel<64, false>},
    {64, 1, mk::at_chain_kernel<64, true>},
    {128, 0, mk::at_chain_kernel<128, false>},
    {128, 1, mk::at_chain_kernel<128, true>},
};

extern "C" const mk_chain_attn_variant* mk_chain_attn(int* n) {
  *n = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
  return kVariants;
}
