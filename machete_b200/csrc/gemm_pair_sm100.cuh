// The compute-bound form of the GEMM tile: C[M,N] = act(A[M,K] · B[N,K]^T) for prompts, where every
// weight byte is used by hundreds of rows.  Included by gemm_sm100.cu, whose helpers it uses.
//
// Two CTAs (the two SMs of a TPC) form a cluster and share one tile of 256 weight rows x `bn` activation
// rows (bn <= 256) with tcgen05.mma.cta_group::2: each CTA holds 128 weight rows and bn / 2 activation
// rows of every 64-wide K step in its own shared memory and the accumulator of its own 128 weight rows
// in its own tensor memory, so a K step brings 16 KB + bn * 64 bytes into an SM instead of
// 16 KB + bn * 128.  The pairs are persistent: each walks the tiles t, t + pairs, ..., the accumulator is
// double-buffered (2 x 256 tensor-memory columns), and the epilogue of a tile runs under the products of
// the next one.
//
//   warp 0 (both CTAs)   TMA producer of the CTA's own half; completion counts on the leader's barrier
//   warp 1 (leader)      issues the MMAs of the pair; commits reach both CTAs' barriers
//   warps 2-9 (both)     epilogue: tensor-memory lane = weight row, column = activation row
//
// A problem with few tiles splits K as well: the pairs of one tile form one cluster, each takes a range of the
// K steps, and their fp32 partial tiles are summed through distributed shared memory (reduce_slice).
//
// What bounds it: the tensor pipe and, in a stream of large products, the power cap.  2048 x 4096 -> 14336: 160.6 us
// alone (the tensor pipe active in 93 % of the SMs' active cycles, 12.8 TB/s from L2, DRAM 14 %; the clock at
// 1.55 GHz), 178.6 us one after another: 1347 TFLOP/s of the 1383 that cuBLAS sustains under the cap.  The single
// kernel, which draws 48 KB a K step into an SM instead of 32, takes 229.
#pragma once

namespace mkg {

constexpr int kPairRows = 256;     // weight rows per tile (both CTAs)
constexpr int kPairStages = 7;
constexpr int kPairEpiWarps = 8;
constexpr int kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr int kMaxPairSplit = 4;   // 2 * split CTAs form one portable cluster

struct PairParams {
  __nv_bfloat16* c;
  int32_t* status;
  int64_t ldc;
  int M, N, K;
  int k_tiles, stages;
  int split_k;                     // pairs that share one tile's K range (1: persistent pairs, many tiles each)
  uint32_t ring_bytes;             // the stages, or the fp32 partial tile if that is larger (split-K)
  int bn;                          // activation rows per tile, a multiple of 16
  int m_tiles, tiles;
  int activation;
  int b_packed;
  int wide_store;                  // C rows and base are 4-byte aligned and N is even
  uint64_t timeout_ns;
};

struct PairShared {
  uint64_t full[kPairStages], empty[kPairStages], acc_full[2], drained, acc_empty[2];   // initialised side by side, one lane each
  uint32_t tmem_base;
  int32_t abort_flag;
  int32_t other_issued;            // leader: the K steps that the other CTA's producer has issued, once it is through
};

// TMA loads of a CTA pair: the data goes to this CTA's shared memory, the completion to `bar`, which may
// lie in the other CTA of the pair (a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(tmap), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* tmap, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                            uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
// One arrival on the barrier at this offset in BOTH CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint16_t ranks, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar),
      "h"(ranks), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = mk::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;          // the same offset in every CTA of the cluster
  const uint32_t a_bytes = (uint32_t)(p.bn >> 1) * kTileK * 2;
  const uint32_t stage_bytes = kWBytes + a_bytes;        // bn is a multiple of 16: a multiple of 1 KB
  PairShared* sh = reinterpret_cast<PairShared*>(smem_raw + (base - raw) + p.ring_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int crank = (int)cluster_ctarank();
  const int rank = crank & 1;                            // which half of the pair
  const uint32_t lead = (uint32_t)(crank & ~1);          // cluster rank of the pair's leader
  const int csize = 2 * p.split_k;
  const int first = (int)blockIdx.x / csize, step = (int)gridDim.x / csize;
  // this pair's K steps
  const int per = (p.k_tiles + p.split_k - 1) / p.split_k;
  const int kt0 = (crank >> 1) * per, kt1 = min(p.k_tiles, kt0 + per);

  const uint32_t full0 = mk::smem_u32(&sh->full[0]), empty0 = mk::smem_u32(&sh->empty[0]);
  if (warp == 0) {
    constexpr int kOnes = 2 * kPairStages + 3;
    if (lane < kOnes + 2) mk::mbar_init(full0 + 8u * lane, lane < kOnes ? 1 : 2 * kPairEpiWarps);
    if (lane == 0) sh->abort_flag = 0, sh->other_issued = -1;
    mk::fence_mbar_init();
  }
  if (warp == 1) tmem_alloc_pair(mk::smem_u32(&sh->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                     // both CTAs' barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);
  mk::prior_work_done();
  // at once: a CTA fills an SM, so nothing lands beside it (1309 x 14320 -> 4424 166.9 us; with the last load 175.3)
  mk::next_may_start();

  // Producer and MMA warps walk their loops as whole warps and one elected lane issues (see tc_mma_bf16).
  if (warp == 0) {
    int it = 0, s = 0;
    uint32_t ph = 0;
    bool ok = true;
    const uint32_t lead_full0 = peer_smem(full0, lead);
    for (int t = first; t < p.tiles && ok; t += step) {
      const int w_row = (t / p.m_tiles) * kPairRows + rank * kTileN;
      const int a_row = (t % p.m_tiles) * p.bn + rank * (p.bn >> 1);
      for (int kt = kt0; kt < kt1; ++kt, ++it) {
        ok = wait_bar_warp(p, sh, empty0 + 8u * s, ph ^ 1u, GEMM_ST_TIMEOUT_EMPTY, 0, it);
        if (!ok) break;
        if (elect_one()) {
          const uint32_t dst = base + (uint32_t)s * stage_bytes, bar = lead_full0 + 8u * s;
          if (rank == 0) mk::mbar_arrive_expect_tx(full0 + 8u * s, 2u * stage_bytes);
          if (p.b_packed)
            tma_load_3d_pair(dst, &map_b, 0, w_row, kt, bar);
          else
            tma_load_2d_pair(dst, &map_b, kt * kTileK, w_row, bar);
          tma_load_2d_pair(dst + kWBytes, &map_a, kt * kTileK, a_row, bar);
        }
        __syncwarp();
        if (++s == p.stages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
    if (lane == 0 && rank == 1) st_cluster_u32(peer_smem(mk::smem_u32(&sh->other_issued), lead), (uint32_t)it);
    if (lane == 0 && rank == 0 && *reinterpret_cast<volatile int32_t*>(&sh->abort_flag)) {
      // Shared memory must outlive the copies in flight.  Both CTAs' copies are counted on the leader's barriers and
      // neither CTA leaves before the leader is at the cluster barrier, so the leader waits (bounded) for each
      // slot's last use: once the other producer's count is known, a step that only the other CTA issued is armed
      // for that half alone.
      const uint64_t t0 = mk::globaltimer_ns();
      const volatile int32_t* other = &sh->other_issued;
      while (*other < 0 && mk::globaltimer_ns() - t0 < 2 * p.timeout_ns) {
      }
      const int last = max(it, (int)*other);
      for (int i = max(0, last - p.stages); i < last; ++i) {
        const uint32_t bar = full0 + 8u * (i % p.stages);
        if (i >= it) mk::mbar_arrive_expect_tx(bar, stage_bytes);
        while (!mk::mbar_try_wait(bar, (uint32_t)(i / p.stages) & 1u) && mk::globaltimer_ns() - t0 < 3 * p.timeout_ns) {
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(kPairRows >> 4) << 24);
      const uint16_t both = (uint16_t)(3u << lead);
      const uint32_t elected = elect_one() ? 1u : 0u;
      int it = 0, s = 0, n = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = first; t < p.tiles && ok; t += step, ++n) {
        const int buf = n & 1;
        ok = wait_bar_warp(p, sh, mk::smem_u32(&sh->acc_empty[buf]), (((uint32_t)n >> 1) & 1u) ^ 1u, GEMM_ST_TIMEOUT_ACC, 1, it);
        if (!ok) break;
        tc_fence_after();
        const uint32_t acc = tmem + (uint32_t)buf * 256u;
        for (int kt = kt0; kt < kt1; ++kt, ++it) {
          ok = wait_bar_warp(p, sh, full0 + 8u * s, ph, GEMM_ST_TIMEOUT_FULL, 1, it);
          if (!ok) break;
          tc_fence_after();
          const uint32_t w_addr = base + (uint32_t)s * stage_bytes;
          const uint64_t dw = smem_desc_sw128(w_addr), da = smem_desc_sw128(w_addr + kWBytes);
#pragma unroll
          for (int k = 0; k < kTileK / 16; ++k) tc_mma_pair(acc, dw + 2u * k, da + 2u * k, idesc, (kt > kt0 || k > 0) ? 1u : 0u, elected);
          tc_commit_pair(empty0 + 8u * s, both, elected);
          if (++s == p.stages) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (ok && kt1 > kt0) tc_commit_pair(mk::smem_u32(&sh->acc_full[buf]), both, elected);
      }
      // Whoever has given up: the products in flight still read both CTAs' shared memory and write their tensor memory.
      tc_commit_pair(mk::smem_u32(&sh->drained), both, elected);
      wait_drained(p, mk::smem_u32(&sh->drained));
    }
  } else {
    const int q = warp & 3;                               // warp w may touch tensor-memory lanes 32 * (w % 4) ..
    const int half = (warp - 2) >> 2;                     // and takes every second block of 32 activation rows
    int n = 0;
    for (int t = first; t < p.tiles; t += step, ++n) {
      const int buf = n & 1;
      // an empty K range (split_k beyond the K steps) adds nothing
      const bool some = kt1 > kt0;
      const bool ok = !some || wait_bar_warp(p, sh, mk::smem_u32(&sh->acc_full[buf]), ((uint32_t)n >> 1) & 1u, GEMM_ST_TIMEOUT_ACC, 2, n);
      if (!ok) break;
      tc_fence_after();
      const int nl = q * 32 + lane;
      const int col = (t / p.m_tiles) * kPairRows + rank * kTileN + nl;
      const int m0 = (t % p.m_tiles) * p.bn;
      const int rows = min(p.bn, p.M - m0);
      const uint32_t acc = tmem + (uint32_t)buf * 256u + ((uint32_t)(q * 32) << 16);
      float* part = reinterpret_cast<float*>(smem_raw + (base - raw)) + nl;
      for (int c = half * 32; c < rows; c += 64) {
        uint32_t r[32];
        if (some) {
          tmem_ld32(acc + (uint32_t)c, r);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        if (p.split_k > 1) {
          // the stage ring is free: every copy was consumed before the accumulator was declared ready
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c + j < rows) part[(c + j) * kTileN] = __uint_as_float(r[j]);
        } else {
          with_act(p.activation, [&](auto act) {
            store_columns<decltype(act)::value>(p.c, p.ldc, r, m0 + c, rows - c, col, col < p.N, p.wide_store != 0, lane);
          });
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(peer_smem(mk::smem_u32(&sh->acc_empty[buf]), lead));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();                                         // nobody leaves while the pair may still signal it
  if (p.split_k > 1) {
    const int m0 = (first % p.m_tiles) * p.bn, n0 = (first / p.m_tiles) * kPairRows + rank * kTileN;
    reduce_slice(p, base, min(p.bn, p.M - m0), rank, 2, crank >> 1, m0, n0, min(p.N, n0 + kTileN), kPairThreads);
    cluster_arrive();
  }
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
  if (p.split_k > 1) cluster_wait();                      // nor while a peer may still read its partial tile
}

}  // namespace mkg
