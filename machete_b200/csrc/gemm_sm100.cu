// bf16 GEMM on the 5th-generation tensor cores: C[M,N] = A[M,K] · B[N,K]^T.
//
// The decode path's own matvec ops cover M <= 32 with mma.sync; any M is taken here,
// by one of two kernels (plan_for chooses).  Up to some 256 rows the problem is bound
// by the weight's bytes, so the tile is laid out around the weight stream: the WEIGHT
// rows are the 128-row "M" operand of tcgen05.mma and the activation rows are its "N"
// operand (16..256 columns), i.e. the kernels compute C^T tile by tile.  More rows run
// as CTA pairs on tiles of 256 weight rows (gemm_pair_sm100.cuh).  In the kernel of
// this file one CTA owns 128 weight rows x one K range:
//
//   warp 0   TMA producer: per 64-wide K step one 128 x 64 weight box and one
//            Mpad x 64 activation box (128-byte swizzle) into a ring of stages;
//   warp 1   allocates tensor memory, issues tcgen05.mma (as a whole warp, one
//            elected lane by predicate), hands stages back with tcgen05.commit;
//   all warps epilogue: tcgen05.ld of the fp32 accumulator (TMEM lane = weight
//            row, column = activation row) and bf16 stores.
//
// One SM draws some 0.16 MB/us through its stages (85 CTAs 3.4 TB/s of HBM, 72 with
// fewer activation rows a step 5.1), and a K step takes 0.2 us at least, so a weight
// with few 128-row tiles is also split along K: the CTAs of one output tile form a
// thread-block cluster, each leaves its fp32 partial tile in its own shared memory
// (the stage ring is free by then), and after a cluster barrier every CTA sums one
// slice of the rows over all peers through distributed shared memory and stores it.
// No global workspace and no atomics are involved.
//
// Takes the place of the reference's GemmSm100Op (src/machete/kernels/gemm/
// gemm_sm100.py:56-658), which tiles (S, N) with a double-buffered K loop inside
// its interpreter; this one is a plain launch next to the decode megakernel.
//
// Every wait is bounded: a wait that runs out records a status, raises a CTA-wide
// abort flag, and all roles fall through to the common exit, where tensor memory
// is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/machete_b200.h"
#include "prims.cuh"

namespace mkg {

constexpr int kThreads = 256;
constexpr int kTileN = 128;        // weight rows per CTA (the MMA's M)
constexpr int kTileK = 64;         // one 128-byte swizzle atom of bf16
constexpr int kMaxM = 256;         // activation rows per CTA (the MMA's N)
constexpr int kMaxStages = 8;
constexpr int kMaxSplit = 8;       // CTAs of one output tile (a portable cluster)
constexpr int kBars = 2 * kMaxStages + 2;
constexpr uint32_t kWBytes = kTileN * kTileK * 2;

struct Params {
  __nv_bfloat16* c;
  int32_t* status;       // [0] code, [1] cta, [2] role, [3] aux
  int64_t ldc;
  int M, N, K;
  int split_k, k_tiles;
  int stages;
  uint32_t ring_bytes;   // stages x stage bytes, or the fp32 partial tile if that is larger (split-K)
  int activation;        // applied to the fp32 sum before the bf16 store: 0 none, 1 relu, 2 silu
  int b_packed;          // the weight is stored K-tile-major: [K/64][N][64] (one box = 16 KB contiguous)
  int wide_store;        // C allows two-column stores
  int m_box;             // rows of one activation box (what one TMA copy delivers, whatever this CTA uses of it)
  uint64_t timeout_ns;
};

enum { GEMM_ST_OK = 0, GEMM_ST_TIMEOUT_EMPTY = 1, GEMM_ST_TIMEOUT_FULL = 2, GEMM_ST_TIMEOUT_ACC = 3 };

struct Shared {
  uint64_t full[kMaxStages];      // the barriers are initialised side by side, one lane each
  uint64_t empty[kMaxStages];
  uint64_t acc_ready;
  uint64_t drained;
  uint32_t tmem_base;
  int32_t abort_flag;
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(tmap), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const void* tmap, int c0, int c1, uint32_t bar, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
      "l"(tmap), "r"(c0), "r"(c1), "r"(bar), "l"(pol)
      : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of `addr` (a shared address of this CTA) in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// The issuing warp runs these as a whole and `elected` (elect_one(), taken once) predicates the instruction
// itself: without a branch around it the warp stays converged and the descriptors stay in uniform registers.
// Clocks per K step of four MMAs on 128 x N x 16, N = 64 / 128 / 256: 197 / 261 / 517 like this, 258 / 272 / 518
// with a branch on elect.sync, 460 / 460 / 518 with one lane in the loop; the first row is what the tensor
// pipe takes.
__device__ __forceinline__ void tc_commit(uint32_t bar, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(elected)
      : "memory");
}
// D[tmem] (+)= A[smem desc] x B[smem desc]^T, both operands K-major bf16, fp32 accumulate.
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                            uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
// 32 consecutive fp32 columns of this warp's 32 TMEM lanes: thread t gets lane t, columns c..c+31.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major bf16 tile stored as 128-byte rows with the
// 128-byte swizzle (what the TMA boxes above write): 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);          // start address, 16-byte units
  d |= (uint64_t)1 << 16;                           // leading-dimension offset: unused for swizzled K-major
  d |= (uint64_t)(1024 >> 4) << 32;                 // stride between 8-row groups
  d |= (uint64_t)1 << 46;                           // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                           // SWIZZLE_128B
  return d;
}
// kind::f16 instruction descriptor: fp32 accumulator, bf16 x bf16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t instr_desc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileN >> 4) << 24);
}

template <class P, class S>
__device__ __forceinline__ void give_up(const P& p, S* sh, int code, int role, int aux) {
  if (atomicCAS(&p.status[0], 0, code) == 0) {
    p.status[1] = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    p.status[2] = role;
    p.status[3] = aux;
  }
  atomicExch(&sh->abort_flag, 1);
  __threadfence();
}
// One thread waits for an mbarrier phase; false = aborted or out of time (recorded).
template <class P, class S>
__device__ __forceinline__ bool wait_bar(const P& p, S* sh, uint32_t bar, uint32_t parity, int code, int role, int aux) {
  // The clock is read only after a batch of failed polls: reading the global timer costs about as
  // much as a whole K step, and almost every wait succeeds within a few polls.
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    if (mk::mbar_try_wait(bar, parity)) return true;
    if ((spin & 255u) == 255u) {
      if (*reinterpret_cast<volatile int32_t*>(&sh->abort_flag)) return false;
      const uint64_t now = mk::globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > p.timeout_ns) {
        give_up(p, sh, code, role, aux);
        return false;
      }
    }
  }
}

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// The same wait for a whole warp: every lane polls, the outcome is the same for all.
template <class P, class S>
__device__ __forceinline__ bool wait_bar_warp(const P& p, S* sh, uint32_t bar, uint32_t parity, int code, int role, int aux) {
  if (__all_sync(0xffffffffu, mk::mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, wait_bar(p, sh, bar, parity, code, role, aux));
}

// The MMA warp waits, for a limited time, until the products that it issued are done: whether all is well (the
// epilogue waits for the same) or somebody has given up.
template <class P>
__device__ __forceinline__ void wait_drained(const P& p, uint32_t bar) {
  if (__all_sync(0xffffffffu, mk::mbar_try_wait(bar, 0))) return;
  const uint64_t t0 = mk::globaltimer_ns();
  while (!__all_sync(0xffffffffu, mk::mbar_try_wait(bar, 0)) && __all_sync(0xffffffffu, mk::globaltimer_ns() - t0 < p.timeout_ns)) {
  }
}

template <int ACT>
__device__ __forceinline__ float apply_act(float v) {
  if (ACT == 1) return fmaxf(v, 0.f);
  if (ACT == 2) return v / (1.f + __expf(-v));
  return v;
}
// Calls f with the activation as a compile-time constant: a branch per value costs more than the value.
template <class F>
__device__ __forceinline__ void with_act(int act, F f) {
  if (act == 0) f(std::integral_constant<int, 0>{});
  else if (act == 1) f(std::integral_constant<int, 1>{});
  else f(std::integral_constant<int, 2>{});
}

// 32 accumulator columns of one warp (lane = weight row `col`, register = activation row) -> C.  With `wide`
// neighbouring lanes swap every second value, so that a store is two columns of C and a warp writes two rows
// of 64 bytes at once.
template <int ACT>
__device__ __forceinline__ void store_columns(__nv_bfloat16* c, int64_t ldc, const uint32_t (&r)[32], int m, int rows, int col,
                                              bool col_ok, bool wide, int lane) {
  if (wide) {
    const int odd = lane & 1;
    __nv_bfloat16* dst = c + (int64_t)(m + odd) * ldc + (col - odd);
    const bool all = rows >= 32;
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float v0 = apply_act<ACT>(__uint_as_float(r[j])), v1 = apply_act<ACT>(__uint_as_float(r[j + 1]));
      const float other = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
      const uint32_t pk = mk::pack_bf16(odd ? other : v0, odd ? v1 : other);
      if (col_ok && (all || j + odd < rows)) *reinterpret_cast<uint32_t*>(dst) = pk;
      dst += 2 * ldc;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < rows && col_ok) c[(int64_t)(m + j) * ldc + col] = __float2bfloat16_rn(apply_act<ACT>(__uint_as_float(r[j])));
  }
}

// ---- split-K sum through distributed shared memory -----------------------------------------------------------
// The CTAs of one output tile each leave their fp32 partial, [row][128 weight rows], at `part` in their own shared
// memory (the stage ring is free by then); after a cluster barrier CTA `mine` of them sums its slice of the rows
// over all partials, in cluster order, and stores it.  All copies of a float4 are requested before the first is
// added: one trip instead of `split`.  (Pushing the slices into their owners' shared memory with st.async instead
// saves the barriers but runs far below the rate of these loads: 256 x 4096 x 4096 21.7 us against 15.8.)
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
template <class P>
__device__ __forceinline__ void reduce_slice(const P& p, uint32_t part, int rows, int first, int stride, int mine, int m0, int n0,
                                             int n_end, int threads) {
  const int per = (rows + p.split_k - 1) / p.split_k;
  const int lo = mine * per, hi = min(rows, lo + per);
  const bool wide = ((reinterpret_cast<uint64_t>(p.c) | (uint64_t)(p.ldc * 2)) & 7) == 0;
  with_act(p.activation, [&](auto act) {
    constexpr int ACT = decltype(act)::value;
    for (int idx = threadIdx.x; idx < (hi - lo) * (kTileN / 4); idx += threads) {
      const int ml = lo + (idx >> 5), nl = (idx & 31) * 4;
      const uint32_t off = part + (uint32_t)(ml * kTileN + nl) * 4u;
      float4 v[kMaxSplit];
#pragma unroll
      for (int i = 0; i < kMaxSplit; ++i)
        if (i < p.split_k) v[i] = ld_cluster_f4(peer_smem(off, (uint32_t)(first + stride * i)));
      float4 acc = v[0];
#pragma unroll
      for (int i = 1; i < kMaxSplit; ++i)
        if (i < p.split_k) acc.x += v[i].x, acc.y += v[i].y, acc.z += v[i].z, acc.w += v[i].w;
      const int n = n0 + nl;
      const float f[4] = {apply_act<ACT>(acc.x), apply_act<ACT>(acc.y), apply_act<ACT>(acc.z), apply_act<ACT>(acc.w)};
      __nv_bfloat16* dst = p.c + (int64_t)(m0 + ml) * p.ldc + n;
      if (wide && n + 4 <= n_end) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(mk::pack_bf16(f[0], f[1]), mk::pack_bf16(f[2], f[3]));
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < n_end) dst[e] = __float2bfloat16_rn(f[e]);
      }
    }
  });
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace mkg

#include "gemm_pair_sm100.cuh"

namespace mkg {

__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  // stages first (1024-byte aligned for the swizzle), the control block after them
  const uint32_t raw = mk::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw);
  const int m0 = blockIdx.z * kMaxM;
  const int m_here = min(kMaxM, p.M - m0);
  const int mpad = (m_here + 15) & ~15;                       // the MMA's N: a multiple of 16
  const uint32_t a_bytes = (uint32_t)p.m_box * kTileK * 2;
  const uint32_t stage_bytes = (kWBytes + a_bytes + 1023u) & ~1023u;
  Shared* sh = reinterpret_cast<Shared*>(smem + p.ring_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kTileN;
  const int n_end = min(p.N, n0 + kTileN);
  // this CTA's K steps
  const int per = (p.k_tiles + p.split_k - 1) / p.split_k;
  const int kt0 = blockIdx.y * per, kt1 = min(p.k_tiles, kt0 + per);
  const int n_steps = max(0, kt1 - kt0);
  uint32_t tmem_cols = 32;
  while ((int)tmem_cols < mpad) tmem_cols <<= 1;
  const uint32_t full0 = mk::smem_u32(&sh->full[0]), empty0 = mk::smem_u32(&sh->empty[0]);

  // The loads need only the barriers, so warp 0 initialises those and fills the ring before the CTA meets;
  // tensor memory is allocated meanwhile.
  const uint64_t pol = mk::l2_evict_first_policy();
  auto load = [&](int i, int s) {
    const uint32_t dst = base + (uint32_t)s * stage_bytes, bar = full0 + 8u * s;
    mk::mbar_arrive_expect_tx(bar, kWBytes + a_bytes);
    if (p.b_packed)
      mk::tma_load_3d(dst, &map_b, 0, n0, kt0 + i, bar, pol);
    else
      tma_load_2d_hint(dst, &map_b, (kt0 + i) * kTileK, n0, bar, pol);
    tma_load_2d(dst + kWBytes, &map_a, (kt0 + i) * kTileK, m0, bar);
  };
  const int ahead = min(p.stages, n_steps);
  if (warp == 0) {
    if (lane < kBars) mk::mbar_init(full0 + 8u * lane, 1);
    if (lane == 0) sh->abort_flag = 0;
    mk::fence_mbar_init();
    __syncwarp();
    mk::prior_work_done();
    if (elect_one())
      for (int i = 0; i < ahead; ++i) load(i, i);
  }
  if (warp == 1) tmem_alloc(mk::smem_u32(&sh->tmem_base), tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);
  mk::prior_work_done();

  if (warp == 0) {
    int issued = ahead, s = ahead == p.stages ? 0 : ahead;
    uint32_t ph = 0;                                          // the parity a reused slot's release is waited with
    for (int i = ahead; i < n_steps; ++i, ++issued) {
      if (!wait_bar_warp(p, sh, empty0 + 8u * s, ph, GEMM_ST_TIMEOUT_EMPTY, 0, i)) break;
      if (elect_one()) load(i, s);
      __syncwarp();
      if (++s == p.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
    mk::next_may_start();
    if (lane == 0 && *reinterpret_cast<volatile int32_t*>(&sh->abort_flag)) {
      // shared memory must outlive the copies still in flight: wait (bounded) for the stages that
      // were issued but perhaps never consumed
      for (int i = max(0, issued - p.stages); i < issued; ++i) {
        const uint32_t bar = full0 + 8u * (i % p.stages);
        const uint64_t t0 = mk::globaltimer_ns();
        while (!mk::mbar_try_wait(bar, (uint32_t)(i / p.stages) & 1u) && mk::globaltimer_ns() - t0 < p.timeout_ns) {
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(mpad), elected = elect_one() ? 1u : 0u;
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n_steps; ++i) {
      ok = wait_bar_warp(p, sh, full0 + 8u * s, ph, GEMM_ST_TIMEOUT_FULL, 1, i);
      if (!ok) break;
      tc_fence_after();
      const uint32_t w_addr = base + (uint32_t)s * stage_bytes;
      const uint64_t dw = smem_desc_sw128(w_addr), da = smem_desc_sw128(w_addr + kWBytes);
#pragma unroll
      for (int k = 0; k < kTileK / 16; ++k)     // 16 bf16 = 32 bytes = 2 descriptor units per MMA
        tc_mma_bf16(tmem, dw + 2u * k, da + 2u * k, idesc, (i > 0 || k > 0) ? 1u : 0u, elected);
      tc_commit(empty0 + 8u * s, elected);      // the stage is free once these MMAs have read it
      if (++s == p.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
    if (ok && n_steps > 0) tc_commit(mk::smem_u32(&sh->acc_ready), elected);
    // Whoever has given up: the products in flight still read shared memory and write tensor memory.
    tc_commit(mk::smem_u32(&sh->drained), elected);
    wait_drained(p, mk::smem_u32(&sh->drained));
  }
  // Epilogue on all eight warps: warp w may touch TMEM lanes 32 * (w % 4) .. and takes every second block of
  // 32 activation rows.
  {
    const int q = warp & 3;
    bool ready = n_steps > 0 && wait_bar_warp(p, sh, mk::smem_u32(&sh->acc_ready), 0, GEMM_ST_TIMEOUT_ACC, 2, warp);
    tc_fence_after();
    const int nl = q * 32 + lane, n = n0 + nl;
    // the stage ring is free: every copy was consumed before the accumulator was declared ready
    float* part = reinterpret_cast<float*>(smem) + nl;
    for (int c = (warp >> 2) * 32; c < mpad; c += 64) {
      uint32_t r[32];
      if (ready) {
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c, r);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = 0u;      // an empty K range (or an aborted CTA) adds nothing
      }
      if (p.split_k > 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c + j < mpad) part[(c + j) * kTileN] = __uint_as_float(r[j]);
      } else if (ready) {
        with_act(p.activation, [&](auto act) {
          store_columns<decltype(act)::value>(p.c, p.ldc, r, m0 + c, m_here - c, n, n < n_end, p.wide_store != 0, lane);
        });
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (p.split_k > 1) {
    // the CTAs of an output tile are one cluster, its rank = the K split
    cluster_arrive();
    cluster_wait();
    reduce_slice(p, base, m_here, 0, 1, (int)blockIdx.y, m0, n0, n_end, kThreads);
    cluster_arrive();
  }
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, tmem_cols);
  if (p.split_k > 1) cluster_wait();        // nobody leaves while a peer may still read its partial tile
}

static int ceil_div(int a, int b) { return (a + b - 1) / b; }
static int round_up(int a, int b) { return ceil_div(a, b) * b; }

static std::string g_err;
static int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(sym);
  return fn;
}
// Encoding a map costs about 2 us of host time, as much as the launch.  Each thread keeps the last maps it encoded
// by their sizes alone, direct-mapped by a hash; the address is put in on every call.
typedef CUresult (*ReplaceAddressFn)(CUtensorMap*, void*);
static ReplaceAddressFn replace_fn() {
  static ReplaceAddressFn fn = nullptr;
  if (fn) return fn;
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapReplaceAddress", &sym, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<ReplaceAddressFn>(sym);
  return fn;
}
struct MapKey {
  int64_t ld;
  int32_t rows, cols, box, kind;
  bool operator==(const MapKey& o) const {
    return ld == o.ld && rows == o.rows && cols == o.cols && box == o.box && kind == o.kind;
  }
};
template <class F>
static int cached_map(CUtensorMap* out, const void* base, const MapKey& key, F encode) {
  constexpr int kSlots = 64;
  struct Slot {
    MapKey key = {};
    CUtensorMap map;
  };
  static thread_local Slot slots[kSlots];
  uint64_t h = (uint64_t)key.ld * 0xC2B2AE3D27D4EB4Full ^ ((uint64_t)(uint32_t)key.rows << 32) ^
               (uint64_t)(uint32_t)(key.cols * 31 + key.box * 7 + key.kind);
  h ^= h >> 29;
  Slot& s = slots[(h * 0xBF58476D1CE4E5B9ull) >> 58];
  if (!(s.key == key)) {        // an unused slot has no columns
    const int rc = encode(&s.map);
    s.key = rc ? MapKey{} : key;
    if (rc) return rc;
    *out = s.map;
    return 0;
  }
  *out = s.map;
  ReplaceAddressFn fn = replace_fn();
  if (!fn) return fail(-5, "cuTensorMapReplaceAddress is not available from this driver");
  const CUresult r = fn(out, const_cast<void*>(base));
  if (r != CUDA_SUCCESS) return fail(-5, "cuTensorMapReplaceAddress failed with CUresult %d", (int)r);
  return 0;
}
// A row-major bf16 matrix [rows, K] with row stride `ld` elements; one box = 64 K values x box_rows rows.
static int encode_bf16_map(CUtensorMap* map, const void* base, int rows, int K, int64_t ld, int box_rows) {
  return cached_map(map, base, MapKey{ld, rows, K, box_rows, 1}, [&](CUtensorMap* out) -> int {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(-5, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)kTileK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(-5, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return 0;
  });
}

// The same matrix stored K-tile-major, [K/64][N][64]: dims (64, N, K/64), one box = 128 rows of one K tile,
// which is one contiguous 16 KB piece of memory.
static int encode_packed_map(CUtensorMap* map, const void* base, int N, int k_tiles) {
  return cached_map(map, base, MapKey{0, N, k_tiles, kTileN, 2}, [&](CUtensorMap* out) -> int {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(-5, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[3] = {(cuuint64_t)kTileK, (cuuint64_t)N, (cuuint64_t)k_tiles};
    cuuint64_t strides[2] = {(cuuint64_t)kTileK * 2, (cuuint64_t)N * kTileK * 2};
    cuuint32_t box[3] = {(cuuint32_t)kTileK, (cuuint32_t)kTileN, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(-5, "cuTensorMapEncodeTiled (packed weight) failed with CUresult %d", (int)r);
    return 0;
  });
}

struct Layout {
  uint64_t status_off, total;     // the workspace holds the status block only
};
static Layout layout_of(int, int) {
  Layout l;
  l.status_off = 0;
  l.total = 256;
  return l;
}

}  // namespace mkg

extern "C" {

const char* mk_gemm_last_error(void) { return mkg::g_err.c_str(); }

uint64_t mk_gemm_bf16_workspace_bytes(int M, int N, int K) {
  (void)K;
  if (M < 1 || N < 1) return 0;
  return mkg::layout_of(M, N).total;
}

}  // extern "C"

namespace mkg {

// What a launch needs to know of its device, read once per device (the kernels' shared-memory limits are
// raised at the same time).  Entries are written under the lock and never change afterwards.
struct Device {
  int sms = 0, smem_optin = 0, cc = 0;
  int clusters[kMaxSplit + 1] = {};           // clusters of this many CTAs of the split-K kernel that run at once
  int pair_clusters[kMaxPairSplit + 1] = {};  // clusters of this many pairs of the pair kernel
};
template <class F>
static int resident_clusters(F* kernel, int ctas, int threads, int smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}
static const Device* device_facts(int dev) {
  constexpr int kMax = 64;
  static Device facts[kMax];
  static std::atomic<bool> known[kMax];
  static std::mutex lock;
  if (dev < 0 || dev >= kMax) return nullptr;
  if (!known[dev].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> g(lock);
    if (!known[dev].load(std::memory_order_relaxed)) {
      Device d;
      if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
          cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
          cudaDeviceGetAttribute(&d.cc, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess)
        return nullptr;
      if (d.cc == 10) {
        if (cudaFuncSetAttribute(gemm_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, d.smem_optin) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, d.smem_optin) != cudaSuccess)
          return nullptr;
        d.clusters[1] = d.sms;
        for (int s = 2; s <= kMaxSplit; ++s) d.clusters[s] = resident_clusters(gemm_bf16_kernel, s, kThreads, d.smem_optin);
        for (int s = 1; s <= kMaxPairSplit; ++s) d.pair_clusters[s] = resident_clusters(gemm_pair_kernel, 2 * s, kPairThreads, d.smem_optin);
      }
      facts[dev] = d;
      known[dev].store(true, std::memory_order_release);
    }
  }
  return &facts[dev];
}

// Which kernel, and how the work is cut.  The model's terms were fitted to 5700 timings of every cut of 330 shapes
// (M 33..2048, N and K 1024..14336, the weight in HBM and in L2; half of them within 3 %, nine tenths within 8 %): a
// fixed part (launch, barriers, first load, tear-down), the K steps that a CTA walks one after another, the store of
// `cols` accumulator columns, and the exchange of a split.  A K step takes the longest of 0.197 us, its MMAs, its
// bytes at what one SM draws (0.16 MB/us), and all CTAs' bytes at what L2 gives (21.5 TB/s); a 128-byte piece of a
// row that does not begin on a 128-byte line costs more of both.  Where the weight comes from HBM its bytes set a floor under the
// steps, and near that floor both count.  The library cannot know where the weight lies, so a plan is judged by the
// mean of the two.  (By the longer of steps and bytes alone, every cut of a call near the floor costs the same and
// the fewest CTAs win: 66 x 5576 -> 8616 28.9 us unsplit on 68 CTAs, 23.9 split in two on 136; 59 x 10760 -> 5392
// 31.1 and 24.9, with pairs 24.2.)  Clusters that do not all run at once cost a second pass, so a split is taken
// only where they do; clusters that take every place there is wait for the very last of the kernel before them
// (3 to 20 % over the model, 42 x 1040 -> 5680 in three 7.6 us against 5.8 unsplit) and are charged 8 %.
struct Plan {
  bool pair = false;
  int split = 1, rows = 0;       // rows: activation rows per tile (pair kernel)
  float us = 1e30f;
};
static float line_cost(const void* base, int64_t row_elems) {
  const uint64_t bits = (uint64_t)base | (uint64_t)row_elems * 2;
  return bits % 128 == 0 ? 1.f : bits % 64 == 0 ? 1.08f : bits % 32 == 0 ? 1.24f : 1.85f;
}
static float modelled_us(float fixed, int steps, float bytes_per_step, int ctas, double weight_bytes, int cols, int split) {
  const float bytes = std::max(bytes_per_step / 0.16e6f, bytes_per_step * (float)ctas / 21.5e6f);
  const float walk = (float)steps * std::max(std::max(0.197f, 0.045f + 0.256f * (float)cols / kMaxM), bytes);
  const float hbm = (float)(weight_bytes / 6.5e6), w2 = walk * walk, h2 = hbm * hbm;
  const float cold = std::sqrt(std::sqrt(w2 * w2 + h2 * h2));
  return fixed + 0.5f * (walk + cold) + cols * 0.009f + (split > 1 ? 1.0f + cols * 0.0095f : 0.f);
}
static Plan plan_single(int M, int N, int K, const Device& d, int split, float line) {
  Plan best;
  const int k_tiles = ceil_div(K, kTileK), mt = ceil_div(M, kMaxM), mpad = round_up(std::min(M, kMaxM), 16);
  const int tiles = ceil_div(N, kTileN) * mt;
  for (int s = split > 0 ? split : 1; s <= (split > 0 ? split : kMaxSplit); ++s) {
    if (split == 0 && s > 1 && (s > k_tiles / 2 || d.clusters[s] < tiles)) break;
    const int steps = ceil_div(tiles, std::max(1, d.clusters[s])) * ceil_div(k_tiles, s);
    const float us = modelled_us(2.2f, steps, line * (float)((int)kWBytes + mpad * kTileK * 2), std::min(tiles * s, d.sms),
                                 2.0 * N * K, mpad, s) * (s > 1 && d.clusters[s] == tiles ? 1.08f : 1.f);
    if (us < best.us) best.split = s, best.us = us;
  }
  return best;
}
static Plan plan_pair(int M, int N, int K, const Device& d, float line) {
  Plan best;
  best.pair = true;
  const int k_tiles = ceil_div(K, kTileK), nt = ceil_div(N, kPairRows), mt0 = ceil_div(M, kMaxM);
  for (int mt = mt0; mt <= mt0 + 3; ++mt) {
    const int bn = round_up(ceil_div(M, mt), 16), tiles = ceil_div(M, bn) * nt;
    for (int s = 1; s <= kMaxPairSplit; ++s) {
      const int room = d.pair_clusters[s];
      if (room < 1 || (s > 1 && (s > k_tiles / 2 || tiles > room))) break;
      const int steps = ceil_div(tiles, room) * ceil_div(k_tiles, s);
      const float us = modelled_us(3.35f, steps, line * (float)((int)kWBytes + bn * kTileK), std::min(2 * tiles * s, d.sms),
                                   2.0 * N * K, bn, s);
      if (us < best.us) best.split = s, best.rows = bn, best.us = us;
    }
  }
  return best;
}
static Plan plan_for(int M, int N, int K, const Device& d, int split_k, float line) {
  const Plan single = plan_single(M, N, K, d, std::max(0, split_k), line);
  if (split_k > 0) return single;
  const Plan pair = plan_pair(M, N, K, d, line);
  return pair.us < single.us ? pair : single;
}

template <class F, class P>
static int launch(F* kernel, dim3 grid, dim3 cluster, int threads, size_t smem, void* stream, const CUtensorMap& map_a,
                  const CUtensorMap& map_b, const P& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  // The kernel may be placed while the one before it in the stream drains; it waits (prior_work_done) before its
  // first access to memory.
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster.x;
  attr[1].val.clusterDim.y = cluster.y;
  attr[1].val.clusterDim.z = cluster.z;
  cfg.attrs = attr;
  cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return fail(-(int)e - 1000, "mk_gemm_bf16 launch: %s", cudaGetErrorString(e));
  return 0;
}

static int pair_launch(const void* a, const void* b, void* c, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                       void* workspace, const Plan& plan, int timeout_ms, void* stream, bool b_packed, int activation,
                       const Device& d) {
  CUtensorMap map_a, map_b;
  const int k_tiles = ceil_div(K, kTileK), bn = plan.rows;
  int rc = encode_bf16_map(&map_a, a, M, K, lda, bn / 2);
  if (rc) return rc;
  rc = b_packed ? encode_packed_map(&map_b, b, N, k_tiles) : encode_bf16_map(&map_b, b, N, K, ldb, kTileN);
  if (rc) return rc;
  const uint32_t stage_bytes = kWBytes + (uint32_t)(bn / 2) * kTileK * 2;
  const int stages = std::min(kPairStages, (d.smem_optin - 1024 - (int)sizeof(PairShared)) / (int)stage_bytes);
  if (stages < 2) return fail(-4, "mk_gemm_bf16: shared memory holds fewer than two stages");
  PairParams p;
  p.c = reinterpret_cast<__nv_bfloat16*>(c);
  p.status = reinterpret_cast<int32_t*>(workspace);
  p.ldc = ldc;
  p.M = M, p.N = N, p.K = K;
  p.k_tiles = k_tiles, p.stages = stages, p.bn = bn, p.split_k = plan.split;
  p.ring_bytes = (uint32_t)stages * stage_bytes;
  if (plan.split > 1) p.ring_bytes = std::max(p.ring_bytes, (uint32_t)bn * kTileN * 4u);
  p.m_tiles = ceil_div(M, bn);
  p.tiles = p.m_tiles * ceil_div(N, kPairRows);
  p.activation = activation;
  p.b_packed = b_packed ? 1 : 0;
  p.wide_store = (N % 2 == 0 && ldc % 2 == 0 && ((uint64_t)c & 3) == 0) ? 1 : 0;
  p.timeout_ns = (uint64_t)(timeout_ms > 0 ? timeout_ms : 1000) * 1000000ull;
  const int clusters = plan.split > 1 ? p.tiles : std::min(p.tiles, d.pair_clusters[1]);
  // a pair holds all 512 columns of both its SMs: no CTA of the other kernel (38 KB or more) may share one with it
  const size_t smem = std::max(1024 + (size_t)p.ring_bytes + sizeof(PairShared), (size_t)d.smem_optin - 32768);
  return launch(gemm_pair_kernel, dim3((unsigned)(2 * plan.split * clusters)), dim3((unsigned)(2 * plan.split)), kPairThreads, smem,
                stream, map_a, map_b, p);
}

static int gemm_launch(const void* a, const void* b, void* c, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                       void* workspace, uint64_t workspace_bytes, int split_k, int timeout_ms, void* cuda_stream,
                       bool b_packed, int activation) {
  if (!a || !b || !c || !workspace) return fail(-1, "mk_gemm_bf16: null pointer");
  if (activation < 0 || activation > 2) return fail(-2, "mk_gemm_bf16: activation must be 0 (none), 1 (relu) or 2 (silu)");
  if (M < 1 || N < 1 || K < 1) return fail(-2, "mk_gemm_bf16: M, N, K must be positive (got %d, %d, %d)", M, N, K);
  if (K % 8 || lda % 8 || ldb % 8 || ((uint64_t)a & 15) || ((uint64_t)b & 15))
    return fail(-2, "mk_gemm_bf16: K and the row strides of A and B must be multiples of 8 elements, bases 16-byte aligned");
  if (lda < K || ldb < K || ldc < N) return fail(-2, "mk_gemm_bf16: a row stride is shorter than its row");
  if (((uint64_t)workspace & 255) != 0) return fail(-2, "mk_gemm_bf16: workspace must be 256-byte aligned");
  const Layout l = layout_of(M, N);
  if (workspace_bytes < l.total) return fail(-2, "mk_gemm_bf16: workspace of %llu bytes, need %llu",
                                             (unsigned long long)workspace_bytes, (unsigned long long)l.total);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(-1001, "cudaGetDevice failed");
  const Device* d = device_facts(dev);
  if (!d) return fail(-1001, "mk_gemm_bf16: cannot read the attributes of device %d", dev);
  if (d->cc != 10) return fail(-6, "mk_gemm_bf16 needs an sm_100 device (compute capability %d.x found)", d->cc);
  const int smem_optin = d->smem_optin;
  const int k_tiles = (K + kTileK - 1) / kTileK;
  if (split_k > k_tiles) split_k = k_tiles;
  if (split_k > kMaxSplit) return fail(-2, "mk_gemm_bf16: split_k is at most 8 (one portable thread-block cluster)");
  const Plan plan = plan_for(M, N, K, *d, split_k, b_packed ? 1.f : line_cost(b, ldb));
  if (plan.pair)
    return pair_launch(a, b, c, M, N, K, lda, ldb, ldc, workspace, plan, timeout_ms, cuda_stream, b_packed, activation, *d);
  split_k = plan.split;
  const int m_box = ((M < kMaxM ? M : kMaxM) + 15) & ~15;
  CUtensorMap map_a, map_b;
  int rc = encode_bf16_map(&map_a, a, M, K, lda, m_box);
  if (rc) return rc;
  rc = b_packed ? encode_packed_map(&map_b, b, N, k_tiles) : encode_bf16_map(&map_b, b, N, K, ldb, kTileN);
  if (rc) return rc;
  const uint32_t stage_bytes = (kWBytes + (uint32_t)m_box * kTileK * 2 + 1023u) & ~1023u;
  int stages = (smem_optin - 2048) / (int)stage_bytes;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages < 2) return fail(-4, "mk_gemm_bf16: shared memory holds fewer than two stages");
  const int per = (k_tiles + split_k - 1) / split_k;
  if (stages > per) stages = per < 2 ? 2 : per;
  uint32_t ring_bytes = (uint32_t)stages * stage_bytes;
  if (split_k > 1) ring_bytes = std::max(ring_bytes, (uint32_t)m_box * kTileN * 4u);
  size_t smem = 1024 + (size_t)ring_bytes + sizeof(Shared);
  if (split_k > 1) {
    // CTAs of a cluster wait for one another while they hold tensor memory: no more of them (of this launch or of
    // one in another stream) may share an SM than its 512 columns serve, or they could wait in a circle.
    int cols = 32;
    while (cols < m_box) cols <<= 1;
    smem = std::max(smem, std::min((size_t)smem_optin, (size_t)smem_optin * cols / 512 + 1024));
  }
  Params p;
  uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
  p.c = reinterpret_cast<__nv_bfloat16*>(c);
  p.status = reinterpret_cast<int32_t*>(ws + l.status_off);
  p.ldc = ldc;
  p.M = M, p.N = N, p.K = K;
  p.split_k = split_k, p.k_tiles = k_tiles, p.stages = stages, p.m_box = m_box, p.b_packed = b_packed ? 1 : 0;
  p.ring_bytes = ring_bytes;
  p.activation = activation;
  p.wide_store = (N % 2 == 0 && ldc % 2 == 0 && ((uint64_t)c & 3) == 0) ? 1 : 0;
  p.timeout_ns = (uint64_t)(timeout_ms > 0 ? timeout_ms : 1000) * 1000000ull;
  return launch(gemm_bf16_kernel, dim3((unsigned)ceil_div(N, kTileN), (unsigned)split_k, (unsigned)ceil_div(M, kMaxM)),
                dim3(1, (unsigned)split_k, 1), kThreads, smem, cuda_stream, map_a, map_b, p);
}
}  // namespace mkg

extern "C" {

int mk_gemm_bf16(const void* a, const void* b, void* c, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                 void* workspace, uint64_t workspace_bytes, int split_k, int activation, int timeout_ms,
                 void* cuda_stream) {
  return mkg::gemm_launch(a, b, c, M, N, K, lda, ldb, ldc, workspace, workspace_bytes, split_k, timeout_ms, cuda_stream,
                          false, activation);
}

int mk_gemm_bf16_packed(const void* a, const void* b_packed, void* c, int M, int N, int K, int64_t lda, int64_t ldc,
                        void* workspace, uint64_t workspace_bytes, int split_k, int activation, int timeout_ms,
                        void* cuda_stream) {
  if (K % 64) return mkg::fail(-2, "mk_gemm_bf16_packed: K must be a multiple of 64 (the packer pads with zeros)");
  return mkg::gemm_launch(a, b_packed, c, M, N, K, lda, K, ldc, workspace, workspace_bytes, split_k, timeout_ms,
                          cuda_stream, true, activation);
}

int mk_gemm_bf16_call(const void* call) {
  if (!call) return mkg::fail(-1, "mk_gemm_bf16_call: null pointer");
  mk_gemm_call_t c;
  memcpy(&c, call, sizeof(c));
  const void *a = reinterpret_cast<const void*>(c.a), *b = reinterpret_cast<const void*>(c.b);
  void *out = reinterpret_cast<void*>(c.c), *ws = reinterpret_cast<void*>(c.workspace), *stream = reinterpret_cast<void*>(c.cuda_stream);
  if (c.packed)
    return mk_gemm_bf16_packed(a, b, out, c.M, c.N, c.K, c.lda, c.ldc, ws, c.workspace_bytes, (int)c.split_k, c.activation,
                               (int)c.timeout_ms, stream);
  return mk_gemm_bf16(a, b, out, c.M, c.N, c.K, c.lda, c.ldb, c.ldc, ws, c.workspace_bytes, (int)c.split_k, c.activation,
                      (int)c.timeout_ms, stream);
}

int mk_gemm_bf16_plan(int M, int N, int K, int64_t ldb, int32_t out[4]) {
  using namespace mkg;
  if (!out || M < 1 || N < 1 || K < 1) return fail(-2, "mk_gemm_bf16_plan: M, N, K must be positive and out given");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(-1001, "cudaGetDevice failed");
  const Device* d = device_facts(dev);
  if (!d) return fail(-1001, "mk_gemm_bf16_plan: cannot read the attributes of device %d", dev);
  if (d->cc != 10) return fail(-6, "mk_gemm_bf16_plan needs an sm_100 device (compute capability %d.x found)", d->cc);
  const Plan plan = plan_for(M, N, K, *d, 0, ldb > 0 ? line_cost(nullptr, ldb) : 1.f);
  const int rows = plan.pair ? plan.rows : std::min(M, kMaxM), tiles = ceil_div(M, rows) * ceil_div(N, plan.pair ? kPairRows : kTileN);
  out[0] = plan.pair ? 1 : 0;
  out[1] = plan.split;
  out[2] = rows;
  out[3] = tiles;
  return 0;
}

int mk_gemm_bf16_status(const void* workspace, int32_t out[4]) {
  using namespace mkg;
  if (!workspace || !out) return fail(-1, "mk_gemm_bf16_status: null pointer");
  if (cudaDeviceSynchronize() != cudaSuccess) return fail(-1001, "mk_gemm_bf16_status: device synchronise failed");
  if (cudaMemcpy(out, workspace, 16, cudaMemcpyDeviceToHost) != cudaSuccess)
    return fail(-1001, "mk_gemm_bf16_status: copy failed");
  return 0;
}

}  // extern "C"
