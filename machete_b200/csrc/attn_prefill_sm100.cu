// Prefill attention on the 5th-generation tensor cores: O = softmax(scale · Q Kᵀ) V for a block of
// query rows against a KV cache, bf16, causal or not, grouped-query heads.
//
// The decode megakernel's own attention op streams K/V once per KV head for a handful of query rows
// (mma.sync).  A prompt has hundreds of query rows per head, which is tensor-core work: this kernel
// takes the place of the reference's FlashAttentionSm100Op (src/machete/kernels/attention/
// sm_100.py:88-…, dispatch attention/__init__.py:16-130) as a launch of its own, so that a prompt can
// fill the KV cache the decode kernel then reads.
//
// A tile is 128 query rows of one batch entry, the rows being 128 / g queries of the g query heads that share a KV head (the
// power of two in the group); KV tiles of 64 tokens.  Two forms:
//   * one tile a CTA, two CTAs to an SM (<= 97 KB of shared memory and 256 tensor-memory columns each), two S accumulators;
//   * (head dim 64) three tiles a CTA, one CTA to an SM, which share the K and V tiles: each tile has one S accumulator and
//     room for P behind it (160 columns), and S(j + 1) is issued as soon as the row threads hold S(j).  Three row warps a
//     scheduler hide more of one another's latencies than two (777 queries behind 2223 tokens, two sequences, us: three CTAs of
//     one accumulator each, whose S waited for the P V before, 58.7; so 50.5; 4096 x 4096 102 / 90).
//
//   load warp     TMA: Q once, then K and V tiles (four each, at 128 two; K one tile ahead of V) as 64-column boxes, 128-byte
//                 swizzle;
//   product warps one a tile, tcgen05.mma: S(j) = Q K(j)^T one tile ahead of the softmax, and O += P(j) V(j) with P read
//                 FROM TENSOR MEMORY (the M x K operand) and V as the N operand in MN-major form (its head dimension is
//                 contiguous in shared memory exactly as the cache stores it);
//   row warps     four a tile, one thread per query row (= tensor-memory lane): one tcgen05.ld of the row of S(j), mask,
//                 maximum, P = exp2(scale * s - reference) with packed f32x2 arithmetic, running sum in
//                 registers (no shuffles: a thread owns its row), P stored as bf16 pairs (tcgen05.st; with two accumulators
//                 over the first half of the one it came from), O rescaled in tensor memory only when a row
//                 maximum outgrew the exponent reference by 2^8; normalised bf16 store at the end.
//
// The row threads hardly wait for P V: while the tensor cores run P(j) V(j) and the next S they are already on tile j + 1, so the
// exponentials (the scarce unit: 16 per clock and SM) and the products overlap inside one tile, and the other tiles of the
// SM fill what is left.  What bounds it: at head dim 64 the row threads' instructions (some 360 a warp and KV tile; ncu on the
// chunk above: issue slots 60 %, exp2 unit 50 %, fma 45 %, alu 40 %, tensor pipe 53 % of active cycles); at 128 the tensor pipe, whose
// 64-wide S products are held up by shared memory.  Measured and left out: KV tiles of 128 tokens (4096 x 4096, head dim 64
// 109 -> 116 us, 128 124 -> 141: the same instructions with more registers); the maximum taken beside the exponentials, and these
// taken again where it grew (50.5 -> 55); one warp for all tiles' products (no change).
//
// Every wait is bounded; on expiry the CTA records a status, raises its abort flag, all roles fall
// through to the common exit and tensor memory is freed.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
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

namespace mkp {

constexpr int kBM = 128;   // query rows of a tile
constexpr int kBN = 64;    // tokens per KV tile
constexpr uint32_t kBox = 128 * 64 * 2;   // one 128-row x 64-column bf16 box

struct Params {
  __nv_bfloat16* o;
  float* lse;            // [B, H, M] or null
  int32_t* status;
  int64_t o_sb, o_sh, o_sm;
  int B, H, Hkv, M, N;
  uint32_t negate_q;     // the product descriptor's bit that takes -Q (a negative scale)
  int causal;
  int row_tiles;
  int pack, pack_log2;   // query heads of a KV head in one tile: row r is query r >> pack_log2 of head r & (pack - 1)
  int next_early;        // the kernel behind this one may be placed from the start (else: with the last load)
  float scale_log2;      // |scale| * log2(e), > 0
  uint64_t timeout_ns;
};

enum { PF_ST_TIMEOUT_EMPTY = 1, PF_ST_TIMEOUT_FULL = 2, PF_ST_TIMEOUT_S = 3, PF_ST_TIMEOUT_P = 4, PF_ST_TIMEOUT_O = 5 };

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* tmap, int c0, int c1, int c2, int c3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
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
// The issuing warp runs these as a whole and `elected` (one lane of it) predicates the instruction itself: with
// one lane in the loop, or a branch around the instruction, the descriptors leave the uniform registers and an
// MMA costs 115 clocks of issue, more than the tensor pipe takes for it (128 x 64 x 16: 48 clocks).
__device__ __forceinline__ void tc_commit(uint32_t bar, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                       uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate,
                                          uint32_t elected) {
  // the M x K operand comes from tensor memory (lane = row, one 32-bit column = two bf16 along K)
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.ftz.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
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
// one row of a 64-column accumulator; the wait is part of the statement so that nothing reads r before it
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&r)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 {"
      "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
      "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Two fp32 operations per instruction (the packed f32x2 forms of sm_100): the softmax of one score costs the
// issue slots of half a multiply-add, one exp2, half an add and half a conversion.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// 2^x for two values on the FMA and integer pipes instead of the exp2 unit (16 results per clock and SM,
// the scarce unit at head dim 64): x = n + f with n = round(x) by the 1.5 * 2^23 addition, f in [-0.5, 0.5];
// 2^f by a cubic fitted here for the smallest maximal relative error (7.5e-5, far inside bf16's 2^-9), and
// n added to the exponent field.  x <= 8 by construction; below -126 it is clamped (the result, ~1e-38,
// rounds into nothing next to the row's maximum of at least 2^-8).
// Measured at 32 heads x 4096 x 4096: head dim 64, every third pair of scores on this path, 113 -> 109 us
// (every second: 114); head dim 128, where the tensor pipe is the bound, 131 -> 135 us: used at 64 only.
#ifndef MK_PF_POLY
#define MK_PF_POLY 3      /* head dim 64: every MK_PF_POLY-th pair of scores takes this path on unmasked tiles (0 = none) */
#endif
__device__ __forceinline__ void exp2_poly2(uint64_t x2, float& e0, float& e1) {
  float x0, x1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(x2));
  x0 = fmaxf(x0, -126.f);
  x1 = fmaxf(x1, -126.f);
  uint64_t xc, r, t, f, pl;
  asm("mov.b64 %0, {%1, %2};" : "=l"(xc) : "f"(x0), "f"(x1));
  const uint64_t magic = 0x4B4000004B400000ull, nmagic = 0xCB400000CB400000ull, neg1 = 0xBF800000BF800000ull;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(xc), "l"(magic));
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(t) : "l"(r), "l"(nmagic));
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(f) : "l"(t), "l"(neg1), "l"(xc));
  // Horner: ((c3 f + c2) f + c1) f + c0
  const uint64_t c3 = 0x3D61FBB03D61FBB0ull, c2 = 0x3E786F0D3E786F0Dull, c1 = 0x3F31798D3F31798Dull, c0 = 0x3F7FFB493F7FFB49ull;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(pl) : "l"(c3), "l"(f), "l"(c2));
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(pl) : "l"(pl), "l"(f), "l"(c1));
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(pl) : "l"(pl), "l"(f), "l"(c0));
  uint32_t p0, p1, r0, r1;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(p0), "=r"(p1) : "l"(pl));
  asm("mov.b64 {%0, %1}, %2;" : "=r"(r0), "=r"(r1) : "l"(r));
  e0 = __uint_as_float(p0 + (r0 << 23));
  e1 = __uint_as_float(p1 + (r1 << 23));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// K-major bf16 tile of 128-byte swizzled rows (8-row groups 1024 bytes apart): Q, K and P.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
// MN-major bf16 tile: V as stored, [token][64 head-dim values = 128 bytes], 128-byte swizzle.  Along K (tokens)
// the 8-row groups are 1024 bytes apart (stride offset); along N (head dim) the next 64 values are the next
// box, `next_box` bytes further (leading offset).
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t addr, uint32_t next_box) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((next_box >> 4) & 0x3FFF) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// kind::f16, fp32 accumulate, bf16 operands, M = 128, N = n; b_mn = the N operand is MN-major.
__device__ __forceinline__ uint32_t idesc_bf16(int n, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}

__device__ __forceinline__ void give_up(const Params& p, int32_t* abort_flag, int code, int aux) {
  if (atomicCAS(&p.status[0], 0, code) == 0) {
    p.status[1] = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    p.status[2] = threadIdx.x >> 5;
    p.status[3] = aux;
  }
  atomicExch(abort_flag, 1);
  __threadfence();
}
__device__ __forceinline__ bool wait_bar(const Params& p, int32_t* abort_flag, uint32_t bar, uint32_t parity, int code, int aux) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    if (mk::mbar_try_wait(bar, parity)) return true;
    if ((spin & 255u) == 255u) {
      if (*reinterpret_cast<volatile int32_t*>(abort_flag)) return false;
      const uint64_t now = mk::globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > p.timeout_ns) {
        give_up(p, abort_flag, code, aux);
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

__device__ __forceinline__ void arrive_if(uint32_t bar, bool yes) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"((uint32_t)yes)
               : "memory");
}
// Waits that find their phase complete, which most do, run straight on, and what is rare stands out of line: by device clocks a taken
// branch in the row threads' loop costs some forty of them.  (With the slow paths in the loop and so, us: a tile that has its SM to
// itself, 128 queries behind 3968 tokens, head dim 64 42.2 / 38.4, 128 50.8 / 44.8; 777 queries behind 2223 tokens, two sequences, head
// dim 128 78.6 / 70.1.  Of the lone tile at 128, ncu, stalled warps an issue: fixed latencies 2.47 / 1.96, long scoreboard 1.19 / 1.03, branches
// being resolved 0.56 / 0.46, no instruction 0.30 / 0.27: it is the branches' own latency more than the fetch behind them.)
__device__ __noinline__ bool wait_cold(const Params& p, int32_t* abort_flag, uint32_t bar, uint32_t parity, int code, int aux) {
  return __all_sync(0xffffffffu, wait_bar(p, abort_flag, bar, parity, code, aux));
}
__device__ __forceinline__ bool wait_hot(const Params& p, int32_t* abort_flag, uint32_t bar, uint32_t parity, int code, int aux) {
  if (__builtin_expect(__all_sync(0xffffffffu, mk::mbar_try_wait(bar, parity)), 1)) return true;
#pragma unroll 1
  for (int i = 0; i < 64; ++i)
    if (mk::mbar_try_wait(bar, parity)) break;
  if (__all_sync(0xffffffffu, mk::mbar_try_wait(bar, parity))) return true;
  return wait_cold(p, abort_flag, bar, parity, code, aux);
}
// O of this thread's row times alpha, once the P V that `bar` tells of has finished with it.
template <int D>
__device__ __noinline__ bool rescale(const Params& p, int32_t* abort_flag, uint32_t o_addr, float alpha, uint32_t bar, uint32_t parity, int j) {
  if (!wait_hot(p, abort_flag, bar, parity, PF_ST_TIMEOUT_O, j)) return false;
  tc_fence_after();
#pragma unroll 1
  for (int c = 0; c < D; c += 32) {
    uint32_t o[32];
    tmem_ld32(o_addr + (uint32_t)c, o);
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
    tmem_st32(o_addr + (uint32_t)c, o);
  }
  return true;
}

// A CTA's shape: T tiles of 128 query rows that share the K and V tiles, each with four warps of row threads and a warp that
// issues its products, and a warp for the loads.
template <int D, int T>
struct Form {
  static constexpr int kThreads = (5 * T + 1) * 32;
  static constexpr int kPerSm = T == 1 ? 2 : 1;
  static constexpr int NB = D / 64;                       // 64-column boxes of a row
  static constexpr uint32_t kQTile = NB * kBox, kKVBox = kBN * 64 * 2, kKVTile = NB * kKVBox;
  static constexpr int KS = D == 128 ? 2 : 4, VS = KS;   // K and V tiles in flight
  // tensor memory of a tile: O, then two S accumulators of which P (bf16 pairs) takes the first half, or (three tiles) one and P behind it
  static constexpr int SB = T == 1 ? 2 : 1;
  static constexpr uint32_t kTileCols = D + (SB == 2 ? 2 * kBN : kBN + kBN / 2), kCols = T == 1 ? 256 : 512;
  static_assert(T * kTileCols <= kCols, "accumulators must fit the allocation");
  struct Shared {
    uint64_t q_full[T], s_full[2 * T], s_free[T], p_ready[2 * T], pv_done[2 * T], k_full[KS], k_empty[KS], v_full[VS], v_empty[VS];
    uint32_t tmem_base;
    int32_t abort_flag;
  };
  static constexpr size_t kSmem = (size_t)T * kQTile + (size_t)(KS + VS) * kKVTile + sizeof(Shared);
};

template <int D, int T>
__global__ void __launch_bounds__(Form<D, T>::kThreads, Form<D, T>::kPerSm)
prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ Params p) {
  using F = Form<D, T>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t q_s = mk::smem_u32(smem), k_s = q_s + T * F::kQTile, v_s = k_s + F::KS * F::kKVTile;
  typename F::Shared* sh = reinterpret_cast<typename F::Shared*>(smem + T * F::kQTile + (F::KS + F::VS) * F::kKVTile);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kLoadWarp = 5 * T;
  // Blocks are handed out in the order x, y, z: the query tiles are the slowest index and run from the LAST tile
  // down, so that under a causal mask the tiles with the most KV tiles start first and the short ones fill the
  // tail (longest job first).
  // The tile's 128 rows are 128 / pack queries of `pack` heads that share a KV head: a prompt of 777 queries and four
  // heads a KV head is 25 tiles, not 4 x 7, and fewer pairs lie behind the diagonal (32 / 8 heads, causal, us with one head a
  // tile and four: 2190 x 2190 head dim 128 50.6 / 46.3, 64 39.4 / 35.5; 1960 of 2045, four sequences, 170.4 / 156.2 and 120.5 / 106.5;
  // 4096 x 4096 137.8 / 135.7 and 95.9 / 94.4).
  const int h0 = blockIdx.x * p.pack, b = blockIdx.y;
  const int kvh = h0 / (p.H / p.Hkv);
  const int tile_m = kBM >> p.pack_log2;
  auto first_row = [&](int i) { return (p.row_tiles - 1 - ((int)blockIdx.z * T + i)) * tile_m; };   // negative: no such tile
  // KV tiles that a query tile can see: of all N tokens, or (causal) up to the diagonal of its last row
  auto kv_tiles = [&](int i) {
    const int m0 = first_row(i);
    if (m0 < 0) return 0;
    const int n_vis = p.causal ? min(p.N, p.N - p.M + m0 + tile_m) : p.N;
    return n_vis > 0 ? (n_vis + kBN - 1) / kBN : 0;
  };
  int n_tiles[T];
#pragma unroll
  for (int i = 0; i < T; ++i) n_tiles[i] = kv_tiles(i);
  const int n_most = n_tiles[0];

  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < T; ++i) {
      mk::mbar_init(mk::smem_u32(&sh->q_full[i]), 1);
      mk::mbar_init(mk::smem_u32(&sh->s_free[i]), 4);
      for (int k = 2 * i; k < 2 * i + 2; ++k) {
        mk::mbar_init(mk::smem_u32(&sh->s_full[k]), 1);
        mk::mbar_init(mk::smem_u32(&sh->p_ready[k]), 4);
        mk::mbar_init(mk::smem_u32(&sh->pv_done[k]), 1);
      }
    }
    for (int s = 0; s < F::KS; ++s) {
      mk::mbar_init(mk::smem_u32(&sh->k_full[s]), 1);
      mk::mbar_init(mk::smem_u32(&sh->k_empty[s]), T);
    }
    for (int s = 0; s < F::VS; ++s) {
      mk::mbar_init(mk::smem_u32(&sh->v_full[s]), 1);
      mk::mbar_init(mk::smem_u32(&sh->v_empty[s]), T);
    }
    sh->abort_flag = 0;
    mk::fence_mbar_init();
  }
  __syncwarp();
  if (warp == kLoadWarp) tmem_alloc(mk::smem_u32(&sh->tmem_base), F::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&sh->tmem_base);
  constexpr int SB = F::SB;
  constexpr uint32_t kSCol = D, kPCol = D + (SB == 2 ? 0 : kBN);
  int32_t* flag = &sh->abort_flag;
  mk::prior_work_done();
  if (p.next_early) mk::next_may_start();

  if (warp == kLoadWarp) {
    if (lane == 0) {
      auto load_q = [&](int i) {
        if (n_tiles[i] == 0) return;
        const uint32_t qb = mk::smem_u32(&sh->q_full[i]);
        mk::mbar_arrive_expect_tx(qb, F::kQTile);
        for (int x = 0; x < F::NB; ++x) tma_load_4d(q_s + i * F::kQTile + x * kBox, &map_q, x * 64, h0, first_row(i), b, qb);
      };
      auto load_kv = [&](int j, bool is_v) -> bool {
        const int n = is_v ? F::VS : F::KS, s = j % n;
        const uint32_t ph = (uint32_t)(j / n) & 1u;
        uint64_t* empty = is_v ? &sh->v_empty[s] : &sh->k_empty[s];
        uint64_t* full = is_v ? &sh->v_full[s] : &sh->k_full[s];
        if (!wait_bar(p, flag, mk::smem_u32(empty), ph ^ 1u, PF_ST_TIMEOUT_EMPTY, j)) return false;
        const uint32_t fb = mk::smem_u32(full);
        mk::mbar_arrive_expect_tx(fb, F::kKVTile);
        const uint32_t dst = (is_v ? v_s : k_s) + (uint32_t)s * F::kKVTile;
        for (int x = 0; x < F::NB; ++x) tma_load_4d(dst + x * F::kKVBox, is_v ? &map_v : &map_k, x * 64, j * kBN, kvh, b, fb);
        return true;
      };
      // K runs one tile ahead of V: S(j + 1) is issued before P(j) V(j)
      load_q(0);
      bool pok = n_most > 0 ? load_kv(0, false) : true;
#pragma unroll
      for (int i = 1; i < T; ++i) load_q(i);
      for (int j = 0; j < n_most && pok; ++j) {
        if (j + 1 < n_most && !load_kv(j + 1, false)) break;
        if (!load_kv(j, true)) break;
      }
      mk::next_may_start();
      if (*reinterpret_cast<volatile int32_t*>(flag)) {
        // shared memory must outlive the copies in flight: a bounded wait for whatever was issued last
        const uint64_t t0 = mk::globaltimer_ns();
        while (mk::globaltimer_ns() - t0 < 20000ull) {
        }
      }
    }
  } else if (warp >= 4 * T) {
    // products of tile i, in the order S(0), S(1), P V(0), S(2), P V(1), ...
    // (By the whole warp at head dim 128 as well.  us, one lane that waits and issues / the warp, causal: 512 x 512 11.7 / 10.7, 300 behind 1700
    // tokens 30.3 / 26.0, 2190 x 2190 50.7 / 49.9, 4096 x 4096 153.2 / 149.7, no mask 311 / 271.)
    // (the tile, and with it every descriptor, is known to be uniform: see tc_mma)
    const int i = T == 1 ? 0 : __shfl_sync(0xffffffffu, warp - 4 * T, 0), nt = kv_tiles(i);
    const uint32_t id_s = idesc_bf16(kBN, false) | p.negate_q, id_o = idesc_bf16(D, true), elected = elect_one() ? 1u : 0u;
    const uint32_t o = tmem + i * F::kTileCols, q = q_s + i * F::kQTile;
    const uint32_t s_full = mk::smem_u32(&sh->s_full[2 * i]), s_free = mk::smem_u32(&sh->s_free[i]);
    const uint32_t p_ready = mk::smem_u32(&sh->p_ready[2 * i]), pv_done = mk::smem_u32(&sh->pv_done[2 * i]);
    auto issue_s = [&](int j) -> bool {
      const int s = j % F::KS;
      if (!wait_hot(p, flag, mk::smem_u32(&sh->k_full[s]), (uint32_t)(j / F::KS) & 1u, PF_ST_TIMEOUT_FULL, j)) return false;
      if (SB == 1 && j > 0 && !wait_hot(p, flag, s_free, (uint32_t)(j - 1) & 1u, PF_ST_TIMEOUT_S, j)) return false;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const uint32_t in_box = (uint32_t)(k & 3) * 32u;
        tc_mma(o + kSCol + (uint32_t)(j % SB) * kBN, desc_kmajor(q + (uint32_t)(k >> 2) * kBox + in_box),
               desc_kmajor(k_s + s * F::kKVTile + (uint32_t)(k >> 2) * F::kKVBox + in_box), id_s, k > 0 ? 1u : 0u, elected);
      }
      tc_commit(s_full + (uint32_t)(j % SB) * 8u, elected);
      tc_commit(mk::smem_u32(&sh->k_empty[s]), elected);
      return true;
    };
    bool ok = nt == 0 || (wait_hot(p, flag, mk::smem_u32(&sh->q_full[i]), 0, PF_ST_TIMEOUT_FULL, -1) && issue_s(0));
#pragma unroll 1
    for (int j = 0; j < nt && ok; ++j) {
      if (__builtin_expect(j + 1 < nt, 1)) ok = issue_s(j + 1);
      if (!ok) break;
      const int s = j % F::VS;
      // O += P V once the row threads have written P (and rescaled O)
      ok = wait_hot(p, flag, p_ready + (uint32_t)(j % SB) * 8u, (uint32_t)(j / SB) & 1u, PF_ST_TIMEOUT_P, j) &&
           wait_hot(p, flag, mk::smem_u32(&sh->v_full[s]), (uint32_t)(j / F::VS) & 1u, PF_ST_TIMEOUT_FULL, j);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < kBN / 16; ++k) {
        // P: 16 tokens = 8 tensor-memory columns of bf16 pairs; V: MN-major, 16 tokens = 16 rows of 128 bytes
        const uint64_t dv = desc_mnmajor(v_s + (uint32_t)s * F::kKVTile + (uint32_t)k * 2048u, F::kKVBox);
        tc_mma_ts(o, o + kPCol + (uint32_t)(j % SB) * kBN + (uint32_t)k * 8u, dv, id_o, (j > 0 || k > 0) ? 1u : 0u, elected);
      }
      tc_commit(pv_done + (uint32_t)(j % SB) * 8u, elected);
      tc_commit(mk::smem_u32(&sh->v_empty[s]), elected);
    }
    // of the KV tiles that only the longer tiles have, this one is done with each slot as soon as it is filled
    for (int j = nt; j < n_most && ok; ++j) {
      ok = wait_hot(p, flag, mk::smem_u32(&sh->k_full[j % F::KS]), (uint32_t)(j / F::KS) & 1u, PF_ST_TIMEOUT_FULL, j);
      if (ok && elected) mk::mbar_arrive(mk::smem_u32(&sh->k_empty[j % F::KS]));
      ok = ok && wait_hot(p, flag, mk::smem_u32(&sh->v_full[j % F::VS]), (uint32_t)(j / F::VS) & 1u, PF_ST_TIMEOUT_FULL, j);
      if (ok && elected) mk::mbar_arrive(mk::smem_u32(&sh->v_empty[j % F::VS]));
    }
  } else if (first_row(warp >> 2) >= 0) {
    // row threads: warp w may touch tensor-memory lanes 32 * (w % 4) ..
    const int ti = warp >> 2, qd = warp & 3;
    const int nt = kv_tiles(ti);
    const int row = qd * 32 + lane;                 // query row inside the tile = TMEM lane
    const int m = first_row(ti) + (row >> p.pack_log2), h = h0 + (row & (p.pack - 1));
    const int lim = p.causal ? (p.N - p.M + m) : (p.N - 1);   // last visible token of this row
    // Only the tiles on the causal diagonal and the last one of a ragged cache need the per-score mask; the first n_open
    // do not.  They take another mix of exponentials (exp2_poly2), so which they are is a matter of results: it goes by
    // blocks of 32 queries, whatever the heads in a tile.  (Every row of a warp is in one block.)
    const int n_open = min(p.causal ? p.N - p.M + (m & ~31) + 1 : p.N, p.N) / kBN;
    const uint32_t lane_addr = tmem + (uint32_t)ti * F::kTileCols + ((uint32_t)(qd * 32) << 16);
    const uint32_t s_full = mk::smem_u32(&sh->s_full[2 * ti]), s_free = mk::smem_u32(&sh->s_free[ti]);
    const uint32_t p_ready = mk::smem_u32(&sh->p_ready[2 * ti]), pv_done = mk::smem_u32(&sh->pv_done[2 * ti]);
    const uint64_t scale2 = pack2(p.scale_log2, p.scale_log2);
    float mx = -INFINITY, sum = 0.f;
    bool ok = true;
    // One KV tile, in straight code (see wait_hot); masked tiles have a copy of their own.
    const int n_plain = min(nt, __shfl_sync(0xffffffffu, n_open, 0));   // (known to be uniform)
    auto kv_tile = [&](int j, auto is_open) -> bool {
      constexpr bool kOpen = decltype(is_open)::value;
      if (!wait_hot(p, flag, s_full + (uint32_t)(j % SB) * 8u, (uint32_t)(j / SB) & 1u, PF_ST_TIMEOUT_S, j)) return false;
      tc_fence_after();
      const uint32_t s_addr = lane_addr + kSCol + (uint32_t)(j % SB) * kBN;
      uint32_t r[kBN];                               // this row of S, then of P (bf16 pairs in r[0 .. 32))
      tmem_ld64(s_addr, r);
      if constexpr (SB == 1) {
        // S(j + 1) may follow
        tc_fence_before();
        arrive_if(s_free, lane == 0);
      }
      if constexpr (!kOpen) {
#pragma unroll
        for (int i = 0; i < kBN; ++i) {
          const int tok = j * kBN + i;
          if (!(tok <= lim && tok < p.N)) r[i] = 0xff800000u;          // -inf: exp2 gives 0
        }
      }
      float t4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < kBN; i += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u) t4[u] = max3(t4[u], __uint_as_float(r[i + 2 * u]), __uint_as_float(r[i + 2 * u + 1]));
      }
      const float tmax = max3(fmaxf(t4[0], t4[1]), t4[2], t4[3]) * p.scale_log2;   // positive: see mk_flash_prefill_bf16
      // mx is the exponent reference in use, not the running maximum: it moves only when a maximum has grown
      // by more than 2^8 since it was set, so O is rescaled rarely (and no P exceeds 2^8).
      if (__builtin_expect(__any_sync(0xffffffffu, tmax > mx + 8.f), 0)) {     // also the first visible tile (mx = -inf)
        const bool grown = tmax > mx + 8.f;
        const float alpha = grown ? exp2f(mx - tmax) : 1.f;                    // 0 when mx = -inf
        mx = grown ? tmax : mx;
        sum *= alpha;
        // (With two accumulators S(j) was issued after P V(j - 2), so the parity of that barrier is unambiguous.)
        if (j > 0 && !rescale<D>(p, flag, lane_addr, alpha, pv_done + (uint32_t)((j - 1) % SB) * 8u, (uint32_t)((j - 1) / SB) & 1u, j)) return false;
      }
      const float muse = mx == -INFINITY ? 0.f : mx;
      const uint64_t ref2 = pack2(-muse, -muse);
      // P = exp2(s * scale - reference), two scores per multiply-add, add and conversion
      uint64_t ts[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < kBN; i += 2) {
        const uint64_t x2 = fma2(pack2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), scale2, ref2);
        float e0, e1;
        // masked tiles keep the exp2 unit for every score: exp2(-inf) is exactly 0 there
        if (MK_PF_POLY > 0 && D == 64 && kOpen && (i >> 1) % (MK_PF_POLY > 0 ? MK_PF_POLY : 1) == 0) {   // compile-time pattern
          exp2_poly2(x2, e0, e1);
        } else {
          float x0, x1;
          unpack2(x2, x0, x1);
          e0 = exp2f(x0);
          e1 = exp2f(x1);
        }
        const __nv_bfloat162 pk = __floats2bfloat162_rn(e0, e1);
        // the row sum is taken before the rounding to bf16 (an unbiased 2^-9 relative error per term)
        ts[(i >> 1) & 3] = add2(ts[(i >> 1) & 3], pack2(e0, e1));
        r[i >> 1] = *reinterpret_cast<const uint32_t*>(&pk);
      }
      float t0, t1;
      unpack2(add2(add2(ts[0], ts[1]), add2(ts[2], ts[3])), t0, t1);
      sum += t0 + t1;
      if constexpr (SB == 1) {
        // P(j - 1) has been read
        if (!wait_hot(p, flag, pv_done, (uint32_t)(j - 1) & 1u, PF_ST_TIMEOUT_O, j)) return false;
        tc_fence_after();
      }
      tmem_st32(SB == 1 ? lane_addr + kPCol : s_addr, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      // (a warp may be a tile ahead of the others: S(j + 1) does not wait for all of P(j) with two accumulators, so each has its barrier)
      arrive_if(p_ready + (uint32_t)(j % SB) * 8u, lane == 0);
      return true;
    };
    int j = 0;
#pragma unroll 1
    for (; j < n_plain && ok; ++j) ok = kv_tile(j, std::true_type{});
#pragma unroll 1
    for (; j < nt && ok; ++j) ok = kv_tile(j, std::false_type{});
    // epilogue: O / sum -> bf16
    if (ok && nt > 0) ok = wait_hot(p, flag, pv_done + (uint32_t)((nt - 1) % SB) * 8u, (uint32_t)((nt - 1) / SB) & 1u, PF_ST_TIMEOUT_O, nt);
    tc_fence_after();
    if (ok) {
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
      __nv_bfloat16* dst = p.o + (int64_t)b * p.o_sb + (int64_t)h * p.o_sh + (int64_t)m * p.o_sm;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t o[32];
        if (nt > 0) {
          tmem_ld32(lane_addr + (uint32_t)c, o);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        if (m < p.M) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint32_t w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const __nv_bfloat162 pk = __floats2bfloat162_rn(__uint_as_float(o[i + 2 * u]) * inv,
                                                              __uint_as_float(o[i + 2 * u + 1]) * inv);
              w[u] = *reinterpret_cast<const uint32_t*>(&pk);
            }
            *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      if (p.lse != nullptr && m < p.M)
        p.lse[((int64_t)b * p.H + h) * p.M + m] = sum > 0.f ? (mx + log2f(sum)) * 0.6931471805599453f : -INFINITY;
    }
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  if (warp == kLoadWarp) tmem_dealloc(tmem, F::kCols);
}

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
// The query rows with the heads inside: dims (D, heads, rows, batch), one box = 64 columns x `pack` heads x 128 / pack
// queries, which lands as 128 rows of 128 bytes, the heads of a query one behind the other.
static int encode_query_map(CUtensorMap* out, const void* base, int D, int rows, int heads, int batch, int64_t s_r,
                            int64_t s_h, int64_t s_b, int pack) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(-5, "cuTensorMapEncodeTiled is not available from this driver");
  if (((uint64_t)base & 15) || (s_r * 2) % 16 || (s_h * 2) % 16 || (s_b * 2) % 16 || s_r <= 0 || s_h <= 0 || s_b <= 0)
    return fail(-2, "mk_flash_prefill_bf16: q must be 16-byte aligned with positive row / head / batch strides that are "
                    "multiples of 8 elements");
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)heads, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[3] = {(cuuint64_t)s_h * 2, (cuuint64_t)s_r * 2, (cuuint64_t)s_b * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)pack, (cuuint32_t)(kBM / pack), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(-5, "cuTensorMapEncodeTiled (q) failed with CUresult %d", (int)r);
  return 0;
}

// [batch][head][row][D] with element strides (s_b, s_h, s_r), D contiguous: dims (D, rows, heads, batch),
// one box = 64 columns x `box_rows` rows of one head of one batch entry.
static int encode_rows_map(CUtensorMap* out, const void* base, int D, int rows, int heads, int batch, int64_t s_r,
                           int64_t s_h, int64_t s_b, int box_rows, const char* what) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(-5, "cuTensorMapEncodeTiled is not available from this driver");
  if (((uint64_t)base & 15) || (s_r * 2) % 16 || (s_h * 2) % 16 || (s_b * 2) % 16 || s_r <= 0 || s_h <= 0 || s_b <= 0)
    return fail(-2, "mk_flash_prefill_bf16: %s must be 16-byte aligned with positive row / head / batch strides that are "
                    "multiples of 8 elements", what);
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)rows, (cuuint64_t)heads, (cuuint64_t)batch};
  cuuint64_t strides[3] = {(cuuint64_t)s_r * 2, (cuuint64_t)s_h * 2, (cuuint64_t)s_b * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(-5, "cuTensorMapEncodeTiled (%s) failed with CUresult %d", what, (int)r);
  return 0;
}

// What a launch needs to know of its device, read once per device (the kernels' shared-memory limits are raised
// at the same time).  Entries are written under the lock and never change afterwards.
struct Device {
  int sms = 0, smem_optin = 0, cc = 0;
};
static const void* kernel_of(int D, int T) {
  return reinterpret_cast<const void*>(D == 128 ? &prefill_kernel<128, 1> : (T == 3 ? &prefill_kernel<64, 3> : &prefill_kernel<64, 1>));
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
      if (d.cc == 10)
        for (const void* f : {kernel_of(64, 1), kernel_of(64, 3), kernel_of(128, 1)})
          if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, d.smem_optin) != cudaSuccess) return nullptr;
      facts[dev] = d;
      known[dev].store(true, std::memory_order_release);
    }
  }
  return &facts[dev];
}

}  // namespace mkp

namespace mkp {

// How a call is cut.
struct Plan {
  int pack;         // query heads of a KV head in one tile
  int row_tiles;
  int64_t tiles;    // of all heads and batch entries
  bool three;       // the form with three tiles a CTA
};

static Plan plan(int B, int H, int Hkv, int M, int N, int D, bool causal, int sms) {
  Plan r;
  // the largest power of two that divides the group, as long as the tiles fit the grid
  r.pack = (H / Hkv) & -(H / Hkv);
  while (r.pack > kBM || (r.pack > 1 && (M + kBM / r.pack - 1) / (kBM / r.pack) > 65535)) r.pack >>= 1;
  const int tile_m = kBM / r.pack;
  const int64_t per_row = (int64_t)(H / r.pack) * B;
  r.row_tiles = (M + tile_m - 1) / tile_m;
  r.tiles = per_row * r.row_tiles;
  // Which form.  One KV tile of a CTA takes 0.8 us where two tiles share the SM and 1.05 us where three do.  Where all tiles fit
  // the device at once as threes and two an SM need a second round, that round is the two shortest of a slot's tiles, one behind the other: it
  // must be the longer way by more than the longest tile's loss and what the threes lose by beginning later (us with one / three tiles a CTA,
  // 32 / 8 heads, causal, 1408 x 1408 20.7 / 26.4, 1600 behind 700 tokens 38.1 / 41.2, behind 2496 81.8 / 68.3; no mask, 1300 x 1300
  // 33.8 / 27.4, 1760 x 4096 89.2 / 85.2).  Above, by the KV tiles of the busiest of a few slots when CTAs are dealt out there and
  // back, the longest first (no mask, 1900 x 1900 54.8 / 67.1, 3000 x 3000 117.9 / 100.6; causal, 2048 x 2048 31.9 / 37.1,
  // 2600 x 2600 46.9 / 45.5, 4096 x 4096 102.1 / 92.5): of 63 such sizes the choice was 1.1 % over the better form on average.
  r.three = false;
  const int64_t slots = 2 * (int64_t)sms;
  if (D == 64 && r.tiles > slots) {
    auto kv_tiles = [&](int64_t rank, int group) {   // of the rank-th CTA, the longest first
      const int64_t rows_end = (r.row_tiles - rank / per_row * group) * tile_m;
      return ((causal ? std::min<int64_t>(N, N - M + rows_end) : N) + kBN - 1) / kBN;
    };
    auto busiest = [&](int group, int64_t n_slots) {
      const int64_t n = per_row * ((r.row_tiles + group - 1) / group);
      // Of more than 64 rounds one stands for an odd number around it, so that both forms are looked at over all their CTAs (us with one /
      // three tiles a CTA, no mask, 24 x 4096 x 4096 5670 / 4390; causal, 32 x 4096 x 4096 3950 / 3140, 4000 x 300 x 300 6600 / 6380).
      const int64_t step = ((n + n_slots - 1) / n_slots - 1) / 64 * 2 + 1;
      int64_t most = 0;
      for (int64_t q = 0; q < 5; ++q) {
        const int64_t slot = q * (n_slots - 1) / 4;
        int64_t sum = 0;
        for (int64_t round = step / 2; round * n_slots < n; round += step) {
          const int64_t rank = round * n_slots + (round & 1 ? n_slots - 1 - slot : slot);
          if (rank < n) sum += step * kv_tiles(rank, group);
        }
        most = std::max(most, sum);
      }
      return most;
    };
    if (r.tiles <= 3 * (int64_t)sms) r.three = 5 * (kv_tiles(slots - 1, 1) + kv_tiles(slots, 1)) > 7 * kv_tiles(0, 1);
    else r.three = 5 * busiest(3, sms) < 4 * busiest(1, slots);
  }
  return r;
}

}  // namespace mkp

extern "C" {

const char* mk_flash_prefill_last_error(void) { return mkp::g_err.c_str(); }

int mk_flash_prefill_bf16(const void* q, const void* k, const void* v, void* o, float* lse, int B, int H, int Hkv, int M,
                          int N, int D, const int64_t q_strides[3], const int64_t k_strides[3],
                          const int64_t v_strides[3], const int64_t o_strides[3], float scale, int causal,
                          void* workspace, uint64_t workspace_bytes, int timeout_ms, void* cuda_stream) {
  using namespace mkp;
  if (!q || !k || !v || !o || !workspace || !q_strides || !k_strides || !v_strides || !o_strides)
    return fail(-1, "mk_flash_prefill_bf16: null pointer");
  if (B < 1 || H < 1 || Hkv < 1 || M < 1 || N < 1 || H % Hkv)
    return fail(-2, "mk_flash_prefill_bf16: B, H, Hkv, M, N must be positive and H a multiple of Hkv");
  if (D != 64 && D != 128) return fail(-2, "mk_flash_prefill_bf16: head dim must be 64 or 128, got %d", D);
  if (B > 65535 || (M + 127) / 128 > 65535) return fail(-2, "mk_flash_prefill_bf16: at most 65535 batch entries and 65535 query tiles of 128 rows");
  const float scale_log2 = scale * 1.4426950408889634f;
  if (!std::isfinite(scale_log2)) return fail(-2, "mk_flash_prefill_bf16: the scale must be finite");
  if (causal && M > N) return fail(-2, "mk_flash_prefill_bf16: causal attention needs M <= N (the queries are the last M tokens)");
  if (workspace_bytes < 256 || ((uint64_t)workspace & 255)) return fail(-2, "mk_flash_prefill_bf16: workspace of 256 aligned bytes");
  if (((uint64_t)o & 15) || o_strides[2] % 8 || o_strides[1] % 8 || o_strides[0] % 8)
    return fail(-2, "mk_flash_prefill_bf16: o must be 16-byte aligned with strides that are multiples of 8 elements");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(-1001, "cudaGetDevice failed");
  const Device* d = device_facts(dev);
  if (!d) return fail(-1001, "mk_flash_prefill_bf16: cannot read the attributes of device %d", dev);
  if (d->cc != 10) return fail(-6, "mk_flash_prefill_bf16 needs an sm_100 device (compute capability %d.x found)", d->cc);
  const int smem_optin = d->smem_optin;
  CUtensorMap mq, mkk, mv;
  const Plan pl = plan(B, H, Hkv, M, N, D, causal != 0, d->sms);
  const int pack = pl.pack;
  int rc = encode_query_map(&mq, q, D, M, H, B, q_strides[2], q_strides[1], q_strides[0], pack);
  if (rc) return rc;
  rc = encode_rows_map(&mkk, k, D, N, Hkv, B, k_strides[2], k_strides[1], k_strides[0], kBN, "k");
  if (rc) return rc;
  rc = encode_rows_map(&mv, v, D, N, Hkv, B, v_strides[2], v_strides[1], v_strides[0], kBN, "v");
  if (rc) return rc;
  const int T = pl.three ? 3 : 1;
  const size_t smem = D == 128 ? Form<128, 1>::kSmem : (T == 3 ? Form<64, 3>::kSmem : Form<64, 1>::kSmem);
  if ((int)smem > smem_optin) return fail(-4, "mk_flash_prefill_bf16: %zu bytes of shared memory needed, %d available", smem, smem_optin);
  Params p;
  p.o = reinterpret_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.status = reinterpret_cast<int32_t*>(workspace);
  p.o_sb = o_strides[0], p.o_sh = o_strides[1], p.o_sm = o_strides[2];
  p.B = B, p.H = H, p.Hkv = Hkv, p.M = M, p.N = N;
  p.causal = causal ? 1 : 0;
  p.row_tiles = pl.row_tiles;
  p.pack = pack;
  p.pack_log2 = 0;
  while ((1 << p.pack_log2) < pack) ++p.pack_log2;
  // The row threads take the maximum of the scores before they scale it, and mask with -inf: the factor there is positive.  The sign of the
  // scale goes to the products, and zero becomes the smallest normal number, times which no score differs from another.
  p.scale_log2 = std::max(std::fabs(scale_log2), FLT_MIN);
  p.negate_q = scale < 0.f ? 1u << 13 : 0u;
  p.timeout_ns = (uint64_t)(timeout_ms > 0 ? timeout_ms : 1000) * 1000000ull;
  const dim3 grid(H / pack, B, (pl.row_tiles + T - 1) / T);
  // Where this grid leaves slots empty (two CTAs an SM), the next one is let in late: its CTAs would pile up on the SMs that are
  // free now (us back to back, causal, 32 / 8 heads, early / late: head dim 64 777 x 777, 200 tiles 12.6 / 10.9, 1024 x 1024, 256 tiles 16.7 /
  // 13.6; 128 1024 x 1024 20.4 / 16.7).  Just above one round late is still the better one, at head dim 64 by more than the rule takes (1185 x
  // 1185, 304 tiles 19.1 / 16.8, 1500 x 1500, 376 tiles 22.7 / 20.4; 128 1600 x 1600, 400 tiles 29.3 / 28.0).  From one and a half rounds on
  // early is up to 1.5 % faster (64 2048 x 2048 31.7 / 31.9, 2400 x 2400 41.2 / 41.7; 128 2048 x 2048 41.4 / 41.8, 2190 x 2190 46.9 / 47.6), from
  // three on neither by more than the runs differ (128 3000 x 3000 78.7 / 79.7, 4096 x 4096 137.0 / 137.2, four sequences of 2048 154.5 / 153.1).
  const int64_t sms = d->sms;
  p.next_early = !pl.three && (D == 64 ? pl.tiles >= 2 * sms : pl.tiles > 3 * sms) ? 1 : 0;
  // the kernel may be placed while the one before it in the stream drains (it waits before it touches memory)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((5 * T + 1) * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = reinterpret_cast<cudaStream_t>(cuda_stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* args[4] = {&mq, &mkk, &mv, &p};
  cudaError_t e = cudaLaunchKernelExC(&cfg, kernel_of(D, T), args);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return fail(-(int)e - 1000, "mk_flash_prefill_bf16 launch: %s", cudaGetErrorString(e));
  return 0;
}

int mk_flash_prefill_call(const void* call) {
  if (!call) return mkp::fail(-1, "mk_flash_prefill_call: null pointer");
  mk_flash_prefill_call_t c;
  memcpy(&c, call, sizeof(c));
  auto ptr = [](uint64_t p) { return reinterpret_cast<void*>(p); };
  return mk_flash_prefill_bf16(ptr(c.q), ptr(c.k), ptr(c.v), ptr(c.o), reinterpret_cast<float*>(c.lse), c.B, c.H, c.Hkv, c.M, c.N, c.D,
                               c.q_strides, c.k_strides, c.v_strides, c.o_strides, (float)c.scale, c.causal, ptr(c.workspace),
                               c.workspace_bytes, (int)c.timeout_ms, ptr(c.cuda_stream));
}

int mk_flash_prefill_plan(int B, int H, int Hkv, int M, int N, int D, int causal, int sms, int32_t out[4]) {
  using namespace mkp;
  if (!out || B < 1 || H < 1 || Hkv < 1 || M < 1 || N < 1 || H % Hkv || (D != 64 && D != 128) || (causal && M > N) || sms < 1)
    return fail(-2, "mk_flash_prefill_plan: bad sizes");
  const Plan pl = plan(B, H, Hkv, M, N, D, causal != 0, sms);
  out[0] = pl.three ? 3 : 2, out[1] = pl.pack, out[2] = pl.row_tiles;
  out[3] = (int32_t)std::min<int64_t>(pl.tiles, INT32_MAX);
  return 0;
}

int mk_flash_prefill_status(const void* workspace, int32_t out[4]) {
  if (!workspace || !out) return mkp::fail(-1, "mk_flash_prefill_status: null pointer");
  if (cudaDeviceSynchronize() != cudaSuccess) return mkp::fail(-1001, "mk_flash_prefill_status: device synchronise failed");
  if (cudaMemcpy(out, workspace, 16, cudaMemcpyDeviceToHost) != cudaSuccess)
    return mkp::fail(-1001, "mk_flash_prefill_status: copy failed");
  return 0;
}

}  // extern "C"
