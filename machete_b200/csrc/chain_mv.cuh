// Matvec launches of a program that runs as a chain of kernels (see chain.inc): the ops that one launch holds are
// the same MK_OP_MATVEC records that the persistent kernel runs, with the same sums in the same order, bit for bit.
//
// What a launch is bound by is HBM for a long product and, for the short ones of a decode step, the way from the end
// of the kernel before to the first product and from the last product to the end of this one.  So:
//   * weights do not depend on the kernel before: the ring of pages is filled before the wait for that kernel, as far as the
//     rows' way is not blocked by it (see MvLaunch::ahead);
//   * what a launch needs to know is read before it waits for the kernel before (records are written by copies only, which
//     no launch overtakes); in the parameters they would cost the host 0.6 us a KB of them at every launch;
//   * a page is shared by AS warps.  The persistent kernel's warp rotates its products over independent accumulators
//     (so that no product waits for the one before); here those accumulators are dealt to different warps, which keeps
//     the order of every sum and takes the time of a page by AS;
//   * 9 warps of at most 96 registers and, where that is room enough, at most 113 KB of shared memory: two CTAs share an SM,
//     the second one being the next launch's or another of this one where that has units enough; 17 warps where the rows
//     leave room for one CTA only (see chain_matvec_step).  (8 warps of 128 registers
//     of which the one that handed a page back last requested the next: some 0.8 us a page on the products' path.)
#pragma once
#include "op_matvec.cuh"

namespace mk {

// A kernel's W consumer warps, and one more that loads.
template <int W>
constexpr int kChainThreads = (W + 1) * 32;
constexpr int kEwWarps = 8;                                 // row-wise ops: a unit each
// A kernel's ROWS: one activation row, or up to 8, 16 or 32; its n-tiles of 8 rows.
__host__ __device__ constexpr int chain_nt(int rows) { return rows <= 8 ? 1 : rows / 8; }
constexpr uint32_t kChainBarrier = 1, kChainReady = 2;   // named barriers: the consumers'; all threads', once
constexpr int kChainOps = 8;                          // ops of one launch: Q, K and V of a layer, or the K blocks of a product
constexpr int kChainMaxStages = 12;

enum { kChainEarlyLoads = 1,   // the weights may be read before the kernel before has finished
       kChainLast = 2 };       // the program's last launch: counts it

struct ChainHead {             // what the loader needs to know of an op: it does not wait for the records
  int64_t out_h;                 // output stride of a head
  int32_t mode, hd, d2, tiles;   // row mapping, head dim, its half, K-tiles of a page
  int32_t rows, flags;           // output rows; kEpi...
};
struct MvLaunch {
  ProgramView pv;                  // status block, time limit, cache position, op records (from first_op on)
  const uint8_t* maps;             // the tensor maps of the first op; 512 bytes an op
  ChainHead head[kChainOps];
  int32_t unit_end[kChainOps];     // units of ops 0..i
  int32_t cta_end[kChainOps];      // K blocks: CTAs of blocks 0..i; zero where the ops share the CTAs and what they stage
  int32_t pages[kChainOps], parts[kChainOps];   // pages of a unit, and the partial sums they meet in
  int32_t spread;                               // the partial sums of a unit are dealt to different warps
  int32_t n_ops, flags, res_op, first_op;       // res_op: the op whose residual_out this launch writes, or -1
  int32_t stages, page_bytes, sets_log2;        // ring slots, and sets of slots for partial sums
  int32_t slot_off, act_off, page_off;          // shared memory, bytes
  // n / d as (n * magic) >> 22 for the small numbers here: rows by tokens a sequence, threads by 16-byte chunks of a row
  int32_t s_magic, stage_magic, chunk_magic[kChainOps];   // (stage: pages by ring slots, see ring_lap)
  int32_t ahead;                                          // pages that are requested before the rows are staged
  int32_t norm_off, res_off;                              // the norm's weights' and residual rows' place in the ring behind those pages, or -1
  int32_t pad[8];
};
// What a launch costs the host goes by where its parameters end: 24 or 32 bytes behind a multiple of 64 2.0 us, elsewhere 2.4 (NVIDIA
// driver 580, 488 to 768 bytes, the stream idle; 16 x 1024 -> 1024 through Megakernel.run 5.3 us a pass with 600 bytes, 5.7 with 616).  Hence the pad:
// fields of 16 bits or in one word with the flags, which make it 608, cost the kernels registers (1B shape batch 1 689 to 694 us,
// 8B NVFP4 batch 1 2250 to 2272).
static_assert(sizeof(MvLaunch) % 64 == 24 || sizeof(MvLaunch) % 64 == 32, "a launch with these parameters costs the host 0.4 us more");

// What a CTA works out once, while it waits for the kernel before, so that no division and no chain of loads stands on the
// way from there to the first product, or at its end.
struct ChainRow {
  int64_t out, er, tab;    // where row m of an op's results, of its residual and of its RoPE tables begins (elements)
};
struct ChainIn {
  int64_t x, ri, ro;       // the same for the staged rows: input, residual input, residual output
};
struct ChainUnit {
  int32_t op, rowA0, rowB0, offA, offB, chunk;   // op of the launch, and MvOut
  int32_t flags, valid;                          // kChainEpi...; valid rows of the two halves, nA | nB << 8
};
// What an op's epilogue does, in one word that comes with the unit.
enum { kEpiNormed = 1, kEpiScaled = 2, kEpiPair = 4, kEpiRope = 8, kEpiSiluMul = 16, kEpiRelu = 32, kEpiSilu = 64, kEpiResidual = 128,
       kEpiTop1 = 256, kEpiFp32 = 512, kEpiFp16 = 1024, kEpiKsum = 2048 };
__device__ __forceinline__ int small_div(int n, int magic) { return (int)(((uint32_t)n * (uint32_t)magic) >> 22); }
// How often the ring has gone round before a CTA's page: page / stages.  The product has 64 bits, as a CTA's pages are as many as its
// share of the weights has (in 32 bits it wraps at 1024 pages a slot); exact below 2^30 / kChainMaxStages pages, of which a chain
// has fewer (kChainMaxPages).
__host__ __device__ constexpr uint32_t ring_magic(int stages) { return ((1u << 30) + (uint32_t)stages - 1u) / (uint32_t)stages; }
__host__ __device__ constexpr uint32_t ring_lap(uint32_t page, uint32_t magic) { return (uint32_t)(((uint64_t)page * magic) >> 30); }
constexpr int64_t kChainMaxPages = 1 << 26;      // of a launch
static_assert(kChainMaxPages * kChainMaxStages <= 1 << 30, "ring_lap must be exact");
constexpr int kChainUnits = 32;   // units between the loader's and the last finisher's: at most 12 pages + 4 slot sets
struct ChainTab {
  ChainIn in[32];
  ChainUnit unit[kChainUnits];
  mk_op_t op[1];           // n_ops records, then 32 ChainRow for each
};

__device__ __forceinline__ uint32_t lds64_lo_hi(uint32_t addr, uint32_t& hi) {
  uint32_t lo;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(addr));
  return lo;
}
__device__ __forceinline__ uint4 ldcg128(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }

// Whether a wait has run out in a launch before: nothing runs any more then, as in the persistent kernel.  Every launch looks before it
// waits for the one before, where it costs no time (behind that wait it cost a step 0.3 to 1 %); the launch that stands behind the
// failed one already may have looked too early, and runs.  One thread of a CTA decides.
__device__ __forceinline__ int launch_failed(const ProgramView& pv) { return *reinterpret_cast<const volatile int32_t*>(&pv.state->abort_flag); }

// Row stride of the staged activations and the place of 16-byte chunk `ch` of row m.  Dense weights: as mv_row_stride.
// NVFP4: the eight lanes of a shared-memory phase read two rows at four chunks that lie 128 bytes apart; the chunk
// number's low bits, exclusive-or with which 128 bytes it lies in and with the row, keep the eight on different banks
// (without it every load takes four times as long, which at 8 rows is more than the weights' own time).
template <int WF>
__device__ __forceinline__ uint32_t chain_row_stride(int K) { return (uint32_t)K * 2u + (WF == 2 ? 0u : 16u); }
template <int WF>
__device__ __forceinline__ uint32_t chain_chunk(int m, int ch) {
  return (uint32_t)(WF == 2 ? ch ^ (((ch >> 3) & 3) | ((m & 1) << 2)) : ch) * 16u;
}

// ---- staging -------------------------------------------------------------------------
// The sums of squares are those of mv_stage: its 224 threads take chunks tid, tid + 224, ... of a row, and a warp's sum
// goes to red[row * 7 + warp].  Here (row, one of those seven warps) is a job, and the W warps take jobs in turn, R at
// a time, so that a batch's rows are requested together.
template <int ROWS, int WF, int R, int H, int W>
__device__ __forceinline__ void chain_stage_rms(Ctx& c, const mk_op_t* op, const ChainIn* in, const mk_op_t* res_op) {
  constexpr int T = kConsumerWarps * 32;
  constexpr bool fused = WF == 0;
  const int K = op->i[MK_MV_K], M = ROWS == 1 ? 1 : op->i[MK_MV_M];
  const uint32_t xs = chain_row_stride<WF>(K);
  const int chunks = K >> 3;
  const uint16_t* x = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_X]);
  const uint16_t* ri = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_RES_IN]);
  const uint16_t* nw = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_NORM_W]);
  const bool add = op->i[MK_MV_PRO] == MK_PRO_ADD_RMS && ri != nullptr;
  uint16_t* ro = add && res_op ? reinterpret_cast<uint16_t*>(res_op->p[MK_MV_P_RES_OUT]) : nullptr;
  const int jobs = kConsumerWarps * M;
  const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll 1
  for (int j0 = c.warp; j0 < jobs; j0 += R * W) {
    int row[R], ch0[R];
    ChainIn at[R];
    float sum[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int job = j0 + j * W;
      row[j] = job < jobs ? (ROWS == 1 ? 0 : job / kConsumerWarps) : -1;
      const int m = max(row[j], 0);
      ch0[j] = row[j] < 0 ? chunks : (job - m * kConsumerWarps) * 32 + c.lane;   // (a missing job has no chunks)
      at[j] = in[m];
      sum[j] = 0.f;
    }
#pragma unroll 1
    for (int base = 0; base < chunks; base += H * T) {
      uint4 v[R][H], r[R][H], wv[fused ? R : 1][fused ? H : 1];
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int ch = base + h * T + ch0[j];
          const bool ok = ch < chunks;
          v[j][h] = ok ? ldcg128(x + at[j].x + ch * 8) : z;
          r[j][h] = ok && add ? ldcg128(ri + at[j].ri + ch * 8) : z;
          if (fused) wv[fused ? j : 0][fused ? h : 0] = ok ? *reinterpret_cast<const uint4*>(nw + ch * 8) : z;
          else if (ok) asm volatile("prefetch.global.L1 [%0];" ::"l"(nw + ch * 8));
        }
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int ch = base + h * T + ch0[j];
          if (ch >= chunks) continue;
          uint4 o = v[j][h];
          if (add) {
            o = add8(o, r[j][h], MK_T_BF16);
            if (ro) *reinterpret_cast<uint4*>(ro + at[j].ro + ch * 8) = o;
          }
          float f[8];
          unpack8(o, MK_T_BF16, f);
#pragma unroll
          for (int i = 0; i < 8; ++i) sum[j] += f[i] * f[i];
          if (fused) o = mul8_bf16(o, wv[fused ? j : 0][fused ? h : 0]);
          sts128(c.act_u32 + (uint32_t)row[j] * xs + chain_chunk<WF>(row[j], ch), o);
        }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const float t = warp_sum(sum[j]);
      if (c.lane == 0 && row[j] >= 0) c.ctrl->red[j0 + j * W] = t;   // = row * 7 + the job's warp
    }
  }
  if constexpr (!fused) {
    // second pass over the chunks that this thread wrote: normalise and convert to the products' type
    named_bar_sync(kChainBarrier, W * 32);
    const float eps = op->f[MK_MV_F_EPS];
#pragma unroll 1
    for (int j0 = c.warp; j0 < jobs; j0 += W) {
      const int m = ROWS == 1 ? 0 : j0 / kConsumerWarps;
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < kConsumerWarps; ++w) tot += c.ctrl->red[m * kConsumerWarps + w];
      const float rstd = rsqrtf(tot / (float)K + eps);
      const uint32_t row = c.act_u32 + (uint32_t)m * xs;
#pragma unroll 1
      for (int base = (j0 - m * kConsumerWarps) * 32 + c.lane; base < chunks; base += H * T) {
        uint4 v[H], wq[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const int ch = base + h * T;
          v[h] = ch < chunks ? lds128(row + chain_chunk<WF>(m, ch)) : z;
          wq[h] = ch < chunks ? *reinterpret_cast<const uint4*>(nw + ch * 8) : z;
        }
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const int ch = base + h * T;
          if (ch >= chunks) break;
          float f[8], w[8];
          unpack8(v[h], MK_T_BF16, f);
          unpack8(wq[h], MK_T_BF16, w);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = f[i] * rstd * w[i];
          sts128(row + chain_chunk<WF>(m, ch), pack8(f, MK_T_FP16));
        }
      }
    }
  }
}

// Without a prologue: thread `tid` takes 16-byte chunks tid, tid + (the CTA's consumer threads), ... of all rows laid end to end: (m0, ch0) is its
// first, and each step is (dm, dch) on.
struct ChainWalk {
  int m0, ch0, dm, dch;
};
template <int WF>
__device__ __forceinline__ void chain_stage_plain(Ctx& c, const mk_op_t* op, int M, const ChainIn* in, const ChainWalk& w) {
  const int K = op->i[MK_MV_K];
  const uint32_t xs = chain_row_stride<WF>(K);
  const int chunks = K >> 3;
  const uint16_t* x = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_X]);
  int m = w.m0, ch = w.ch0;
  auto step = [&]() {
    m += w.dm;
    ch += w.dch;
    if (ch >= chunks) {
      ch -= chunks;
      ++m;
    }
  };
#pragma unroll 2
  for (; m < M; step()) cp_async16(c.act_u32 + (uint32_t)m * xs + chain_chunk<WF>(m, ch), x + in[m].x + ch * 8);
  cp_async_wait_all();
  if constexpr (WF == 2) {
    // another type for the products: every thread converts the chunks that it copied, four side by side
    m = w.m0, ch = w.ch0;
#pragma unroll 1
    while (m < M) {
      uint4 v[4];
      uint32_t at[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        at[j] = m < M ? c.act_u32 + (uint32_t)m * xs + chain_chunk<WF>(m, ch) : 0u;
        if (m < M) v[j] = lds128_sync(at[j]);
        step();
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (at[j] == 0u) break;
        float f[8];
        unpack8(v[j], MK_T_BF16, f);
        sts128(at[j], pack8(f, MK_T_FP16));
      }
    }
  }
}

// Whether a kernel's rows come by bulk copies: nine rows and more of dense weights, and NVFP4 rows of sixteen warps.  (us a step, rows
// through registers and by copies: 8B NVFP4 batch 8 3391 / 3206, batch 6 - / 2421; 1B shape batch 16 1136 / 1113, batch 8 787 / 789,
// batch 4 732 / 753, batch 2 694 / 711; one row, and NVFP4 4 x 4096 -> 14336 by eight warps, 13.7 / 14.8, are slower so too.)
__host__ __device__ constexpr bool chain_fetches(int rows, int wf, int warps) { return warps == 16 && (rows == 16 || wf == 2); }
// The rows come by bulk copies, a lane's row each, to where they are staged; residual rows
// and the norm's weights to ring slots that the loader leaves empty until then.  They are there after some 2000 clocks, and
// what is left is arithmetic: every warp's jobs side by side, a norm weight unpacked once for all rows.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// A warp has given up its wait for them, or something has gone wrong elsewhere.  The copies must have landed before the CTA exits, so it
// waits on, with a limit.  Where they do not come the CTA stores nothing of them: its copies of the records lose their residual
// outputs, which a warp reads behind this, and its units get an arrival count that no sum waits for.
static __device__ __noinline__ void rows_late(const MvLaunch* L, Ctrl* ctrl, uint32_t bar) {
  const uint64_t t0 = globaltimer_ns();
  for (;;) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, 0u))) return;
    if (__any_sync(0xffffffffu, globaltimer_ns() - t0 > L->pv.timeout_ns)) break;
  }
  if ((threadIdx.x & 31) == 0) {
    for (int set = 0; set < 4; ++set) atomicOr(&ctrl->mv_arrive[set], 0x80000000u);
    mk_op_t* ops = reinterpret_cast<ChainTab*>(reinterpret_cast<uint8_t*>(ctrl) + kCtrlStructBytes)->op;
    for (int i = 0; i < L->n_ops; ++i) *reinterpret_cast<volatile uint64_t*>(&ops[i].p[MK_MV_P_RES_OUT]) = 0;
  }
  __syncwarp();
}
template <int WF>
__device__ __forceinline__ void chain_fetch_rows(Ctx& c, const MvLaunch& L, const mk_op_t* op, int M, const ChainIn* in) {
  const int K = op->i[MK_MV_K];
  const uint32_t bytes = (uint32_t)K * 2u, bar = smem_u32(&c.ctrl->rows_in);
  const uint16_t* x = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_X]);
  const uint16_t* ri = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_RES_IN]);
  const bool norm = op->i[MK_MV_PRO] != MK_PRO_NONE && L.norm_off >= 0;
  const bool add = op->i[MK_MV_PRO] == MK_PRO_ADD_RMS && ri != nullptr && L.res_off >= 0;
  if (c.warp == 0) {
    if (c.lane == 0) {
      mbar_arrive_expect_tx(bar, ((uint32_t)M * (add ? 2u : 1u) + (norm ? 1u : 0u)) * bytes);
      if (norm) bulk_load(c.pages_u32 + (uint32_t)L.norm_off, reinterpret_cast<const void*>(op->p[MK_MV_P_NORM_W]), bytes, bar);
    }
    __syncwarp();
    if (c.lane < M) {
      bulk_load(c.act_u32 + (uint32_t)c.lane * chain_row_stride<WF>(K), x + in[c.lane].x, bytes, bar);
      if (add) bulk_load(c.pages_u32 + (uint32_t)L.res_off + (uint32_t)c.lane * bytes, ri + in[c.lane].ri, bytes, bar);
    }
    __syncwarp();
  }
  uint64_t t0 = 0;
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (__builtin_expect(__all_sync(0xffffffffu, mbar_try_wait(bar, 0u)), 1)) return;
    if (give_up_check(c, t0, MK_ST_TIMEOUT_PAGE_FULL, -1, 0)) {
      rows_late(&L, c.ctrl, bar);
      c.dead = true;
      return;
    }
  }
}

// chain_stage_rms for rows that lie in shared memory, with the same jobs and sums.  Rows are changed where they lie: a warp reads
// 32 chunks and writes them back, NVFP4 rows to other places among the same eight (see chain_chunk).
template <int WF, int R, int W>
__device__ __forceinline__ void chain_norm_rows(Ctx& c, const MvLaunch& L, const mk_op_t* op, const ChainIn* in, const mk_op_t* res_op) {
  constexpr int T = kConsumerWarps * 32;
  const int K = op->i[MK_MV_K], M = op->i[MK_MV_M];
  const uint32_t xs = chain_row_stride<WF>(K);
  const int chunks = K >> 3;
  const uint16_t* ri = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_RES_IN]);
  const uint16_t* nw = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_NORM_W]);
  const bool add = op->i[MK_MV_PRO] == MK_PRO_ADD_RMS && ri != nullptr;
  uint16_t* ro = add && res_op ? reinterpret_cast<uint16_t*>(res_op->p[MK_MV_P_RES_OUT]) : nullptr;
  const uint4 z = make_uint4(0, 0, 0, 0);
  auto norm_w = [&](int ch) { return L.norm_off >= 0 ? lds128(c.pages_u32 + (uint32_t)L.norm_off + (uint32_t)ch * 16u) : *reinterpret_cast<const uint4*>(nw + ch * 8); };
  const int jobs = kConsumerWarps * M;
#pragma unroll 1
  for (int j0 = c.warp; j0 < jobs; j0 += R * W) {
    int row[R], part[R];
    float sum[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int job = j0 + j * W;
      row[j] = job / kConsumerWarps;
      part[j] = job < jobs ? (job - row[j] * kConsumerWarps) * 32 : chunks;   // (a missing job has no chunks)
      sum[j] = 0.f;
    }
#pragma unroll 1
    for (int base = 0; base < chunks; base += T) {
      bool any = false;
#pragma unroll
      for (int j = 0; j < R; ++j) any |= base + part[j] < chunks;
      if (!any) break;
      uint4 v[R], r[R], wv[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int ch = base + part[j] + c.lane;
        const bool ok = ch < chunks;
        v[j] = ok ? lds128(c.act_u32 + (uint32_t)row[j] * xs + (uint32_t)ch * 16u) : z;
        r[j] = wv[j] = z;
        if (ok && add) r[j] = L.res_off >= 0 ? lds128(c.pages_u32 + (uint32_t)L.res_off + (uint32_t)(row[j] * chunks + ch) * 16u) : ldcg128(ri + in[row[j]].ri + ch * 8);
        if (WF == 0 && ok) wv[j] = norm_w(ch);
      }
      if (WF == 2) __syncwarp();
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int ch = base + part[j] + c.lane;
        if (ch >= chunks) continue;
        uint4 o = v[j];
        if (add) {
          o = add8(o, r[j], MK_T_BF16);
          if (ro) *reinterpret_cast<uint4*>(ro + in[row[j]].ro + ch * 8) = o;
        }
        float f[8];
        unpack8(o, MK_T_BF16, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) sum[j] += f[i] * f[i];
        if (WF == 0) o = mul8_bf16(o, wv[j]);
        sts128(c.act_u32 + (uint32_t)row[j] * xs + chain_chunk<WF>(row[j], ch), o);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < R; ++j) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (c.lane == 0 && j0 + j * W < jobs) c.ctrl->red[j0 + j * W] = sum[j];   // = row * 7 + the job's warp
  }
  if constexpr (WF == 2) {
    // second pass: normalise and convert to the products' type, a thread the same chunk of every row
    named_bar_sync(kChainBarrier, W * 32);
    float rstd = 0.f;                      // of row `lane`
    if (c.lane < M) {
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < kConsumerWarps; ++w) tot += c.ctrl->red[c.lane * kConsumerWarps + w];
      rstd = rsqrtf(tot / (float)K + op->f[MK_MV_F_EPS]);
    }
#pragma unroll 1
    for (int ch0 = c.warp * 32; ch0 < chunks; ch0 += W * 32) {
      const int ch = ch0 + c.lane;
      const bool ok = ch < chunks;
      float w[8];
      unpack8(ok ? norm_w(ch) : z, MK_T_BF16, w);
#pragma unroll 4
      for (int m = 0; m < M; ++m) {
        const float rs = __shfl_sync(0xffffffffu, rstd, m);
        const uint32_t at = c.act_u32 + (uint32_t)m * xs + chain_chunk<WF>(m, ok ? ch : 0);
        float f[8];
        unpack8(ok ? lds128(at) : z, MK_T_BF16, f);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = f[i] * rs * w[i];
        if (ok) sts128(at, pack8(f, MK_T_FP16));
      }
    }
  }
}

// Fetched rows without a prologue are staged as they come, but for NVFP4 weights, whose products take f16: a thread's chunks as in
// chain_stage_plain, four a turn.  (Eight chunks that change places are one warp's, in one turn: all are read before one is written.)
template <int W>
__device__ __forceinline__ void chain_to_f16(Ctx& c, const mk_op_t* op, int M, const ChainWalk& w) {
  const int K = op->i[MK_MV_K];
  const uint32_t xs = chain_row_stride<2>(K);
  const int chunks = K >> 3;
  int m = w.m0, ch = w.ch0;
#pragma unroll 1
  for (int done = 0; done < M * chunks; done += 4 * W * 32) {
    uint4 v[4];
    uint32_t at[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      at[j] = 0u;
      if (m < M) {
        v[j] = lds128(c.act_u32 + (uint32_t)m * xs + (uint32_t)ch * 16u);
        at[j] = c.act_u32 + (uint32_t)m * xs + chain_chunk<2>(m, ch);
      }
      m += w.dm;
      ch += w.dch;
      if (ch >= chunks) {
        ch -= chunks;
        ++m;
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (at[j] == 0u) break;
      float f[8];
      unpack8(v[j], MK_T_BF16, f);
      sts128(at[j], pack8(f, MK_T_FP16));
    }
  }
}

// ---- products ------------------------------------------------------------------------
// The accumulators of mv_unit (NA of them per n-tile: 4, 2 or 1 for 1, 2 or 4 n-tiles) and which of them warp h of AS
// takes.  UN x JN are the tiles of a pair and the chunks of a tile (dense), QN the words of a chunk (NVFP4), NN the n-tiles.
template <int NT, int AS>
struct ChainCut {
  static constexpr int NA = NT == 1 ? 4 : (NT == 2 ? 2 : 1);
  static constexpr int AH = NA < AS ? NA : AS;         // warps that the accumulators are dealt to
  static constexpr int AN = NA / AH;                   // accumulators of a warp
  static constexpr int NN = NT / (AS / AH);            // n-tiles of a warp
  static constexpr int UN = NT == 1 ? 2 / (AH >= 2 ? 2 : 1) : 2;
  static constexpr int JN = NT == 1 ? (AH == 4 ? 1 : 2) : (NT == 2 && AH == 2 ? 1 : 2);
  static constexpr int QN = 4 / AH;
};

// acc[a][n]: accumulator a of this warp's n-tile n.  `h` = which of the AS warps.
template <int NT, int WF, int AS>
__device__ __forceinline__ void chain_page_dense(float (&acc)[ChainCut<NT, AS>::AN][ChainCut<NT, AS>::NN][4], uint32_t page,
                                                 uint32_t half, int tiles, const uint32_t (&xrow)[ChainCut<NT, AS>::NN],
                                                 uint32_t k0, int h, int lane) {
  using Cut = ChainCut<NT, AS>;
  constexpr int UN = Cut::UN, JN = Cut::JN, NN = Cut::NN;
  const int g = lane >> 2, t = lane & 3, a = h & (Cut::AH - 1);
  const int u0 = NT == 1 && Cut::AH >= 2 ? (Cut::AH == 4 ? a >> 1 : a) : 0;
  const int j0 = JN == 1 ? a & 1 : 0;
  struct Frag {
    uint4 wa[UN][JN], wb[UN][JN], x[NN][UN][JN];
  };
  // running addresses of the pair's first tile (of this warp)
  uint32_t pw[JN], px[NN];
#pragma unroll
  for (int j = 0; j < JN; ++j) pw[j] = page + (uint32_t)u0 * 1024u + (uint32_t)g * 128u + (uint32_t)(((2 * t + j0 + j) ^ g) << 4);
#pragma unroll
  for (int n = 0; n < NN; ++n) px[n] = xrow[n] + k0 * 2u + (uint32_t)u0 * 128u + (uint32_t)(2 * t + j0) * 16u;
  auto load = [&](Frag& f, uint32_t at, int un) {   // the pair `at` pairs behind the running addresses, its first `un` tiles
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      if (u < un) {
#pragma unroll
        for (int j = 0; j < JN; ++j) {
          f.wa[u][j] = lds128(pw[j] + at * 2048u + (uint32_t)u * 1024u);
          f.wb[u][j] = lds128(pw[j] + half + at * 2048u + (uint32_t)u * 1024u);
#pragma unroll
          for (int n = 0; n < NN; ++n) f.x[n][u][j] = lds128(px[n] + at * 256u + (uint32_t)u * 128u + (uint32_t)j * 16u);
        }
      }
    }
  };
  auto products = [&](const Frag& f, int un) {
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        if (u < un) {
#pragma unroll
          for (int j = 0; j < JN; ++j)
#pragma unroll
            for (int n = 0; n < NN; ++n) {
              // accumulator (u * 2 + j) % NA, counted from this warp's first
              float(&d)[4] = acc[Cut::AN == 1 ? 0 : j][n];
              const uint32_t a0 = hf ? f.wa[u][j].z : f.wa[u][j].x, a1 = hf ? f.wb[u][j].z : f.wb[u][j].x;
              const uint32_t a2 = hf ? f.wa[u][j].w : f.wa[u][j].y, a3 = hf ? f.wb[u][j].w : f.wb[u][j].y;
              const uint32_t b0 = hf ? f.x[n][u][j].z : f.x[n][u][j].x, b1 = hf ? f.x[n][u][j].w : f.x[n][u][j].y;
              if constexpr (WF == 0)
                mma_bf16(d, a0, a1, a2, a3, b0, b1);
              else
                mma_f16(d, a0, a1, a2, a3, b0, b1);
            }
        }
      }
  };
  auto advance = [&](uint32_t by) {
#pragma unroll
    for (int j = 0; j < JN; ++j) pw[j] += by * 2048u;
#pragma unroll
    for (int n = 0; n < NN; ++n) px[n] += by * 256u;
  };
  // a warp of one tile a pair has (tiles - u0) / 2 of them, rounded up; one of both may end with a pair of one tile
  const int pairs = UN == 1 ? (tiles - u0 + 1) >> 1 : tiles >> 1;
  if constexpr (NT > 1 && NN * UN * JN >= 4) {   // (two sets of fragments would not fit the registers)
    Frag f;
#pragma unroll 1
    for (int i = 0; i < pairs; ++i) {
      load(f, 0, UN);
      products(f, UN);
      advance(1);
    }
  } else if (pairs > 0) {
    Frag f0, f1;
    load(f0, 0, UN);
#pragma unroll 1
    for (int i = 0;;) {
      if (i + 1 < pairs) load(f1, 1, UN);
      products(f0, UN);
      advance(2);
      if (++i >= pairs) break;
      if (i + 1 < pairs) load(f0, 0, UN);
      products(f1, UN);
      if (++i >= pairs) break;
    }
    if (UN == 2 && (pairs & 1)) advance(-1u);
  }
  if (UN == 2 && (tiles & 1)) {
    Frag f;
    load(f, 0, 1);
    products(f, 1);
  }
}

__device__ __forceinline__ uint32_t e4m3x2(uint32_t v) {   // the two e4m3 values of the low half, as f16
  uint32_t d;
  asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; cvt.rn.f16x2.e4m3x2 %0, lo; }" : "=r"(d) : "r"(v));
  return d;
}

template <int NT, int AS>
__device__ __forceinline__ void chain_page_fp4(float (&acc)[ChainCut<NT, AS>::AN][ChainCut<NT, AS>::NN][4], uint32_t page,
                                               uint32_t half, int tiles, const uint32_t (&xrow)[ChainCut<NT, AS>::NN],
                                               uint32_t k0, int h, int lane, bool f16s) {
  using Cut = ChainCut<NT, AS>;
  constexpr int QN = Cut::QN, NN = Cut::NN;
  constexpr bool kPair = QN == 2 && NT == 1;   // this warp's two words lie side by side, under one scale
  const int g = lane >> 2, t = lane & 3, a = h & (Cut::AH - 1);
  // word q of a chunk goes to accumulator q % NA: this warp's words
  auto word = [&](int i) { return QN == 4 ? i : (NT == 1 ? a * QN + i : a + 2 * i); };
  // running addresses; what one step adds to another is the same for all of them, so that it can stand in the instruction
  const uint32_t sa = page + 2u * half + (uint32_t)g * 128u + (uint32_t)t * 4u;
  uint32_t pw[2], px[NN][2][QN];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    pw[j] = tile_chunk(page, g, 2 * t + j) + (QN == 4 ? 0u : (uint32_t)word(0) * 4u);
#pragma unroll
    for (int n = 0; n < NN; ++n)
#pragma unroll
      for (int i = 0; i < QN; ++i)
        px[n][j][i] = xrow[n] + k0 * 2u + (uint32_t)t * 128u +
                      ((uint32_t)((j << 2) | word(i)) ^ (uint32_t)(t | ((g & 1) << 2))) * 16u;
  }
  // e4m3 scales: which bytes of (j 0, j 1) x (values 0-15, 16-31) a warp of one word or pair takes
  const int s_of = NT == 1 && QN < 4 ? (QN == 2 ? a : a >> 1) : 0;
  const uint32_t pick = s_of ? 0x31u : 0x20u;
  struct Frag {
    uint32_t lo[2][QN], hi[2][QN], slo, shi;
    uint4 x[NN][2][QN];
  };
  auto load = [&](Frag& f, int kt, uint32_t at) {   // tile kt, `at` tiles behind the running addresses
    const uint32_t srow = sa + (uint32_t)((kt ^ g) << 4);
    f.slo = lds32(srow);
    f.shi = lds32(srow + 1024u);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t ta = pw[j] + at * 1024u, tb = ta + half;
      if constexpr (QN == 4) {
        const uint4 p = lds128(ta), q = lds128(tb);
        f.lo[j][0] = p.x, f.lo[j][1] = p.y, f.lo[j][2] = p.z, f.lo[j][3] = p.w;
        f.hi[j][0] = q.x, f.hi[j][1] = q.y, f.hi[j][2] = q.z, f.hi[j][3] = q.w;
      } else if constexpr (kPair) {
        f.lo[j][0] = lds64_lo_hi(ta, f.lo[j][1]);
        f.hi[j][0] = lds64_lo_hi(tb, f.hi[j][1]);
      } else {
#pragma unroll
        for (int i = 0; i < QN; ++i) {
          f.lo[j][i] = lds32(ta + (uint32_t)i * 8u);
          f.hi[j][i] = lds32(tb + (uint32_t)i * 8u);
        }
      }
#pragma unroll
      for (int i = 0; i < QN; ++i)
#pragma unroll
        for (int n = 0; n < NN; ++n) f.x[n][j][i] = lds128(px[n][j][i] + at * 512u);
    }
  };
  auto both = [](uint32_t v, int hi) { return __byte_perm(v, v, hi ? 0x3232 : 0x1010); };
  auto products = [&](const Frag& f) {
    // f16x2 broadcast scales of chunk j, values [0, 16) and [16, 32)
    uint32_t sl[2][2], sh[2][2];
    if (f16s) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        sl[j][0] = sl[j][1] = both(f.slo, j);
        sh[j][0] = sh[j][1] = both(f.shi, j);
      }
    } else if constexpr (NT == 1 && QN < 4) {
      const uint32_t l = e4m3x2(__byte_perm(f.slo, 0u, pick)), hh = e4m3x2(__byte_perm(f.shi, 0u, pick));
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        sl[j][0] = sl[j][1] = both(l, j);
        sh[j][0] = sh[j][1] = both(hh, j);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t l = e4m3x2(f.slo >> (16 * j)), hh = e4m3x2(f.shi >> (16 * j));
        sl[j][0] = both(l, 0), sl[j][1] = both(l, 1);
        sh[j][0] = both(hh, 0), sh[j][1] = both(hh, 1);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int i = 0; i < QN; ++i) {
        // a word's scale is that of half word / 2 of the chunk
        const int sc = QN == 4 ? i >> 1 : (NT == 1 ? 0 : i);
        uint32_t al[4], ah[4];
        e2m1x8_scaled(f.lo[j][i], sl[j][sc], al);
        e2m1x8_scaled(f.hi[j][i], sh[j][sc], ah);
        constexpr int AN = Cut::AN;
        const int ai = NT == 1 ? i % AN : (QN == 4 ? i % AN : 0);
#pragma unroll
        for (int n = 0; n < NN; ++n) {
          const uint4& xb = f.x[n][j][i];
          mma_f16(acc[ai][n], al[0], ah[0], al[1], ah[1], xb.x, xb.y);
          mma_f16(acc[ai][n], al[2], ah[2], al[3], ah[3], xb.z, xb.w);
        }
      }
    }
  };
  auto advance = [&](uint32_t by) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      pw[j] += by * 1024u;
#pragma unroll
      for (int n = 0; n < NN; ++n)
#pragma unroll
        for (int i = 0; i < QN; ++i) px[n][j][i] += by * 512u;
    }
  };
  if constexpr (NT > 1 && NN * QN >= 4) {   // (two sets of fragments would not fit the registers)
    Frag f;
#pragma unroll 1
    for (int kt = 0; kt < tiles; ++kt) {
      load(f, kt, 0);
      products(f);
      advance(1);
    }
    return;
  }
  Frag f0, f1;
  load(f0, 0, 0);
#pragma unroll 1
  for (int kt = 0;;) {
    if (kt + 1 < tiles) load(f1, kt + 1, 1);
    products(f0);
    if (++kt >= tiles) break;
    advance(2);
    if (kt + 1 < tiles) load(f0, kt + 1, 0);
    products(f1);
    if (++kt >= tiles) break;
  }
}

// First weight rows of a unit's two halves, and where its results go (see fill_instr_fast_path).  `unit` is the launch's,
// or, for K blocks, the op's own.
__device__ __forceinline__ ChainUnit chain_unit(const MvLaunch& L, int op0, int unit) {
  ChainUnit r;
  r.op = op0;
  if (L.cta_end[0] == 0) {
    while (unit >= L.unit_end[r.op]) ++r.op;
    if (r.op) unit -= L.unit_end[r.op - 1];
  }
  const ChainHead& op = L.head[r.op];
  r.chunk = 0;
  if (op.mode == MK_MV_PLAIN) {
    r.rowA0 = unit * 16;
    r.rowB0 = unit * 16 + 8;
  } else if (op.mode == MK_MV_PAIR) {
    r.rowA0 = r.rowB0 = unit * 8;
  } else {
    const int upb = op.d2 / 8, hh = unit / upb;
    r.chunk = unit - hh * upb;
    r.rowA0 = hh * op.hd + r.chunk * 8;
    r.rowB0 = r.rowA0 + op.d2;
  }
  r.offA = r.rowA0;
  r.offB = r.rowB0;
  if (r.rowB0 >= op.hd) {
    const int qa = r.rowA0 / op.hd, qb = r.rowB0 / op.hd;
    r.offA = (int)((int64_t)qa * op.out_h + (r.rowA0 - qa * op.hd));
    r.offB = (int)((int64_t)qb * op.out_h + (r.rowB0 - qb * op.hd));
  }
  r.flags = op.flags;
  const int na = op.mode == MK_MV_ROPE ? 8 : clamp8(op.rows - r.rowA0), nb = op.mode == MK_MV_ROPE ? 8 : clamp8(op.rows - r.rowB0);
  r.valid = na | nb << 8;
  return r;
}

// Row m = token t of sequence b; `pos` is the sequence's device-resident position.
__device__ __forceinline__ ChainRow chain_row(const mk_op_t* op, int b, int t, int pos) {
  const int dyn = op->i[MK_MV_DYNPOS];
  ChainRow r;
  r.out = b * op->s[MK_MV_S_O_B] + (int64_t)(t + op->i[MK_MV_POS] + ((dyn & MK_MV_DYN_OUT) ? pos : 0)) * op->s[MK_MV_S_O_S];
  r.er = b * op->s[MK_MV_S_ER_B] + t * op->s[MK_MV_S_ER_S];
  r.tab = (int64_t)(t + ((dyn & MK_MV_DYN_TABLES) ? pos : 0)) * op->s[MK_MV_S_COS];
  return r;
}

// mv_epilogue for results that are stored.  What an op asks for is asked once, around loops over the rows that are unrolled
// and hold no branch: one warp runs this for a unit, and for a launch of a unit or two a CTA it is the launch's end.
template <int ROWS, int WF>
__device__ __forceinline__ void chain_epilogue(Ctx& c, const mk_op_t* op, const ChainRow* rows, const ChainUnit& r,
                                               const float (&sum)[chain_nt(ROWS)][4]) {
  constexpr int Q = ROWS == 1 ? 1 : 2 * chain_nt(ROWS);   // rows of a lane
  const int g = c.lane >> 2, t = c.lane & 3;
  const int M = ROWS == 1 ? 1 : op->i[MK_MV_M];
  const int fl = r.flags;
  constexpr bool bf = WF != 1;   // the activations' type
  const bool va = g < (r.valid & 255), vb = g < (r.valid >> 8) && !(fl & kEpiSiluMul);
  auto row_of = [&](int q) { return (q >> 1) * 8 + 2 * t + (q & 1); };
  auto value = [&](uint32_t v) { return bf ? bf16lo(v) : f16lo(v); };
  float a[Q], b[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) a[q] = sum[q >> 1][q & 1], b[q] = sum[q >> 1][2 + (q & 1)];
  if (WF == 0 && (fl & kEpiNormed)) {
    // the rows' RMSNorm scales, from the sums of squares that the staging left
    const float k = (float)op->i[MK_MV_K], eps = op->f[MK_MV_F_EPS];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float* rs = c.ctrl->red + row_of(q) * kConsumerWarps;
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < kConsumerWarps; ++w) tot += rs[w];
      const float scale = rsqrtf(tot / k + eps);
      a[q] *= scale;
      b[q] *= scale;
    }
  }
  if (WF == 2 && (fl & kEpiScaled)) {
    const float gs = op->f[MK_MV_F_GSCALE], gsb = fl & kEpiPair ? op->f[MK_MV_F_GSCALE1] : gs;
#pragma unroll
    for (int q = 0; q < Q; ++q) a[q] *= gs, b[q] *= gsb;
  }
  if (fl & kEpiRope) {
    const uint16_t* cs = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_COS]) + r.chunk * 8 + g;
    const uint16_t* sn = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_SIN]) + r.chunk * 8 + g;
    uint16_t cq[Q], sq[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const bool ok = row_of(q) < M;
      const int64_t off = ok ? rows[row_of(q)].tab : 0;
      cq[q] = ok ? cs[off] : (uint16_t)0;
      sq[q] = ok ? sn[off] : (uint16_t)0;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float cv = value(cq[q]), sv = value(sq[q]);
      const float a2 = a[q] * cv - b[q] * sv, b2 = b[q] * cv + a[q] * sv;
      a[q] = a2;
      b[q] = b2;
    }
  } else if (fl & kEpiSiluMul) {
#pragma unroll
    for (int q = 0; q < Q; ++q) a[q] = silu_f(a[q]) * b[q];
  } else if (fl & kEpiRelu) {
#pragma unroll
    for (int q = 0; q < Q; ++q) a[q] = fmaxf(a[q], 0.f), b[q] = fmaxf(b[q], 0.f);
  } else if (fl & kEpiSilu) {
#pragma unroll
    for (int q = 0; q < Q; ++q) a[q] = silu_f(a[q]), b[q] = silu_f(b[q]);
  }
  if (fl & kEpiResidual) {
    const uint16_t* er = reinterpret_cast<const uint16_t*>(op->p[MK_MV_P_EPI_RES]) + g;
    uint16_t ra[Q], rb[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const bool ok = row_of(q) < M;
      const int64_t off = ok ? rows[row_of(q)].er : 0;
      ra[q] = ok && va ? er[off + r.rowA0] : (uint16_t)0;
      rb[q] = ok && vb ? er[off + r.rowB0] : (uint16_t)0;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) a[q] += value(ra[q]), b[q] += value(rb[q]);
  }
  if (fl & kEpiTop1) {
    const int idx0 = op->i[MK_MV_IDX0];
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(op->p[MK_MV_P_OUT]);
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      float qa = 0.f, qb = 0.f;
#pragma unroll
      for (int i = 0; i < Q; ++i)
        if (i == q) qa = a[i], qb = b[i];
      unsigned long long key = 0ull;
      if (va) key = top1_key(qa, idx0 + r.rowA0 + g);
      if (vb) key = max(key, top1_key(qb, idx0 + r.rowB0 + g));
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
      if (g == 0 && row_of(q) < M) atomicMax(keys + row_of(q), key);
    }
    return;
  }
  char* out = reinterpret_cast<char*>(op->p[MK_MV_P_OUT]);
  if (fl & kEpiFp32) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (row_of(q) >= M) continue;
      float* o = reinterpret_cast<float*>(out) + rows[row_of(q)].out + g;
      if (va) o[r.offA] = a[q];
      if (vb) o[r.offB] = b[q];
    }
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const bool ok = row_of(q) < M;
      uint16_t* o = reinterpret_cast<uint16_t*>(out) + (ok ? rows[row_of(q)].out : 0) + g;
      const uint32_t v = fl & kEpiFp16 ? pack_f16(a[q], b[q]) : pack_bf16(a[q], b[q]);
      if (ok && va) o[r.offA] = (uint16_t)v;
      if (ok && vb) o[r.offB] = (uint16_t)(v >> 16);
    }
  }
}

// All partial sums of a unit are in: add them in the order of mv_unit (a participant's accumulators, then the participants),
// free the slot set and store.
template <int ROWS, int WF, int NA, bool KS>
__device__ __forceinline__ void chain_finish(Ctx& c, const mk_op_t* ops, const ChainRow* rows, const ChainUnit cu, int unit,
                                             const float4* mine, int parts, uint32_t set, uint32_t gen) {
  constexpr int NT = chain_nt(ROWS);
  const mk_op_t* op = ops + cu.op;
  float sum[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) sum[n][0] = sum[n][1] = sum[n][2] = sum[n][3] = 0.f;
#pragma unroll 1
  for (int j = 0; j < parts; ++j) {
    float4 v[NA][NT];
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int n = 0; n < NT; ++n) v[a][n] = mine[((j * NA + a) * NT + n) * 32];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float4 s = v[0][n];
#pragma unroll
      for (int a = 1; a < NA; ++a) s.x += v[a][n].x, s.y += v[a][n].y, s.z += v[a][n].z, s.w += v[a][n].w;
      sum[n][0] += s.x, sum[n][1] += s.y, sum[n][2] += s.z, sum[n][3] += s.w;
    }
  }
  __syncwarp();
  if (c.lane == 0) {
    c.ctrl->mv_arrive[set] = 0;
    __threadfence_block();
    *reinterpret_cast<volatile uint32_t*>(&c.ctrl->mv_done[set]) = gen + 1u;
  }
  if constexpr (KS) {
    if ((cu.flags & kEpiKsum) && !mv_kblock_sum<NT, WF == 1 ? -1 : WF>(c, op, unit, sum)) return;
  }
  chain_epilogue<ROWS, WF>(c, op, rows + cu.op * 32, cu, sum);
}

// Waits until the ring's slot holds its k-th page: when all `handed_back` shares of the earlier ones are in, and only then,
// the barrier's parity says which page is there.  One vote for both, and one straight way through where the page is there.
__device__ __forceinline__ bool chain_page_there(Ctx& c, uint32_t slot, uint32_t k, uint32_t handed_back) {
  const uint32_t released = *reinterpret_cast<volatile uint32_t*>(&c.ctrl->released[slot]);   // (looked at before the barrier)
  const bool there = mbar_try_wait(full_bar(c, slot), k & 1u);
  return __all_sync(0xffffffffu, there & (released >= handed_back));
}
__device__ __forceinline__ bool chain_acquire(Ctx& c, uint32_t slot, uint32_t k, uint32_t handed_back) {
  uint64_t t0 = 0;
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (__builtin_expect(chain_page_there(c, slot, k, handed_back), 1)) return true;
    if (give_up_check(c, t0, MK_ST_TIMEOUT_PAGE_FULL, (int)slot, (int)k)) {
      c.dead = true;
      return false;
    }
  }
}

template <int ROWS, int WF, int AS, bool KS, int W>
__global__ void __launch_bounds__(kChainThreads<W>, ROWS <= 8 && W == 8 ? 2 : 1)
    mv_chain_kernel(const __grid_constant__ MvLaunch L) {
  constexpr int NT = chain_nt(ROWS);
  using Cut = ChainCut<NT, AS>;
  extern __shared__ __align__(1024) uint8_t smem[];
  ChainTab& tab = *reinterpret_cast<ChainTab*>(smem + kCtrlStructBytes);
  mk_op_t* ops = tab.op;
  ChainRow* rows = reinterpret_cast<ChainRow*>(ops + L.n_ops);   // 32 an op
  Ctx c;
  c.pv = &L.pv;
  c.ctrl = reinterpret_cast<Ctrl*>(smem);
  c.act_u32 = smem_u32(smem + L.act_off);
  c.pages_u32 = smem_u32(smem + L.page_off);
  c.warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  c.lane = threadIdx.x & 31;
  c.instr_idx = L.first_op;
  c.dead = false;
  c.trace_base = nullptr;
  c.trace_n = c.trace_cap = 0;
  if (!plan_in_force(L.pv)) {
    prior_work_done();
    return;
  }
  const uint32_t page_bytes = (uint32_t)L.page_bytes;

  // this CTA's units: every `count`-th of `total` from `local` on, of ops [op0, ...)
  int op0 = 0, local = (int)blockIdx.x, count = (int)gridDim.x, total = L.unit_end[L.n_ops - 1];
  if (L.cta_end[0] > 0) {
    while (local >= L.cta_end[op0]) ++op0;
    const int c0 = op0 ? L.cta_end[op0 - 1] : 0;
    count = L.cta_end[op0] - c0;
    local -= c0;
    total = L.unit_end[op0] - (op0 ? L.unit_end[op0 - 1] : 0);
  }
  const int units = local < total ? (total - local + count - 1) / count : 0;
  const int P = L.pages[op0], parts = L.parts[op0];
  // shares of a unit that its sum waits for, and pages that are the last of a partial sum
  const int arrivals = L.spread ? parts * AS : AS, last_pages = L.spread ? parts : 1;

  const bool early = (L.flags & kChainEarlyLoads) != 0;
  if (c.warp == W) {
    // ---- loader
    if (c.lane < L.stages) {
      mbar_init(smem_u32(&c.ctrl->full[c.lane]), 32);
      mbar_init(smem_u32(&c.ctrl->empty[c.lane]), AS);
      c.ctrl->released[c.lane] = 0;
    }
    if (c.lane == 0) {
      mbar_init(smem_u32(&c.ctrl->staged), 1);
      mbar_init(smem_u32(&c.ctrl->rows_in), 1);
    }
    if (c.lane < 4) c.ctrl->mv_arrive[c.lane] = c.ctrl->mv_done[c.lane] = 0;
    if (c.lane == 0) c.ctrl->abort_flag = c.ctrl->pos_bad = 0;
    fence_mbar_init();
    named_bar_arrive(kChainReady, kChainThreads<W>);
    __syncwarp();
    int leader;
    if (elect_one(leader)) {
      const uint64_t policy = l2_evict_first_policy();
      uint32_t slot = 0, k = 0, issued = 0;
      bool dead = false;
      for (int u = 0; u < units && !dead; ++u) {
        const ChainUnit cu = chain_unit(L, op0, local + u * count);
        tab.unit[u & (kChainUnits - 1)] = cu;     // (ordered before the arrivals on the unit's pages)
        const uint8_t* maps = L.maps + cu.op * 512;
        const bool pair = L.head[cu.op].mode == MK_MV_PAIR;
        MvLoad ml;
        ml.fp4 = WF == 2;
        ml.tm_a = maps;
        ml.tm_b = maps + (pair ? 128 : 0);
        ml.ts_a = maps + 256;
        ml.ts_b = maps + (pair ? 384 : 256);
        ml.rowA0 = cu.rowA0;
        ml.rowB0 = cu.rowB0;
        ml.tiles_per_page = L.head[cu.op].tiles;
        ml.half = (uint32_t)ml.tiles_per_page * 1024u;
        if (u == 0 && !early) prior_work_done();
#pragma unroll 1
        for (int p = 0; p < P; ++p) {
          if ((issued == (uint32_t)L.ahead && !wait_mbar_one(c, smem_u32(&c.ctrl->staged), 0u, MK_ST_TIMEOUT_PAGE_EMPTY, (int)issued)) ||
              (k > 0 && !wait_mbar_one(c, empty_bar(c, slot), (k & 1u) ^ 1u, MK_ST_TIMEOUT_PAGE_EMPTY, (int)issued))) {
            dead = true;
            break;
          }
          mv_load_issue(ml, p, c.pages_u32 + slot * page_bytes, full_bar(c, slot), policy);
          ++issued;
          if (++slot == (uint32_t)L.stages) {
            slot = 0;
            ++k;
          }
        }
      }
      // every copy has landed before the CTA may exit (the consumers wait for all of them, unless a wait ran out)
      for (uint32_t i = 0; i < min(issued, (uint32_t)L.stages); ++i) {
        if (slot == 0) {
          slot = (uint32_t)L.stages;
          --k;
        }
        --slot;
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(full_bar(c, slot), k & 1u))
          if (globaltimer_ns() - t0 > L.pv.timeout_ns) break;
      }
    }
    return;
  }

  // ---- consumers
  const int failed = threadIdx.x == 0 ? launch_failed(L.pv) : 0;
  for (int i = threadIdx.x; i < L.n_ops * (int)(sizeof(mk_op_t) / 16); i += W * 32)
    reinterpret_cast<uint4*>(ops)[i] = ldcg128(reinterpret_cast<const uint4*>(L.pv.ops + L.first_op) + i);
  named_bar_sync(kChainReady, kChainThreads<W>);      // the records, and the loader's barriers
  if (failed) c.ctrl->pos_bad = -1;
  const mk_op_t* sop = ops + op0;
  const int K = sop->i[MK_MV_K], M = ROWS == 1 ? 1 : sop->i[MK_MV_M], Kc = sop->i[MK_MV_KC], pro = sop->i[MK_MV_PRO];
  ChainWalk walk;
  {
    const int tid = (int)threadIdx.x, m = tid & 31, chunks = K >> 3;
    const int b = ROWS == 1 ? 0 : small_div(m, L.s_magic), t = ROWS == 1 ? 0 : m - b * sop->i[MK_MV_S];
    int pos = 0;
    if (L.pv.dyn_pos != nullptr) {
      // one position per sequence, or one for all; every launch looks at all of them
      prior_work_done();
      const volatile int32_t* at = reinterpret_cast<const volatile int32_t*>(L.pv.dyn_pos);
      const int any = at[min(m, L.pv.pos_count - 1)];
      pos = at[min(b, L.pv.pos_count - 1)];
      if (m < L.pv.pos_count && (uint32_t)any >= (uint32_t)L.pv.pos_limit) c.ctrl->pos_bad = 1 + m;
      if (tid < 32) c.ctrl->pos[m] = any;
    }
#pragma unroll 1
    for (int o = tid >> 5; o < L.n_ops; o += W)
      if (m < M) rows[o * 32 + m] = chain_row(ops + o, b, t, pos);
    if (tid < M) {
      const mk_op_t* ro = ops + max(L.res_op, 0);
      tab.in[m].x = b * sop->s[MK_MV_S_X_B] + t * sop->s[MK_MV_S_X_S];
      tab.in[m].ri = b * sop->s[MK_MV_S_RI_B] + t * sop->s[MK_MV_S_RI_S];
      tab.in[m].ro = b * ro->s[MK_MV_S_RO_B] + t * ro->s[MK_MV_S_RO_S];
    }
    walk.m0 = small_div(tid, L.chunk_magic[op0]);
    walk.ch0 = tid - walk.m0 * chunks;
    walk.dm = small_div(W * 32, L.chunk_magic[op0]);
    walk.dch = W * 32 - walk.dm * chunks;
  }
  named_bar_sync(kChainBarrier, W * 32);
  const int bad = c.ctrl->pos_bad;
  prior_work_done();
  if ((L.flags & kChainLast) && blockIdx.x == 0 && threadIdx.x == 0) L.pv.state->launches += 1;
  if (bad) {
    // a position outside the caches, or a launch before has failed: nothing runs, the residual output included
    // (the report raises the abort flag, at which the loader stops)
    if (threadIdx.x == 0) {
      if (bad > 0) report(c, MK_ST_BAD_POSITION, c.ctrl->pos[bad - 1], L.pv.pos_limit);
      else atomicExch(&c.ctrl->abort_flag, 1);
    }
    return;
  }
  if (units > 0) {
    const mk_op_t* res_op = L.res_op >= 0 && blockIdx.x == 0 ? ops + L.res_op : nullptr;
    if constexpr (chain_fetches(ROWS, WF, W)) {
      chain_fetch_rows<WF>(c, L, sop, M, tab.in);
      if (pro == MK_PRO_NONE) {
        if constexpr (WF == 2) chain_to_f16<W>(c, sop, M, walk);
      } else if constexpr (WF != 1) {
        chain_norm_rows<WF, 4, W>(c, L, sop, tab.in, res_op);
      }
    } else if (pro == MK_PRO_NONE) {
      chain_stage_plain<WF>(c, sop, M, tab.in, walk);
    } else if constexpr (WF != 1) {
      // rows' parts, and chunks of each, requested together
      constexpr int R = ROWS == 1 ? 1 : (WF == 0 && NT != 1 ? 3 : 2), H = ROWS == 1 || WF == 2 ? 3 : (NT == 1 ? 2 : 1);
      chain_stage_rms<ROWS, WF, R, H, W>(c, sop, tab.in, res_op);
    }
  }
  named_bar_sync(kChainBarrier, W * 32);
  // The next launch starts, and begins to fetch its weights, only now: its copies would stand in the way of this launch's
  // activations.  (No launch behind the first starts before all CTAs of this one have come here, behind the wait: what ran
  // before the program is visible to every load of the later launches, early or not.)
  if (threadIdx.x == 0) mbar_arrive(smem_u32(&c.ctrl->staged));
  next_may_start();

  const int g = c.lane >> 2;
  const uint32_t xs = chain_row_stride<WF>(K);
  const uint32_t half = mv_half_bytes(WF == 2 ? (int)MK_W_NVFP4_E4M3S16 : (int)MK_W_BF16, Kc);
  const bool f16s = WF == 2 && sop->i[MK_MV_WFMT] == MK_W_NVFP4_F16S32;
  constexpr int NA = Cut::NA, AN = Cut::AN, NN = Cut::NN;
  float4* slots = reinterpret_cast<float4*>(smem + L.slot_off);
  // Groups of AS warps take the CTA's partial sums in turn (dealt out), or its units, and walk straight from one of their pages
  // to the next.  Looking at all pages for those that are its own cost a warp some 1500 clocks between two pages of 4000
  // clocks of products (NVFP4 1 x 4096 -> 14336), by device clocks: 8B NVFP4 step us batch 1 2255 ->
  // 2194, batch 8 3516 -> 3410, 1B shape batch 16 1185 -> 1165.  (Aligned groups: with one warp more from unit to unit, so
  // that the one that adds a unit up sits the next one out, 2233, 3487 and 1190.)
  constexpr int G = W / AS;
  const int h = c.warp & (AS - 1), grp = c.warp / AS;
  const int a0 = (h & (Cut::AH - 1)) * AN, n0 = (h / Cut::AH) * NN;   // this warp's accumulators and n-tiles
  // (rows past M read row 0: their columns of the accumulators are never stored.  The row's parity, which places
  // its chunks, is the lane's: an odd lane of a missing row finds other values of row 0, as good as any.)
  uint32_t xrow[NN];
#pragma unroll
  for (int n = 0; n < NN; ++n) {
    const int m = (n0 + n) * 8 + g;
    xrow[n] = c.act_u32 + (uint32_t)(m < M ? m : 0) * xs;
  }
  const int spread = L.spread;
  const int u_step = spread ? 1 : G, q_step = spread ? G : 1;
  int q0 = spread ? grp : 0;         // this group's first partial sum of unit u
#pragma unroll 1
  for (int u = spread ? 0 : grp; u < units && !c.dead; u += u_step) {
    const uint32_t set = (uint32_t)u & ((1u << L.sets_log2) - 1u), gen = (uint32_t)u >> L.sets_log2;
    float4* mine = slots + (size_t)set * (uint32_t)(parts * NA * NT) * 32u + c.lane;
    bool entered = false;
#pragma unroll 1
    for (int lap = 0; lap < P; lap += parts) {      // (pages of a unit beyond its partial sums go round again, in the ring's order)
#pragma unroll 1
      for (int part = q0; part < parts && lap + part < P; part += q_step) {
        const int p = lap + part;
        const uint32_t page_no = (uint32_t)(u * P + p), k = ring_lap(page_no, (uint32_t)L.stage_magic), slot = page_no - k * (uint32_t)L.stages;
        const uint32_t page = c.pages_u32 + slot * page_bytes;
        if (!chain_acquire(c, slot, k, k * AS)) goto out;
        const ChainUnit& cu = tab.unit[u & (kChainUnits - 1)];
        if (p == 0 && h == 0 && (cu.flags & (kEpiRope | kEpiResidual)) && c.lane < M) {
          // what the unit's epilogue reads: into L1 now
          const mk_op_t* op = ops + cu.op;
          const ChainRow& row = rows[cu.op * 32 + c.lane];
          if (cu.flags & kEpiRope) {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(op->p[MK_MV_P_COS] + (uint64_t)(row.tab + cu.chunk * 8) * 2u));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(op->p[MK_MV_P_SIN] + (uint64_t)(row.tab + cu.chunk * 8) * 2u));
          } else {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(op->p[MK_MV_P_EPI_RES] + (uint64_t)(row.er + cu.rowA0) * 2u));
          }
        }
        auto rec = [&](int a, int n) -> float4& { return mine[((part * NA + a0 + a) * NT + n0 + n) * 32]; };
        float acc[AN][NN][4];
#pragma unroll
        for (int a = 0; a < AN; ++a)
#pragma unroll
          for (int n = 0; n < NN; ++n) acc[a][n][0] = acc[a][n][1] = acc[a][n][2] = acc[a][n][3] = 0.f;
        if (__builtin_expect(lap > 0, 0)) {   // a further page of the same partial sum: this warp left it here
#pragma unroll
          for (int a = 0; a < AN; ++a)
#pragma unroll
            for (int n = 0; n < NN; ++n) {
              const float4 v = rec(a, n);
              acc[a][n][0] = v.x, acc[a][n][1] = v.y, acc[a][n][2] = v.z, acc[a][n][3] = v.w;
            }
        }
        const int k0 = p * Kc, kc = min(Kc, K - k0);
        if constexpr (WF == 2)
          chain_page_fp4<NT, AS>(acc, page, half, kc >> 8, xrow, (uint32_t)k0, h, c.lane, f16s);
        else
          chain_page_dense<NT, WF, AS>(acc, page, half, kc >> 6, xrow, (uint32_t)k0, h, c.lane);
        __syncwarp();
        if (c.lane == 0) {
          mbar_arrive(empty_bar(c, slot));
          atomicAdd(&c.ctrl->released[slot], 1u);
        }
        if (!entered && gen > 0 && !wait_smem_ge(c, &c.ctrl->mv_done[set], gen, u)) goto out;   // the set's previous user must have been summed
        entered = true;
#pragma unroll
        for (int a = 0; a < AN; ++a)
#pragma unroll
          for (int n = 0; n < NN; ++n) rec(a, n) = make_float4(acc[a][n][0], acc[a][n][1], acc[a][n][2], acc[a][n][3]);
        if (p + last_pages >= P) {
          // this warp's last page of the partial sum, or of the unit
          __syncwarp();
          int last = 0;
          if (c.lane == 0) {
            uint32_t old;
            asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(old) : "r"(smem_u32(&c.ctrl->mv_arrive[set])) : "memory");
            last = old == (uint32_t)(arrivals - 1);
          }
          last = __shfl_sync(0xffffffffu, last, 0);
          if (last) chain_finish<ROWS, WF, NA, KS>(c, ops, rows, cu, local + u * count, mine, parts, set, gen);
        }
      }
    }
    if (spread) {
      q0 -= parts;
      while (q0 < 0) q0 += G;
    }
  }
out:;
}

}  // namespace mk

// One compiled kernel: <activation rows, weight family (0 bf16, 1 fp16, 2 NVFP4), warps a page, with the sum of K blocks,
// consumer warps>.
typedef void (*mk_chain_fn)(const mk::MvLaunch);
struct mk_chain_variant {
  int rows, as, ks, warps;
  mk_chain_fn fn;
};
#define MK_CHAIN_KERNEL(ROWS, WF, AS, KS, W) {ROWS, AS, KS, W, mk::mv_chain_kernel<ROWS, WF, AS, KS, W>}
// (K blocks of up to 8 rows on eight warps: NVFP4 only, two CTAs a multiprocessor)
#define MK_CHAIN_TABLE(name, WF, ...)                                                                     \
  extern "C" const mk_chain_variant* name(int* n) {                                                       \
    static const mk_chain_variant v[] = {                                                                 \
        MK_CHAIN_KERNEL(1, WF, 2, false, 8),   MK_CHAIN_KERNEL(1, WF, 4, false, 8),                       \
        MK_CHAIN_KERNEL(8, WF, 2, false, 8),   MK_CHAIN_KERNEL(8, WF, 4, false, 8),                       \
        MK_CHAIN_KERNEL(8, WF, 2, false, 16),  MK_CHAIN_KERNEL(8, WF, 4, false, 16),                      \
        MK_CHAIN_KERNEL(16, WF, 2, false, 16), MK_CHAIN_KERNEL(16, WF, 4, false, 16),                     \
        MK_CHAIN_KERNEL(32, WF, 2, false, 8),  MK_CHAIN_KERNEL(32, WF, 4, false, 8),                      \
        MK_CHAIN_KERNEL(8, WF, 2, true, 16),   MK_CHAIN_KERNEL(16, WF, 2, true, 16),                      \
        MK_CHAIN_KERNEL(32, WF, 2, true, 8),   ##__VA_ARGS__};                                            \
    *n = (int)(sizeof(v) / sizeof(v[0]));                                                                 \
    return v;                                                                                             \
  }
