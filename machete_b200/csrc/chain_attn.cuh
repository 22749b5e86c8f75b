// Split-KV attention launches of a program that runs as a chain of kernels (see chain.inc): one CTA a unit, with the pages,
// participants, partial states and combine of at_unit, bit for bit.
//
// What a launch of one token's attention is bound by, besides the cache's bytes, is what follows the last page: the states of
// up to seven warps are merged, the partial goes to memory and the last CTA of a (batch, KV head) group combines the
// group's splits.  The persistent kernel does each of these on one warp (12 us of a layer's 20 at head dim 128, 8192 tokens);
// here all warps of the CTA, the loader's included, share them: a merge takes n-tiles of the output in turn, a combine pairs of values, and
// neither changes the order of any sum.  The cache does not depend on the kernel before, except for the rows that it
// appends: the loader fills the ring before it waits, and waits at the first page that holds such a row.  The query rows go
// through shared memory, normalised and rotated once for all warps, which also leaves 128 registers a thread enough for
// head dim 128: two CTAs share an SM.
#pragma once
#include "chain_mv.cuh"
#include "op_attn.cuh"

namespace mk {

// Participants and a loader.  Seven participants, of which two CTAs share a multiprocessor; or four, and three or four CTAs, for
// launches of many units of few pages (see chain_attn_step).
template <int PARTS>
constexpr int kAtChainThreads = (PARTS + 1) * 32;
// Shared memory of each: 228 KB a multiprocessor, 1 KB of a CTA's the system's.
constexpr int at_chain_smem(int ctas) { return (228 / ctas - 1) * 1024; }
constexpr int kAtChainMaxStages = 16;

struct AtLaunch {
  ProgramView pv;               // n_pages: ring slots; page_bytes: a K and a V block
  int32_t flags, index;
  int32_t tn, most_parts;       // tokens a page; participants of a unit at most
  int32_t q_off, comb_off, page_off;   // shared memory, bytes: query fragments; combine weights; ring
  const uint8_t* maps;                 // the K and the V cache's tensor maps
};

// Per-head RMSNorm and rotation of the query rows, as in at_unit, for k-steps `w` and `w` + D/32 (the two halves that a
// split-half rotation pairs): one warp each.
struct AtTables {
  uint32_t w0[2], w1[2], cs[2], sn[2];   // norm weights of both halves, cos, sin: values 2t and 2t + 8 of the k-step
};
template <int D>
__device__ __forceinline__ AtTables at_query_tables(const mk_op_t* op, int w, int t, int64_t tab_off) {
  const uint16_t* nw = reinterpret_cast<const uint16_t*>(op->p[MK_AT_P_QNW]);
  const uint16_t* cs = reinterpret_cast<const uint16_t*>(op->p[MK_AT_P_COS]) + tab_off;
  const uint16_t* sn = reinterpret_cast<const uint16_t*>(op->p[MK_AT_P_SIN]) + tab_off;
  AtTables r;
#pragma unroll
  for (int h2 = 0; h2 < 2; ++h2) {
    const int col = w * 16 + 2 * t + 8 * h2;
    r.w0[h2] = *reinterpret_cast<const uint32_t*>(nw + col);
    r.w1[h2] = *reinterpret_cast<const uint32_t*>(nw + col + D / 2);
    r.cs[h2] = *reinterpret_cast<const uint32_t*>(cs + col);
    r.sn[h2] = *reinterpret_cast<const uint32_t*>(sn + col);
  }
  return r;
}
template <int D>
__device__ __forceinline__ void at_norm_query(const mk_op_t* op, const uint32_t (&qf)[D / 16][4], const AtTables& tb, int w,
                                              uint32_t (&lo)[4], uint32_t (&hi)[4]) {
  constexpr int KS = D / 16;
  float ss[2] = {0.f, 0.f};
#pragma unroll
  for (int ks = 0; ks < KS; ++ks)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float vl = bf16lo(qf[ks][r]), vh = bf16hi(qf[ks][r]);
      ss[r & 1] += vl * vl + vh * vh;
    }
  float rstd[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 1);
    ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 2);
    rstd[e] = rsqrtf(ss[e] / (float)D + op->f[MK_AT_F_EPS]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) lo[i] = hi[i] = 0u;
#pragma unroll
  for (int ks = 0; ks < KS / 2; ++ks)
    if (ks == w) {
#pragma unroll
      for (int i = 0; i < 4; ++i) lo[i] = qf[ks][i], hi[i] = qf[ks + KS / 2][i];
    }
#pragma unroll
  for (int h2 = 0; h2 < 2; ++h2) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint32_t r0 = lo[e + 2 * h2], r1 = hi[e + 2 * h2];
      const uint32_t w0 = tb.w0[h2], w1 = tb.w1[h2], cc = tb.cs[h2], sc2 = tb.sn[h2];
      const float n0l = bf16_round(bf16lo(r0) * rstd[e] * bf16lo(w0)), n0h = bf16_round(bf16hi(r0) * rstd[e] * bf16hi(w0));
      const float n1l = bf16_round(bf16lo(r1) * rstd[e] * bf16lo(w1)), n1h = bf16_round(bf16hi(r1) * rstd[e] * bf16hi(w1));
      const float cl = bf16lo(cc), ch = bf16hi(cc), sl = bf16lo(sc2), sh = bf16hi(sc2);
      lo[e + 2 * h2] = pack_bf16(n0l * cl - n1l * sl, n0h * ch - n1h * sh);
      hi[e + 2 * h2] = pack_bf16(n1l * cl + n0l * sl, n1h * ch + n0h * sh);
    }
  }
}

// PARTS: participants; one more warp loads.  CTAS: that share a multiprocessor.
template <int D, bool QNORM, int PARTS, int CTAS>
__global__ void __launch_bounds__(kAtChainThreads<PARTS>, CTAS) at_chain_kernel(const __grid_constant__ AtLaunch L) {
  constexpr int KS = D / 16, ND = D / 8, TN = (D == 64) ? 64 : 32, NS = TN / 8;
  constexpr uint32_t kStateBytes = (ND + 1) * 512;
  extern __shared__ __align__(1024) uint8_t smem[];
  Ctx c;
  c.pv = &L.pv;
  c.ctrl = reinterpret_cast<Ctrl*>(smem);
  c.pages_u32 = smem_u32(smem + L.page_off);
  c.act_u32 = 0;
  c.warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  c.lane = threadIdx.x & 31;
  c.instr_idx = L.index;
  c.dead = false;
  c.trace_base = nullptr;
  c.trace_n = c.trace_cap = 0;
  if (!plan_in_force(L.pv)) {
    prior_work_done();
    return;
  }
  const int NPG = L.pv.n_pages;
  static_assert(!QNORM || PARTS >= KS / 2, "a warp for each pair of query fragments");
  if (threadIdx.x == 0) {
    for (int i = 0; i < NPG; ++i) {
      mbar_init(smem_u32(&c.ctrl->full[i]), 32);
      mbar_init(smem_u32(&c.ctrl->empty[i]), 1);
      c.ctrl->released[i] = 0;
    }
    c.ctrl->abort_flag = 0;
    c.ctrl->is_last = 0;
    c.ctrl->pos_bad = launch_failed(L.pv);
    fence_mbar_init();
  }
  if (threadIdx.x < sizeof(mk_op_t) / 16)
    reinterpret_cast<uint4*>(&c.ctrl->op_cache[0])[threadIdx.x] =
        ldcg128(reinterpret_cast<const uint4*>(L.pv.ops + L.index) + threadIdx.x);
  __syncthreads();
  const bool early = (L.flags & kChainEarlyLoads) != 0;
  if (!early) prior_work_done();
  if (c.ctrl->pos_bad) {     // a launch before has failed
    prior_work_done();
    if ((L.flags & kChainLast) && blockIdx.x == 0 && threadIdx.x == 0) L.pv.state->launches += 1;
    return;
  }
  const mk_op_t* op = &c.ctrl->op_cache[0];

  AtUnit u = at_decode(op, (int)blockIdx.x);
  const int M = op->i[MK_AT_M], H = op->i[MK_AT_H], G = op->i[MK_AT_GROUP], S = op->i[MK_AT_SPLITS];
  const bool dyn = op->i[MK_AT_DYNPOS] != 0;
  // (the position changes at the end of a program at the earliest: a launch behind the first may read it before it waits)
  int pos = 0;
  if (L.pv.dyn_pos != nullptr) {
    pos = reinterpret_cast<const volatile int32_t*>(L.pv.dyn_pos)[min(u.b, L.pv.pos_count - 1)];
    // every launch of the program sees a position outside the caches, and none runs
    bool bad = false;
    int worst = 0;
    for (int i = 0; i < L.pv.pos_count; ++i) {
      const int v = reinterpret_cast<const volatile int32_t*>(L.pv.dyn_pos)[i];
      if ((uint32_t)v >= (uint32_t)L.pv.pos_limit) bad = true, worst = v;
    }
    if (bad) {
      prior_work_done();
      if (threadIdx.x == 0) {
        if ((L.flags & kChainLast) && blockIdx.x == 0) L.pv.state->launches += 1;
        report(c, MK_ST_BAD_POSITION, worst, L.pv.pos_limit);
      }
      return;
    }
  }
  const int N = dyn ? min(op->i[MK_AT_N], pos + M) : op->i[MK_AT_N];
  u.t_begin = min(u.t_begin, N);
  u.t_end = min(u.t_end, N);
  const int tn = L.tn;
  const int np = (u.t_end - u.t_begin + tn - 1) / tn;
  const int parts = max(1, min(L.most_parts, np));

  uint32_t qf_at = smem_u32(smem + L.q_off) + (uint32_t)c.lane * 16u;   // query fragment of k-step ks: 512 bytes each
  const int g = c.lane >> 2, t = c.lane & 3;
  const float sc = op->f[MK_AT_F_SCALE];
  const float c2 = sc * 1.4426950408889634f;
  // rows of this thread: r0 = mt*16 + g, r1 = r0 + 8 -> (m, head)
  int rm[2], rh[2];
  bool rv[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = u.mt * 16 + g + 8 * e;
    rv[e] = r < M * G;
    rm[e] = (rv[e] && M != 1) ? r / G : 0;
    rh[e] = u.kvh * G + (rv[e] ? (M != 1 ? r % G : r) : 0);
  }

  if (c.warp == PARTS) {
    // ---- loader
    int leader;
    if (elect_one(leader)) {
      const uint64_t policy = l2_evict_first_policy();
      const int moved = op->i[kAtWaitDyn] ? pos : 0, w0 = op->i[kAtWaitLo] + moved, w1 = op->i[kAtWaitHi] + moved;
      bool waited = !early;
      uint32_t slot = 0, k = 0;
      int p = 0;
#pragma unroll 1
      for (; p < np; ++p) {
        const int tok0 = u.t_begin + p * tn;
        if (!waited && w0 < tok0 + tn && w1 > tok0) {
          prior_work_done();
          fence_proxy_async_all();   // the rows were written by plain stores
          waited = true;
        }
        if (k > 0 && !wait_mbar_one(c, empty_bar(c, slot), (k & 1u) ^ 1u, MK_ST_TIMEOUT_PAGE_EMPTY, p)) break;
        at_load_issue(L.maps, L.maps + 128, D == 128, tn, tok0, u.kvh, u.b, c.pages_u32 + slot * (uint32_t)L.pv.page_bytes,
                      full_bar(c, slot), policy);
        if (++slot == (uint32_t)NPG) {
          slot = 0;
          ++k;
        }
      }
      // every copy has landed before the ring serves for the states, and before the CTA may exit
      for (int i = 0; i < min(p, NPG); ++i) {
        if (slot == 0) {
          slot = (uint32_t)NPG;
          --k;
        }
        --slot;
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(full_bar(c, slot), k & 1u))
          if (globaltimer_ns() - t0 > L.pv.timeout_ns) break;
      }
    }
    __syncwarp();
  } else {
    // ---- query rows: fragments of the A operand, a k-step (or, normalised and rotated, a pair of them) a warp.  The tables
    // do not depend on the kernel before.
    const int64_t tab_off = dyn ? (int64_t)pos * op->i[MK_AT_NEW_TOK] : 0;
    AtTables tb = {};
    if constexpr (QNORM) {
      if (c.warp < KS / 2) tb = at_query_tables<D>(op, c.warp, t, tab_off);
      // (and what the new k row wants, close by)
      if (c.warp == PARTS - 1 && c.lane < D / 64)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(op->p[MK_AT_P_KNW] + (uint64_t)c.lane * 128u));
    }
    const uint16_t* q = reinterpret_cast<const uint16_t*>(op->p[MK_AT_P_Q]) + u.b * op->s[MK_AT_S_Q_B];
    const uint16_t* q0 = q + rm[0] * op->s[MK_AT_S_Q_M] + rh[0] * op->s[MK_AT_S_Q_H] + 2 * t;
    const uint16_t* q1 = q + rm[1] * op->s[MK_AT_S_Q_M] + rh[1] * op->s[MK_AT_S_Q_H] + 2 * t;
    auto fetch = [&](int ks, uint32_t (&f)[4]) {
      f[0] = rv[0] ? __ldcg(reinterpret_cast<const uint32_t*>(q0 + ks * 16)) : 0u;
      f[1] = rv[1] ? __ldcg(reinterpret_cast<const uint32_t*>(q1 + ks * 16)) : 0u;
      f[2] = rv[0] ? __ldcg(reinterpret_cast<const uint32_t*>(q0 + ks * 16 + 8)) : 0u;
      f[3] = rv[1] ? __ldcg(reinterpret_cast<const uint32_t*>(q1 + ks * 16 + 8)) : 0u;
    };
    prior_work_done();
    if ((L.flags & kChainLast) && blockIdx.x == 0 && threadIdx.x == 0) L.pv.state->launches += 1;
    if constexpr (QNORM) {
      if (c.warp < KS / 2) {
        uint32_t qf[KS][4], lo[4], hi[4];
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) fetch(ks, qf[ks]);
        at_norm_query<D>(op, qf, tb, c.warp, lo, hi);
        sts128(qf_at + (uint32_t)c.warp * 512u, make_uint4(lo[0], lo[1], lo[2], lo[3]));
        sts128(qf_at + (uint32_t)(c.warp + KS / 2) * 512u, make_uint4(hi[0], hi[1], hi[2], hi[3]));
      }
    } else {
#pragma unroll 1
      for (int ks = c.warp; ks < KS; ks += PARTS) {
        uint32_t f[4];
        fetch(ks, f);
        sts128(qf_at + (uint32_t)ks * 512u, make_uint4(f[0], f[1], f[2], f[3]));
      }
    }
    named_bar_sync(kConsumerBarrier, PARTS * 32);
    next_may_start();     // (not before: the next launch's weights would stand in the way of the query rows)
  }

  // ---- this participant's pages
  float o[ND][4];
#pragma unroll
  for (int i = 0; i < ND; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
  float mrow[2] = {-INFINITY, -INFINITY};
  float lrow[2] = {0.f, 0.f};   // per-lane partial row sums (summed over the quad at the end)
  if (c.warp < parts) {
    int lim[2];   // causal limit per row: token index <= N - M + m
#pragma unroll
    for (int e = 0; e < 2; ++e) lim[e] = op->i[MK_AT_CAUSAL] ? (N - M + rm[e]) : (N - 1);
    const uint32_t tile_bytes = (uint32_t)tn * (uint32_t)D * 2u;
    // Where this lane's rows of an 8 x 8 matrix lie: token row r of the tile, 16-byte chunk 2 * step + (which matrix) under the
    // 128-byte swizzle, which repeats every four steps; `sub` is the next 64 values of the head dim.
    const int mat = c.lane >> 3, r8 = c.lane & 7;
    const uint32_t sub = (uint32_t)tn * 128u;
    const uint32_t krow = (uint32_t)((mat >> 1) * 8 + r8) * 128u, vrow = tile_bytes + (uint32_t)((mat & 1) * 8 + r8) * 128u;
    uint32_t kx[4], vx[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      kx[i] = krow + (uint32_t)(((2 * i + (mat & 1)) ^ r8) << 4);
      vx[i] = vrow + (uint32_t)(((2 * i + (mat >> 1)) ^ r8) << 4);
    }
    RingPos rp;
    rp.slot = rp.k = 0;
    ring_advance(rp, c.warp, NPG);
#pragma unroll 1
    for (int p = c.warp; p < np; p += parts, ring_advance(rp, parts, NPG)) {
      uint32_t page;
      if (!page_acquire(c, rp, page)) break;
      const int tp0 = u.t_begin + p * tn;
      if constexpr (QNORM) {
        const int nt = dyn ? pos : op->i[MK_AT_NEW_TOK];
        if (nt >= tp0 && nt < tp0 + tn && nt < u.t_end)
          at_fix_k_row<D>(c, op, u, page, tn, nt - tp0, nt, dyn ? (int64_t)nt * op->i[MK_AT_NEW_TOK] : 0);
      }
#pragma unroll 1
      for (int blk = 0; blk * TN < tn; ++blk) {
        const int tb0 = tp0 + blk * TN;       // token of column 0 of the block
        if (tb0 >= u.t_end) break;
        const uint32_t at = page + (uint32_t)(blk * TN) * 128u;
        float s[NS][4];
#pragma unroll
        for (int i = 0; i < NS; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[i][e] = 0.f;
        // S = Q K^T
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          const uint4 qv = lds128(qf_at + (uint32_t)ks * 512u);
#pragma unroll
          for (int pr = 0; pr < NS / 2; ++pr) {
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4(at + kx[ks & 3] + (ks >= 4 ? sub : 0u) + (uint32_t)pr * 2048u, b0, b1, b2, b3);
            mma_bf16(s[2 * pr], qv.x, qv.y, qv.z, qv.w, b0, b1);
            mma_bf16(s[2 * pr + 1], qv.x, qv.y, qv.z, qv.w, b2, b3);
          }
        }
        // mask + row max
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < NS; ++i) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int tok = tb0 + i * 8 + 2 * t + (e & 1);
            const int row = e >> 1;
            if (tok >= u.t_end || tok > lim[row]) s[i][e] = -INFINITY;
            mx[row] = fmaxf(mx[row], s[i][e]);
          }
        }
        float corr[2], muse[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
          mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
          const float mnew = fmaxf(mrow[e], mx[e]);
          muse[e] = (mnew == -INFINITY) ? 0.f : mnew;
          corr[e] = fast_exp2((mrow[e] - muse[e]) * c2);
          mrow[e] = mnew;
          lrow[e] *= corr[e];
        }
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          o[i][0] *= corr[0];
          o[i][1] *= corr[0];
          o[i][2] *= corr[1];
          o[i][3] *= corr[1];
        }
        // P = exp2(S*c2 - m*c2), packed as bf16 A fragments
        uint32_t pf[NS / 2][4];
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          float pv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = e >> 1;
            pv[e] = fast_exp2(s[i][e] * c2 - muse[row] * c2);
            lrow[row] += pv[e];
          }
          pf[i >> 1][(i & 1) * 2 + 0] = pack_bf16(pv[0], pv[1]);
          pf[i >> 1][(i & 1) * 2 + 1] = pack_bf16(pv[2], pv[3]);
        }
        // O += P V
#pragma unroll
        for (int kk = 0; kk < NS / 2; ++kk) {
#pragma unroll
          for (int dp = 0; dp < ND / 2; ++dp) {
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4_trans(at + vx[dp & 3] + (dp >= 4 ? sub : 0u) + (uint32_t)kk * 2048u, b0, b1, b2, b3);
            mma_bf16(o[2 * dp], pf[kk][0], pf[kk][1], pf[kk][2], pf[kk][3], b0, b1);
            mma_bf16(o[2 * dp + 1], pf[kk][0], pf[kk][1], pf[kk][2], pf[kk][3], b2, b3);
          }
        }
      }
      page_release(c, rp);
    }
  }

  // ---- states, merged in participant order; a warp takes every W-th n-tile of the output
  __syncthreads();      // all pages are consumed: the ring is free
  if (c.warp < parts) {
    const uint32_t park = c.pages_u32 + (uint32_t)c.warp * kStateBytes;
#pragma unroll
    for (int i = 0; i < ND; ++i)
      sts128(park + (uint32_t)(i * 32 + c.lane) * 16u,
             make_uint4(__float_as_uint(o[i][0]), __float_as_uint(o[i][1]), __float_as_uint(o[i][2]), __float_as_uint(o[i][3])));
    sts128(park + (uint32_t)(ND * 32 + c.lane) * 16u, make_uint4(__float_as_uint(mrow[0]), __float_as_uint(mrow[1]),
                                                                 __float_as_uint(lrow[0]), __float_as_uint(lrow[1])));
  }
  __syncthreads();
  constexpr int W = PARTS + 1, MT = (ND + PARTS) / W;
  float om[MT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i) om[i][0] = om[i][1] = om[i][2] = om[i][3] = 0.f;
  mrow[0] = mrow[1] = -INFINITY;
  lrow[0] = lrow[1] = 0.f;
  {
    // everything that is read is requested first; the running maximum and the weights do not depend on the values
    uint4 ml[PARTS], v[PARTS][MT];
#pragma unroll
    for (int j = 0; j < PARTS; ++j) {
      if (j >= parts) break;
      const uint32_t src = c.pages_u32 + (uint32_t)j * kStateBytes + (uint32_t)c.lane * 16u;
      ml[j] = lds128_sync(src + (uint32_t)ND * 512u);
#pragma unroll
      for (int i = 0; i < MT; ++i)
        if (c.warp + W * i < ND) v[j][i] = lds128_sync(src + (uint32_t)(c.warp + W * i) * 512u);
    }
#pragma unroll
    for (int j = 0; j < PARTS; ++j) {
      if (j >= parts) break;
      const float mj[2] = {__uint_as_float(ml[j].x), __uint_as_float(ml[j].y)};
      const float lj[2] = {__uint_as_float(ml[j].z), __uint_as_float(ml[j].w)};
      float wa[2], wb[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float mnew = fmaxf(mrow[e], mj[e]);
        const float muse = (mnew == -INFINITY) ? 0.f : mnew;
        wa[e] = fast_exp2((mrow[e] - muse) * c2);
        wb[e] = fast_exp2((mj[e] - muse) * c2);
        mrow[e] = mnew;
        lrow[e] = lrow[e] * wa[e] + lj[e] * wb[e];
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        om[i][0] = om[i][0] * wa[0] + __uint_as_float(v[j][i].x) * wb[0];
        om[i][1] = om[i][1] * wa[0] + __uint_as_float(v[j][i].y) * wb[0];
        om[i][2] = om[i][2] * wa[1] + __uint_as_float(v[j][i].z) * wb[1];
        om[i][3] = om[i][3] * wa[1] + __uint_as_float(v[j][i].w) * wb[1];
      }
    }
  }
  // normalised partial + lse
  float* op_ = reinterpret_cast<float*>(op->p[MK_AT_P_OPART]);
  float* lp_ = reinterpret_cast<float*>(op->p[MK_AT_P_LSEPART]);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    float l = lrow[e];
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    if (!rv[e]) continue;
    const float inv = l > 0.f ? 1.f / l : 0.f;
    const int64_t base = ((((int64_t)u.b * H + rh[e]) * S + u.sp) * M + rm[e]);
    float* dst = op_ + base * D;
#pragma unroll
    for (int i = 0; i < MT; ++i)
      if (c.warp + W * i < ND)
        *reinterpret_cast<float2*>(dst + (c.warp + W * i) * 8 + 2 * t) = make_float2(om[i][2 * e] * inv, om[i][2 * e + 1] * inv);
    if (t == 0 && c.warp == 0) lp_[base] = l > 0.f ? mrow[e] * sc + __logf(l) : -INFINITY;
  }
  if (!op->i[MK_AT_FUSE_COMBINE]) return;

  // ---- count this split in; whoever completes the group combines it
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t* arrive = reinterpret_cast<int32_t*>(op->p[MK_AT_P_ARRIVE]) + ((size_t)u.b * op->i[MK_AT_HKV] + u.kvh) * op->i[MK_AT_MT] + u.mt;
    // one acq_rel atomic: releases the partial (all threads' stores, ordered by the barrier) and acquires the others'
    int32_t old;
    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(old) : "l"(arrive) : "memory");
    if (old == S - 1) *arrive = 0;   // ready for the next launch
    c.ctrl->is_last = old == S - 1;
  }
  __syncthreads();
  if (!c.ctrl->is_last) return;
  // As at_combine_group, with a pair of values a thread: splits are added in order.  Row r's weights: comb[r * S + s].  The
  // first splits' values are requested before the weights are worked out.
  constexpr int UN = 18;
  float* comb = reinterpret_cast<float*>(smem + L.comb_off);
  float* inv_of = reinterpret_cast<float*>(c.ctrl->red);
  const int rows = min(16, M * G - u.mt * 16);
  auto pair_at = [&](int i, int64_t& off) -> const float* {   // the pair's partial values, and where its result goes
    const int r0 = i / (D / 2), d = (i % (D / 2)) * 2;
    const int r = u.mt * 16 + r0, m = M != 1 ? r / G : 0, h = u.kvh * G + (M != 1 ? r % G : r);
    off = u.b * op->s[MK_AT_S_O_B] + m * op->s[MK_AT_S_O_M] + h * op->s[MK_AT_S_O_H] + d;
    return op_ + ((((int64_t)u.b * H + h) * S) * M + m) * D + d;
  };
  const int64_t stride = (int64_t)M * D;
  float2 v[UN];
  auto fetch_pairs = [&](const float* base, int s0) {
#pragma unroll
    for (int k = 0; k < UN; ++k)
      v[k] = s0 + k < S ? __ldcg(reinterpret_cast<const float2*>(base + (s0 + k) * stride)) : make_float2(0.f, 0.f);
  };
  int pair = threadIdx.x;
  int64_t off = 0;
  const float* base = pair < rows * (D / 2) ? pair_at(pair, off) : nullptr;
  if (base) fetch_pairs(base, 0);
  for (int r0 = c.warp; r0 < rows; r0 += W) {
    const int r = u.mt * 16 + r0, m = M != 1 ? r / G : 0, h = u.kvh * G + (M != 1 ? r % G : r);
    const float* ls = lp_ + ((int64_t)u.b * H + h) * S * M + m;
    float* w = comb + r0 * S;
    float lv[4], mx = -INFINITY;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      lv[q] = c.lane + 32 * q < S ? __ldcg(ls + (int64_t)(c.lane + 32 * q) * M) : -INFINITY;
      mx = fmaxf(mx, lv[q]);
    }
    mx = warp_max(mx);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c.lane + 32 * q < S) w[c.lane + 32 * q] = mx != -INFINITY ? __expf(lv[q] - mx) : 0.f;
    __syncwarp();
    float sum = 0.f;
#pragma unroll 4
    for (int s = 0; s < S; ++s) sum += w[s];
    if (c.lane == 0) {
      inv_of[r0] = sum > 0.f ? 1.f / sum : 0.f;
      float* lse_out = reinterpret_cast<float*>(op->p[MK_AT_P_LSE]);
      if (lse_out) lse_out[((int64_t)u.b * H + h) * M + m] = (sum > 0.f) ? mx + __logf(sum) : -INFINITY;
    }
  }
  __syncthreads();
  const int ot = op->i[MK_AT_O_T];
#pragma unroll 1
  while (base) {
    const float inv = inv_of[pair / (D / 2)];
    const float* w = comb + pair / (D / 2) * S;
    float a0 = 0.f, a1 = 0.f;
#pragma unroll 1
    for (int s0 = 0;;) {
#pragma unroll
      for (int k = 0; k < UN; ++k) {
        const float ws = s0 + k < S ? w[s0 + k] * inv : 0.f;
        a0 += ws * v[k].x;
        a1 += ws * v[k].y;
      }
      s0 += UN;
      if (s0 >= S) break;
      fetch_pairs(base, s0);
    }
    if (ot == MK_T_FP32)
      *reinterpret_cast<float2*>(reinterpret_cast<float*>(op->p[MK_AT_P_O]) + off) = make_float2(a0, a1);
    else
      *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(op->p[MK_AT_P_O]) + off) = ot == MK_T_BF16 ? pack_bf16(a0, a1) : pack_f16(a0, a1);
    pair += kAtChainThreads<PARTS>;
    base = pair < rows * (D / 2) ? pair_at(pair, off) : nullptr;
    if (base) fetch_pairs(base, 0);
  }
}

}  // namespace mk

typedef void (*mk_chain_attn_fn)(const mk::AtLaunch);
struct mk_chain_attn_variant {
  int d, qnorm, parts, ctas;
  mk_chain_attn_fn fn;
};
