// Row-wise ops, the split-KV combine and the top-1 finalise as launches of their own in a program that runs as a chain of
// kernels: one warp a unit, the unit code of the persistent kernel.
#pragma once
#include "chain_mv.cuh"
#include "op_attn.cuh"
#include "op_elementwise.cuh"

namespace mk {

struct EwLaunch {
  ProgramView pv;
  int32_t flags, index;
};

static __global__ void __launch_bounds__(kEwWarps * 32) ew_chain_kernel(const __grid_constant__ EwLaunch L) {
  __shared__ Ctrl ctrl;
  __shared__ mk_op_t rec;
  Ctx c;
  c.pv = &L.pv;
  c.ctrl = &ctrl;
  c.warp = threadIdx.x >> 5;
  c.lane = threadIdx.x & 31;
  c.instr_idx = L.index;
  c.dead = false;
  c.trace_base = nullptr;
  c.trace_n = c.trace_cap = 0;
  if (!plan_in_force(L.pv)) {
    prior_work_done();
    return;
  }
  if (threadIdx.x == 0) ctrl.abort_flag = launch_failed(L.pv), ctrl.pos_bad = 0;
  if (threadIdx.x < sizeof(mk_op_t) / 16)
    reinterpret_cast<uint4*>(&rec)[threadIdx.x] = ldcg128(reinterpret_cast<const uint4*>(L.pv.ops + L.index) + threadIdx.x);
  __syncthreads();
  prior_work_done();
  next_may_start();
  if (threadIdx.x < 32) {
    if (L.pv.dyn_pos != nullptr) {
      const int v = reinterpret_cast<const volatile int32_t*>(L.pv.dyn_pos)[min(c.lane, L.pv.pos_count - 1)];
      if (c.lane < L.pv.pos_count && (uint32_t)v >= (uint32_t)L.pv.pos_limit) ctrl.pos_bad = 1 + c.lane;
      ctrl.pos[c.lane] = v;
    }
    // The top-1 looks again, behind the wait: no token is chosen or fed back behind a launch that failed (a row of which no unit
    // has left a maximum would name token -1)
    if (rec.opcode == MK_OP_TOP1_FINAL && launch_failed(L.pv) && c.lane == 0) ctrl.abort_flag = 1;
    if ((L.flags & kChainLast) && blockIdx.x == 0 && c.lane == 0) L.pv.state->launches += 1;
  }
  __syncthreads();
  if (ctrl.pos_bad) {
    if (threadIdx.x == 0) report(c, MK_ST_BAD_POSITION, ctrl.pos[ctrl.pos_bad - 1], L.pv.pos_limit);
    return;
  }
  if (ctrl.abort_flag) return;
  const int unit = (int)blockIdx.x * kEwWarps + c.warp;
  const mk_op_t* op = &rec;
  if (unit >= op->n_units) return;
  switch (op->opcode) {
    case MK_OP_RMSNORM: ew_rmsnorm(c, op, unit); break;
    case MK_OP_ROPE: ew_rope(c, op, unit); break;
    case MK_OP_QKNORM_ROPE: ew_qknorm_rope(c, op, unit); break;
    case MK_OP_GLU: ew_glu(c, op, unit); break;
    case MK_OP_ADD: ew_add(c, op, unit); break;
    case MK_OP_ATTN_COMBINE: at_combine_unit(c, op, unit); break;
    case MK_OP_TOP1_FINAL: ew_top1_final(c, op, unit); break;
    default: break;
  }
}

}  // namespace mk
