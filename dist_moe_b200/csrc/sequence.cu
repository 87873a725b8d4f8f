// The launches of one training pass or BF16 forward behind one call.  Host code only: small layers wait for the host, not
// for the GPU, and a call through the foreign-function interface costs more than the launch it is for.
//
// Launch order as in the reference's orchestration (BF16: dist_moe/api.py:1844-2188 forward, 2205-2609 backward; MXFP8:
// dist_moe/_blockscaled.py:1309-1931, 1951-2541).  Nothing here reads a device value, so a pass can be captured in a CUDA
// graph.
#include <cuda_runtime.h>

#include "../../include/dist_moe_b200.h"

namespace {

struct Sequence {
  const dm_layer_context& c;
  uint32_t steps;
  int32_t* report;  // launches made, step that failed
  void* stream;
  int rc = 0;

  // Runs `fn` (returning a library code) when `step` is asked for and nothing failed before; it makes `launches` launches.
  template <class Fn>
  void step(uint32_t bit, int launches, Fn&& fn) {
    if ((steps & bit) == 0 || rc != 0) return;
    rc = fn();
    if (rc != 0)
      report[1] = static_cast<int32_t>(bit);
    else
      report[0] += launches;
  }
  void barrier(uint32_t bit, const uint64_t* pads, const int* cond) {
    if (c.ep > 1)
      step(bit, 1, [&] { return dm_barrier(pads, c.rank, c.ep, 0, cond, c.barrier_timeout_ns, c.status, stream); });
  }
  // num_sms of a dispatch GEMM
  int dispatch_sms() const {
    if (!c.gather_flags_kept_clear) return c.num_sms;
    return DM_GATHER_FLAGS_KEPT_CLEAR | (c.num_sms < 0 ? 0 : c.num_sms > 0xffff ? 0xffff : c.num_sms);
  }
  dm_operand arena(const int64_t* offset) const { return dm_operand{c.arena, c.arena_bytes, offset}; }
};

const dm_operand kNone{nullptr, 0, nullptr};

}  // namespace

extern "C" int dm_bf16_forward(const dm_layer_context* ctx, const dm_layer_call* call, uint32_t steps, int32_t* report,
                               void* stream) {
  if (!ctx || !call || !report) return -1;
  const dm_layer_context& c = *ctx;
  const dm_layer_call& k = *call;
  report[0] = report[1] = 0;
  Sequence s{c, steps, report, stream};
  const int64_t stride = c.D * 2;
  int64_t* fs = k.fwd_state;
  const int route_launches = DM_ROUTE_LAUNCHES(c.ep, k.T, c.e_local, dm_route_decode_kernel_enabled());
  s.step(DM_FWD_PUBLISH, 1, [&] {
    return dm_publish(k.x, k.ids, k.ids_are_int64, c.dispatch, c.routing, k.T, c.D, c.K, c.E, k.validate_ids, c.status, stream);
  });
  s.barrier(DM_FWD_PUBLISH, c.dispatch_pads, nullptr);
  s.step(DM_FWD_ROUTE, route_launches, [&] {
    return dm_route(c.routing_ptrs, c.dispatch_ptrs, c.combine_ptrs, c.rank, c.ep, k.T, c.K, c.E, stride, stride, stride, 0,
                    c.capacity_rows, k.ptrs_size, k.counts, k.per_rank, k.expert_offsets, k.fwd_ptrs, k.bwd_ptrs, k.sct_ptrs,
                    c.route_workspace, c.route_workspace_words, c.status, stream);
  });
  const int32_t* recv = k.expert_offsets + c.e_local;
  s.step(DM_FWD_ROUTE, 1, [&] {
    return dm_plan_fwd_bf16(recv, k.per_rank, c.saved_bytes, c.buffer_offsets, c.peak_min_free, k.need, k.cond, fs,
                            c.slot_selector, c.moe_layer_id, c.ep, c.T_max, c.K, c.D, c.F, c.slot_bytes, c.num_slots,
                            k.num_layers, k.scratch_only | DM_PLAN_BOUNDED, c.status, stream);
  });
  if (!k.scratch_only)
    s.step(DM_FWD_SAVE_X, 1, [&] { return dm_cond_copy(k.x, nullptr, c.arena, fs, k.T * c.D * 2, k.cond, 1, stream); });
  // dispatch + W13: gather warps pull the routed rows (peer loads) while the tensor cores run; a forward without a backward
  // has no reader of h1: the fused epilogue then writes h2 alone
  s.step(DM_FWD_W13, k.separate_gather ? 2 : 1, [&] {
    const dm_operand xg = s.arena(fs + 1), h1 = k.fuse_swiglu && k.scratch_only ? kNone : s.arena(fs + 2);
    const dm_operand h2 = k.fuse_swiglu ? s.arena(fs + 3) : kNone;
    if (!k.separate_gather)
      return dm_gemm_fprop_dispatch(k.fwd_ptrs, c.gather_flags, xg, k.w13, h1, h2, k.expert_offsets, c.e_local, k.max_rows,
                                    2 * c.F, c.D, k.fuse_swiglu, c.clamped, c.alpha, c.limit, nullptr, s.dispatch_sms(), c.status,
                                    stream);
    const int rc = dm_gather_rows(k.fwd_ptrs, recv, c.arena, fs + 1, stride, k.max_rows, nullptr, stream);
    if (rc != 0) return rc;
    return dm_gemm_fprop(xg, k.w13, h1, h2, nullptr, k.expert_offsets, c.e_local, k.max_rows, 2 * c.F, c.D, k.fuse_swiglu,
                         c.clamped, c.alpha, c.limit, nullptr, c.num_sms, c.status, stream);
  });
  if (!k.fuse_swiglu)
    s.step(DM_FWD_SWIGLU, 1, [&] {
      return dm_swiglu_fwd(c.arena, fs + 2, c.arena, fs + 3, recv, k.max_rows, c.F, c.clamped, c.alpha, c.limit, k.clip_stats,
                           k.clip_limit, nullptr, stream);
    });
  s.step(DM_FWD_W2, 1, [&] {
    return dm_gemm_fprop(s.arena(fs + 3), k.w2, kNone, kNone, k.sct_ptrs, k.expert_offsets, c.e_local, k.max_rows, c.D, c.F, 0,
                         0, 1.0f, 0.0f, nullptr, c.num_sms, c.status, stream);
  });
  s.barrier(DM_FWD_COMBINE, c.combine_pads, nullptr);
  s.step(DM_FWD_REDUCE, 1, [&] {
    return dm_scale_and_sum(c.combine, k.scores, k.scores_are_bf16, k.ids, k.ids_are_int64, k.out, k.T, c.K, c.D,
                            k.scratch_only ? nullptr : c.arena, k.scratch_only ? nullptr : fs + 4,
                            k.scratch_only ? nullptr : k.cond, 0, stream);
  });
  return s.rc;
}

extern "C" int dm_bf16_backward(const dm_layer_context* ctx, const dm_layer_call* call, uint32_t steps, int32_t* report,
                                void* stream) {
  if (!ctx || !call || !report) return -1;
  const dm_layer_context& c = *ctx;
  const dm_layer_call& k = *call;
  report[0] = report[1] = 0;
  Sequence s{c, steps, report, stream};
  const int64_t stride = c.D * 2;
  const int64_t* fs = k.fwd_state;
  int64_t* bo = k.bwd_offsets;  // [xg, h1, h2, grad_h2, grad_h3_gathered, grad_h1]
  const int32_t* recv = k.expert_offsets + c.e_local;
  const int64_t x_bytes = k.T * c.D * 2;
  s.step(DM_BWD_PLAN, 1, [&] {
    return dm_plan_bwd_bf16(recv, k.per_rank, c.saved_bytes, c.buffer_offsets, c.peak_min_free, k.need, fs, bo, c.moe_layer_id,
                            c.ep, c.T_max, c.K, c.D, c.F, c.slot_bytes, c.num_slots, c.status, stream);
  });
  // ---- recompute block (device-predicated on the planner's decision) ------------------------------------------------
  s.step(DM_BWD_REPUBLISH, 1, [&] { return dm_cond_copy(c.arena, fs, c.dispatch, nullptr, x_bytes, k.cond, 1, stream); });
  s.barrier(DM_BWD_REPUBLISH, c.dispatch_pads, k.cond);
  s.step(DM_BWD_W13_AGAIN, k.separate_gather ? 2 : 1, [&] {
    if (!k.separate_gather)
      return dm_gemm_fprop_dispatch(k.fwd_ptrs, c.gather_flags, s.arena(bo), k.w13, s.arena(bo + 1), kNone, k.expert_offsets,
                                    c.e_local, k.max_rows, 2 * c.F, c.D, 0, c.clamped, c.alpha, c.limit, k.cond, s.dispatch_sms(),
                                    c.status, stream);
    const int rc = dm_gather_rows(k.fwd_ptrs, recv, c.arena, bo, stride, k.max_rows, k.cond, stream);
    if (rc != 0) return rc;
    return dm_gemm_fprop(s.arena(bo), k.w13, s.arena(bo + 1), kNone, nullptr, k.expert_offsets, c.e_local, k.max_rows, 2 * c.F,
                         c.D, 0, c.clamped, c.alpha, c.limit, k.cond, c.num_sms, c.status, stream);
  });
  // h2 is always rebuilt from h1: only x_gathered, h1 and h3 are ever saved
  s.step(DM_BWD_SWIGLU_AGAIN, 1, [&] {
    return dm_swiglu_fwd(c.arena, bo + 1, c.arena, bo + 2, recv, k.max_rows, c.F, c.clamped, c.alpha, c.limit, nullptr, 0.0f,
                         nullptr, stream);
  });
  s.step(DM_BWD_W2_AGAIN, 1, [&] {
    return dm_gemm_fprop(s.arena(bo + 2), k.w2, kNone, kNone, k.sct_ptrs, k.expert_offsets, c.e_local, k.max_rows, c.D, c.F, 0,
                         0, 1.0f, 0.0f, k.cond, c.num_sms, c.status, stream);
  });
  s.barrier(DM_BWD_W2_AGAIN, c.combine_pads, k.cond);
  s.step(DM_BWD_LOAD_H3, 1, [&] {
    return dm_cond_copy(c.arena, fs + 4, c.combine, nullptr, k.T * c.K * c.D * 2, k.cond, 0, stream);
  });
  // ---- gradient of the expert outputs and the scores: saved outputs are read where they were saved (chosen on the device)
  s.step(DM_BWD_GRAD_H3, 1, [&] {
    if (k.grad_scores != nullptr && !k.h3_in_combine)
      return dm_broadcast_and_scale_select(k.grad_out, k.scores, k.scores_are_bf16, k.ids, k.ids_are_int64, c.arena, fs + 4,
                                           c.combine, k.cond, c.combine, k.grad_scores, k.T, c.K, c.D, stream);
    return dm_broadcast_and_scale(k.grad_out, k.scores, k.scores_are_bf16, k.ids, k.ids_are_int64,
                                  k.grad_scores != nullptr ? c.combine : nullptr, nullptr, c.combine, k.grad_scores, k.T, c.K,
                                  c.D, stream);
  });
  s.barrier(DM_BWD_COMBINE, c.combine_pads, nullptr);
  // ---- W2 -----------------------------------------------------------------------------------------------------------
  s.step(DM_BWD_W2_DGRAD, k.separate_gather ? 2 : 1, [&] {
    if (!k.separate_gather)
      return dm_gemm_dgrad_dispatch(k.sct_ptrs, c.gather_flags, s.arena(bo + 4), k.w2, s.arena(bo + 3), k.expert_offsets,
                                    c.e_local, k.max_rows, c.F, c.D, nullptr, s.dispatch_sms(), c.status, stream);
    const int rc = dm_gather_rows(k.sct_ptrs, recv, c.arena, bo + 4, stride, k.max_rows, nullptr, stream);
    if (rc != 0) return rc;
    return dm_gemm_dgrad(s.arena(bo + 4), k.w2, s.arena(bo + 3), nullptr, k.expert_offsets, c.e_local, k.max_rows, c.F, c.D,
                         nullptr, c.num_sms, c.status, stream);
  });
  s.step(DM_BWD_W2_WGRAD, 1, [&] {
    return dm_gemm_wgrad(s.arena(bo + 4), s.arena(bo + 2), k.dw2, k.dw2_is_fp32, k.dw2_accumulate, k.expert_offsets, c.e_local,
                         k.max_rows, c.D, c.F, c.num_sms, c.status, stream);
  });
  // ---- SwiGLU backward, W13 input gradient (scattered to the owners) and weight gradient -----------------------------
  s.step(DM_BWD_SWIGLU, 1, [&] {
    return dm_swiglu_bwd(c.arena, bo + 1, c.arena, bo + 3, c.arena, bo + 5, recv, k.max_rows, c.F, c.clamped, c.alpha, c.limit,
                         stream);
  });
  s.step(DM_BWD_W13_DGRAD, 1, [&] {
    return dm_gemm_dgrad(s.arena(bo + 5), k.w13, kNone, k.bwd_ptrs, k.expert_offsets, c.e_local, k.max_rows, c.D, 2 * c.F,
                         nullptr, c.num_sms, c.status, stream);
  });
  s.step(DM_BWD_W13_WGRAD, 1, [&] {
    return dm_gemm_wgrad(s.arena(bo + 5), s.arena(bo), k.dw13, k.dw13_is_fp32, k.dw13_accumulate, k.expert_offsets, c.e_local,
                         k.max_rows, 2 * c.F, c.D, c.num_sms, c.status, stream);
  });
  // The closing barrier is unconditional (dist_moe/api.py:2580): peers may still be pulling grad_h3 out of this rank's
  // combine buffer, and the next call on this context overwrites it.
  s.barrier(DM_BWD_CLOSE, c.dispatch_pads, nullptr);
  s.step(DM_BWD_REDUCE, 1, [&] {
    return dm_scale_and_sum(c.dispatch, nullptr, 0, k.ids, k.ids_are_int64, k.grad_x, k.T, c.K, c.D, nullptr, nullptr, nullptr,
                            0, stream);
  });
  return s.rc;
}

// MXFP8 training on the device planner's placement: entry `i` of group `g` of an offset table names an operand in the arena.
namespace {
enum { kAQ, kBQ, kC, kASf, kBSf, kSrcX, kSrcY, kColQ, kColSf, kEntries };
inline const int64_t* at(const int64_t* table, int group, int entry) { return table + group * kEntries + entry; }
}  // namespace

extern "C" int dm_mxfp8_forward(const dm_layer_context* ctx, const dm_layer_call* call, uint32_t steps, int32_t* report,
                                void* stream) {
  if (!ctx || !call || !report) return -1;
  const dm_layer_context& c = *ctx;
  const dm_layer_call& k = *call;
  report[0] = report[1] = 0;
  Sequence s{c, steps, report, stream};
  const int64_t stride = c.D * 2;
  int64_t *fs = k.fwd_state, *ft = k.fwd_table;
  const int route_launches = DM_ROUTE_LAUNCHES(c.ep, k.T, c.e_local, dm_route_decode_kernel_enabled());
  s.step(DM_FWD_PUBLISH, 1, [&] {
    return dm_publish(k.x, k.ids, k.ids_are_int64, c.dispatch, c.routing, k.T, c.D, c.K, c.E, k.validate_ids, c.status, stream);
  });
  s.barrier(DM_FWD_PUBLISH, c.dispatch_pads, nullptr);
  s.step(DM_FWD_ROUTE, route_launches, [&] {
    return dm_route_counted(c.routing_ptrs, c.dispatch_ptrs, c.combine_ptrs, c.rank, c.ep, k.T, c.K, c.E, stride, stride,
                            stride, 128, c.capacity_rows, k.ptrs_size, k.counts, k.real_counts, k.per_rank, k.expert_offsets,
                            k.fwd_ptrs, k.bwd_ptrs, k.sct_ptrs, c.route_workspace, c.route_workspace_words, c.status, stream);
  });
  const int32_t* recv = k.expert_offsets + c.e_local;
  s.step(DM_FWD_ROUTE, 1, [&] {
    return dm_plan_fwd_blockscaled(recv, k.per_rank, nullptr, c.saved_bytes, c.buffer_offsets, c.peak_min_free, k.need, k.cond,
                                   fs, ft, c.slot_selector, c.moe_layer_id, c.ep, c.T_max, c.K, c.D, c.F, c.storage,
                                   c.capacity_rows, c.slot_bytes, c.num_slots, k.num_layers, 0, 0, DM_PLAN_BOUNDED, 0, 0,
                                   c.status, stream);
  });
  // a layer that will be recomputed keeps only its dense input
  s.step(DM_FWD_SAVE_X, 1, [&] { return dm_cond_copy(k.x, nullptr, c.arena, fs, k.T * c.D * 2, k.cond, 1, stream); });
  // dispatch: the routed rows are pulled through the pointer table by the quantiser itself
  s.step(DM_FWD_W13, 1, [&] {
    return dm_quant_mxfp8_rowcol_gather_at(k.fwd_ptrs, recv, k.max_rows, c.D, s.arena(at(ft, 0, kAQ)), s.arena(at(ft, 0, kASf)),
                                           s.arena(at(ft, 0, kColQ)), s.arena(at(ft, 0, kColSf)), nullptr, stream);
  });
  s.step(DM_FWD_W13, 1, [&] {
    return dm_gemm_blockscaled_counted(0, s.arena(at(ft, 0, kAQ)), s.arena(at(ft, 0, kASf)), k.w13, k.w13_sf,
                                       s.arena(at(ft, 0, kC)), kNone, nullptr, kNone, nullptr, k.expert_offsets, k.real_counts,
                                       c.e_local, k.max_rows, 2 * c.F, c.D, 0, 0, 1.0f, 0.0f, nullptr, c.num_sms, c.status,
                                       stream);
  });
  s.step(DM_FWD_SWIGLU, 1, [&] {
    return dm_swiglu_fwd_quant_mxfp8_rowcol_at(s.arena(at(ft, 1, kSrcX)), recv, k.max_rows, c.F, c.clamped, c.alpha, c.limit,
                                               s.arena(at(ft, 1, kAQ)), s.arena(at(ft, 1, kASf)), s.arena(at(ft, 1, kColQ)),
                                               s.arena(at(ft, 1, kColSf)), nullptr, stream);
  });
  s.step(DM_FWD_W2, 1, [&] {
    return dm_gemm_blockscaled_counted(0, s.arena(at(ft, 1, kAQ)), s.arena(at(ft, 1, kASf)), k.w2, k.w2_sf, kNone, kNone,
                                       k.sct_ptrs, kNone, nullptr, k.expert_offsets, k.real_counts, c.e_local, k.max_rows, c.D,
                                       c.F, 0, 0, 1.0f, 0.0f, nullptr, c.num_sms, c.status, stream);
  });
  s.barrier(DM_FWD_COMBINE, c.combine_pads, nullptr);
  // the expert outputs go to the slot (when the layer is saved) only if the score gradient will read them
  s.step(DM_FWD_REDUCE, 1, [&] {
    return dm_scale_and_sum(c.combine, k.scores, k.scores_are_bf16, k.ids, k.ids_are_int64, k.out, k.T, c.K, c.D,
                            k.keep_h3 ? c.arena : nullptr, k.keep_h3 ? fs + 4 : nullptr, k.keep_h3 ? k.cond : nullptr, 0,
                            stream);
  });
  return s.rc;
}

extern "C" int dm_mxfp8_backward(const dm_layer_context* ctx, const dm_layer_call* call, uint32_t steps, int32_t* report,
                                 void* stream) {
  if (!ctx || !call || !report) return -1;
  const dm_layer_context& c = *ctx;
  const dm_layer_call& k = *call;
  report[0] = report[1] = 0;
  Sequence s{c, steps, report, stream};
  const int64_t* fs = k.fwd_state;
  int64_t* bt = k.bwd_table;
  const int32_t* recv = k.expert_offsets + c.e_local;
  auto A = [&](int group, int entry) { return s.arena(at(bt, group, entry)); };
  s.step(DM_BWD_PLAN, 1, [&] {
    return dm_plan_bwd_blockscaled(recv, k.per_rank, c.saved_bytes, c.buffer_offsets, c.peak_min_free, k.need, fs, k.bwd_offsets,
                                   bt, c.moe_layer_id, c.ep, c.T_max, c.K, c.D, c.F, c.storage, c.capacity_rows, c.slot_bytes,
                                   c.num_slots, 0, 0, c.status, stream);
  });
  // ---- recompute block: every launch is a no-op unless the forward chose to recompute this layer ---------------------
  s.step(DM_BWD_REPUBLISH, 1, [&] {
    return dm_cond_copy(c.arena, fs, c.dispatch, nullptr, k.T * c.D * 2, k.cond, 1, stream);
  });
  s.barrier(DM_BWD_REPUBLISH, c.dispatch_pads, k.cond);
  s.step(DM_BWD_W13_AGAIN, 1, [&] {
    return dm_quant_mxfp8_rowcol_gather_at(k.fwd_ptrs, recv, k.max_rows, c.D, A(0, kAQ), A(0, kASf), A(0, kColQ), A(0, kColSf),
                                           k.cond, stream);
  });
  s.step(DM_BWD_W13_AGAIN, 1, [&] {
    return dm_gemm_blockscaled_counted(0, A(0, kAQ), A(0, kASf), k.w13, k.w13_sf, A(0, kC), kNone, nullptr, kNone, nullptr,
                                       k.expert_offsets, k.real_counts, c.e_local, k.max_rows, 2 * c.F, c.D, 0, 0, 1.0f, 0.0f,
                                       k.cond, c.num_sms, c.status, stream);
  });
  s.step(DM_BWD_SWIGLU_AGAIN, 1, [&] {
    return dm_swiglu_fwd_quant_mxfp8_rowcol_at(A(1, kSrcX), recv, k.max_rows, c.F, c.clamped, c.alpha, c.limit, A(1, kAQ),
                                               A(1, kASf), A(1, kColQ), A(1, kColSf), k.cond, stream);
  });
  s.step(DM_BWD_W2_AGAIN, 1, [&] {  // the expert outputs again, scattered to their owners' combine buffers
    return dm_gemm_blockscaled_counted(0, A(1, kAQ), A(1, kASf), k.w2, k.w2_sf, kNone, kNone, k.sct_ptrs, kNone, nullptr,
                                       k.expert_offsets, k.real_counts, c.e_local, k.max_rows, c.D, c.F, 0, 0, 1.0f, 0.0f,
                                       k.cond, c.num_sms, c.status, stream);
  });
  s.barrier(DM_BWD_W2_AGAIN, c.combine_pads, k.cond);
  s.step(DM_BWD_LOAD_H3, 1, [&] {
    return dm_cond_copy(c.arena, fs + 4, c.combine, nullptr, k.T * c.K * c.D * 2, k.cond, 0, stream);
  });
  // ---- gradient of the expert outputs and the scores -------------------------------------------------------------
  s.step(DM_BWD_GRAD_H3, 1, [&] {
    if (k.grad_scores != nullptr)
      return dm_broadcast_and_scale_select(k.grad_out, k.scores, k.scores_are_bf16, k.ids, k.ids_are_int64, c.arena, fs + 4,
                                           c.combine, k.cond, c.combine, k.grad_scores, k.T, c.K, c.D, stream);
    return dm_broadcast_and_scale(k.grad_out, k.scores, k.scores_are_bf16, k.ids, k.ids_are_int64, nullptr, nullptr, c.combine,
                                  nullptr, k.T, c.K, c.D, stream);
  });
  s.barrier(DM_BWD_COMBINE, c.combine_pads, nullptr);
  // ---- W2 -----------------------------------------------------------------------------------------------------------
  s.step(DM_BWD_W2_DGRAD, 1, [&] {
    return dm_quant_mxfp8_rowcol_gather_at(k.sct_ptrs, recv, k.max_rows, c.D, A(2, kAQ), A(2, kASf),
                                           k.want_w2 ? A(2, kColQ) : kNone, k.want_w2 ? A(2, kColSf) : kNone, nullptr, stream);
  });
  s.step(DM_BWD_W2_DGRAD, 1, [&] {
    return dm_gemm_blockscaled_dgrad_counted(A(2, kAQ), A(2, kASf), k.w2, k.w2_dgrad_sf, A(2, kC), nullptr, k.expert_offsets,
                                             k.real_counts, c.e_local, k.max_rows, c.F, c.D, nullptr, c.num_sms, c.status,
                                             stream);
  });
  s.step(DM_BWD_W2_WGRAD, 1, [&] {
    return dm_gemm_blockscaled_wgrad_compact(A(3, kAQ), A(3, kASf), A(3, kBQ), A(3, kBSf), k.dw2, k.dw2_is_fp32,
                                             k.dw2_accumulate, k.expert_offsets, c.e_local, k.max_rows, c.D, c.F, nullptr,
                                             c.num_sms, c.status, stream);
  });
  // ---- SwiGLU backward, W13 -----------------------------------------------------------------------------------------
  s.step(DM_BWD_SWIGLU, 1, [&] {
    return dm_swiglu_bwd_quant_mxfp8_at(A(4, kSrcY), A(4, kSrcX), recv, k.max_rows, c.F, c.clamped, c.alpha, c.limit,
                                        k.want_x ? A(4, kAQ) : kNone, k.want_x ? A(4, kASf) : kNone,
                                        k.want_w13 ? A(4, kColQ) : kNone, k.want_w13 ? A(4, kColSf) : kNone, stream);
  });
  s.step(DM_BWD_W13_DGRAD, 1, [&] {
    return dm_gemm_blockscaled_dgrad_counted(A(4, kAQ), A(4, kASf), k.w13, k.w13_dgrad_sf, kNone, k.bwd_ptrs, k.expert_offsets,
                                             k.real_counts, c.e_local, k.max_rows, c.D, 2 * c.F, nullptr, c.num_sms, c.status,
                                             stream);
  });
  s.step(DM_BWD_W13_WGRAD, 1, [&] {
    return dm_gemm_blockscaled_wgrad_compact(A(5, kAQ), A(5, kASf), A(5, kBQ), A(5, kBSf), k.dw13, k.dw13_is_fp32,
                                             k.dw13_accumulate, k.expert_offsets, c.e_local, k.max_rows, 2 * c.F, c.D, nullptr,
                                             c.num_sms, c.status, stream);
  });
  // unconditional, as in the reference (dist_moe/api.py:2580): peers may still be reading this rank's combine buffer
  s.barrier(DM_BWD_CLOSE, c.dispatch_pads, nullptr);
  s.step(DM_BWD_REDUCE, 1, [&] {
    return dm_scale_and_sum(c.dispatch, nullptr, 0, k.ids, k.ids_are_int64, k.grad_x, k.T, c.K, c.D, nullptr, nullptr, nullptr,
                            0, stream);
  });
  return s.rc;
}
