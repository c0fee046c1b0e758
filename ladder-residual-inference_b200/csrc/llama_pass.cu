// The layers of one forward pass of a Llama-shaped model on one GPU, launched from native code: the order of kernels that
// gpt_fast/engine.py documents for its schedules (dense, ladder, ladder on two streams, parallel, desync with nothing to reduce).
//
// A decode step of a small model is a chain of 2 to 4 us kernels; called one by one from Python each costs 8 us of host time (stories110M,
// 125 launches: 1004 us a step for 290 us of device time).  One call per pass leaves the launches themselves.  Nothing is kept between
// calls: every pointer comes from the caller, who reads it from the model's tensors for this pass.
#include "common.cuh"

using namespace lri;

namespace {

enum LayerPointer { kAttentionNorm, kQkv, kWo, kMlpNorm, kW1, kW2, kKCache, kVCache, kPointers };

struct Pass {
  const lri_llama_pass& p;
  int64_t rows;
  int rc = LRI_OK;

  const void* at(int layer, int which) const { return p.layers[static_cast<int64_t>(layer) * kPointers + which]; }
  bool ok(int r) { return (rc = r) == LRI_OK; }
  bool cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    rc = fail(LRI_ERR_CUDA, "llama_pass: %s failed: %s", what, cudaGetErrorString(e));
    return false;
  }
  // residual += adds (in place), normed = RMSNorm(residual) * weight
  bool norm(const void* weight, const void* add1, const void* add2, bool write, void* normed, lri_stream_t st) {
    void* res_out = write && (add1 || add2) ? p.resid : nullptr;
    return ok(lri_add_rmsnorm(p.dtype, p.resid, add1, add2, 1.0f, weight, p.eps, res_out, normed, rows, p.dim, st));
  }
  bool attention(int l) {
    void *kc = const_cast<void*>(at(l, kKCache)), *vc = const_cast<void*>(at(l, kVCache));
    if (!ok(lri_qkv_rope_kvcache(p.dtype, p.normed, at(l, kQkv), p.rope_table, p.input_pos, p.pos_is_i64, p.q, kc, vc, p.B, p.S, p.dim, p.n_head,
                                 p.n_kv, p.head_dim, p.smax, p.table_rows, 0, p.ws_qkv, p.ws_qkv_bytes, p.stream)))
      return false;
    const bool done =
        p.S == 1 ? ok(lri_attn_decode(p.dtype, p.q, kc, vc, p.input_pos, p.pos_is_i64, p.y, p.B, p.n_head, p.n_kv, p.head_dim, p.smax, p.splits,
                                      p.scratch, p.scratch_bytes, p.stream))
                 : ok(lri_attn_prefill(p.dtype, p.q, kc, vc, p.input_pos, p.pos_is_i64, p.y, p.B, p.S, p.n_head, p.n_kv, p.head_dim, p.smax, p.stream));
    return done && ok(lri_linear(p.dtype, p.y, at(l, kWo), nullptr, p.part_a, rows, p.dim, p.n_head * p.head_dim, p.ws_wo, p.ws_wo_bytes, p.stream));
  }
  bool mlp(int l, const void* normed, const void* addend, lri_stream_t st) {
    return ok(lri_gateup_swiglu(p.dtype, normed, at(l, kW1), p.h, rows, p.inter, p.dim, p.ws_ug, p.ws_ug_bytes, st)) &&
           ok(lri_linear(p.dtype, p.h, at(l, kW2), addend, p.part_m, rows, p.dim, p.inter, p.ws_w2, p.ws_w2_bytes, st));
  }
  bool record(int i, lri_stream_t st) {
    return cuda(cudaEventRecord(static_cast<cudaEvent_t>(p.events[i]), static_cast<cudaStream_t>(st)), "cudaEventRecord");
  }
  bool wait(int i, lri_stream_t st) {
    return cuda(cudaStreamWaitEvent(static_cast<cudaStream_t>(st), static_cast<cudaEvent_t>(p.events[i]), 0), "cudaStreamWaitEvent");
  }

  bool dense() {
    const void* pending = nullptr;
    for (int l = 0; l < p.n_layer; ++l) {
      if (!norm(at(l, kAttentionNorm), pending, nullptr, true, p.normed, p.stream) || !attention(l)) return false;
      if (!norm(at(l, kMlpNorm), p.part_a, nullptr, true, p.normed, p.stream) || !mlp(l, p.normed, nullptr, p.stream)) return false;
      pending = p.part_m;
    }
    return norm(p.final_norm, pending, nullptr, false, p.normed, p.stream);
  }
  bool ladder() {
    for (int l = 0; l < p.n_layer; ++l) {
      if (!norm(at(l, kAttentionNorm), l ? p.part_a : nullptr, nullptr, true, p.normed, p.stream) || !attention(l)) return false;
      if (!norm(at(l, kMlpNorm), l ? p.part_m : nullptr, nullptr, true, p.normed, p.stream) || !mlp(l, p.normed, nullptr, p.stream)) return false;
    }
    return norm(p.final_norm, p.part_a, p.part_m, false, p.normed, p.stream);
  }
  // the attention chain of a layer on `stream`, its MLP chain on `side`: see Engine._run_ladder_two_streams
  bool ladder_two_streams() {
    if (!record(0, p.stream) || !wait(0, p.side)) return false;
    int n = 1;
    for (int l = 0; l < p.n_layer; ++l, n += 2) {
      if (!norm(at(l, kAttentionNorm), l ? p.part_a : nullptr, nullptr, true, p.normed, p.stream) || !record(n, p.stream) || !attention(l)) return false;
      if (!wait(n, p.side) || !norm(at(l, kMlpNorm), l ? p.part_m : nullptr, nullptr, true, p.normed_m, p.side) || !record(n + 1, p.side) ||
          !mlp(l, p.normed_m, nullptr, p.side) || !wait(n + 1, p.stream))
        return false;
    }
    return record(n, p.side) && wait(n, p.stream) && norm(p.final_norm, p.part_a, p.part_m, false, p.normed, p.stream);
  }
  bool parallel() {
    const void* pending = nullptr;
    for (int l = 0; l < p.n_layer; ++l) {
      if (!norm(at(l, kAttentionNorm), pending, nullptr, true, p.normed, p.stream) || !attention(l) || !mlp(l, p.normed, p.part_a, p.stream)) return false;
      pending = p.part_m;
    }
    return norm(p.final_norm, pending, nullptr, false, p.normed, p.stream);
  }
  // where a sublayer reduces, its partial is added to the residual first, and the sum (here: itself) is the new residual
  bool fold(const void* partial) {
    return ok(lri_add_rmsnorm(p.dtype, p.resid, partial, nullptr, 1.0f, nullptr, p.eps, p.resid, nullptr, rows, p.dim, p.stream));
  }
  bool desync() {
    const void* pending = nullptr;
    for (int l = 0; l < p.n_layer; ++l) {
      if (!norm(at(l, kAttentionNorm), pending, nullptr, true, p.normed, p.stream) || !attention(l)) return false;
      pending = p.part_a;
      if (p.reduces[2 * l]) {
        if (!fold(pending)) return false;
        pending = nullptr;
      }
      if (!norm(at(l, kMlpNorm), pending, nullptr, true, p.normed, p.stream) || !mlp(l, p.normed, nullptr, p.stream)) return false;
      pending = p.part_m;
      if (p.reduces[2 * l + 1]) {
        if (!fold(pending)) return false;
        pending = nullptr;
      }
    }
    return norm(p.final_norm, pending, nullptr, false, p.normed, p.stream);
  }
};

}  // namespace

extern "C" int lri_llama_run(const lri_llama_pass* pass) {
  LRI_REQUIRE(pass != nullptr && pass->layers != nullptr, LRI_ERR_ARG, "llama_pass: NULL pointer");
  LRI_REQUIRE(pass->n_layer >= 0 && pass->B >= 0 && pass->S >= 0, LRI_ERR_ARG, "llama_pass: n_layer=%d B=%d S=%d", pass->n_layer, pass->B, pass->S);
  LRI_REQUIRE(pass->schedule != LRI_LADDER_TWO_STREAMS || (pass->events != nullptr && pass->normed_m != nullptr), LRI_ERR_ARG,
              "llama_pass: two streams need events and a second buffer");
  LRI_REQUIRE(pass->schedule != LRI_DESYNC || pass->reduces != nullptr, LRI_ERR_ARG, "llama_pass: NULL flags");
  Pass run{*pass, static_cast<int64_t>(pass->B) * pass->S};
  switch (pass->schedule) {
    case LRI_DENSE: run.dense(); break;
    case LRI_LADDER: run.ladder(); break;
    case LRI_LADDER_TWO_STREAMS: run.ladder_two_streams(); break;
    case LRI_PARALLEL: run.parallel(); break;
    case LRI_DESYNC: run.desync(); break;
    default: return fail(LRI_ERR_ARG, "llama_pass: schedule %d", pass->schedule);
  }
  return run.rc;
}
