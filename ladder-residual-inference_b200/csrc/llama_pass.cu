// The layers of one forward pass of a Llama-shaped model on one GPU, launched from native code: the order of kernels that
// gpt_fast/engine.py documents for its schedules (dense, ladder, ladder on two streams, parallel, desync with nothing to reduce).
//
// A decode step of a small model is a chain of 2 to 4 us kernels; called one by one from Python each costs 8 us of host time (stories110M,
// 125 launches: 1004 us a step for 290 us of device time).  One call per pass leaves the launches themselves.  Nothing is kept between
// calls: every pointer comes from the caller, who reads it from the model's tensors for this pass.
#include "linear.cuh"

using namespace lri;

namespace {

enum LayerPointer { kAttentionNorm, kQkv, kWo, kMlpNorm, kW1, kW2, kKCache, kVCache, kPointers };

struct Pass {
  const lri_llama_pass& p;
  int64_t rows;
  void* row_ws;
  int rc = LRI_OK;
  Share share{};  // see early() and where two streams run

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
    return ok(lri::qkv_rope_kvcache(p.dtype, p.normed, at(l, kQkv), p.rope_table, p.input_pos, p.pos_is_i64, p.q, kc, vc, p.B, p.S, p.dim, p.n_head,
                                   p.n_kv, p.head_dim, p.smax, p.table_rows, 0, p.ws_qkv, p.ws_qkv_bytes, share, p.stream)) &&
           attend(l);
  }
  // from the queries and the caches to the output projection
  bool attend(int l) {
    void *kc = const_cast<void*>(at(l, kKCache)), *vc = const_cast<void*>(at(l, kVCache));
    const bool done =
        p.S == 1 ? ok(lri_attn_decode(p.dtype, p.q, kc, vc, p.input_pos, p.pos_is_i64, p.y, p.B, p.n_head, p.n_kv, p.head_dim, p.smax, p.splits,
                                      p.scratch, p.scratch_bytes, p.stream))
                 : ok(lri_attn_prefill(p.dtype, p.q, kc, vc, p.input_pos, p.pos_is_i64, p.y, p.B, p.S, p.n_head, p.n_kv, p.head_dim, p.smax, p.stream));
    return done && ok(lri::linear(p.dtype, p.y, at(l, kWo), nullptr, p.part_a, rows, p.dim, p.n_head * p.head_dim, p.ws_wo, p.ws_wo_bytes, share, p.stream));
  }
  bool mlp(int l, const void* normed, const void* addend, lri_stream_t st) {
    return ok(lri::gateup_swiglu(p.dtype, normed, at(l, kW1), p.h, rows, p.inter, p.dim, p.ws_ug, p.ws_ug_bytes, share, st)) &&
           ok(lri::linear(p.dtype, p.h, at(l, kW2), addend, p.part_m, rows, p.dim, p.inter, p.ws_w2, p.ws_w2_bytes, share, st));
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
    // Half of the ring for each (gemm_streamk.cu), but not in wide models where attention over a long cache is what runs beside 9 to 16 rows.  8B, us a
    // captured step, whole / half: 9 sequences at 1000, 2000, 4000 positions 2967 / 2924, 3200 / 3202, 3648 / 3679; 12 2983 / 2961, 3234 / 3254, 3728 / 3818;
    // 16 3054 / 3012, 3364 / 3394, 3983 / 4055; but 8 at 7000 3778 / 3738, 24 at 2600 4193 / 4184, 64 at 900 4648 / 4565; 1B, 16 at 1900 852 / 819.  The
    // position is not known here, the cache's length is.
    share = {false, !(p.dim >= 4096 && rows > 8 && rows <= 16 && p.smax > 1600)};
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

  // the gate/up projection beside the attention chain: both read the norm
  bool parallel_two_streams() {
    const void* pending = nullptr;
    // us a captured step, whole / half ring.  8B: 16, 32 sequences 3251 / 3176, 3488 / 3400, but 33, 40, 48, 64 3542 / 3609, 3777 / 3851, 3848 / 3950, 4025 /
    // 4120; 3B: 2, 4 1677 / 1779, 1785 / 1903, 9, 40, 48 1842 / 1785, 2712 / 2702, 2798 / 2797, 64 3241 / 3258; 1B: 9, 16, 32 787 / 756, 795 / 777, 869 / 845,
    // 48, 64 943 / 944, 1048 / 1056, but called eagerly 1173 / 1118 (on another machine 1162 / 1152).
    share = {false, rows > 8 && rows <= (p.dim >= 4096 ? 32 : p.dim > 2048 ? 48 : kSplitKMaxRows)};
    for (int l = 0; l < p.n_layer; ++l) {
      if (!norm(at(l, kAttentionNorm), pending, nullptr, true, p.normed, p.stream) || !record(2 * l, p.stream) || !wait(2 * l, p.side)) return false;
      if (!attention(l) ||
          !ok(lri::gateup_swiglu(p.dtype, p.normed, at(l, kW1), p.h, rows, p.inter, p.dim, p.ws_ug, p.ws_ug_bytes, share, p.side)) ||
          !record(2 * l + 1, p.side) || !wait(2 * l + 1, p.stream) ||
          !ok(lri::linear(p.dtype, p.h, at(l, kW2), p.part_a, p.part_m, rows, p.dim, p.inter, p.ws_w2, p.ws_w2_bytes, share, p.stream)))
        return false;
      pending = p.part_m;
    }
    return norm(p.final_norm, pending, nullptr, false, p.normed, p.stream);
  }

  // ---- one row, called eagerly: norms taken by the projections behind them ----------------------------------------
  // Small models called eagerly are bound by the host, 2.3 us a launch: five launches a layer instead of seven take 49 of the 195 us that the
  // launches of a stories110M step take (step 302 -> 250 us).  On the device the chain gets no shorter, because each of a projection's CTAs
  // works out the norm after the wait (captured: 196 us with kernels for the norms, 209 without; Ladder-Llama 1B 457 and 623).  So captured
  // steps and wider models keep them.  The results are the same bits.
  const void* cur = nullptr;  // the residual, and where the next sum goes: every CTA of a projection reads the one, so it is not written
  void* other = nullptr;
  bool folds() const { return option(OPT_FOLD_NORM) && p.n_layer > 0 && row_ws && rows == 1 && gemv_norm_supports(1, p.dim) && eager(); }
  bool eager() const {
    cudaStreamCaptureStatus status;
    return cudaStreamIsCapturing(static_cast<cudaStream_t>(p.stream), &status) == cudaSuccess && status == cudaStreamCaptureStatusNone;
  }
  // One stream: where the kernels behind small-batch projections come early (gemm_streamk.cu).  us, late / early.
  // Captured steps: 8B dense, 9, 16, 20 sequences 3272 / 3218, 3359 / 3277, 3491 / 3420, 24 the same (0.989 to 1.013 in three comparisons), but 28, 40, 64
  // 3569 / 3596, 3900 / 3961, 4133 / 4177; 3B dense, 16, 24, 28 2179 / 2167, 2367 / 2338, 2536 / 2513, but 32, 48, 64 2539 / 2560, 2971 / 3007, 3475 / 3511; narrower models at any
  // number: 1B 16, 32, 64 902 / 833, 963 / 910, 1136 / 1127, stories110M 371 / 351, 409 / 394, 576 / 558.
  // Eager passes lose by it: 8B dense, 16 and 64 sequences 3402 / 3477, 4293 / 4389, a prompt of 16 tokens 3414 / 3466; 3B 2269 / 2348, 3555 / 3601,
  // 2081 / 2116; 1B 896 / 917, 1174 / 1227, 896 / 922; stories110M 404 / 425, 603 / 625, 407 / 417.  But not short prompts through parallel blocks: 3B,
  // 9, 16, 32 tokens 2027 / 1998, 2055 / 2033, 2167 / 2181; 8B 3338 / 3297, 3379 / 3373, 3573 / 3605; 1B, 9, 16, 32, 64 890 / 870, 895 / 884, 943 / 922,
  // 1061 / 1054.
  bool early() const {
    if (eager()) return p.schedule == LRI_PARALLEL && p.S > 1 && rows <= (p.dim > 2048 ? 16 : kSplitKMaxRows);
    return rows <= (p.dim >= 4096 ? 24 : p.dim > 2048 ? 28 : kSplitKMaxRows);
  }
  bool folded_qkv(int l, const void* add1, bool write) {
    void *kc = const_cast<void*>(at(l, kKCache)), *vc = const_cast<void*>(at(l, kVCache));
    const NormArgs nm{cur, add1, nullptr, at(l, kAttentionNorm), write ? other : nullptr, p.eps};
    return ok(norm_qkv_rope_kvcache(p.dtype, nm, at(l, kQkv), p.rope_table, p.input_pos, p.pos_is_i64, p.q, kc, vc, p.dim, p.n_head, p.n_kv,
                                    p.head_dim, p.smax, p.table_rows, static_cast<cudaStream_t>(p.stream)));
  }
  bool folded_up(int l, const void* add1, const void* add2, bool write) {
    const NormArgs nm{cur, add1, add2, at(l, kMlpNorm), write ? other : nullptr, p.eps};
    return ok(norm_gateup_swiglu(p.dtype, nm, at(l, kW1), p.h, p.inter, p.dim, static_cast<cudaStream_t>(p.stream)));
  }
  bool down(int l, const void* addend) {
    return ok(lri_linear(p.dtype, p.h, at(l, kW2), addend, p.part_m, rows, p.dim, p.inter, p.ws_w2, p.ws_w2_bytes, p.stream));
  }
  void written() {
    void* was = const_cast<void*>(cur);
    cur = other, other = was;
  }
  bool last_norm(const void* add1, const void* add2) {
    return ok(lri_add_rmsnorm(p.dtype, cur, add1, add2, 1.0f, p.final_norm, p.eps, nullptr, p.normed, rows, p.dim, p.stream));
  }
  bool folded_dense() {
    const void* pending = nullptr;
    for (int l = 0; l < p.n_layer; ++l) {
      if (!folded_qkv(l, pending, pending)) return false;
      if (pending) written();
      if (!attend(l) || !folded_up(l, p.part_a, nullptr, true)) return false;
      written();
      if (!down(l, nullptr)) return false;
      pending = p.part_m;
    }
    return last_norm(pending, nullptr);
  }
  // both sublayers start from the residual before the layer; the MLP's projection adds the results of the layer before and writes the sum
  bool folded_ladder() {
    for (int l = 0; l < p.n_layer; ++l) {
      const void *add1 = l ? p.part_a : nullptr, *add2 = l ? p.part_m : nullptr;
      if (!folded_qkv(l, add1, false) || !folded_up(l, add1, add2, l > 0)) return false;
      if (l) written();
      if (!attend(l) || !down(l, nullptr)) return false;
    }
    return last_norm(p.part_a, p.part_m);
  }
  bool folded_parallel() {
    const void* pending = nullptr;
    for (int l = 0; l < p.n_layer; ++l) {
      if (!folded_qkv(l, pending, false) || !attend(l) || !folded_up(l, pending, nullptr, pending != nullptr)) return false;
      if (pending) written();
      if (!down(l, p.part_a)) return false;
      pending = p.part_m;
    }
    return last_norm(pending, nullptr);
  }
};

}  // namespace

extern "C" int lri_llama_run(const lri_llama_pass* pass) { return lri_llama_run_row(pass, nullptr); }

extern "C" int lri_llama_run_row(const lri_llama_pass* pass, void* row_ws) {
  LRI_REQUIRE(pass != nullptr && pass->layers != nullptr, LRI_ERR_ARG, "llama_pass: NULL pointer");
  LRI_REQUIRE(pass->n_layer >= 0 && pass->B >= 0 && pass->S >= 0, LRI_ERR_ARG, "llama_pass: n_layer=%d B=%d S=%d", pass->n_layer, pass->B, pass->S);
  LRI_REQUIRE(pass->schedule != LRI_LADDER_TWO_STREAMS || (pass->events != nullptr && pass->normed_m != nullptr), LRI_ERR_ARG,
              "llama_pass: two streams need events and a second buffer");
  LRI_REQUIRE(pass->schedule != LRI_PARALLEL_TWO_STREAMS || (pass->events != nullptr && pass->side != nullptr), LRI_ERR_ARG,
              "llama_pass: two streams need events and a second stream");
  LRI_REQUIRE(pass->schedule != LRI_DESYNC || pass->reduces != nullptr, LRI_ERR_ARG, "llama_pass: NULL flags");
  Pass run{*pass, static_cast<int64_t>(pass->B) * pass->S, row_ws};
  if (run.folds()) {
    run.cur = pass->resid, run.other = row_ws;
    switch (pass->schedule) {
      case LRI_DENSE:
      case LRI_DESYNC: run.folded_dense(); return run.rc;
      case LRI_LADDER:
      case LRI_LADDER_TWO_STREAMS: run.folded_ladder(); return run.rc;
      case LRI_PARALLEL:
      case LRI_PARALLEL_TWO_STREAMS: run.folded_parallel(); return run.rc;
    }
  }
  run.share.early = run.rows > 8 && run.early();  // (few rows: see gemm_streamk.cu)
  // From 129 rows on (or 65, where the option forces it) the projections of two streams would run on pairs of SMs beside each other, which is not
  // done (gemm_pair.cu): such a pass runs on one stream, with the same results.
  const bool two = run.rows <= (option(OPT_GEMM_PAIR) > 1 ? kSplitKMaxRows : 128);
  switch (pass->schedule) {
    case LRI_DENSE:
    // on one GPU a partial that is reduced at once and one that is added by the next norm are the same sums
    case LRI_DESYNC: run.dense(); break;
    case LRI_LADDER: run.ladder(); break;
    case LRI_LADDER_TWO_STREAMS: two ? run.ladder_two_streams() : run.ladder(); break;
    case LRI_PARALLEL: run.parallel(); break;
    case LRI_PARALLEL_TWO_STREAMS: two ? run.parallel_two_streams() : run.parallel(); break;
    default: return fail(LRI_ERR_ARG, "llama_pass: schedule %d", pass->schedule);
  }
  return run.rc;
}
