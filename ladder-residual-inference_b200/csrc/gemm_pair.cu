// tcgen05 GEMM on pairs of SMs (cta_group::2):  C[m, n] = sum_k A[m, k] * W[n, k], both operands K-major.
//
// A cluster of two CTAs works through output tiles of 256 tokens x bn outputs.  Each CTA fetches its own 128 tokens and its
// own half of the tile's weight rows into its shared memory; one instruction, issued by the first CTA, multiplies 256 x bn x 16
// and leaves 128 rows of the result in the tensor memory of each.
//
// What bounds a 128 x 256 x 64 step of the single-CTA kernel (gemm_tcgen05.cu) beside the tensor pipe's 512 cycles is moving 48 KB
// into shared memory and 48 KB out of it.  Here a step of the same work per SM moves 32 KB each way, because the two halves of
// the weight tile are read once per pair.  Measured on B200, 4096 x 28672 x 4096, operands zero (the clock stays at 1965 MHz): 726 cycles a
// step there, 563 here (2100 TFLOP/s); random operands, where the 1000 W cap sets the clock, 2048 x 28672 x 4096: 394 -> 363 us,
// 16384 x 28672 x 4096: 3100 -> 2782 us, 999 x 2048 x 8192: 38.7 -> 29.4 us.
//
// Roles per CTA: warp 0 fetches (TMA, no multicast), warp 1 owns the tensor memory and, in the first CTA, issues the products,
// warps 2-5 store.  The first CTA's `full` barriers count the bytes of both CTAs' copies; commits free a stage, and hand over
// an accumulator, in both CTAs at once; the stores of both CTAs hand the accumulator back to the first.
// Every wait on an mbarrier is bounded (device status word, see lri_gemm_status).  Not bounded are the allocation of tensor memory, the
// cluster barriers and the wait for the preceding kernel.  The allocation is one operation of both CTAs, so each first waits until
// the other runs, and it finds the tensor memory of its SMs free: no tensor-memory kernel of this library fits on an SM beside
// kOwnSmem.  The barriers are reached by both CTAs in every case.
//
// Beside a tensor-memory kernel of another stream: prompt passes that ran the prompt attention of latent_attention_tc.cu on a second
// stream while products of one K step ran here stopped for good (the form that allocated before the other CTA was known to run).
// Whether that was the cause is not known, and the engines do not bring the two together: designs with side-by-side mixers
// ask for single SMs (LRI_ONE_SM).  Option gemm_pair = 0 does the same for a program that runs passes on several streams at a time.
#include "gemm_tile.cuh"

namespace lri {
namespace {

using namespace tc;

__device__ int g_pair_status = 0;

constexpr int kMaxStages = 8;
constexpr int kTile = kBM * kBK * 2;    // bytes of 128 operand rows
constexpr int kAccCols = 256;           // TMEM columns of one of the two accumulators
constexpr int kMaxBn = 256;
constexpr int kSmemLimit = 226 * 1024;  // of the 227 KB of an SM; the barriers take the rest
constexpr int kOwnSmem = 181 * 1024;    // the smallest other tensor-memory kernel (prompt attention, heads of 64) takes 49 KB

__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `bar` may lie in either CTA of the pair
__device__ __forceinline__ void tma_load_pair(uint32_t smem_dst, const CUtensorMap* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_pair_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void arrive_in_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

template <typename T, int EPI>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, T* __restrict__ c,
                 GemmShape shape, GemmGrid grid, int bn, uint32_t stages, const LinearParams lin) {
  constexpr bool kGlu = EPI == EPI_SWIGLU || EPI == EPI_GLU;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment; the same in both CTAs
  __shared__ uint64_t bars[2 * kMaxStages + 4];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // uniform for the compiler too
  const int lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int num_kt = (shape.k + kBK - 1) / kBK;
  const int half = bn >> 1;
  const uint32_t stage_bytes = static_cast<uint32_t>(kTile + half * kBK * 2);  // 128 token rows and bn / 2 weight rows

  const uint32_t full0 = smem_u32(&bars[0]);
  const uint32_t empty0 = smem_u32(&bars[kMaxStages]);
  const uint32_t acc_full0 = smem_u32(&bars[2 * kMaxStages]);       // products -> stores, one per accumulator
  const uint32_t acc_empty0 = smem_u32(&bars[2 * kMaxStages + 2]);  // stores -> products (first CTA)

  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (uint32_t s = 0; s < stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full0 + 8 * a, 1);
      mbar_init(acc_empty0 + 8 * a, 8);  // four warps of each CTA
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // the other CTA runs
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(2 * kAccCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();  // the barriers of both CTAs exist before either is used from the other
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
  pdl_wait();
  pdl_launch_dependents();
  const int items = grid.tiles_p * grid.tiles_q;

  // Fetching and issuing are serial work of one warp, and set the pace of a step unless they are short: a loop run by one lane, with
  // the place in the ring divided out, took 458 cycles for the barriers alone and 74 for each product.  So the loops are
  // warp-uniform (one elected lane issues), addresses and descriptors stay in uniform registers, and the place is counted.
  if (warp == 0) {
    const uint32_t full_first = in_cta(full0, 0);
    uint32_t s = 0, parity = 1;  // a fresh barrier passes a wait on parity 1, so the first round does not block
    bool ok = true;
    for (int item = pair; item < items && ok; item += pairs) {
      const WorkItem w = work_item(item, grid);
      // the weight rows of this CTA: half of the tile's, or all its up rows (first CTA) and all its gate rows (second)
      const int w_row = kGlu ? static_cast<int>(rank) * lin.n + w.tile_q * half : w.tile_q * bn + static_cast<int>(rank) * half;
      const int a_row = w.tile_p * 2 * kBM + static_cast<int>(rank) * kBM;
      for (int kt = 0; kt < num_kt; ++kt) {
        ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, parity, &abort_flag, 21, &g_pair_status));
        if (!ok) break;
        if (elect_one()) {
          // (the second CTA's bytes may arrive before this: the phase cannot end before the arrival counted here)
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * stage_bytes);
          const uint32_t dst = base + s * stage_bytes;
          tma_load_pair(dst, &tmap_a, full_first + 8 * s, kt * kBK, a_row);
          tma_load_pair(dst + kTile, &tmap_w, full_first + 8 * s, kt * kBK, w_row);
        }
        if (++s == stages) s = 0, parity ^= 1u;
      }
    }
    // the commits that free the last stages arrive in both CTAs: neither leaves before it has seen its own
    for (uint32_t left = 0; left < stages && ok; ++left) {
      ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, parity, &abort_flag, 25, &g_pair_status));
      if (++s == stages) s = 0, parity ^= 1u;
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // fp32 accumulate, A and B of type T, both K-major, M = 256, N = bn
      constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (kFmt << 7) | (kFmt << 10) | (static_cast<uint32_t>(bn >> 3) << 17) | (static_cast<uint32_t>(2 * kBM >> 4) << 24);
      uint32_t s = 0, parity = 0;
      bool ok = true;
      int it = 0;
      for (int item = pair; item < items && ok; item += pairs, ++it) {
        const uint32_t a = it & 1;
        const uint32_t use = static_cast<uint32_t>(it) >> 1;
        // the stores of both CTAs must have drained this accumulator (its first use does not block)
        ok = __all_sync(0xffffffffu, mbar_wait(acc_empty0 + 8 * a, (use & 1u) ^ 1u, &abort_flag, 24, &g_pair_status));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d_tmem = tmem_base + a * kAccCols;
        for (int kt = 0; kt < num_kt; ++kt) {
          ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, parity, &abort_flag, 22, &g_pair_status));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (elect_one()) {
            const uint64_t adesc = smem_desc_sw128(base + s * stage_bytes);
            const uint64_t wdesc = smem_desc_sw128(base + s * stage_bytes + kTile);
#pragma unroll
            for (int kk = 0; kk < kBK / kUmmaK; ++kk)
              umma_pair_f16(d_tmem, adesc + 2 * kk, wdesc + 2 * kk, idesc, (kt > 0 || kk > 0) ? 1u : 0u);
            umma_commit_pair(empty0 + 8 * s);  // both CTAs' stage is free once these products have read it
            if (kt == num_kt - 1) umma_commit_pair(acc_full0 + 8 * a);
          }
          __syncwarp();
          if (++s == stages) s = 0, parity ^= 1u;
        }
      }
    }
  } else {
    const int quarter = warp & 3;  // the TMEM lanes a warp may read are fixed by warp id mod 4
    const int i = quarter * 32 + lane;
    int it = 0;
    for (int item = pair; item < items; item += pairs, ++it) {
      const WorkItem w = work_item(item, grid);
      const uint32_t a = it & 1;
      const uint32_t use = static_cast<uint32_t>(it) >> 1;
      // the tcgen05.ld of the epilogue are warp-collective: the warp leaves together or not at all
      const bool ready = mbar_wait(acc_full0 + 8 * a, use & 1u, &abort_flag, 23, &g_pair_status);
      if (!__all_sync(0xffffffffu, ready)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tacc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * kAccCols;
      store_row<T, EPI>(lin, c, shape, static_cast<int64_t>(w.tile_p) * 2 * kBM + rank * kBM + i, w.tile_q, bn, tacc);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive_in_cluster(in_cta(acc_empty0 + 8 * a, 0));
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    // give copies that were already issued time to land before the pair's shared memory is released
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
  }
  __syncthreads();
  cluster_barrier();  // the products read both CTAs' shared memory, and the stores arrive on the first CTA's barriers
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * kAccCols) : "memory");
  }
}

// rounds of tiles that the busiest pair works through
int64_t waves(int64_t m, int64_t cols, int bn, int pairs) {
  const int64_t tiles = ((m + 2 * kBM - 1) / (2 * kBM)) * ((cols + bn - 1) / bn);
  return (tiles + pairs - 1) / pairs;
}

template <typename T, int EPI>
int launch(int dtype, const LinearParams& lin, int64_t m, int n_rows, int bn, cudaStream_t st) {
  constexpr bool kGlu = EPI == EPI_SWIGLU || EPI == EPI_GLU;
  CUtensorMap ta, tw;
  int rc = make_tmap(&ta, dtype, lin.x, m, lin.k, kBM);
  if (rc != LRI_OK) return rc;
  rc = make_tmap(&tw, dtype, lin.w, n_rows, lin.k, bn / 2);
  if (rc != LRI_OK) return rc;
  auto kern = gemm_pair_kernel<T, EPI>;
  static std::atomic<unsigned long long> attr_set{0};  // per template instantiation, one bit per device
  LRI_ONCE_PER_DEVICE(attr_set, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
  const int stage_bytes = kTile + bn / 2 * kBK * 2;
  int stages = (kSmemLimit - 1024) / stage_bytes;
  stages = stages > kMaxStages ? kMaxStages : stages;

  const int64_t tiles_p = (m + 2 * kBM - 1) / (2 * kBM);
  const int64_t tiles_q = kGlu ? (lin.n + bn / 2 - 1) / (bn / 2) : (n_rows + bn - 1) / bn;
  const int64_t items = tiles_p * tiles_q;
  if (items >= (1ll << 31)) return fail(LRI_ERR_UNSUPPORTED, "gemm: %lld output tiles", (long long)items);
  // panel of token tiles: about 32 MB of tokens, between 2 and 16 tiles (LRI_GEMM_GROUP, in tiles of 128 rows, overrides).
  // 16384 x 28672 x 4096: 3284 / 2960 / 2822 / 2782 us at 2 / 4 / 8 / 16 tiles; at k = 14336 no panel is 2 % from another.
  const int forced_group = option(OPT_GEMM_GROUP);
  int64_t group = (32ll << 20) / (4ll * kBM * lin.k);
  group = group < 2 ? 2 : (group > 16 ? 16 : group);
  if (forced_group > 0) group = (forced_group + 1) / 2;
  group = group > tiles_p ? tiles_p : group;
  GemmGrid grid{static_cast<int>(tiles_p), static_cast<int>(tiles_q), static_cast<int>(group), nullptr, 0};
  GemmShape shape{static_cast<int>(m), n_rows, lin.k};
  int usable = (sm_count() - option(OPT_GEMM_RESERVE_SMS)) / 2;
  usable = usable < 1 ? 1 : usable;
  const int64_t clusters = items < usable ? items : usable;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * clusters));
  cfg.blockDim = dim3(kGemmThreads);
  const int smem = stages * stage_bytes + 1024;
  cfg.dynamicSmemBytes = static_cast<size_t>(smem > kOwnSmem ? smem : kOwnSmem);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  LRI_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tw, static_cast<T*>(lin.y), shape, grid, bn, static_cast<uint32_t>(stages), lin));
  LRI_LAUNCH_CHECK("gemm_pair_kernel");
  return LRI_OK;
}

template <typename T>
int launch_epi(int dtype, int epi, const LinearParams& lin, int64_t m, int n_rows, int bn, cudaStream_t st) {
  switch (epi) {
    case EPI_SWIGLU: return launch<T, EPI_SWIGLU>(dtype, lin, m, n_rows, bn, st);
    case EPI_GLU: return launch<T, EPI_GLU>(dtype, lin, m, n_rows, bn, st);
    case EPI_QKV: return launch<T, EPI_QKV>(dtype, lin, m, n_rows, bn, st);
    case EPI_F32: return launch<T, EPI_F32>(dtype, lin, m, n_rows, bn, st);
    default: return launch<T, EPI_PLAIN>(dtype, lin, m, n_rows, bn, st);
  }
}

}  // namespace

// Up to 128 rows half of the pair's tile would be padding, and the single-CTA kernel is the better one (128 x 28672 x 4096: 47.1 us
// there, 52.4 here); above, this one (200 x 28672 x 4096: 66.9 there, 54.1 here).
// The width: a step costs about bn + 64 columns' worth (337, 382, 436, 505, 563 cycles at 128 .. 256 by 32), so the narrower tile
// wins where it fills the last round: 999 x 2048 x 8192 takes 29.4 us at 128 and 44.1 at 256, 2048 x 5120 x 2048 37.9 at 192 and 42.6 at
// 256, 2048 x 28672 x 4096 363 at 224 and at 256 and 405 at 128.
// Short sums: a launch costs about a microsecond more here.  Wide tiles do not make up for it below a depth of 512 (us, one SM a tile / here:
// 2048 x 4096 x 256 10.1 / 11.5, 4096 x 4096 x 384 19.6 / 21.5, 2048 x 4096 x 1024 17.6 / 16.9), narrow ones, which fill a last round, do
// (1000 x 3072 x 256 8.3 / 7.7).  One or two K steps stay with one SM in any case (2048 x 4096 x 128 9.4 / 10.6, 1000 x 3072 x 128 7.5 / 7.1): they are
// what ran when passes stopped, see the head of this file.
constexpr int kMinDepth = 2 * kBK, kMinWideDepth = 512, kWide = 224;

int gemm_pair_bn(int64_t m, int64_t cols, int k) {
  const int forced = option(OPT_GEMM_PAIR);
  if (forced == 0) return 0;
  if (forced > 1) return forced / 32 * 32;
  if (m <= kBM || k <= kMinDepth) return 0;
  const int pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  int best = kMaxBn;
  int64_t cost = 0;
  for (int bn = kMaxBn; bn >= 64; bn -= 32) {
    const int64_t c = waves(m, cols, bn, pairs) * (bn + 64);
    if (bn == kMaxBn || c < cost) best = bn, cost = c;
  }
  return best >= kWide && k < kMinWideDepth ? 0 : best;
}

// lin.x [m, k], lin.w [n_rows, k]; lin.n outputs where the epilogue counts them
int gemm_pair_launch(int dtype, int epi, const LinearParams& lin, int64_t m, int n_rows, int bn, cudaStream_t st) {
  return dtype == LRI_BF16 ? launch_epi<__nv_bfloat16>(dtype, epi, lin, m, n_rows, bn, st)
                           : launch_epi<__half>(dtype, epi, lin, m, n_rows, bn, st);
}

int gemm_pair_status_read_and_clear(int* status_out) {
  int v = 0;
  LRI_CUDA(cudaMemcpyFromSymbol(&v, g_pair_status, sizeof(int)));
  if (v != 0) {
    int zero = 0;
    LRI_CUDA(cudaMemcpyToSymbol(g_pair_status, &zero, sizeof(int)));
  }
  *status_out = v;
  return LRI_OK;
}

}  // namespace lri
