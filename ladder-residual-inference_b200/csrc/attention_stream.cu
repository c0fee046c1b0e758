// F3, several sequences: decode attention as a stream of cache rows, with the query heads of a KV head as the rows of tensor-core
// tiles.
//
// From some tens of (sequence, KV head) pairs on the K/V bytes of a layer are MBs to hundreds of MB and what counts is that every
// SM has copies in flight from the first microsecond to the last.  One warp fetches (TMA, 128-byte swizzle, a 64 KB ring of K and V
// tiles of 32 positions, each given back as soon as it has been read), four warps compute, two to a tile: S = Q K^T and O += P V as
// m16n8k16 products, online softmax per warp.  Two CTAs share an SM.  How the work is cut:
//   few pairs            a pair goes to a cluster of 2, 4 or 8 CTAs, which merge through distributed shared memory
//   up to 2 a SM         one CTA a pair
//   more                 the (pair, tile) units are numbered pair-major and dealt out in equal contiguous runs, so that no last round
//                        of CTAs is nearly empty; a pair that two CTAs share leaves its parts in scratch memory, and the later of
//                        them merges these.  Without scratch memory one CTA a pair.
//
// MASKED: key and value widths below HD, a window or chunk that bounds the visible positions from below, a sink in the
// denominator, row pitch and factor of the output.
// TWO_TERM: probabilities enter the product as the sum of two 16-bit numbers, where the kernel that smaller batches take keeps them in
// 32 bits (masked form, and plain below 128 pairs or without scratch memory): rounded once, they add an error of the size of the result's own
// rounding (8B, 2 sequences at 1025 positions, bf16: 1.98e-3 against 64 bits for 1.66e-3, which is the rounding alone).  The second product
// costs 2 to 4 % of a layer's attention: 16 pairs 7.3 -> 7.65 us, 64 pairs 10.2 -> 10.5, 120 pairs 14.6 -> 15.0.
//
// Bound by HBM, from some 100 MB on at 85 to 92 % of a plain copy's rate; below, by a chain of about 4.5 us (position, descriptors, first tile,
// merge).  Measured on B200, us a layer: 40 sequences x 24 heads of 128, 701 positions (344 MB) 58.0 (77 with one 4-warp CTA a pair), 16 sequences
// x 8 KV heads, 1025 positions (67 MB) 15.2 (20.5), 4000 positions 43.6; masked 16.6 (36.0 with dot products on the FMA pipe).  What a CTA
// gets is what it has in flight: tiles of 16 positions, held until both products were done, gave 34 bytes a ns to a CTA, this form 41 and
// more; scores computed a tile ahead hold two tiles and were slower (19.8 us for 15.2).

// Cache rows past the newest position may hold anything: their scores are masked, their values replaced by zeros.
#include <cooperative_groups.h>

#include "latent_attention.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace lri {
namespace {

using namespace tc;

__device__ int g_attn_stream_status = 0;

constexpr int kWarps = 4;                        // that compute
constexpr int kThreads = (kWarps + 1) * 32;      // and one that fetches
constexpr int kTile = 16;                        // positions of a warp's products
constexpr int kUnit = 32;                        // positions of a unit: one stage of the ring, two warps' tiles
constexpr int kTeams = kWarps * kTile / kUnit;   // warps that share a unit form a team
constexpr int kRingBytes = 64 * 1024;
constexpr int kMaxGroup = 16;                    // query heads of a KV head
constexpr int kMaxCluster = 8, kMaxGathered = 32;  // CTAs of a cluster, and times the heads of a group
constexpr int kMinCut = 16;                      // units; shorter pairs are not shared by CTAs
constexpr int kHintUnits = kRingBytes / (kUnit * 128 * 4);  // asked into the L2 ahead of time

struct StreamParams {
  const void *q, *k, *v;  // [B, n_head, dim], [pairs, smax, dim], [pairs, smax, vdim]
  const void* input_pos;
  int pos_is_i64;
  void* out;  // [B, n_head, vdim], row pitch out_ld
  int64_t out_ld;
  int pairs, n_head, n_kv, group;
  int64_t smax;
  float scale_log2;
  int cluster;             // CTAs that share a pair
  int slots;               // 2: pairs may be cut where a run ends
  unsigned int* counters;  // [pairs]
  float* part_ml;          // [pairs][slots][group][2]
  float* part_o;           // [pairs][slots][group][HD]
  // MASKED
  int dim, vdim;
  int64_t window, chunk;
  const void* sink;
  float out_scale;
};

__device__ __forceinline__ void warps_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory"); }
__device__ __forceinline__ void load_matrix(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void load_matrix_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// What a CTA works through: the units [begin, end) of the pair-major order.
struct Deal {
  int64_t ctx, lo, units, begin, end;
  int tiles;  // units of a pair
};
__device__ __forceinline__ Deal deal(const StreamParams& p, int64_t pos, bool masked) {
  Deal d;
  d.ctx = pos + 1;
  d.ctx = d.ctx < 0 ? 0 : (d.ctx > p.smax ? p.smax : d.ctx);
  d.lo = masked && d.ctx > 0 ? first_visible(d.ctx - 1, p.window, p.chunk) : 0;
  d.tiles = d.ctx > d.lo ? static_cast<int>((d.ctx - d.lo + kUnit - 1) / kUnit) : 1;  // without positions one that is masked
  d.units = static_cast<int64_t>(p.pairs) * d.tiles;
  if (p.cluster > 1) {
    const int64_t pair = blockIdx.x / p.cluster, rank = blockIdx.x % p.cluster;
    d.begin = pair * d.tiles + d.tiles * rank / p.cluster, d.end = pair * d.tiles + d.tiles * (rank + 1) / p.cluster;
  } else if (p.slots > 1 && d.tiles >= kMinCut) {
    d.begin = d.units * blockIdx.x / gridDim.x, d.end = d.units * (blockIdx.x + 1) / gridDim.x;
  } else {
    d.begin = static_cast<int64_t>(p.pairs) * blockIdx.x / gridDim.x * d.tiles, d.end = static_cast<int64_t>(p.pairs) * (blockIdx.x + 1) / gridDim.x * d.tiles;
  }
  return d;
}

template <typename T, int HD, bool MASKED, bool TWO_TERM, int PER_SM>
__global__ void __launch_bounds__(kThreads, PER_SM)
attn_decode_stream_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const StreamParams p) {
  constexpr int KB = HD / 16;
  constexpr int OB = HD / 8;
  constexpr int kChunks = HD / 64;                 // 128-byte column chunks of a row
  constexpr uint32_t kChunkBytes = kUnit * 128;    // [32 rows][128 B]
  constexpr uint32_t kHalf = kChunks * kChunkBytes;
  constexpr uint32_t kStages = kRingBytes / kHalf;  // a tile of K or of V each
  static_assert(kStages % (2 * kTeams) == 0, "a team's tiles lie in its own stages");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float* sm_o = reinterpret_cast<float*>(smem_raw + (ring - smem_u32(smem_raw)) + kRingBytes);  // [warps][group][HD]
  float* gather_o = sm_o + kWarps * p.group * HD;                                                // [cluster][group][HD], in its first CTA
  float* gather_ml = gather_o + p.cluster * p.group * HD;                                        // [cluster][group][2]
  __shared__ uint64_t bars[2 * kStages];
  __shared__ float sm_m[kWarps][kMaxGroup], sm_l[kWarps][kMaxGroup];
  __shared__ int abort_flag;
  __shared__ unsigned int ticket;

  cg::cluster_group cluster = cg::this_cluster();
  if (p.cluster > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first remote store
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kStages]);
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (uint32_t s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, kWarps / kTeams);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (warp == kWarps) {
    if (elect_one()) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_k) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_v) : "memory");
    }
    __syncwarp();
  } else {
    // While the preceding kernel still runs: ask the L2 for the first units of the run, all but whose newest row were written by
    // earlier steps.  The position read here may still be the previous step's; it only steers a hint.
    const Deal d = deal(p, p.pos_is_i64 ? *static_cast<const volatile int64_t*>(p.input_pos) : *static_cast<const volatile int32_t*>(p.input_pos), MASKED);
    const int64_t last = d.end < d.begin + kHintUnits ? d.end : d.begin + kHintUnits;
    for (int64_t u = d.begin; u < last; ++u) {
      const int pair = static_cast<int>(u / d.tiles);
      const int64_t at = d.lo + (u - static_cast<int64_t>(pair) * d.tiles) * kUnit + (threadIdx.x >> 2);
      if (at >= d.ctx) continue;
      const int part = threadIdx.x & 3;  // a line of the row's key or value
      const int width = MASKED ? (part & 1 ? p.vdim : p.dim) : HD;
      const char* row = static_cast<const char*>(part & 1 ? p.v : p.k) + ((pair * p.smax + at) * width + (part >> 1) * 64) * 2;
      if ((part >> 1) * 64 < width) asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
    }
  }
  pdl_launch_dependents();
  pdl_wait();  // q and the newest cache rows come from the preceding kernel

  const Deal d = deal(p, load_pos(p.input_pos, p.pos_is_i64, 0), MASKED);
  const int64_t ctx = d.ctx, lo = d.lo, u0 = d.begin, u1 = d.end;
  const int tiles = d.tiles;

  // result of elements e, e + 1 of head h of a pair's group from their maximum, sum and weighted values
  auto store = [&](int pair, int h, int e, float m, float l, float2 v) {
    const int vd = MASKED ? p.vdim : HD, b = pair / p.n_kv, head0 = (pair - b * p.n_kv) * p.group;
    float mm = m, f = 1.f;
    if (MASKED && p.sink) {
      const float sk = Num<T>::to_f(static_cast<const T*>(p.sink)[head0 + h]) * 1.4426950408889634f;
      mm = fmaxf(m, sk);
      f = m == -INFINITY ? 0.f : exp2f(m - mm);
      l = l * f + exp2f(sk - mm);
    }
    const float inv = l > 0.f ? f / l : 0.f;
    if (MASKED) {
      T* dst = static_cast<T*>(p.out) + static_cast<int64_t>(b) * p.out_ld + static_cast<int64_t>(head0 + h) * vd + e;
      if (e < vd) dst[0] = Num<T>::from_f(v.x * inv * p.out_scale);
      if (e + 1 < vd) dst[1] = Num<T>::from_f(v.y * inv * p.out_scale);
    } else {
      *reinterpret_cast<uint32_t*>(static_cast<T*>(p.out) + static_cast<int64_t>(b) * p.out_ld + static_cast<int64_t>(head0 + h) * HD + e) =
          pack2<T>(v.x * inv, v.y * inv);
    }
  };
  // the same from n parts, part(i, ml, v) fetching one
  auto store_merged = [&](int pair, int h, int e, int n, auto part) {
    float mm = -INFINITY, ll = 0.f;
    float2 sum = make_float2(0.f, 0.f);
    for (int i = 0; i < n; ++i) {
      float2 ml, v;
      part(i, ml, v);
      const float m_new = fmaxf(mm, ml.x);
      const float w_old = mm == -INFINITY ? 0.f : exp2f(mm - m_new), w = ml.x == -INFINITY ? 0.f : exp2f(ml.x - m_new);
      ll = ll * w_old + ml.y * w;
      sum.x = sum.x * w_old + v.x * w, sum.y = sum.y * w_old + v.y * w;
      mm = m_new;
    }
    store(pair, h, e, mm, ll, sum);
  };

  if (warp == kWarps) {
    uint32_t s = 0, parity = 1;  // a fresh barrier passes a wait on parity 1
    int pair = static_cast<int>(u0 / tiles), t = static_cast<int>(u0 - static_cast<int64_t>(pair) * tiles);
    for (int64_t u = u0; u < u1; ++u) {
      bool ok = true;
#pragma unroll
      for (int half = 0; half < 2 && ok; ++half) {
        ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * (s + half), parity, &abort_flag, 31, &g_attn_stream_status));
        if (ok && elect_one()) {
          mbar_expect_tx(full0 + 8 * (s + half), kHalf);
          const int row = static_cast<int>(pair * p.smax + lo) + t * kUnit;
#pragma unroll
          for (int c = 0; c < kChunks; ++c)
            tma_load_2d(ring + (s + half) * kHalf + c * kChunkBytes, half ? &tmap_v : &tmap_k, full0 + 8 * (s + half), c * 64, row);
        }
        __syncwarp();
      }
      if (!ok) break;
      s += 2;
      if (s == kStages) s = 0, parity ^= 1u;
      if (++t == tiles) t = 0, ++pair;
    }
  } else {
    const int g = p.group, kd = MASKED ? p.dim : HD;
    const int r0 = lane >> 2, r1 = r0 + 8;  // the rows (heads) whose scores this thread holds
    const int sub = warp & 1;  // which half of a unit
    uint32_t s = 2 * (warp >> 1), parity = 0;  // the stage of K; V is in the next one
    bool ok = true;
    int64_t next = u0 + (warp >> 1);  // this team's next unit
    int64_t u = u0;
    for (bool more = u0 < u1 || p.cluster > 1; more; more = u < u1) {  // a cluster's CTA without units still takes part in its merge
      const int pair = p.cluster > 1 ? static_cast<int>(blockIdx.x) / p.cluster : static_cast<int>(u / tiles);
      const int64_t first = static_cast<int64_t>(pair) * tiles;
      const int64_t end = first + tiles < u1 ? first + tiles : u1;
      const int b = pair / p.n_kv, head0 = (pair - b * p.n_kv) * g;

      // ---- Q: head h of the group is row h; rows from g up are zero ---------------------------------------------
      uint32_t qa[KB][4];
      {
        const T* qg = static_cast<const T*>(p.q) + (static_cast<int64_t>(b) * p.n_head + head0) * kd + (lane & 3) * 2;
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = (e & 1) ? r1 : r0, col = kb * 16 + (e >> 1) * 8;
            qa[kb][e] = r < g && (!MASKED || col < kd) ? *reinterpret_cast<const uint32_t*>(qg + static_cast<int64_t>(r) * kd + col) : 0u;
          }
      }
      float o[OB][4];
#pragma unroll
      for (int i = 0; i < OB; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
      float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};

      auto arrived = [&](uint32_t stage) {
        return __all_sync(0xffffffffu, mbar_wait(full0 + 8 * stage, parity, &abort_flag, 32, &g_attn_stream_status)) != 0;
      };
      auto give_back = [&](uint32_t stage) {
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * stage);
      };
      for (; next < end && ok; next += kTeams) {
        const int64_t left = ctx - lo - (next - first) * kUnit - sub * kTile;
        const int valid = left < kTile ? (left > 0 ? static_cast<int>(left) : 0) : kTile;
        ok = arrived(s);
        if (!ok) break;
        // ---- scores 16 heads x 16 positions, four accumulation chains ---------------------------------------------------
        float sc[2][2][4];
#pragma unroll
        for (int i = 0; i < 16; ++i) sc[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
        {
          const int row = (lane & 7) + (lane >> 4) * 8;
          const uint32_t at = ring + s * kHalf + (sub * kTile + row) * 128;
#pragma unroll
          for (int kb = 0; kb < KB; ++kb) {
            const int unit = (kb & 3) * 2 + ((lane >> 3) & 1);
            uint32_t bf[4];
            load_matrix(at + (kb >> 2) * kChunkBytes + ((unit ^ (row & 7)) << 4), bf);
            mma16816<T>(sc[kb & 1][0], qa[kb][0], qa[kb][1], qa[kb][2], qa[kb][3], bf[0], bf[1]);
            mma16816<T>(sc[kb & 1][1], qa[kb][0], qa[kb][1], qa[kb][2], qa[kb][3], bf[2], bf[3]);
          }
        }
        give_back(s);
        // ---- scale, mask ---------------------------------------------------------------------------------------------------
        float x[2][4], mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          const int key = nb * 8 + (lane & 3) * 2;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            x[nb][e] = key + (e & 1) < valid ? (sc[0][nb][e] + sc[1][nb][e]) * p.scale_log2 : -INFINITY;
            mx[e >> 1] = fmaxf(mx[e >> 1], x[nb][e]);
          }
        }
        // ---- online softmax ---------------------------------------------------------------------------------------------
        float corr[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
          mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
          const float m_new = fmaxf(m_run[r], mx[r]);
          const float m_use = m_new == -INFINITY ? 0.f : m_new;
          corr[r] = exp2f(m_run[r] - m_use);
          m_run[r] = m_new;
          mx[r] = m_use;
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {  // a maximum moved: seldom after the first tiles
#pragma unroll
          for (int r = 0; r < 2; ++r) l_run[r] *= corr[r];
#pragma unroll
          for (int i = 0; i < OB; ++i) {
            o[i][0] *= corr[0];
            o[i][1] *= corr[0];
            o[i][2] *= corr[1];
            o[i][3] *= corr[1];
          }
        }
        uint32_t pa[4], pl[4];
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          float pv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            pv[e] = exp2f(x[nb][e] - mx[e >> 1]);
            l_run[e >> 1] += pv[e];
          }
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            pa[nb * 2 + r] = pack2<T>(pv[2 * r], pv[2 * r + 1]);
            if (TWO_TERM) {
              float h0, h1;
              Num<T>::unpack2(pa[nb * 2 + r], h0, h1);
              pl[nb * 2 + r] = pack2<T>(pv[2 * r] - h0, pv[2 * r + 1] - h1);
            }
          }
        }
        // ---- O += P V (16 positions = one k block) --------------------------------------------------------------------
        ok = arrived(s + 1);
        if (!ok) break;
        const uint32_t sv = ring + (s + 1) * kHalf + sub * kTile * 128;
        if (valid < kTile) {
          // values past the newest position may be anything, and 0 x NaN is not 0
          for (int i = valid * 8 + lane; i < kTile * 8; i += 32)
#pragma unroll
            for (int c = 0; c < kChunks; ++c)
              asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(sv + c * kChunkBytes + i * 16), "r"(0u) : "memory");
          __syncwarp();
        }
        {
          const int row = (lane & 7) + ((lane >> 3) & 1) * 8;
          const uint32_t at = sv + row * 128;
#pragma unroll
          for (int ob2 = 0; ob2 < OB / 2; ++ob2) {
            const int unit = (ob2 & 3) * 2 + (lane >> 4);
            uint32_t bf[4];
            load_matrix_trans(at + (ob2 >> 2) * kChunkBytes + ((unit ^ (row & 7)) << 4), bf);
            mma16816<T>(o[2 * ob2], pa[0], pa[1], pa[2], pa[3], bf[0], bf[1]);
            mma16816<T>(o[2 * ob2 + 1], pa[0], pa[1], pa[2], pa[3], bf[2], bf[3]);
            if (TWO_TERM) {
              mma16816<T>(o[2 * ob2], pl[0], pl[1], pl[2], pl[3], bf[0], bf[1]);
              mma16816<T>(o[2 * ob2 + 1], pl[0], pl[1], pl[2], pl[3], bf[2], bf[3]);
            }
          }
        }
        if (valid < kTile) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the zeros, before the next copy
        give_back(s + 1);
        s += 2 * kTeams;
        if (s >= kStages) s -= kStages, parity ^= 1u;
      }

      // ---- merge the warps --------------------------------------------------------------------------------------------
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
        l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
      }
      warps_sync();  // the arrays' previous contents have been read
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int h = r ? r1 : r0;
        if (h < g) {
          if ((lane & 3) == 0) sm_m[warp][h] = m_run[r], sm_l[warp][h] = l_run[r];
          float* d = sm_o + (warp * g + h) * HD + (lane & 3) * 2;
#pragma unroll
          for (int i = 0; i < OB; ++i) *reinterpret_cast<float2*>(d + i * 8) = make_float2(o[i][2 * r], o[i][2 * r + 1]);
        }
      }
      warps_sync();
      // the CTAs that share this pair
      const bool whole = p.cluster > 1 || (u == first && end == first + tiles);
      const int64_t c_first = whole ? blockIdx.x : ((first + 1) * gridDim.x - 1) / d.units;
      const int parts = whole ? 1 : static_cast<int>(((first + tiles) * gridDim.x - 1) / d.units - c_first) + 1;
      const int64_t part0 = static_cast<int64_t>(pair) * p.slots * g;
      const int64_t mine = part0 + (blockIdx.x - c_first) * g;
      if (p.cluster > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // the first CTA has started
      for (int idx = threadIdx.x; idx < g * (HD / 2); idx += kWarps * 32) {
        const int h = idx / (HD / 2), e = idx % (HD / 2) * 2;
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, sm_m[w][h]);
        float ll = 0.f;
        float2 v = make_float2(0.f, 0.f);
        if (mm > -INFINITY) {
#pragma unroll
          for (int w = 0; w < kWarps; ++w) {
            const float wt = exp2f(sm_m[w][h] - mm);  // 0 for warps that saw no position
            const float2 ow = *reinterpret_cast<const float2*>(sm_o + (w * g + h) * HD + e);
            ll += sm_l[w][h] * wt;
            v.x += ow.x * wt, v.y += ow.y * wt;
          }
        }
        if (p.cluster > 1) {
          const int rank = static_cast<int>(cluster.block_rank());
          *reinterpret_cast<float2*>(cluster.map_shared_rank(gather_o, 0) + (rank * g + h) * HD + e) = v;
          if (e == 0) *reinterpret_cast<float2*>(cluster.map_shared_rank(gather_ml, 0) + (rank * g + h) * 2) = make_float2(mm, ll);
        } else if (parts == 1) {
          store(pair, h, e, mm, ll, v);
        } else {
          *reinterpret_cast<float2*>(p.part_o + (mine + h) * HD + e) = v;
          if (e == 0) *reinterpret_cast<float2*>(p.part_ml + (mine + h) * 2) = make_float2(mm, ll);
        }
      }
      if (parts > 1) {
        // ---- the last CTA of this pair merges the parts -----------------------------------------------------------------
        warps_sync();
        if (threadIdx.x == 0) {
          unsigned int before;  // the barrier orders the other threads' stores before this release, and their loads behind it
          asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(p.counters + pair) : "memory");
          ticket = before;
        }
        warps_sync();
        if (ticket == static_cast<unsigned int>(parts - 1)) {
          for (int idx = threadIdx.x; idx < g * (HD / 2); idx += kWarps * 32) {
            const int h = idx / (HD / 2), e = idx % (HD / 2) * 2;
            store_merged(pair, h, e, parts, [&](int i, float2& ml, float2& v) {
              ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + (part0 + i * g + h) * 2));
              v = __ldcg(reinterpret_cast<const float2*>(p.part_o + (part0 + i * g + h) * HD + e));
            });
          }
          if (threadIdx.x == 0) p.counters[pair] = 0u;  // ready for the next call
        }
      }
      u = end;
    }
  }
  if (p.cluster > 1) {
    if (warp == kWarps) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    cluster.sync();  // every part has landed in the first CTA's shared memory
    if (cluster.block_rank() == 0 && warp < kWarps)
      for (int idx = threadIdx.x; idx < p.group * (HD / 2); idx += kWarps * 32) {
        const int h = idx / (HD / 2), e = idx % (HD / 2) * 2;
        store_merged(static_cast<int>(blockIdx.x) / p.cluster, h, e, p.cluster, [&](int i, float2& ml, float2& v) {
          ml = *reinterpret_cast<const float2*>(gather_ml + (i * p.group + h) * 2);
          v = *reinterpret_cast<const float2*>(gather_o + (i * p.group + h) * HD + e);
        });
      }
  }
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 2000; ++i) __nanosleep(100);  // let copies in flight land before shared memory is released
  }
  __syncthreads();
}

template <typename T, int HD, bool MASKED, bool TWO_TERM, int PER_SM>
int launch(int dtype, const StreamParams& p, int64_t grid, cudaStream_t st) {
  CUtensorMap tk, tv;
  int rc = make_tmap(&tk, dtype, p.k, p.pairs * p.smax, p.dim, kUnit);
  if (rc != LRI_OK) return rc;
  rc = make_tmap(&tv, dtype, p.v, p.pairs * p.smax, p.vdim, kUnit);
  if (rc != LRI_OK) return rc;
  const int smem = 1024 + kRingBytes + kWarps * p.group * HD * 4 + p.cluster * p.group * (HD + 2) * 4;
  auto kern = attn_decode_stream_kernel<T, HD, MASKED, TWO_TERM, PER_SM>;
  static std::atomic<unsigned long long> attr_set{0};  // per template instantiation, one bit per device
  LRI_ONCE_PER_DEVICE(attr_set, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     1024 + kRingBytes + kWarps * kMaxGroup * HD * 4 + kMaxGathered * (HD + 2) * 4));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(p.cluster);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  LRI_CUDA(cudaLaunchKernelEx(&cfg, kern, tk, tv, p));
  LRI_LAUNCH_CHECK("attn_decode_stream_kernel");
  return LRI_OK;
}

// CTAs of a cluster that share a pair, with `room` CTAs on the GPU: as many (a power of two) as fit at once.  Clusters of 2 find room for all
// CTAs that would fit singly (8 KV heads, 1025 positions, 136 and 144 pairs: 18.8 and 18.9 us singly, 15.7 and 16.3 in clusters; of 64
// elements, three CTAs an SM, 216 pairs: 17.1 and 12.8), of 4 for 7 of 8, of 8 for half of them (72 pairs: 17.1 us in 288 CTAs, 11.8 in 144; 32 pairs:
// 13.1 in 256, 9.0 in 128).
int cluster_size(const StreamParams& p, int64_t room, int forced) {
  int size = 1;
  for (int c = 2; c <= kMaxCluster; c *= 2)
    if (static_cast<int64_t>(p.pairs) * c <= (c == 2 ? room : c == 4 ? room / 8 * 7 : room / 2) && p.group * c <= kMaxGathered && (forced == 0 || c <= forced)) size = c;
  return size;
}

// CTAs: two of them share an SM.  Rows of 64 elements, whose tiles are half as large, take three where that gives a pair more CTAs or shortens
// the run of a CTA (us a layer, two / three, 1025 positions: 144 pairs 16.6 / 11.8, 384 26.3 / 19.9, 768 43.6 / 38.7).  Where it does not, two have
// the registers of three, and a third does not fit: CTAs would come to lie three on one SM and one on another (40 pairs 7.6 / 8.4, 240 pairs
// 16.9 / 18.5).
// From more pairs than fit on, and with room for their parts, all CTAs get equal runs, each at least a pair long.
template <bool MASKED, bool TWO_TERM>
int dispatch(int dtype, StreamParams& p, int forced, cudaStream_t st) {
  const int64_t sms = device_sm_count();
  const bool narrow = p.dim <= 64 && p.vdim <= 64;
  int per_sm = 2;
  p.cluster = cluster_size(p, 2 * sms, forced);
  if (narrow && p.group <= 4) {  // more heads take more shared memory than a third of an SM's
    const int of_three = cluster_size(p, 3 * sms, forced);
    // pairs of a CTA, times its neighbours, if pairs are not cut
    const int64_t two_deep = (p.pairs + 2 * sms - 1) / (2 * sms) * 2, three_deep = (p.pairs + 3 * sms - 1) / (3 * sms) * 3;
    const bool cut = p.slots > 1 && p.smax >= kMinCut * kUnit;
    if (of_three > p.cluster || (p.pairs > 2 * sms && (cut || three_deep < two_deep))) per_sm = 3;
    if (of_three > p.cluster) p.cluster = of_three;
  }
  const int64_t room = per_sm * sms;
  if (p.cluster > 1 || p.pairs <= room) p.slots = 1;
  const int64_t grid = p.slots > 1 ? room : static_cast<int64_t>(p.pairs) * p.cluster;
  if (dtype == LRI_BF16) {
    if (!narrow) return launch<__nv_bfloat16, 128, MASKED, TWO_TERM, 2>(dtype, p, grid, st);
    return per_sm == 3 ? launch<__nv_bfloat16, 64, MASKED, TWO_TERM, 3>(dtype, p, grid, st) : launch<__nv_bfloat16, 64, MASKED, TWO_TERM, 2>(dtype, p, grid, st);
  }
  if (!narrow) return launch<__half, 128, MASKED, TWO_TERM, 2>(dtype, p, grid, st);
  return per_sm == 3 ? launch<__half, 64, MASKED, TWO_TERM, 3>(dtype, p, grid, st) : launch<__half, 64, MASKED, TWO_TERM, 2>(dtype, p, grid, st);
}

}  // namespace

// row coordinates of the tensor maps are 32-bit
bool attn_decode_stream_supports(int64_t pairs, int group, int64_t smax) {
  return group <= kMaxGroup && pairs * smax + kUnit < (1ll << 31) && pairs < (1 << 24);
}

// counters: zero, and left zero; parts: room for part_slots parts of every pair; two_term: probabilities of more than 16 bits
int attn_decode_stream_launch(int dtype, const void* q, const void* k_cache, const void* v_cache, const void* input_pos, int pos_is_i64,
                              void* out, int B, int n_head, int n_kv, int head_dim, int64_t smax, float scale_log2, unsigned int* counters,
                              float* parts, int64_t part_slots, bool two_term, cudaStream_t st) {
  StreamParams p{};
  p.q = q, p.k = k_cache, p.v = v_cache, p.input_pos = input_pos, p.pos_is_i64 = pos_is_i64, p.out = out, p.out_ld = static_cast<int64_t>(n_head) * head_dim;
  p.pairs = B * n_kv, p.n_head = n_head, p.n_kv = n_kv, p.group = n_head / n_kv, p.smax = smax, p.scale_log2 = scale_log2;
  p.dim = p.vdim = head_dim;
  p.slots = part_slots < 2 ? 1 : 2;
  p.counters = counters;
  p.part_ml = parts;
  p.part_o = parts + (static_cast<int64_t>(B) * n_head * p.slots * 2 + 3) / 4 * 4;
  return two_term ? dispatch<false, true>(dtype, p, option(OPT_DECODE_SPLITS), st) : dispatch<false, false>(dtype, p, option(OPT_DECODE_SPLITS), st);
}

int attn_decode_stream_masked_launch(int dtype, const WindowParams& w, int B, cudaStream_t st) {
  StreamParams p{};
  p.q = w.q, p.k = w.k, p.v = w.v, p.input_pos = w.input_pos, p.pos_is_i64 = w.pos_is_i64, p.out = w.out, p.out_ld = w.out_ld;
  p.n_head = w.H, p.n_kv = w.H / w.group, p.pairs = B * p.n_kv, p.group = w.group, p.smax = w.k_rows;
  p.scale_log2 = w.scale * 1.4426950408889634f;
  p.slots = 1;
  p.dim = w.d1, p.vdim = w.dv, p.window = w.window, p.chunk = w.chunk, p.sink = w.sink, p.out_scale = w.out_scale;
  return dispatch<true, true>(dtype, p, option(OPT_DECODE_SPLITS), st);
}

int attn_decode_stream_status_read_and_clear(int* status_out) {
  int v = 0;
  LRI_CUDA(cudaMemcpyFromSymbol(&v, g_attn_stream_status, sizeof(int)));
  if (v != 0) {
    int zero = 0;
    LRI_CUDA(cudaMemcpyToSymbol(g_attn_stream_status, &zero, sizeof(int)));
  }
  *status_out = v;
  return LRI_OK;
}

}  // namespace lri
