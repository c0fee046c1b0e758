// What the prefill GEMM kernels share: the order of the output tiles and the fused epilogues, which take a row of fp32
// accumulators from tensor memory to its place in the output.
#pragma once

#include "linear.cuh"
#include "tcgen05.cuh"

namespace lri {
namespace tc {

struct GemmShape {
  int m, n, k;
};

// One unit of work of a persistent CTA (or pair of CTAs): an output tile.
struct WorkItem {
  int tile_p, tile_q;
};
struct GemmGrid {
  int tiles_p, tiles_q;
  int group;  // P tiles per panel
  // expert tiles: the number of P tiles in use and the weight matrix of each are read from the device
  const int* tiles;
  int matrix_rows;
};
// Order of the output tiles.  The P tiles are taken in panels of `group`; inside a panel the
// Q tile is the slow index.  The CTAs that run at the same time then share one panel of P
// (a few MB, stays in L2) and a handful of Q tiles, each of which all of them use at once, so
// that both operands come from DRAM about once per panel instead of once per P tile.
__device__ __forceinline__ WorkItem work_item(int item, const GemmGrid& g) {
  WorkItem w;
  const int panel_items = g.group * g.tiles_q;
  const int panel = item / panel_items;
  const int r = item - panel * panel_items;
  const int p0 = panel * g.group;
  const int gm = min(g.group, g.tiles_p - p0);
  w.tile_q = r / gm;
  w.tile_p = p0 + (r - w.tile_q * gm);
  return w;
}

// Stores one row of an output tile of bn columns (a multiple of 32) from the TMEM lane at `tacc`; row = the token's row of A.
//   EPI_SWIGLU  columns [0, bn/2) are up rows and [bn/2, bn) the matching gate rows of w1: the thread finds up_j and gate_j of
//               its token in one accumulator row and stores silu(gate) * up to h [m, I] (lin.y, lin.n = I)
//   EPI_GLU     as SWIGLU with the clamped unit, on fp32 accumulators (scaled per row for experts)
//   EPI_F32     stores the fp32 accumulators
//   EPI_QKV     rotates the 16 adjacent pairs of each 32-column chunk with the table row of the token's position and stores
//               them to q_out / k-cache / v-cache
// The loads are warp-collective: the lanes meet before each of them, rows outside the problem store nothing.
template <typename T, int EPI>
__device__ __forceinline__ void store_row(const LinearParams& lin, T* c, const GemmShape& shape, int64_t row, int tile_q, int bn, uint32_t tacc) {
  if (EPI == EPI_SWIGLU || EPI == EPI_GLU) {
    const float sc = EPI == EPI_GLU && lin.ex.row_scale && row < shape.m ? lin.ex.row_scale[row] : 1.f;
#pragma unroll 1
    for (int cc = 0; cc < bn / 2; cc += 16) {
      uint32_t up[16], gate[16];
      __syncwarp();
      tmem_ld16_issue(tacc + cc, up);
      tmem_ld16_issue(tacc + bn / 2 + cc, gate);
      tmem_wait_ld();
      const int64_t j0 = static_cast<int64_t>(tile_q) * (bn / 2) + cc;
      if (row < shape.m && j0 < lin.n) {
        T* dst = static_cast<T*>(lin.y) + row * lin.n + j0;
        __align__(16) T out[16];
#pragma unroll
        for (int e = 0; e < 16; ++e)
          out[e] = EPI == EPI_GLU ? Num<T>::from_f(clamped_glu(sc * __uint_as_float(gate[e]), sc * __uint_as_float(up[e]), lin.ex.glu))
                                  : swiglu_rounded<T>(rnd<T>(__uint_as_float(up[e])), rnd<T>(__uint_as_float(gate[e])));
        if (j0 + 16 <= lin.n && (lin.n & 7) == 0) {
#pragma unroll
          for (int v = 0; v < 2; ++v) reinterpret_cast<uint4*>(dst)[v] = reinterpret_cast<const uint4*>(out)[v];
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (j0 + e < lin.n) dst[e] = out[e];
        }
      }
    }
  } else if (EPI == EPI_QKV) {
    const int hd = lin.head_dim;
    const int64_t nq = static_cast<int64_t>(lin.n_head) * hd, nk = static_cast<int64_t>(lin.n_kv) * hd;
    const int64_t b = row / lin.S, sq = row - b * lin.S;
    int64_t pos = 0, trow = 0;
    bool live = row < shape.m;
    if (live) {
      pos = load_pos(lin.input_pos, lin.pos_is_i64, sq);
      trow = lin.table_gathered ? sq : pos;
      live = pos >= 0 && pos < lin.smax && trow < lin.table_rows;
    }
#pragma unroll 1
    for (int cc = 0; cc < bn; cc += 32) {
      uint32_t r[32];
      __syncwarp();
      tmem_ld32(tacc + cc, r);
      const int64_t n = static_cast<int64_t>(tile_q) * bn + cc;  // a 32-column chunk never straddles a head
      if (live && n < shape.n) {
        float f[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) f[e] = rnd<T>(__uint_as_float(r[e]));
        T* dst;
        if (n < nq + nk) {
          const int64_t nn = n < nq ? n : n - nq;
          const int e0 = static_cast<int>(nn % hd);
          const uint4* cs = reinterpret_cast<const uint4*>(static_cast<const T*>(lin.rope_table) + (trow * (hd >> 1) + (e0 >> 1)) * 2);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            float t[8];
            unpack8<T>(cs[v], t);  // (cos, sin) of 4 pairs
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float o0, o1;
              rope_pair(f[v * 8 + 2 * q], f[v * 8 + 2 * q + 1], t[2 * q], t[2 * q + 1], o0, o1);
              f[v * 8 + 2 * q] = o0;
              f[v * 8 + 2 * q + 1] = o1;
            }
          }
          dst = n < nq ? static_cast<T*>(lin.q_out) + row * nq + n
                       : static_cast<T*>(lin.k_cache) + ((b * lin.n_kv + nn / hd) * lin.smax + pos) * hd + e0;
        } else {
          const int64_t nn = n - nq - nk;
          dst = static_cast<T*>(lin.v_cache) + ((b * lin.n_kv + nn / hd) * lin.smax + pos) * hd + nn % hd;
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float g8[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) g8[e] = f[v * 8 + e];
          reinterpret_cast<uint4*>(dst)[v] = pack8<T>(g8);
        }
      }
    }
  } else {
#pragma unroll 1
    for (int cc = 0; cc < bn; cc += 32) {
      uint32_t r[32];
      __syncwarp();
      tmem_ld32(tacc + cc, r);
      const int64_t col0 = static_cast<int64_t>(tile_q) * bn + cc;
      if (row < shape.m) {
        if (EPI == EPI_F32) {
          float* dst = static_cast<float*>(lin.y) + row * shape.n + col0;
          if (col0 + 32 <= shape.n) {
#pragma unroll
            for (int v = 0; v < 8; ++v) reinterpret_cast<uint4*>(dst)[v] = make_uint4(r[v * 4], r[v * 4 + 1], r[v * 4 + 2], r[v * 4 + 3]);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (col0 + e < shape.n) dst[e] = __uint_as_float(r[e]);
          }
        } else {
          T* dst = c + row * shape.n + col0;
          if (col0 + 32 <= shape.n) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[v * 8 + e]);
              reinterpret_cast<uint4*>(dst)[v] = pack8<T>(f);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (col0 + e < shape.n) dst[e] = Num<T>::from_f(__uint_as_float(r[e]));
          }
        }
      }
    }
  }
}

}  // namespace tc
}  // namespace lri
