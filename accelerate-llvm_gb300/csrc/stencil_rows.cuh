// stencil_rows.cuh -- how a warp reads a strip of 32 x E columns of one array
// row into registers, with the boundary columns beside it, for the row-streaming
// stencils of stencil.cu.
#pragma once

#include "stencil_common.cuh"

namespace accgb {

// A warp owns the columns x0 .. x0 + 32 E - 1 of an array `in_w` wide.
// VEC: lane l holds the E consecutive columns x0 + l E .. (16-byte loads; the
// rows are 16-byte aligned and in_w is a multiple of E).  Otherwise lane l
// holds columns x0 + l, x0 + l + 32, ... (E single loads, each coalesced over
// the warp, whatever the alignment).  The RX columns on either side of the
// strip are held by the lanes that need them (`halo`).  Columns outside of
// the array are remapped by the boundary (or are the constant) once, when the
// strip is set up: they are the same in every row.
template <class T, int RX, bool VEC> struct StripRow {
  static constexpr int E = 16 / (int)sizeof(T);
  static constexpr int H = RX > 0 ? RX : 1;
  T v[E];
  T halo[H];
};

template <class T, int RX, bool VEC> struct Strip {
  using Row = StripRow<T, RX, VEC>;
  static constexpr int E = Row::E, H = Row::H;
  int64_t off[VEC ? H : E];  // columns this lane reads: VEC: its first (or, outside, the remapped ones); else each
  int64_t hoff[H];           // its halo columns
  uint32_t cmask;            // bits: halo column i (i), column e (8 + e) is the boundary constant
  int lane;
  bool inside;               // VEC: the lane's columns lie in the array
  bool side;                 // the lane holds halo columns
  T cval;

  __device__ __forceinline__ void init(int64_t x0, int64_t in_w, int boundary, T c) {
    lane = threadIdx.x & 31;
    cval = c;
    cmask = 0;
    auto column = [&](int64_t x, int bit) -> int64_t {
      if (x >= 0 && x < in_w) return x;
      if (boundary == ACC_CONSTANT) cmask |= 1u << bit;
      return bound_index(x, in_w, boundary);
    };
    inside = true;
    if constexpr (VEC) {
      const int64_t x = x0 + (int64_t)lane * E;
      inside = x < in_w;
#pragma unroll
      for (int i = 0; i < H; ++i) off[i] = inside ? x : column(x + i, 8 + i);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) off[e] = column(x0 + 32 * e + lane, 8 + e);
    }
    const bool left = VEC ? lane == 0 : lane < RX, right = VEC ? lane == 31 : lane >= 32 - RX;
    side = RX > 0 && (left || right);
#pragma unroll
    for (int i = 0; i < H; ++i) hoff[i] = side ? column(left ? x0 - RX + i : x0 + 32 * E + i, i) : 0;
  }

  // Read one row of the array (`row`: its first column).
  __device__ __forceinline__ void load(const T *row, Row &r) const {
    if constexpr (VEC) {
      if (inside) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(row + off[0]));
        memcpy(r.v, &q, 16);
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e)
          r.v[e] = e < RX ? (((cmask >> (8 + e)) & 1u) ? cval : __ldg(row + off[e < H ? e : 0])) : T(0);
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) r.v[e] = ((cmask >> (8 + e)) & 1u) ? cval : __ldg(row + off[e]);
    }
    if constexpr (RX > 0) {
      if (side) {
#pragma unroll
        for (int i = 0; i < RX; ++i) r.halo[i] = ((cmask >> i) & 1u) ? cval : __ldg(row + hoff[i]);
      }
    }
  }
  // A strip whose columns and halo all lie in the array reads at constant
  // distances from two addresses per lane, p (its first column) and h (its
  // first halo column).
  __device__ __forceinline__ int64_t inner_column(int64_t x0) const { return x0 + (VEC ? lane * E : lane); }
  __device__ __forceinline__ int64_t inner_halo(int64_t x0) const {
    return (VEC ? lane == 0 : lane < RX) ? x0 - RX : x0 + 32 * E;
  }
  __device__ __forceinline__ void load_inner(const T *p, const T *h, Row &r) const {
    if constexpr (VEC) {
      const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
      memcpy(r.v, &q, 16);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) r.v[e] = __ldg(p + 32 * e);
    }
    if constexpr (RX > 0) {
      if (side) {
#pragma unroll
        for (int i = 0; i < RX; ++i) r.halo[i] = __ldg(h + i);
      }
    }
  }
  // A row that lies outside of the array under the constant boundary.
  __device__ __forceinline__ void fill(Row &r) const {
#pragma unroll
    for (int e = 0; e < E; ++e) r.v[e] = cval;
#pragma unroll
    for (int i = 0; i < H; ++i) r.halo[i] = cval;
  }

  // win[RX + d][e]: the value at distance d of this lane's column e (warp-collective).
  __device__ __forceinline__ void window(const Row &r, T (&win)[2 * RX + 1][E]) const {
#pragma unroll
    for (int e = 0; e < E; ++e) win[RX][e] = r.v[e];
    if constexpr (VEC) {
      T lo[H], hi[H];  // columns -RX.. -1 and E .. E + RX - 1 of this lane
#pragma unroll
      for (int i = 0; i < RX; ++i) {
        const T a = shfl_up(r.v[E - RX + i], 1), b = shfl_down(r.v[i], 1);
        lo[i] = lane == 0 ? r.halo[i] : a;
        hi[i] = lane == 31 ? r.halo[i] : b;
      }
#pragma unroll
      for (int d = 1; d <= RX; ++d)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          win[RX - d][e] = e >= d ? r.v[e >= d ? e - d : 0] : lo[e < d ? RX + e - d : 0];
          win[RX + d][e] = e + d < E ? r.v[e + d < E ? e + d : 0] : hi[e + d >= E ? e + d - E : 0];
        }
    } else {
#pragma unroll
      for (int d = 1; d <= RX; ++d) {
        // the halo values of lane l are those at column distances RX - i
        T hl = r.halo[0], hr = r.halo[0];
        if constexpr (RX == 2) {
          hl = (d == 1 || lane == 1) ? r.halo[1] : r.halo[0];
          hr = (d == 2 && lane == 31) ? r.halo[1] : r.halo[0];
        }
        T a[E], b[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          a[e] = shfl_idx(r.v[e], (lane - d) & 31);
          b[e] = shfl_idx(r.v[e], (lane + d) & 31);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
          win[RX - d][e] = lane >= d ? a[e] : (e > 0 ? a[e > 0 ? e - 1 : 0] : hl);
          win[RX + d][e] = lane + d < 32 ? b[e] : (e < E - 1 ? b[e < E - 1 ? e + 1 : 0] : hr);
        }
      }
    }
  }

  // Store the lane's columns of one output row `w` wide (VEC: w a multiple of E).
  __device__ __forceinline__ void store(T *row, int64_t x0, int64_t w, const T (&y)[E]) const {
    if constexpr (VEC) {
      const int64_t x = x0 + (int64_t)lane * E;
      if (x < w) {
        uint4 q;
        memcpy(&q, y, 16);
        __stcs(reinterpret_cast<uint4 *>(row + x), q);
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int64_t x = x0 + 32 * e + lane;
        if (x < w) __stcs(row + x, y[e]);
      }
    }
  }
};

}  // namespace accgb
