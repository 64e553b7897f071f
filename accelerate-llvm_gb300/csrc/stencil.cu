// stencil.cu -- weighted-sum stencils over rank-1 / rank-2 arrays with
// clamp / mirror / wrap / constant boundaries.
//
// The reference launches `stencil_inside` over the interior (one thread per
// output, every tap a separate global load, no shared-memory reuse) and
// 2*rank `stencil_border` kernels on forked streams
// (accelerate-llvm-ptx/src/Data/Array/Accelerate/LLVM/PTX/Execute.hs:686-776,
// PTX/CodeGen/Stencil.hs:113-179).  Here one launch covers the whole array.
// The usual patterns (3x3, 1x3, 3x1, 5x5) stream the rows of a strip of
// columns through a warp's registers (stencil_rows_kernel).  The others, and
// the second pass of stencil2, pull a (TH + 2R) x (TW + 2PX) halo tile per CTA
// into shared memory with one 2-D TMA load (the x start rounded out to a
// 16-byte boundary), overwrite the cells outside of the array with the
// boundary rule (accelerate-llvm/src/Data/Array/Accelerate/LLVM/CodeGen/
// Stencil.hs:195-253), and each thread sweeps a column of outputs, keeping one
// accumulator per output and visiting the taps in the reference's order
// (rows outer, -r..r; CodeGen/Stencil.hs:73-180).
//
// Arithmetic: acc starts at the additive identity (-0.0) and every tap is one
// fused multiply-add, acc = fma(w, x, acc), in tap order, so Float32 / Float64
// results are bit-identical to a sequential C evaluation with C99 fma()
// (correctly rounded).  Taps whose weight is exactly zero are not part of the
// pattern and are not read.
#include "stencil_rows.cuh"

namespace accgb {

constexpr int ST_TW = 64;       // tile width (outputs)
constexpr int ST_TH = 32;       // tile height (outputs)
constexpr int ST_THREADS = 256; // 64 columns x 4 row groups of 8
constexpr int ST_ROWS = ST_TH / (ST_THREADS / ST_TW);

template <class T> struct StencilW { T w[81]; };

struct StencilArgs {
  const void *in;
  void *out;
  int64_t h, w;
  int64_t in_h, in_w;           // extent of the input (boundaries apply here)
  int64_t in_pitch, out_pitch;  // elements
  int ry, rx;
  int boundary;
  uint64_t cval;
  int accumulate;  // add onto out (second input of stencil2)
  int tma;
  uint32_t *err;
};

// RM: the largest radius this instantiation handles (ry, rx <= RM); PX: the
// halo width in x, RM rounded up to 16 bytes.
template <class T, int RM>
__global__ void __launch_bounds__(ST_THREADS)
stencil_kernel(const __grid_constant__ CUtensorMap tin, StencilArgs a, StencilW<T> W) {
  constexpr int PX = ((RM * (int)sizeof(T) + 15) / 16) * 16 / (int)sizeof(T);
  constexpr int SW = ST_TW + 2 * PX;   // smem tile width
  constexpr int SH = ST_TH + 2 * RM;   // smem tile height
  extern __shared__ unsigned char smem_raw[];
  T *tile = reinterpret_cast<T *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  __shared__ uint64_t bar;

  const int64_t tx0 = (int64_t)blockIdx.x * ST_TW, ty0 = (int64_t)blockIdx.y * ST_TH;
  const int64_t gx0 = tx0 - PX, gy0 = ty0 - RM;  // global coords of tile[0][0]
  const T *in = static_cast<const T *>(a.in);
  const bool border = gx0 < 0 || gy0 < 0 || gx0 + SW > a.in_w || gy0 + SH > a.in_h;

  if (a.tma) {
    if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      mbar_expect_tx(&bar, SW * SH * sizeof(T));
      tma_load_2d(tile, &tin, (int)gx0, (int)gy0, &bar);
    }
    if (__syncthreads_or(!mbar_wait_flagged(&bar, 0, a.err))) return;  // the tile never landed
    if (border) {
      // Overwrite the cells the TMA filled with zeros (outside the array).
      for (int k = threadIdx.x; k < SW * SH; k += ST_THREADS) {
        const int sy = k / SW, sx = k % SW;
        const int64_t gy = gy0 + sy, gx = gx0 + sx;
        if (gy >= 0 && gy < a.in_h && gx >= 0 && gx < a.in_w) continue;
        T v;
        if (a.boundary == ACC_CONSTANT) v = from_bits<T>(a.cval);
        else v = in[bound_index(gy, a.in_h, a.boundary) * a.in_pitch + bound_index(gx, a.in_w, a.boundary)];
        tile[sy * SW + sx] = v;
      }
    }
  } else {
    for (int k = threadIdx.x; k < SW * SH; k += ST_THREADS) {
      const int sy = k / SW, sx = k % SW;
      const int64_t gy = gy0 + sy, gx = gx0 + sx;
      T v;
      if (gy >= 0 && gy < a.in_h && gx >= 0 && gx < a.in_w) v = in[gy * a.in_pitch + gx];
      else if (a.boundary == ACC_CONSTANT) v = from_bits<T>(a.cval);
      else v = in[bound_index(gy, a.in_h, a.boundary) * a.in_pitch + bound_index(gx, a.in_w, a.boundary)];
      tile[sy * SW + sx] = v;
    }
  }
  __syncthreads();

  const int col = threadIdx.x % ST_TW;
  const int rg = threadIdx.x / ST_TW;
  const int oy0 = rg * ST_ROWS;  // first output row of this thread (tile coords)
  T acc[ST_ROWS];
  T *out = static_cast<T *>(a.out);
  const int64_t gx = tx0 + col;
#pragma unroll
  for (int r = 0; r < ST_ROWS; ++r) {
    const int64_t gy = ty0 + oy0 + r;
    if (a.accumulate && gy < a.h && gx < a.w) acc[r] = out[gy * a.out_pitch + gx];
    else acc[r] = Prim<ACC_ADD, T>::id();
  }
  const int ry = a.ry, rx = a.rx;
  const int KW = 2 * rx + 1;
  // Input rows oy0-ry .. oy0+ST_ROWS-1+ry (tile coords, offset by RM).
#pragma unroll
  for (int ir = 0; ir < ST_ROWS + 2 * RM; ++ir) {
    const int iy = oy0 + ir - RM;       // input row relative to the tile's first output row
    const int dyl = ir - RM;            // = iy - oy0
    if (dyl < -ry || dyl > ST_ROWS - 1 + ry) continue;
    T xv[2 * RM + 1];
#pragma unroll
    for (int dx = -RM; dx <= RM; ++dx)
      xv[dx + RM] = (dx >= -rx && dx <= rx) ? tile[(iy + RM) * SW + PX + col + dx] : T(0);
#pragma unroll
    for (int r = 0; r < ST_ROWS; ++r) {
      const int dy = dyl - r;  // this input row is tap row dy of output row r
      if (dy < -ry || dy > ry) continue;
#pragma unroll
      for (int dx = -RM; dx <= RM; ++dx) {
        if (dx < -rx || dx > rx) continue;
        const T wk = W.w[(dy + ry) * KW + (dx + rx)];
        if (wk == T(0)) continue;
        acc[r] = fma_tap(wk, xv[dx + RM], acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ST_ROWS; ++r) {
    const int64_t gy = ty0 + oy0 + r;
    if (gy < a.h && gx < a.w) out[gy * a.out_pitch + gx] = acc[r];
  }
}

// ----------------------------------------------------------------- second pass
// The second pass of stencil2 for the usual radii: the same computation from the
// accumulators in `out`, with the radii and the tap pattern known at compile time: PAT 0 = every tap has a non-zero weight, PAT 1 = the cross (5-point
// style: only the corners of the 3x3 are zero), PAT 2 = any pattern (each tap
// tested against a zero mask).  Tiles are 64 x 64 outputs, 16 rows per thread.
constexpr int SF_TW = 64, SF_TH = 64, SF_ROWS = 16;

template <class T, int RY, int RX, int PAT>
__global__ void __launch_bounds__(ST_THREADS, (sizeof(T) == 4 && RY * RX <= 1) ? 4 : 2)
stencil_onto_kernel(const __grid_constant__ CUtensorMap tin, StencilArgs a, StencilW<T> W, uint32_t zmask) {
  constexpr int PX = ((RX * (int)sizeof(T) + 15) / 16) * 16 / (int)sizeof(T) > 0
                         ? ((RX * (int)sizeof(T) + 15) / 16) * 16 / (int)sizeof(T) : 0;
  constexpr int SW = SF_TW + 2 * PX;
  constexpr int SH = SF_TH + 2 * RY;
  constexpr int KW = 2 * RX + 1;
  constexpr int NT = (2 * RY + 1) * KW;
  extern __shared__ unsigned char smem_raw[];
  T *tile = reinterpret_cast<T *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  __shared__ uint64_t bar;

  const int64_t tx0 = (int64_t)blockIdx.x * SF_TW, ty0 = (int64_t)blockIdx.y * SF_TH;
  const int64_t gx0 = tx0 - PX, gy0 = ty0 - RY;
  const T *in = static_cast<const T *>(a.in);
  const bool border = gx0 < 0 || gy0 < 0 || gx0 + SW > a.in_w || gy0 + SH > a.in_h;

  if (a.tma) {
    if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_expect_tx(&bar, SW * SH * sizeof(T));
      tma_load_2d(tile, &tin, (int)gx0, (int)gy0, &bar);
    }
    __syncthreads();
    if (__syncthreads_or(!mbar_wait_flagged(&bar, 0, a.err))) return;  // the tile never landed
    if (border) {
      for (int k = threadIdx.x; k < SW * SH; k += ST_THREADS) {
        const int sy = k / SW, sx = k % SW;
        const int64_t gy = gy0 + sy, gx = gx0 + sx;
        if (gy >= 0 && gy < a.in_h && gx >= 0 && gx < a.in_w) continue;
        tile[sy * SW + sx] = a.boundary == ACC_CONSTANT
                                 ? from_bits<T>(a.cval)
                                 : in[bound_index(gy, a.in_h, a.boundary) * a.in_pitch + bound_index(gx, a.in_w, a.boundary)];
      }
      __syncthreads();
    }
  } else {
    for (int k = threadIdx.x; k < SW * SH; k += ST_THREADS) {
      const int sy = k / SW, sx = k % SW;
      const int64_t gy = gy0 + sy, gx = gx0 + sx;
      T v;
      if (gy >= 0 && gy < a.in_h && gx >= 0 && gx < a.in_w) v = in[gy * a.in_pitch + gx];
      else if (a.boundary == ACC_CONSTANT) v = from_bits<T>(a.cval);
      else v = in[bound_index(gy, a.in_h, a.boundary) * a.in_pitch + bound_index(gx, a.in_w, a.boundary)];
      tile[sy * SW + sx] = v;
    }
    __syncthreads();
  }

  T w[NT];
#pragma unroll
  for (int k = 0; k < NT; ++k) w[k] = W.w[k];
  const int col = threadIdx.x % SF_TW;
  const int oy0 = (threadIdx.x / SF_TW) * SF_ROWS;
  T acc[SF_ROWS];
  T *out = static_cast<T *>(a.out);
  const int64_t gx = tx0 + col;
#pragma unroll
  for (int r = 0; r < SF_ROWS; ++r) {
    const int64_t gy = ty0 + oy0 + r;
    acc[r] = gy < a.h && gx < a.w ? out[gy * a.out_pitch + gx] : Prim<ACC_ADD, T>::id();
  }
  const T *trow = tile + oy0 * SW + PX + col;  // smem row oy0 - RY + RY = oy0 (halo offset)
#pragma unroll
  for (int ir = 0; ir < SF_ROWS + 2 * RY; ++ir) {
    T xv[KW];
#pragma unroll
    for (int dx = 0; dx < KW; ++dx) xv[dx] = trow[ir * SW + dx - RX];
#pragma unroll
    for (int dyi = 0; dyi < 2 * RY + 1; ++dyi) {
      const int r = ir - dyi;  // output row for which this input row is tap row dyi - RY
      if (r < 0 || r >= SF_ROWS) continue;
#pragma unroll
      for (int dx = 0; dx < KW; ++dx) {
        const int k = dyi * KW + dx;
        if constexpr (PAT == 1) {
          if (k == 0 || k == 2 || k == 6 || k == 8) continue;  // corners of the 3x3 cross
        }
        if constexpr (PAT == 2) {
          if ((zmask >> k) & 1u) continue;
        }
        acc[r] = fma_tap(w[k], xv[dx], acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < SF_ROWS; ++r) {
    const int64_t gy = ty0 + oy0 + r;
    if (gy < a.h && gx < a.w) out[gy * a.out_pitch + gx] = acc[r];
  }
}

template <class T, int RY, int RX, int PAT>
int stencil_onto_launch(StencilArgs a, const StencilW<T> &W, uint32_t zmask, cudaStream_t s) {
  constexpr int PX = ((RX * (int)sizeof(T) + 15) / 16) * 16 / (int)sizeof(T);
  constexpr int SW = SF_TW + 2 * PX;
  constexpr int SH = SF_TH + 2 * RY;
  const size_t smem = (size_t)SW * SH * sizeof(T) + 128;
  CUtensorMap tin;
  memset(&tin, 0, sizeof(tin));
  a.tma = encode_2d(&tin, a.in, sizeof(T), (uint64_t)a.in_w, (uint64_t)a.in_h, (uint64_t)a.in_pitch * sizeof(T),
                    SW, SH, false);
  auto kern = stencil_onto_kernel<T, RY, RX, PAT>;
  static std::atomic<uint64_t> attr_done{0};
  smem_attrs_once(kern, (int)smem, attr_done, false);
  const int64_t gx = cdiv_h(a.w, SF_TW), gy = cdiv_h(a.h, SF_TH);
  if (gy > 65535 || gx > (1ll << 31) - 1) return ACC_ERR_TOO_LARGE;
  kern<<<dim3((unsigned)gx, (unsigned)gy), ST_THREADS, smem, s>>>(tin, a, W, zmask);
  return check_launch();
}

// ----------------------------------------------------------------- row streaming
// Every call but the second pass of stencil2, radii up to 2 as instantiated
// below.  A warp owns a strip of 32 x E columns and SR_ROWS output rows, and
// reads the input rows of its range in increasing order straight into
// registers, `ahead` rows ahead; a row's neighbours left and right come from
// the other lanes by shuffle, and each lane keeps the accumulators of the
// 2 RY + 1 output rows that an input row is a tap row of, rotating by the
// unrolled row loop.  No shared memory and no barrier: a warp waits only for
// its own loads.  Every output accumulates its taps rows outer, then columns,
// one fused multiply-add each.  Warps whose halo leaves the array take their
// rows through the boundary rule, one at a time.
//
// Bound: HBM (3x3), issue (5x5).  Measured on a GB300, Float32 8192 x 8192
// (floor 79 us) against halo tiles through shared memory in a two-stage TMA
// pipeline with barriers (and, for 8191 x 8191, which TMA cannot describe, one
// tile per CTA read element by element): 3x3 108 -> 86 us, 5x5 153 -> 129 us;
// 8191 x 8191 360 -> 101 us and 644 -> 164 us.
// Few rows per warp: neighbouring warps then work on neighbouring rows, which
// DRAM and L2 reward (3x3: 10 rows 86 us, 20 rows 90, 64 rows 117, 144 rows --
// whole waves of warps -- 147), against the 2 RY rows that adjacent warps
// both read.  Two warps per CTA, so that a slot is refilled as soon as they end
// (256 threads: 95 us at 16 rows against 90).  Registers: 72 (14 CTAs per SM)
// for 16-byte rows; the strided form needs 91 (10) and takes 9 rows ahead (6
// rows ahead: 105 us).  Float32 taps in pairs (fma.rn.f32x2) were slower (129
// us): the weights then live in registers, twice.
constexpr int SR_THREADS = 64;
template <int RY, bool VEC> constexpr int sr_ahead() { return RY == 0 ? 4 : RY == 2 ? 5 : VEC ? 6 : 9; }  // of 2 RY + 1
template <class T, int RY, bool VEC> constexpr int sr_ctas() {  // 8-byte types: registers without spills
  return sizeof(T) == 8 ? (RY == 2 ? 5 : 8) : RY == 2 ? 8 : VEC ? 14 : 10;
}
// 8-byte types are bound by their multiply-adds, of which the rows that two warps share cost some
// twice; Int64 less so (3x3, 4096 x 4096: 16 rows 72 us, 24 72, 32 74, 48 77)
template <class T, int RY, bool VEC> constexpr int sr_rows() {
  if (std::is_same<T, int64_t>::value && RY > 0) return 24;
  return sizeof(T) == 8 ? (RY == 2 ? 96 : 32) : RY == 2 ? 20 : VEC ? 10 : 12;
}

// One input row (window `win`) applied to the accumulators, whose roles start
// at slot I: output row r - RY + k takes input row r as its tap row 2 RY - k.
template <class T, int RY, int RX, int PAT, int I, int E>
__device__ __forceinline__ void rows_apply(const StencilW<T> &W, uint32_t zmask, const T (&win)[2 * RX + 1][E],
                                           T (&acc)[2 * RY + 1][E]) {
  constexpr int K = 2 * RY + 1, KW = 2 * RX + 1;
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int dx = 0; dx < KW; ++dx) {
      const int q = (2 * RY - k) * KW + dx;
      if constexpr (PAT == 1) {
        if (q == 0 || q == 2 || q == 6 || q == 8) continue;
      }
      if constexpr (PAT == 2) {
        if ((zmask >> q) & 1u) continue;
      }
#pragma unroll
      for (int e = 0; e < E; ++e) acc[(k + I) % K][e] = fma_tap(W.w[q], win[dx][e], acc[(k + I) % K][e]);
    }
}
// f(std::integral_constant<int, 0>()) ... f(N - 1) until f returns false.
template <int N, int I = 0, class F> __device__ __forceinline__ bool rows_unroll(F &&f) {
  if constexpr (I < N) {
    if (!f(std::integral_constant<int, I>())) return false;
    return rows_unroll<N, I + 1>(f);
  } else {
    return true;
  }
}

template <class T, int RY, int RX, int PAT, bool VEC>
__global__ void __launch_bounds__(SR_THREADS, sr_ctas<T, RY, VEC>())
stencil_rows_kernel(const __grid_constant__ StencilArgs a, const __grid_constant__ StencilW<T> W, uint32_t zmask,
                    int64_t strips, int rows) {
  using S = Strip<T, RX, VEC>;
  using Row = typename S::Row;
  constexpr int E = S::E, K = 2 * RY + 1, KW = 2 * RX + 1, D = sr_ahead<RY, VEC>();
  static_assert(D % K == 0, "the accumulators' roles rotate with the unrolled loop");
  const int64_t gw = (int64_t)blockIdx.x * (SR_THREADS / 32) + (threadIdx.x >> 5);
  const int64_t x0 = gw % strips * (32 * E), y0 = gw / strips * rows;
  if (y0 >= a.h) return;
  const int64_t y1 = y0 + rows < a.h ? y0 + rows : a.h;
  S strip;
  strip.init(x0, a.in_w, a.boundary, from_bits<T>(a.cval));
  T acc[K][E];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int e = 0; e < E; ++e) acc[k][e] = Prim<ACC_ADD, T>::id();
  const int n = (int)(y1 - y0) + 2 * RY;  // input rows y0 - RY ..; output row y0 + t - 2 RY is complete after row t
  T *o = static_cast<T *>(a.out) + (y0 - 2 * RY) * a.out_pitch;
  if (x0 >= RX && x0 + 32 * E + RX <= a.in_w && y0 >= RY && y1 + RY <= a.in_h) {
    const T *first = static_cast<const T *>(a.in) + (y0 - RY) * a.in_pitch;
    const T *p = first + strip.inner_column(x0), *h = first + strip.inner_halo(x0);
    Row ring[D];
#pragma unroll
    for (int i = 0; i < D; ++i)
      if (i < n) {
        strip.load_inner(p, h, ring[i]);
        p += a.in_pitch;
        h += a.in_pitch;
      }
    for (int t0 = 0; t0 < n; t0 += D) {
      const bool go = rows_unroll<D>([&](auto ic) -> bool {
        constexpr int I = decltype(ic)::value;
        const int t = t0 + I;
        if (t >= n) return false;
        T win[KW][E];
        strip.window(ring[I], win);
        if (t + D < n) {
          strip.load_inner(p, h, ring[I]);
          p += a.in_pitch;
          h += a.in_pitch;
        }
        rows_apply<T, RY, RX, PAT, I % K, E>(W, zmask, win, acc);
        if (t >= 2 * RY) strip.store(o, x0, a.w, acc[I % K]);
        o += a.out_pitch;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[I % K][e] = Prim<ACC_ADD, T>::id();
        return true;
      });
      if (!go) break;
    }
    return;
  }
  for (int t0 = 0; t0 < n; t0 += K) {
    const bool go = rows_unroll<K>([&](auto ic) -> bool {
      constexpr int I = decltype(ic)::value;
      const int t = t0 + I;
      if (t >= n) return false;
      const int64_t r = y0 - RY + t;
      const bool yin = r >= 0 && r < a.in_h;
      Row row;
      if (!yin && a.boundary == ACC_CONSTANT) strip.fill(row);
      else strip.load(static_cast<const T *>(a.in) + (yin ? r : bound_index(r, a.in_h, a.boundary)) * a.in_pitch, row);
      T win[KW][E];
      strip.window(row, win);
      rows_apply<T, RY, RX, PAT, I, E>(W, zmask, win, acc);
      if (t >= 2 * RY) strip.store(o, x0, a.w, acc[I]);
      o += a.out_pitch;
#pragma unroll
      for (int e = 0; e < E; ++e) acc[I][e] = Prim<ACC_ADD, T>::id();
      return true;
    });
    if (!go) break;
  }
}

template <class T, int RY, int RX, int PAT, bool VEC>
static int stencil_rows_on(const StencilArgs &a, const StencilW<T> &W, uint32_t zmask, cudaStream_t s) {
  constexpr int WARPS = SR_THREADS / 32;
  const int64_t strips = cdiv_h(a.w, 32 * (16 / (int)sizeof(T)));
  // Whole waves of resident warps, as few as keep a warp's rows within sr_rows
  // (one wave, and fewer rows, where the array is small).
  const int64_t resident = (int64_t)device_info().sms * sr_ctas<T, RY, VEC>() * WARPS;
  const int64_t waves = cdiv_h(strips * a.h, resident * sr_rows<T, RY, VEC>());
  const int64_t rows = cdiv_h(strips * a.h, resident * waves);
  const int64_t grid = cdiv_h(strips * cdiv_h(a.h, rows), WARPS);
  if (grid > 0x7fffffffll) return ACC_ERR_TOO_LARGE;
  stencil_rows_kernel<T, RY, RX, PAT, VEC><<<(unsigned)grid, SR_THREADS, 0, s>>>(a, W, zmask, strips, (int)rows);
  return check_launch();
}
template <class T, int RY, int RX, int PAT>
static int stencil_rows_launch(const StencilArgs &a, const StencilW<T> &W, uint32_t zmask, cudaStream_t s) {
  // 16-byte loads and stores: every row of both arrays starts on a 16-byte boundary.
  constexpr int E = 16 / (int)sizeof(T);
  const bool vec = aligned16(a.in) && aligned16(a.out) && a.w % E == 0 && a.in_w % E == 0 && a.in_pitch % E == 0 &&
                   a.out_pitch % E == 0;
  // Int64 3x3 and 5x5 take single loads all the same: 4096 x 4096 107 -> 73 us and 206 -> 163,
  // 8192 x 8192 370 -> 233 and 657 -> 573, from 2048 x 2048 down alike (more rows ahead in 16-byte
  // loads, 9 to 15, 97 to 117 us; 10 CTAs per SM 87).
  if constexpr (!(std::is_same<T, int64_t>::value && RY > 0 && RX > 0)) {
    if (vec) return stencil_rows_on<T, RY, RX, PAT, true>(a, W, zmask, s);
  }
  return stencil_rows_on<T, RY, RX, PAT, false>(a, W, zmask, s);
}

template <class T, int RY, int RX>
int stencil_pat(StencilArgs a, const StencilW<T> &W, cudaStream_t s) {
  constexpr int NT = (2 * RY + 1) * (2 * RX + 1);
  static_assert(NT <= 32, "one mask word");
  uint32_t zeros = 0;  // bit k: the weight of tap k is zero
  for (int k = 0; k < NT; ++k)
    if (W.w[k] == T(0)) zeros |= 1u << k;
  auto pattern = [&](auto pat) {
    constexpr int PAT = decltype(pat)::value;
    return a.accumulate ? stencil_onto_launch<T, RY, RX, PAT>(a, W, zeros, s)
                        : stencil_rows_launch<T, RY, RX, PAT>(a, W, zeros, s);
  };
  if (zeros == 0) return pattern(IC<0>{});
  if constexpr (RY == 1 && RX == 1) {
    if (zeros == ((1u << 0) | (1u << 2) | (1u << 6) | (1u << 8))) return pattern(IC<1>{});
  }
  return pattern(IC<2>{});
}

// ----------------------------------------------------------------- host side
template <class T, int RM>
int stencil_launch(StencilArgs a, const StencilW<T> &W, cudaStream_t s) {
  constexpr int PX = ((RM * (int)sizeof(T) + 15) / 16) * 16 / (int)sizeof(T);
  constexpr int SW = ST_TW + 2 * PX;
  constexpr int SH = ST_TH + 2 * RM;
  const size_t smem = (size_t)SW * SH * sizeof(T) + 128;
  CUtensorMap tin;
  memset(&tin, 0, sizeof(tin));
  a.tma = encode_2d(&tin, a.in, sizeof(T), (uint64_t)a.in_w, (uint64_t)a.in_h, (uint64_t)a.in_pitch * sizeof(T),
                    SW, SH, false);
  auto kern = stencil_kernel<T, RM>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int64_t gx = cdiv_h(a.w, ST_TW), gy = cdiv_h(a.h, ST_TH);
  if (gy > 65535 || gx > (1ll << 31) - 1) return ACC_ERR_TOO_LARGE;
  kern<<<dim3((unsigned)gx, (unsigned)gy), ST_THREADS, smem, s>>>(tin, a, W);
  return check_launch();
}

template <class T>
int stencil_typed(StencilArgs a, const void *weights, cudaStream_t s) {
  StencilW<T> W;
  const int nw = (2 * a.ry + 1) * (2 * a.rx + 1);
  memset(&W, 0, sizeof(W));
  memcpy(W.w, weights, (size_t)nw * sizeof(T));
  if (a.ry == 1 && a.rx == 1) return stencil_pat<T, 1, 1>(a, W, s);
  if (a.ry == 0 && a.rx == 1) return stencil_pat<T, 0, 1>(a, W, s);
  if (a.ry == 1 && a.rx == 0) return stencil_pat<T, 1, 0>(a, W, s);
  if (a.ry == 2 && a.rx == 2) return stencil_pat<T, 2, 2>(a, W, s);
  const int r = a.ry > a.rx ? a.ry : a.rx;
  if (r <= 1) return stencil_launch<T, 1>(a, W, s);
  if (r <= 2) return stencil_launch<T, 2>(a, W, s);
  return stencil_launch<T, 4>(a, W, s);
}

static int stencil_dispatch(int type, StencilArgs a, const void *weights, cudaStream_t s) {
  switch (type) {
    case ACC_F32: return stencil_typed<float>(a, weights, s);
    case ACC_F64: return stencil_typed<double>(a, weights, s);
    case ACC_I32: return stencil_typed<int32_t>(a, weights, s);
    case ACC_I64: return stencil_typed<int64_t>(a, weights, s);
    default: return ACC_ERR_UNSUPPORTED;
  }
}

static int stencil_check(int type, int ry, int rx, int boundary, const void *cval, int64_t h, int64_t w) {
  if (ry < 0 || ry > 4 || rx < 0 || rx > 4) return ACC_ERR_INVALID;
  if (h < 0 || w < 0) return ACC_ERR_INVALID;
  if (boundary < ACC_CLAMP || boundary > ACC_CONSTANT) return ACC_ERR_INVALID;
  if (boundary == ACC_CONSTANT && !cval) return ACC_ERR_INVALID;
  if (type != ACC_F32 && type != ACC_F64 && type != ACC_I32 && type != ACC_I64) return ACC_ERR_UNSUPPORTED;
  return ACC_OK;
}

}  // namespace accgb

using namespace accgb;

extern "C" int acc_stencil2d(int type, int ry, int rx, const void *weights, int boundary, const void *cval,
                             const void *in, void *out, int64_t h, int64_t w, void *stream) {
  int st = stencil_check(type, ry, rx, boundary, cval, h, w);
  if (st) return st;
  if (h == 0 || w == 0) return ACC_OK;
  if (!weights || !in || !out) return ACC_ERR_INVALID;
  StencilArgs a{};
  a.in = in; a.out = out; a.h = h; a.w = w; a.in_h = h; a.in_w = w; a.in_pitch = w; a.out_pitch = w;
  a.ry = ry; a.rx = rx; a.boundary = boundary;
  a.cval = 0;
  if (cval) memcpy(&a.cval, cval, (type == ACC_F64 || type == ACC_I64) ? 8 : 4);
  a.accumulate = 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Workspace *ws = workspace(s, &st);
  if (!ws) return st;
  a.err = ws->words + W_ERR;
  return stencil_dispatch(type, a, weights, s);
}

extern "C" int acc_stencil2d_pair(int type, int ry, int rx, const void *wa_w, const void *wb_w, int boundary_a,
                                  const void *cval_a, int boundary_b, const void *cval_b, const void *a_in,
                                  int64_t ha, int64_t wa, const void *b_in, int64_t hb, int64_t wb, void *out,
                                  void *stream) {
  int st = stencil_check(type, ry, rx, boundary_a, cval_a, ha, wa);
  if (st) return st;
  st = stencil_check(type, ry, rx, boundary_b, cval_b, hb, wb);
  if (st) return st;
  const int64_t h = ha < hb ? ha : hb, w = wa < wb ? wa : wb;
  if (h == 0 || w == 0) return ACC_OK;
  if (!wa_w || !wb_w || !a_in || !b_in || !out) return ACC_ERR_INVALID;
  // The second pass's grid, refused before the first pass writes.
  if (cdiv_h(h, SF_TH) > 65535 || cdiv_h(w, SF_TW) > (1ll << 31) - 1) return ACC_ERR_TOO_LARGE;
  const size_t esz = (type == ACC_F64 || type == ACC_I64) ? 8 : 4;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Workspace *ws = workspace(s, &st);
  if (!ws) return st;
  // Pass 1 evaluates the taps of a; pass 2 continues the same accumulator
  // (read back from out) with the taps of b.  The accumulator is rounded to
  // the element type after every tap either way, so the two passes give the
  // bits of one fused sweep.
  StencilArgs a{};
  a.err = ws->words + W_ERR;
  a.in = a_in; a.out = out; a.h = h; a.w = w; a.in_h = ha; a.in_w = wa; a.in_pitch = wa; a.out_pitch = w;
  a.ry = ry; a.rx = rx; a.boundary = boundary_a; a.cval = 0;
  if (cval_a) memcpy(&a.cval, cval_a, esz);
  a.accumulate = 0;
  st = stencil_dispatch(type, a, wa_w, s);
  if (st) return st;
  a.in = b_in; a.in_h = hb; a.in_w = wb; a.in_pitch = wb; a.boundary = boundary_b; a.cval = 0;
  if (cval_b) memcpy(&a.cval, cval_b, esz);
  a.accumulate = 1;
  return stencil_dispatch(type, a, wb_w, s);
}
