// foldseg.cu -- foldSeg f z / fold1Seg f over a segment-offset array.
//
// The reference picks ONE kernel for the whole array from the average
// segment length: a warp per segment or a CTA per segment
// (accelerate-llvm-ptx/src/Data/Array/Accelerate/LLVM/PTX/Execute.hs:343-374,
// PTX/CodeGen/FoldSeg.hs:79-458), so skewed (lognormal) lengths leave most
// lanes idle or most CTAs waiting on a few long segments.  Here:
//   * a 1-D row with 16-byte aligned values goes through foldseg_tile_kernel,
//     one launch that cuts the VALUES into equal tiles whatever the segment
//     lengths (see "tiled single pass" below);
//   * other shapes (rank >= 2, unaligned values) dispatch each segment by its
//     own length, in two launches:
//       1. seg_classify lists the segments longer than LONG_SEG (atomic
//          append; the order of the list does not matter, each segment is
//          reduced alone);
//       2. foldseg_main: the first CTAs stream the listed long segments, one
//          CTA per segment with 16-byte vector loads; every other warp owns 32
//          consecutive segments and reduces the short ones (<= SHORT_SEG) one
//          per lane, serially, and the medium ones with the whole warp.
// Per segment the result is z `f` (x_u `f` ... `f` x_(v-1)), as the native
// backend's reduceFromTo over [seg[i], seg[i+1]) (accelerate-llvm-native/src/
// Data/Array/Accelerate/LLVM/Native/CodeGen/FoldSeg.hs:103-141).  An empty
// segment gives z with a seed and is left unwritten without one
// (PTX/CodeGen/FoldSeg.hs:170-178).  Offsets that decrease or run past the
// row raise ACC_ERR_INDEX instead of reading out of bounds.
#include <cstdlib>
#include <cstring>

#include "common.cuh"

namespace accgb {

constexpr int SHORT_SEG = 32;
constexpr int64_t LONG_SEG = 2048;

struct SegArgs {
  const void *in;
  const void *off;
  void *out;
  int64_t outer, inner, nseg;
  int off64;
  uint64_t seed;
  int has_seed;
  uint32_t *nlong;     // number of listed long segments
  int64_t *longs;      // listed long segment ids
  int64_t long_ctas;   // CTAs [0, long_ctas) work on the list
  int64_t long_cap;    // capacity of the list
  uint32_t *err;
  const void *in2;     // ZIP kernels: the folded element i is zop(in[i], in2[i])
  int zop;
};

__device__ __forceinline__ int64_t seg_off(const SegArgs &a, int64_t i) {
  return a.off64 ? static_cast<const int64_t *>(a.off)[i] : (int64_t) static_cast<const int32_t *>(a.off)[i];
}

__global__ void seg_classify(SegArgs a) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < a.nseg; s += (int64_t)gridDim.x * blockDim.x) {
    const int64_t u = seg_off(a, s), v = seg_off(a, s + 1);
    if (v - u > LONG_SEG && u >= 0 && v <= a.inner) {
      const uint32_t k = atomicAdd(a.nlong, 1u);
      // Valid offsets give at most inner / LONG_SEG long segments; overlapping
      // (malformed) offsets could give more: never write past the list.
      if ((int64_t)k >= a.long_cap) { raise_error(a.err, DEV_ERR_INDEX); continue; }
      a.longs[k] = s;
    }
  }
}

// Same vector streaming as the fold kernels, 4 x 16 B in flight per thread.
template <class A, class T>
__device__ __forceinline__ typename A::S seg_span(const T *p, int64_t len, int64_t t, int64_t nt) {
  using S = typename A::S;
  constexpr int VEC = 16 / sizeof(T);
  S acc = A::id();
  const uintptr_t addr = reinterpret_cast<uintptr_t>(p);
  int64_t head = (int64_t)(((16u - (addr & 15u)) & 15u) / sizeof(T));
  if (head > len) head = len;
  if (t < head) acc = A::push(acc, ld_stream(p + t));
  const int64_t nvec = (len - head) / VEC;
  const uint4 *qv = reinterpret_cast<const uint4 *>(p + head);
  int64_t i = t;
  for (; i + 3 * nt < nvec; i += 4 * nt) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = ld_stream16(qv + i + u * nt);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      T e[VEC];
      memcpy(e, &v[u], 16);
#pragma unroll
      for (int k = 0; k < VEC; ++k) acc = A::push(acc, e[k]);
    }
  }
  for (; i < nvec; i += nt) {
    uint4 v = ld_stream16(qv + i);
    T e[VEC];
    memcpy(e, &v, 16);
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc = A::push(acc, e[k]);
  }
  const int64_t tail0 = head + nvec * VEC;
  if (tail0 + t < len) acc = A::push(acc, ld_stream(p + tail0 + t));
  return acc;
}

// seg_span over the fused producer zipWith zop p q: the vector body when p
// and q share their 16-byte alignment phase, a scalar stride otherwise.
template <class A, class T>
__device__ __forceinline__ typename A::S seg_span_zip(const T *p, const T *q, int zop, int64_t len, int64_t t,
                                                      int64_t nt) {
  using S = typename A::S;
  constexpr int VEC = 16 / sizeof(T);
  S acc = A::id();
  const uintptr_t addr = reinterpret_cast<uintptr_t>(p);
  if (((addr ^ reinterpret_cast<uintptr_t>(q)) & 15u) != 0u) {
    for (int64_t i = t; i < len; i += nt) acc = A::push(acc, zip_elem(zop, ld_stream(p + i), ld_stream(q + i)));
    return acc;
  }
  int64_t head = (int64_t)(((16u - (addr & 15u)) & 15u) / sizeof(T));
  if (head > len) head = len;
  if (t < head) acc = A::push(acc, zip_elem(zop, ld_stream(p + t), ld_stream(q + t)));
  const int64_t nvec = (len - head) / VEC;
  const uint4 *pv = reinterpret_cast<const uint4 *>(p + head);
  const uint4 *qv = reinterpret_cast<const uint4 *>(q + head);
  for (int64_t i = t; i < nvec; i += nt) {
    const uint4 v = ld_stream16(pv + i), w = ld_stream16(qv + i);
    T e[VEC], f[VEC];
    memcpy(e, &v, 16);
    memcpy(f, &w, 16);
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc = A::push(acc, zip_elem(zop, e[k], f[k]));
  }
  const int64_t tail0 = head + nvec * VEC;
  if (tail0 + t < len) acc = A::push(acc, zip_elem(zop, ld_stream(p + tail0 + t), ld_stream(q + tail0 + t)));
  return acc;
}

// With ZIP the folded array is the fused producer zipWith zop in in2.
template <int OP, class T, int PREC, bool ZIP = false>
__global__ void __launch_bounds__(256) foldseg_main(SegArgs a) {
  using A = Acc<OP, T, PREC>;
  using S = typename A::S;
  const T *in = static_cast<const T *>(a.in);
  const T *in2 = static_cast<const T *>(a.in2);
  (void)in2;
  // Element i of row r, and the fold of a span of row r.
  auto elem = [&](const T *row, const T *row2, int64_t i) -> T {
    if constexpr (ZIP) return zip_elem(a.zop, row[i], row2[i]);
    else { (void)row2; return row[i]; }
  };
  auto span = [&](const T *row, const T *row2, int64_t len, int64_t t, int64_t nt) -> S {
    if constexpr (ZIP) return seg_span_zip<A, T>(row, row2, a.zop, len, t, nt);
    else { (void)row2; return seg_span<A, T>(row, len, t, nt); }
  };
  T *out = static_cast<T *>(a.out);
  const int lane = threadIdx.x & 31;
  __shared__ S s_part[8];

  if ((int64_t)blockIdx.x < a.long_ctas) {
    // ---- long segments: one CTA per (row, listed segment)
    int64_t nl = (int64_t)ld_relaxed_u32(a.nlong);
    if (nl > a.long_cap) nl = a.long_cap;
    for (int64_t job = blockIdx.x; job < nl * a.outer; job += a.long_ctas) {
      const int64_t r = job / nl, s = a.longs[job % nl];
      const int64_t u = seg_off(a, s), v = seg_off(a, s + 1);
      S acc = span(in + r * a.inner + u, ZIP ? in2 + r * a.inner + u : nullptr, v - u, threadIdx.x, blockDim.x);
      acc = warp_reduce<A>(acc);
      if (lane == 0) s_part[threadIdx.x >> 5] = acc;
      __syncthreads();
      if (threadIdx.x == 0) {
        S t = s_part[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = A::comb(t, s_part[w]);
        if (a.has_seed) t = A::comb(A::lift(from_bits<T>(a.seed)), t);
        out[r * a.nseg + s] = A::lower(t);
      }
      __syncthreads();
    }
    return;
  }

  // ---- short and medium segments: a warp per group of 32 segments
  const int64_t groups = (a.nseg + 31) / 32;
  const int64_t gw = (((int64_t)blockIdx.x - a.long_ctas) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (((int64_t)gridDim.x - a.long_ctas) * blockDim.x) >> 5;
  for (int64_t job = gw; job < groups * a.outer; job += nw) {
    const int64_t r = job / groups, g = job % groups;
    const int64_t s = g * 32 + lane;
    const T *row = in + r * a.inner;
    const T *row2 = ZIP ? in2 + r * a.inner : nullptr;
    int64_t u = 0, v = 0;
    bool valid = s < a.nseg;
    if (valid) {
      u = seg_off(a, s);
      v = seg_off(a, s + 1);
      if (u < 0 || v < u || v > a.inner) {
        raise_error(a.err, DEV_ERR_INDEX);
        valid = false;
      }
    }
    const int64_t len = valid ? v - u : 0;
    // short: this lane alone, left to right from the seed
    if (valid && len <= SHORT_SEG) {
      if (len > 0 || a.has_seed) {
        S acc;
        int64_t i = u;
        if (a.has_seed) acc = A::lift(from_bits<T>(a.seed));
        else acc = A::lift(elem(row, row2, i++));
        for (; i < v; ++i) acc = A::push(acc, elem(row, row2, i));
        out[r * a.nseg + s] = A::lower(acc);
      }
    }
    // medium: the whole warp, one segment at a time
    unsigned med = __ballot_sync(0xffffffffu, valid && len > SHORT_SEG && len <= LONG_SEG);
    while (med) {
      const int src = __ffs(med) - 1;
      med &= med - 1;
      const int64_t mu = __shfl_sync(0xffffffffu, u, src);
      const int64_t mv = __shfl_sync(0xffffffffu, v, src);
      S acc = span(row + mu, ZIP ? row2 + mu : nullptr, mv - mu, lane, 32);
      acc = warp_reduce<A>(acc);
      if (lane == 0) {
        if (a.has_seed) acc = A::comb(A::lift(from_bits<T>(a.seed)), acc);
        out[r * a.nseg + g * 32 + src] = A::lower(acc);
      }
    }
  }
}

// ----------------------------------------------------------------- tiled single pass
// 1-D rows with 16-byte aligned values take this path.  The values are cut
// into tiles of 256 rows x 128 B (one 2-D TMA load per 128 rows, 128-byte
// swizzle, as in the scan; each thread owns two adjacent rows), independent of the segment lengths, so every CTA streams the
// same number of bytes however skewed the segmentation is:
//   * a pre-pass (foldseg_tile_index) records for every tile the index of
//     the first offset at or after its start, so a tile knows its offset
//     range [kf, ks) from two loads; the CTA copies those offsets
//     (tile-relative) to shared memory, writing z for the empty segments on
//     the way;
//   * each thread walks its 256 bytes once: a segment boundary inside them
//     closes the segment that was open, whose state the row parks in shared
//     memory when it also saw that segment start; the value before the row's
//     first boundary and after its last one are carried out;
//   * a segmented CTA scan ((f1,v1).(f2,v2) = (f1|f2, f2 ? v2 : v1 `f` v2))
//     gives every row the value carried in from earlier rows of the tile, and
//     the tile's own carried-out value (flag 2 when the tile holds a boundary,
//     1 when it lies inside one segment);
//   * the parked results are written out in one coalesced pass, except the
//     segment that closes at the tile's first boundary, which also needs the
//     values carried in from earlier tiles: its part goes to the tile's slot
//     with the carried-out value, and foldseg_fix completes those segments from
//     the slots, each from the nearest earlier tile that holds a boundary
//     (usually the previous one).
// An extra tile past the last value closes the segments that end at the very
// end of the row.  Three launches: the index pre-pass, the tiles and the
// completion (two where the last tile takes that over); one for short calls.  Offsets that decrease or leave [0, n] raise
// ACC_ERR_INDEX; of a tile that holds such offsets only the z of empty segments may
// have been written, inside of the output.
// Bound: issue (about 30 thread instructions per value, compensated).  A tile
// that completed its first segment itself, by a decoupled look-back, held its
// shared memory for 7,400 cycles of polls and 2,100 of drawing a ticket, of
// 19,800 (2^22 values); the tiles now wait for no one.  2^26 Float32 values in
// 2^20 lognormal segments, compensated: 115 -> 92 us, plain 88 -> 76, Int32 max
// 88 -> 76 (the index pre-pass is about 5 of them, the completion 3).
// DENSE: the tiles of short segments (see ft_dense), 256 threads with one row.
template <bool DENSE = false> constexpr int ft_threads() { return DENSE ? 256 : 128; }
constexpr int FT_ROW_BYTES = 128;
// Tile-relative offsets (and their results) held in shared memory: the walk by
// boundary slots needs all of a tile's, so segments of 11 values and more on
// average take it; 768 is what leaves five CTAs per SM.  With 512, 2^26 Float32
// values in segments of 16 took 179 us (now 126).
constexpr int FT_CAP = 768;
// Adjacent 128-byte rows per thread: two, so that a thread's share of the tile's
// bookkeeping and scans (about as much as the walk of one row) is spread over 64
// 4-byte values, with 128 threads, so that five tiles still fit an SM.  256
// threads with one row (compensated) or two: 100 us where this takes 92, plain 74
// (76), 2^26 Int32 values in segments of 16 231 (110: 16,384 values have more
// boundaries than are kept), 2^25 Float64 140 (116).
// Over a fused zipWith each tile needs the rows of both arrays: one row each.
template <bool ZIP, bool DENSE = false> constexpr int ft_rpt() { return ZIP || DENSE ? 1 : 2; }

// Segments of fewer than 11 values on average leave a tile more offsets than are
// kept, and its threads walk value by value; a thread then carries a compensated
// state over one row only (2^24 Float32 values, compensated, against two: segments of
// 2 197 -> 121 us, of 6 94 -> 66, of 10 73 -> 56, of 12 39 and 41; other states gain nothing).
template <class S> constexpr bool ft_dense() { return std::is_same<S, F2>::value; }

struct SegTileArgs {
  const void *in;
  const void *in2;  // ZIP: the folded element i is zop(in[i], in2[i])
  int zop;
  const void *off;
  void *out;
  int64_t n, nseg;
  int64_t full_rows, ntiles;
  uint64_t seed;
  int has_seed;
  struct SegSlot *slots;  // per tile
  const uint64_t *tidx;  // per tile: epoch tag << 35 | first offset index >= the tile start; small: unused
  int small;             // 1: the CTA keeps all the offsets in shared memory; 2: and scans them from the lengths
  int finish;      // the last tile to get there completes the segments that cross tiles
  uint32_t *done;  // finish: tiles finished (zero between calls)
  uint32_t *err;
  uint32_t epoch;
};

// What a tile leaves for the segments that cross its edges.
struct __align__(16) SegSlot {
  uint64_t carry;    // state carried out to the right (bits)
  uint64_t first;    // state of the part before the tile's first boundary
  int64_t first_id;  // the segment that closes there, or -1
  int64_t boundary;  // 1: the tile holds a boundary, so its carry starts inside it
};

constexpr int TIDX_SHIFT = 35;  // offset indices below 2^35; the epoch above

// Short calls (at most FT_SMALL segments, at most two tiles per SM) take one
// launch: each CTA reads all the offsets (or the lengths, which it scans) into
// shared memory and finds its tile's first and last offset by counting.
// 100,003 Int32 values in 1,562 segments by lengths, device time: 23.4 us in
// three launches (scan of the lengths, index, tiles) -> 11.1; by offsets 17.0
// -> 11.1.  At the limits, 10^6 Float32 values: 4,000 segments by offsets 14.8 ->
// 13.2 us, 15,625 segments (three launches) 15.0 -> 12.1.
constexpr int FT_SMALL = 4096;
// most offsets per thread
template <bool DENSE> constexpr int ft_per() { return (FT_SMALL + ft_threads<DENSE>()) / ft_threads<DENSE>(); }
static_assert(ft_per<false>() % 2 == 1 && ft_per<false>() * ft_threads<false>() >= FT_SMALL + 1 &&
                  ft_per<true>() % 2 == 1 && ft_per<true>() * ft_threads<true>() >= FT_SMALL + 1,
              "an odd number (free of bank conflicts) holds them all");

// Pre-pass: tidx[t] = the first k with off[k] >= t << log_te (t < ntiles), and
// tidx[ntiles] = nseg + 1, each tagged with the call's epoch so that no
// clearing is needed.  Thread k writes the tiles whose start lies in
// (off[k-1], off[k]]; k = nseg + 1 stands for the tiles past the last offset.
// Decreasing offsets leave tiles unwritten (their stale tag is caught later).
template <class OT>
__global__ void foldseg_tile_index(const OT *off, int64_t nseg, int64_t ntiles, int log_te, uint64_t *tidx,
                                   uint32_t epoch) {
  const uint64_t tag = (uint64_t)epoch << TIDX_SHIFT;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k <= nseg + 1;
       k += (int64_t)gridDim.x * blockDim.x) {
    int64_t t0, t1;  // tiles [t0, t1] get k
    if (k == 0) t0 = 0;
    else {
      const int64_t lo = (int64_t)off[k - 1];
      t0 = lo < 0 ? 0 : (lo >> log_te) + 1;
    }
    if (k == nseg + 1) t1 = ntiles - 1;
    else {
      const int64_t hi = (int64_t)off[k];
      t1 = hi < 0 ? -1 : hi >> log_te;
    }
    if (t1 > ntiles - 1) t1 = ntiles - 1;
    for (int64_t t = t0; t <= t1; ++t) tidx[t] = tag | (uint64_t)k;
    if (k == nseg + 1) tidx[ntiles] = tag | (uint64_t)k;
  }
}

// Complete the segment that closes at the first boundary of tile t0 + lane, for
// 32 tiles (warp-collective): the carried-out values of the tiles since the
// nearest earlier boundary, then the tile's own first part.  The previous tile
// usually holds that boundary.  Where it does not, a segmented scan over the warp
// finds it within the 32, and one walk back over the slots before them serves all
// that are open there: 32 slots at a time and, where all NT threads of a CTA call
// (NT > 0), after 128 by the CTA together, 8 NT at a time.  One segment of 2^26 values
// is 8192 tiles: 203 -> 110 us of device time (Float32, compensated), Int32 max 182 ->
// 98; 5 * 10^6 Float32 values in 300 segments of two tiles 18.9 -> 13.0.
template <int OP, class T, int PREC, int NT>
__device__ __forceinline__ void seg_complete(const SegTileArgs &a, int64_t t0) {
  using A = Acc<OP, T, PREC>;
  using S = typename A::S;
  const int lane = threadIdx.x & 31;
  const int64_t t = t0 + lane;
  auto word = [&](const void *p) { return ld_relaxed_u64(static_cast<const uint64_t *>(p)); };
  bool mine = false;
  S carry = A::id();
  bool closed = true;
  if (t < a.ntiles) {
    const SegSlot *prev = a.slots + (t > 0 ? t - 1 : 0);
    const int64_t id = (int64_t)word(&a.slots[t].first_id);
    const uint64_t pc = word(&prev->carry), pb = word(&prev->boundary);
    mine = id >= 0 && id < a.nseg;
    if (t > 0) {
      carry = from_bits<S>(pc);
      closed = pb != 0;
    }
  }
  const bool any_open = __any_sync(0xffffffffu, mine && !closed);
  bool stopped = true;
  if (any_open) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const S ov = shfl_up(carry, d);
      const bool of = __shfl_up_sync(0xffffffffu, closed, d);
      if (lane >= d && !closed) {
        carry = A::comb(ov, carry);
        closed = of;
      }
    }
    stopped = !__any_sync(0xffffffffu, mine && !closed);
  }
  int64_t k = t0 - 2;  // the nearest slot that is not in `carry`
  if (!stopped) {
    S acc = A::id();
    for (int i = 0; !stopped && (NT == 0 || i < 4); ++i, k -= 32) {
      const int64_t q = k - lane;
      S v = A::id();
      bool stop = q < 0;
      if (!stop) {
        v = from_bits<S>(word(&a.slots[q].carry));
        stop = word(&a.slots[q].boundary) != 0;
      }
      const unsigned sm = __ballot_sync(0xffffffffu, stop);
      if (lane > (sm ? __ffs(sm) - 1 : 32)) v = A::id();
      acc = A::comb(shfl_idx(warp_reduce_rev<A>(v), 0), acc);
      stopped = sm != 0u;
    }
    if (!closed) carry = A::comb(acc, carry);
  }
  if constexpr (NT > 0) {
    if (__syncthreads_or(!stopped)) {
      constexpr int U = 8, NW = NT / 32;
      __shared__ S s_v[NW];
      __shared__ int64_t s_from[NW];
      __shared__ unsigned s_near[NW];
      const int tid = threadIdx.x, warp = tid >> 5;
      if (lane == 0) s_from[warp] = stopped ? -1 : k;
      __syncthreads();
      for (int w = 0; w < NW; ++w) {
        S acc = A::id();
        for (int64_t from = s_from[w]; from >= 0; from -= NT * U) {
          S v[U];
          unsigned near = NT * U;  // distance of the nearest slot that holds a boundary
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int64_t q = from - (u * NT + tid);
            v[u] = A::id();
            if (q < 0) continue;
            v[u] = from_bits<S>(word(&a.slots[q].carry));
            if (word(&a.slots[q].boundary) != 0 && near == NT * U) near = u * NT + tid;
          }
          near = __reduce_min_sync(0xffffffffu, near);
          if (lane == 0) s_near[warp] = near;
          __syncthreads();
          for (int i = 0; i < NW; ++i) near = s_near[i] < near ? s_near[i] : near;
          S sum = A::id();
#pragma unroll
          for (int u = U - 1; u >= 0; --u)
            if ((unsigned)(u * NT + tid) <= near) sum = A::comb(sum, v[u]);
          sum = warp_reduce_rev<A>(sum);
          if (lane == 0) s_v[warp] = sum;
          __syncthreads();
          S all = s_v[NW - 1];
          for (int i = NW - 2; i >= 0; --i) all = A::comb(all, s_v[i]);
          acc = A::comb(all, acc);
          __syncthreads();
          if (near < NT * U) break;
        }
        if (w == warp && !closed) carry = A::comb(acc, carry);
      }
    }
  }
  if (mine) {
    const S v = A::comb(carry, from_bits<S>(word(&a.slots[t].first)));
    static_cast<T *>(a.out)[word(&a.slots[t].first_id)] =
        A::lower(a.has_seed ? A::comb(A::lift(from_bits<T>(a.seed)), v) : v);
  }
}
template <int OP, class T, int PREC>
__global__ void __launch_bounds__(256) foldseg_fix(SegTileArgs a) {
  seg_complete<OP, T, PREC, 256>(a, (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll);
}

// ZIP: a thread zips its own rows of the two arrays' tiles in place before the
// walk, its 16-byte pieces in an order of its own (both rows are swizzled alike): all
// lanes on one column would meet on the same banks.
template <class T, int Z>
__device__ __forceinline__ void seg_zip_row(unsigned char *row, const unsigned char *row2, int order) {
  constexpr int VEC = 16 / sizeof(T);
#pragma unroll
  for (int i = 0; i < FT_ROW_BYTES / 16; ++i) {
    const int c = i ^ order;
    uint4 v = reinterpret_cast<const uint4 *>(row)[c];
    const uint4 w = reinterpret_cast<const uint4 *>(row2)[c];
    T x[VEC], y[VEC];
    memcpy(x, &v, 16);
    memcpy(y, &w, 16);
#pragma unroll
    for (int k = 0; k < VEC; ++k) x[k] = Prim<Z, T>::ap(x[k], y[k]);
    memcpy(&v, x, 16);
    reinterpret_cast<uint4 *>(row)[c] = v;
  }
}

template <int OP, class T, int PREC, class OT, bool ZIP = false, bool DENSE = false>
__global__ void __launch_bounds__(ft_threads<DENSE>(), ZIP ? 4 : 5)
foldseg_tile_kernel(const __grid_constant__ CUtensorMap tin, SegTileArgs a, const __grid_constant__ CUtensorMap tin2) {
  using A = Acc<OP, T, PREC>;
  using S = typename A::S;
  constexpr int FT_THREADS = ft_threads<DENSE>(), FT_PER = ft_per<DENSE>();
  constexpr int FT_RPT = ft_rpt<ZIP, DENSE>();
  constexpr int ITEMS = FT_ROW_BYTES / sizeof(T);
  constexpr int VEC = 16 / sizeof(T);
  constexpr int W = FT_RPT * ITEMS;          // values per thread (FT_RPT adjacent rows)
  constexpr int TE = FT_THREADS * W;
  constexpr int SUB_BYTES = FT_THREADS * FT_ROW_BYTES;
  constexpr int NWARP = FT_THREADS / 32;
  constexpr int FAR = 1 << 30;  // beyond every tile-relative position
  extern __shared__ unsigned char smem_raw[];
  unsigned char *buf = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t bar;
  __shared__ int64_t s_kf, s_cnt, s_lo, s_hi, s_first_id;
  __shared__ int16_t s_offs[FT_CAP];  // -1: before the tile (malformed)
  static_assert(TE < 32768, "16-bit tile-relative offsets");
  __shared__ int s_rowh[FT_THREADS];  // per thread: first offset entry at or after its first value
  __shared__ S s_res[FT_CAP];         // per entry (or, in a slot tile, per boundary): a closed segment's state
  __shared__ S s_wv[NWARP], s_first_v, s_tile_v;
  __shared__ int s_wf[NWARP];
  __shared__ int s_has_first, s_tile_f, s_bad;
  __shared__ uint64_t s_bm[FT_THREADS];  // slot tiles: each thread's boundary positions
  __shared__ int16_t s_base[FT_THREADS]; // slot tiles: each thread's first boundary slot
  __shared__ int s_nbw[NWARP];
  __shared__ unsigned s_count;           // small: offsets before the tile, and (high half) before its end
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const OT *off = static_cast<const OT *>(a.off);  // small: in shared memory, below
  T *out = static_cast<T *>(a.out);
  const T idT = Prim<OP, T>::id();

  const int64_t tile = blockIdx.x;
  if (tid == 0) {
    s_has_first = 0;
    s_bad = 0;
    s_count = 0;
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_expect_tx(&bar, (ZIP ? 2 : 1) * FT_RPT * SUB_BYTES);
#pragma unroll
    for (int u = 0; u < FT_RPT; ++u)
      tma_load_2d(buf + u * SUB_BYTES, &tin, 0, (int)((tile * FT_RPT + u) * FT_THREADS), &bar);
    if constexpr (ZIP) tma_load_2d(buf + SUB_BYTES, &tin2, 0, (int)(tile * FT_THREADS), &bar);
  }
  __syncthreads();
  const int64_t tb = tile * TE;
  const bool last_tile = tile == a.ntiles - 1;
  if (a.small) {
    const OT *given = off;
    OT *all = reinterpret_cast<OT *>(buf + (ZIP ? 2 : 1) * FT_RPT * SUB_BYTES);
    const int no = (int)a.nseg + 1, ng = a.small == 2 ? no - 1 : no;
    const int per = ((no + FT_THREADS - 1) / FT_THREADS) | 1;  // consecutive offsets per thread, an odd number
    {
      OT mine[FT_PER];
#pragma unroll
      for (int j = 0; j < FT_PER; ++j) {
        mine[j] = OT(0);
        if (j < per && tid + j * FT_THREADS < ng) mine[j] = given[tid + j * FT_THREADS];
      }
#pragma unroll
      for (int j = 0; j < FT_PER; ++j)
        if (j < per) all[tid + j * FT_THREADS] = mine[j];
    }
    __syncthreads();
    OT *mine = all + tid * per;
    if (a.small == 2) {
      // exclusive scan of the lengths, wrapping as scanl (+) 0 does
      using U = typename IntBits<OT>::U;
      U sum = 0;
      for (int j = 0; j < per; ++j) sum += (U)mine[j];
      const U incl = warp_scan_incl<Acc<ACC_ADD, U, 0>>(sum);
      U *s_sum = reinterpret_cast<U *>(all + FT_PER * FT_THREADS);
      if (lane == 31) s_sum[warp] = incl;
      __syncthreads();
      U run = incl - sum;
      for (int w2 = 0; w2 < warp; ++w2) run += s_sum[w2];
      for (int j = 0; j < per; ++j) {
        const U len = (U)mine[j];
        mine[j] = (OT)run;
        run += len;
      }
    }
    unsigned before = 0;  // of this thread's offsets: before the tile | before its end << 16
    for (int j = 0; j < per; ++j)
      if (tid * per + j < no)
        before += ((int64_t)mine[j] < tb ? 1u : 0u) + ((int64_t)mine[j] < tb + TE ? 0x10000u : 0u);
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) atomicAdd(&s_count, before);
    off = all;
    __syncthreads();
  }
  if (tid < 32) {
    // The offsets inside [tb, te) are [kf, ks); the last tile takes every
    // remaining one (ks = nseg + 1).
    const uint64_t tag = (uint64_t)a.epoch << TIDX_SHIFT, mask = (1ull << TIDX_SHIFT) - 1;
    const uint64_t e0 = a.small ? tag | (s_count & 0xffffu) : a.tidx[tile];
    const uint64_t e1 = a.small ? tag | (last_tile ? (uint64_t)(a.nseg + 1) : (uint64_t)(s_count >> 16)) : a.tidx[tile + 1];
    const int64_t vstart = (int64_t)off[0], vend = (int64_t)off[a.nseg];
    if (lane == 0) {
      const int64_t kf = (int64_t)(e0 & mask), ks = (int64_t)(e1 & mask);
      s_kf = kf;
      s_cnt = ks - kf;
      // Tile-relative value window of the segments, clamped to the tile.
      int64_t lo = vstart - tb, hi = vend - tb;
      s_lo = lo < 0 ? 0 : (lo > TE ? TE : lo);
      s_hi = hi < 0 ? 0 : (hi > TE ? TE : hi);
      if ((e0 & ~mask) != tag || (e1 & ~mask) != tag || ks < kf || ks > a.nseg + 1 || (tile == 0 && kf != 0) ||
          vstart < 0 || vend > a.n || vend < vstart)
        s_bad = 1;
      if (s_bad) s_cnt = 0;
    }
  }
  __syncthreads();
  const int64_t kf = s_kf, cnt = s_cnt > 0 ? s_cnt : 0;
  const T z = from_bits<T>(a.seed);
  // Tile-relative offsets to shared memory (the first FT_CAP of them), the
  // per-thread first entries, checks, and z for the empty segments that
  // start in this tile.  Entry i+1 is the first entry for the threads whose
  // first value lies in (rel_i, rel_(i+1)]; entry 0 for those at or before rel_0.
  if (cnt == 0) s_rowh[tid] = 0;
  bool bad = false;
  for (int64_t i = tid; i < cnt; i += FT_THREADS) {
    const int64_t k = kf + i;
    const int64_t o = (int64_t)off[k];
    const int64_t rel = o - tb;
    if (rel < 0 || (!last_tile && rel >= TE)) bad = true;
    const int r = (int)(rel < 0 ? 0 : (rel > TE ? TE : rel));
    if (i < FT_CAP) s_offs[i] = (int16_t)(rel < 0 ? -1 : r);
    int rn = FAR;  // the next entry, or past the tile
    if (k < a.nseg) {
      const int64_t o1 = (int64_t)off[k + 1];
      if (o1 < o) bad = true;
      else if (o1 == o && a.has_seed) out[k] = z;
      if (i + 1 < cnt) {
        const int64_t reln = o1 - tb;
        rn = (int)(reln < 0 ? 0 : (reln > TE ? TE : reln));
      }
    }
    if (i == 0)
      for (int t = 0; t <= r / W && t < FT_THREADS; ++t) s_rowh[t] = 0;
    const int t_hi = rn >= TE ? FT_THREADS - 1 : rn / W;
    for (int t = r / W + 1; t <= t_hi && t < FT_THREADS; ++t) s_rowh[t] = (int)(i + 1);
  }
  if (bad) s_bad = 1;
  auto rel_at = [&](int64_t h) -> int {
    if (h >= cnt) return FAR;
    if (h < FT_CAP) return s_offs[h];
    const int64_t rel = (int64_t)off[kf + h] - tb;
    return (int)(rel < 0 ? -1 : (rel > TE ? TE : rel));
  };
  // One warp waits for the tile; the others block at the CTA barrier, which
  // costs no issue slots (several CTAs share an SM and the walk is
  // issue-bound).  The barrier orders every thread after the completed load.
  bool landed = true;
  if (warp == 0 && !mbar_wait_sleep(&bar, 0)) {
    if (lane == 0) raise_error(a.err, DEV_ERR_TIMEOUT);
    landed = mbar_wait_sleep(&bar, 0);
  }
  // The tile's slot; a.finish: the last tile to get here completes the
  // segments that cross tiles, for all of them.
  auto finish = [&](uint64_t carry, uint64_t first, int64_t first_id, bool boundary) {
    if (tid == 0) {
      SegSlot sl{carry, first, first_id, boundary ? 1 : 0};
      uint4 q[2];
      memcpy(q, &sl, sizeof(sl));
      reinterpret_cast<uint4 *>(a.slots + tile)[0] = q[0];
      reinterpret_cast<uint4 *>(a.slots + tile)[1] = q[1];
    }
    if (!a.finish) return;
    if (tid == 0) {
      __threadfence();
      s_bad = atomicAdd(a.done, 1u) == (uint32_t)(a.ntiles - 1) ? 2 : 0;
    }
    __syncthreads();
    if (s_bad != 2) return;
    __threadfence();
    if (tid == 0) *a.done = 0u;
    for (int64_t t0 = warp * 32; t0 < a.ntiles; t0 += FT_THREADS) seg_complete<OP, T, PREC, 0>(a, t0);
  };
  // A tile whose load never landed is not read.
  if (__syncthreads_or(!landed)) {
    finish(0, 0, -1, true);
    return;
  }
  if constexpr (ZIP) {
    unsigned char *row = buf + tid * FT_ROW_BYTES;
    const unsigned char *row2 = row + SUB_BYTES;
    switch (a.zop) {
      case ACC_ADD: seg_zip_row<T, ACC_ADD>(row, row2, tid & 7); break;
      case ACC_MUL: seg_zip_row<T, ACC_MUL>(row, row2, tid & 7); break;
      case ACC_MIN: seg_zip_row<T, ACC_MIN>(row, row2, tid & 7); break;
      default: seg_zip_row<T, ACC_MAX>(row, row2, tid & 7); break;
    }
  }
  // The values after the last whole row (TMA left zeros there; the positions
  // past the last value are masked below).
  if (a.full_rows >= tile * (FT_RPT * FT_THREADS) && a.full_rows < (tile + 1) * (FT_RPT * FT_THREADS)) {
    if constexpr (ZIP) __syncthreads();  // after its owner has zipped that row's zeros
    const int64_t gi = a.full_rows * ITEMS + tid;
    if (tid < ITEMS && gi < a.n) {
      const int r = (int)(a.full_rows - tile * (FT_RPT * FT_THREADS)), rr = r % FT_THREADS;
      T v = static_cast<const T *>(a.in)[gi];
      if constexpr (ZIP) v = zip_elem(a.zop, v, static_cast<const T *>(a.in2)[gi]);
      *reinterpret_cast<T *>(buf + (r / FT_THREADS) * SUB_BYTES + rr * FT_ROW_BYTES + (((tid / VEC) ^ (rr & 7)) << 4) +
                             (tid % VEC) * sizeof(T)) = v;
    }
    __syncthreads();
  }
  const bool ok = s_bad == 0;
  if (!ok && tid == 0) raise_error(a.err, DEV_ERR_INDEX);
  const int lo = (int)s_lo, hi = (int)s_hi;

  // ---- the walk over this thread's FT_RPT adjacent rows
  const int tb0 = tid * W;
  int64_t h = s_rowh[tid];
  if (h < 0 || h > cnt) h = cnt;  // only with malformed offsets (nothing is written then)
  int np = rel_at(h);
  S acc = A::id(), left = A::id();
  bool started = false;
  int64_t first_h = -1;
  // A slot tile (the common case: well-formed offsets, all in shared memory,
  // every value of the tile inside the segments, no partial row) parks the
  // closed states by BOUNDARY: thread t's boundaries take slots s_base[t],
  // s_base[t]+1, ... (an exclusive scan of the threads' boundary counts), so
  // the walk keeps one running slot index and has no branch per value;
  // several offsets at one position (empty segments) are one boundary.  The
  // result pass finds a segment's slot from its position.
  const bool slot_tile = ok && cnt <= FT_CAP && lo == 0 && hi == TE &&
                         (tile + 1) * (int64_t)(FT_RPT * FT_THREADS) <= a.full_rows;
  int pbase = 0;
  if (slot_tile) {
    int64_t he = tid + 1 < FT_THREADS ? (int64_t)s_rowh[tid + 1] : cnt;
    if (he < h || he > cnt) he = cnt;
    uint64_t bm = 0;
    for (int64_t e = h; e < he; ++e) {
      const int r = s_offs[e] - tb0;
      if (r >= 0 && r < W) bm |= 1ull << r;
    }
    const int nb = __popcll(bm);
    int incl = nb;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) s_nbw[warp] = incl;
    __syncthreads();
    int wbase = 0;
    for (int w2 = 0; w2 < warp; ++w2) wbase += s_nbw[w2];
    pbase = wbase + incl - nb;
    s_bm[tid] = bm;
    s_base[tid] = (int16_t)pbase;
    int pk = pbase;
    // fully unrolled: every mask bit is tested at a constant position
    const uint32_t bm_lo = (uint32_t)bm, bm_hi = (uint32_t)(bm >> 32);
    const int r0 = FT_RPT * tid;
#pragma unroll
    for (int c = 0; c < W / VEC; ++c) {
      const int r = r0 + c / (ITEMS / VEC);
      const int cc = c % (ITEMS / VEC);
      const int rr = r % FT_THREADS;
      const uint4 v = *reinterpret_cast<const uint4 *>(buf + (r / FT_THREADS) * SUB_BYTES + rr * FT_ROW_BYTES +
                                                       ((cc ^ (rr & 7)) << 4));
      T x[VEC];
      memcpy(x, &v, 16);
#pragma unroll
      for (int q = 0; q < VEC; ++q) {
        const int bit = c * VEC + q;
        const bool bnd = ((bit < 32 ? bm_lo : bm_hi) >> (bit & 31)) & 1u;
        if (bnd) s_res[pk] = acc;
        pk += bnd ? 1 : 0;
        acc = bnd ? A::id() : acc;
        acc = A::push(acc, x[q]);
      }
    }
    started = nb > 0;
    first_h = h;  // the entry of the thread's first boundary
    if (started) left = s_res[pbase];
  } else {
  // A boundary only parks the closed segment's state (the results leave in
  // one coalesced pass after the scan), so a lane that meets one holds its
  // warp up for a few instructions.
  auto boundary = [&](int p) {
    if (!started) {
      left = acc;
      first_h = h;
      started = true;
    } else if (h < FT_CAP) {
      s_res[h] = acc;
    } else if (ok) {  // long offset lists only: write at once
      const int64_t sid = kf + h - 1;
      if (sid >= 0) out[sid] = A::lower(a.has_seed ? A::comb(A::lift(z), acc) : acc);
    }
    acc = A::id();
    do { ++h; np = rel_at(h); } while (np == p);  // several offsets at p: empty segments
  };
  const bool masked = lo > tb0 || hi < tb0 + W;
  auto load_chunk = [&](int c, T (&x)[VEC]) {
    const int r = FT_RPT * tid + c / (ITEMS / VEC);  // row within the tile
    const int cc = c % (ITEMS / VEC);                // 16-byte chunk within the row
    const int rr = r % FT_THREADS;
    const uint4 v = *reinterpret_cast<const uint4 *>(buf + (r / FT_THREADS) * SUB_BYTES + rr * FT_ROW_BYTES +
                                                     ((cc ^ (rr & 7)) << 4));
    memcpy(x, &v, 16);
  };
  // Fast walk: when this thread's offsets are in shared memory they become
  // a bit mask of boundary positions (bm) and the boundaries take entries
  // h, h+1, ... in order, so a boundary costs a shared-memory store and no
  // load; only a position that holds several offsets (empty segments
  // follow) skips its extra entries by reading them (dm marks those).
  static_assert(W <= 64, "one 64-bit boundary mask per thread");
  int64_t h_end = tid + 1 < FT_THREADS ? (int64_t)s_rowh[tid + 1] : cnt;
  if (h_end < h || h_end > cnt) h_end = cnt;
  bool fast = ok && h_end <= FT_CAP;
  uint64_t bm = 0, dm = 0;
  if (fast) {
    for (int64_t e = h; e < h_end; ++e) {
      const int r = s_offs[e] - tb0;
      if (r < 0 || r >= W) fast = false;
      else if ((bm >> r) & 1u) dm |= 1ull << r;
      else bm |= 1ull << r;
    }
  }
  if (fast) {
    // Branch-free walk: every boundary, the row's first included, parks the
    // closed segment's state at its entry; the first one is read back as
    // the value carried out to the left.  Only a boundary followed by empty
    // segments branches (to skip their entries).
    int hh = (int)h;
    const int h0 = hh;
#pragma unroll 1
    for (int c = 0; c < W / VEC; ++c) {
      T x[VEC];
      load_chunk(c, x);
      const uint32_t cb = (uint32_t)(bm >> (c * VEC)) & ((1u << VEC) - 1u);
      const uint32_t cd = (uint32_t)(dm >> (c * VEC)) & ((1u << VEC) - 1u);
#pragma unroll
      for (int q = 0; q < VEC; ++q) {
        const bool bnd = (cb >> q) & 1u;
        if (bnd) s_res[hh] = acc;
        if (bnd && ((cd >> q) & 1u)) {
          const int at = tb0 + c * VEC + q;
          do { ++hh; } while (hh < h_end && s_offs[hh] == at);
        } else {
          hh += bnd ? 1 : 0;
        }
        acc = bnd ? A::id() : acc;
        const int pos = tb0 + c * VEC + q;
        acc = A::push(acc, pos >= lo && pos < hi ? x[q] : idT);
      }
    }
    started = hh != h0;
    first_h = h0;
    if (started) left = s_res[h0];
  } else {
#pragma unroll 1
    for (int c = 0; c < W / VEC; ++c) {
      T x[VEC];
      load_chunk(c, x);
      const int p0 = tb0 + c * VEC;
      if (masked) {
#pragma unroll
        for (int q = 0; q < VEC; ++q) {
          if (p0 + q == np) boundary(p0 + q);
          acc = A::push(acc, (p0 + q >= lo && p0 + q < hi) ? x[q] : idT);
        }
      } else {
#pragma unroll
        for (int q = 0; q < VEC; ++q) {
          if (p0 + q == np) boundary(p0 + q);
          acc = A::push(acc, x[q]);
        }
      }
    }
  }

  }

  // ---- segmented CTA scan of the rows' carried-out values
  S iv = acc;
  bool ifl = started;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const S ov = shfl_up(iv, d);
    const bool of = __shfl_up_sync(0xffffffffu, ifl, d);
    if (lane >= d) {
      if (!ifl) iv = A::comb(ov, iv);
      ifl = ifl || of;
    }
  }
  S ex = shfl_up(iv, 1);
  bool exf = __shfl_up_sync(0xffffffffu, ifl, 1);
  if (lane == 0) { ex = A::id(); exf = false; }
  if (lane == 31) { s_wv[warp] = iv; s_wf[warp] = ifl; }
  __syncthreads();
  S wv = A::id();
  bool wf = false;
  for (int w = 0; w < warp; ++w) {
    wv = s_wf[w] ? s_wv[w] : A::comb(wv, s_wv[w]);
    wf = wf || s_wf[w];
  }
  const S cin = exf ? ex : A::comb(wv, ex);  // value of the segment open at the row start
  const bool cinf = exf || wf;                // that segment started inside the tile
  if (started) {
    const S v = A::comb(cin, left);
    if (cinf) {
      if (slot_tile) s_res[pbase] = v;
      else if (first_h < FT_CAP) s_res[first_h] = v;
      else if (ok) out[kf + first_h - 1] = A::lower(a.has_seed ? A::comb(A::lift(z), v) : v);
    } else {
      s_first_v = v;  // the tile's first boundary: needs the value from earlier tiles
      s_first_id = kf + first_h - 1;
      s_has_first = 1;
    }
  }
  if (tid == FT_THREADS - 1) {
    s_tile_v = started ? acc : A::comb(cin, acc);
    s_tile_f = started || cinf;
  }
  __syncthreads();

  // ---- the parked results leave
  if (ok) {
    const int64_t nres = cnt < FT_CAP ? cnt : FT_CAP;
    for (int64_t e = 1 + tid; e < nres; e += FT_THREADS)
      if (s_offs[e] > s_offs[e - 1]) {  // the first entry at its position closes a segment
        int slot = (int)e;
        if (slot_tile) {
          // the boundary at position p is bit p % W of thread p / W
          const int p = s_offs[e], t = p / W, bit = p % W;
          slot = s_base[t] + __popcll(s_bm[t] & ((1ull << bit) - 1ull));
        }
        const S v = s_res[slot];
        out[kf + e - 1] = A::lower(a.has_seed ? A::comb(A::lift(z), v) : v);
      }
  }
  finish(to_bits(s_tile_v), s_has_first ? to_bits(s_first_v) : 0, s_has_first && ok ? s_first_id : -1, s_tile_f != 0);
}

// One launcher per kernel instantiation, so that each gets its own
// shared-memory attribute (the tile needs more than the default 48 KB).
template <int OP, class T, int PREC, class OT, bool ZIP, bool DENSE>
int launch_foldseg_tile(const CUtensorMap &tin, const SegTileArgs &a, int64_t ntiles, cudaStream_t s,
                        const CUtensorMap &tin2) {
  constexpr int FT_THREADS = ft_threads<DENSE>(), FT_PER = ft_per<DENSE>(), FT_RPT = ft_rpt<ZIP, DENSE>();
  const size_t tile = (size_t)(ZIP ? 2 : 1) * FT_RPT * FT_THREADS * FT_ROW_BYTES + 1024;
  const size_t all = (size_t)(FT_PER * FT_THREADS + FT_THREADS / 32) * sizeof(OT);  // small: the offsets, the warps' sums
  const size_t smem = tile + (a.small ? all : 0);
  auto kern = foldseg_tile_kernel<OP, T, PREC, OT, ZIP, DENSE>;
  static std::atomic<uint64_t> attr_done{0};
  smem_attrs_once(kern, (int)(tile + all), attr_done);
  kern<<<(unsigned)ntiles, FT_THREADS, smem, s>>>(tin, a, tin2);
  const int st = check_launch();
  if (st || a.finish) return st;
  foldseg_fix<OP, T, PREC><<<(unsigned)cdiv_h(ntiles, 256), 256, 0, s>>>(a);
  return check_launch();
}

template <int OP, class T, int PREC, bool ZIP = false, bool DENSE = false>
int foldseg_tile_typed(Workspace *w, const T *in, const void *off, int off64, bool lengths, T *out, int64_t inner,
                       int64_t nseg, bool has_seed, uint64_t seed, cudaStream_t s, bool *taken,
                       const T *in2 = nullptr, int zop = 0) {
  *taken = false;
  // Short segments over a zipWith keep the per-segment kernels, a lane per segment: 2^24
  // Float64 values in equal segments of 4 84 us (206 by tiles), of 14 79 (112); 2^18
  // Float32 values in segments of 8 8.4 (12).  From 16 values on lognormal lengths, whose
  // lanes wait for the longest, gain more than equal ones lose: 2^24 Float64 values in
  // segments of 20, lognormal 254 (118), equal 81 (114).
  if (ZIP && inner < 16 * nseg) return ACC_OK;
  if constexpr (!DENSE && !ZIP && ft_dense<typename Acc<OP, T, PREC>::S>()) {
    if (inner < 11 * nseg)
      return foldseg_tile_typed<OP, T, PREC, ZIP, true>(w, in, off, off64, lengths, out, inner, nseg, has_seed, seed, s,
                                                        taken);
  }
  constexpr int ITEMS = FT_ROW_BYTES / sizeof(T);
  constexpr int FT_THREADS = ft_threads<DENSE>(), FT_RPT = ft_rpt<ZIP, DENSE>();
  constexpr int64_t TE = (int64_t)FT_THREADS * FT_RPT * ITEMS;
  constexpr int LOG_TE = 31 - __builtin_clz((unsigned)TE);
  static_assert(TE == int64_t(1) << LOG_TE, "tiles of a power of two values");
  const int64_t full_rows = inner / ITEMS;
  CUtensorMap tin, tin2;
  memset(&tin, 0, sizeof(tin));
  memset(&tin2, 0, sizeof(tin2));
  if (full_rows == 0 || !encode_2d(&tin, in, sizeof(T), ITEMS, full_rows, FT_ROW_BYTES, ITEMS, FT_THREADS, true) ||
      (ZIP && !encode_2d(&tin2, in2, sizeof(T), ITEMS, full_rows, FT_ROW_BYTES, ITEMS, FT_THREADS, true)))
    return ACC_OK;  // not describable by TMA: the caller uses the per-segment kernels
  // One tile more than the values need when they fill the last tile exactly:
  // that tile holds the boundary at position n.
  const int64_t ntiles = inner / TE + 1;
  if (ntiles * FT_RPT * FT_THREADS >= (1ll << 31)) return ACC_OK;  // TMA row coordinates are 32-bit
  if (nseg + 2 >= (1ll << TIDX_SHIFT)) return ACC_OK;
  const bool small = nseg <= FT_SMALL && ntiles <= 2 * (int64_t)device_info().sms;
  if (lengths && !small) return ACC_OK;  // the caller scans the lengths first
  // Over a zipWith, two arrays' tiles leave too few CTAs per SM for long calls:
  // 67,860 Float32 values 41 -> 16 us, 10^6 28 -> 23, 2^25 115 -> 155.  Float64
  // states are bound by their additions there too (2^24 Float64 212 -> 166).
  if (ZIP && ntiles > 2 * (int64_t)device_info().sms && !std::is_same<typename Acc<OP, T, PREC>::S, double>::value)
    return ACC_OK;
  *taken = true;
  const size_t slot_bytes = (size_t)ntiles * sizeof(SegSlot);
  int st = ws_scratch(w, slot_bytes + (size_t)(ntiles + 1) * sizeof(uint64_t));
  if (st) return st;
  uint64_t *tidx = reinterpret_cast<uint64_t *>(static_cast<char *>(w->scratch) + slot_bytes);
  SegTileArgs a{};
  a.in = in; a.off = off; a.out = out;
  a.in2 = in2; a.zop = zop;
  a.n = inner; a.nseg = nseg;
  a.full_rows = full_rows; a.ntiles = ntiles;
  a.seed = seed; a.has_seed = has_seed;
  a.slots = static_cast<SegSlot *>(w->scratch);
  a.tidx = tidx;
  a.small = small ? (lengths ? 2 : 1) : 0;
  // Up to as many tiles as a CTA's warps complete at once the last one spares the
  // completion's launch: 10^6 Float32 values in 62,500 segments 20.5 -> 18.4 us of device
  // time, 300,000 Int64 in 7,500 18.4 -> 16.4.
  a.finish = small || ntiles <= FT_THREADS;
  a.done = w->words + W_DONE;
  a.err = w->words + W_ERR;
  a.epoch = ws_next_epoch(w, s);
  if (!small) {
    const Device &d = device_info();
    int64_t pb = cdiv_h(nseg + 2, 256);
    if (pb > (int64_t)d.sms * 8) pb = (int64_t)d.sms * 8;
    if (off64)
      foldseg_tile_index<int64_t><<<(unsigned)pb, 256, 0, s>>>(static_cast<const int64_t *>(off), nseg, ntiles, LOG_TE,
                                                                tidx, a.epoch);
    else
      foldseg_tile_index<int32_t><<<(unsigned)pb, 256, 0, s>>>(static_cast<const int32_t *>(off), nseg, ntiles, LOG_TE,
                                                                tidx, a.epoch);
    st = check_launch();
    if (st) return st;
  }
  return off64 ? launch_foldseg_tile<OP, T, PREC, int64_t, ZIP, DENSE>(tin, a, ntiles, s, tin2)
               : launch_foldseg_tile<OP, T, PREC, int32_t, ZIP, DENSE>(tin, a, ntiles, s, tin2);
}

// ----------------------------------------------------------------- host side
// The per-segment path; with ZIP over the fused producer zipWith zop in in2.
template <int OP, class T, int PREC, bool ZIP = false>
int foldseg_typed(Workspace *w, const T *in, const void *off, int off64, T *out, int64_t outer,
                  int64_t inner, int64_t nseg, bool has_seed, uint64_t seed, cudaStream_t s,
                  const T *in2 = nullptr, int zop = 0) {
  const Device &d = device_info();
  // Scratch: the list of long segments (at most inner / LONG_SEG of them).
  int64_t maxlong = inner / LONG_SEG + 1;
  if (maxlong > nseg) maxlong = nseg;
  int st = ws_scratch(w, (size_t)maxlong * sizeof(int64_t) + 256);
  if (st) return st;
  SegArgs a{};
  a.in = in; a.off = off; a.out = out;
  a.outer = outer; a.inner = inner; a.nseg = nseg; a.off64 = off64;
  a.seed = seed; a.has_seed = has_seed;
  a.nlong = w->words + W_SEGBIG;
  a.longs = static_cast<int64_t *>(w->scratch);
  a.long_cap = maxlong;
  a.err = w->words + W_ERR;
  a.in2 = in2;
  a.zop = zop;
  // Only a row longer than LONG_SEG can hold a long segment.
  a.long_ctas = 0;
  if (inner > LONG_SEG) {
    cudaError_t e = cudaMemsetAsync(a.nlong, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return cuda_status(e);
    int64_t cb = cdiv_h(nseg, 256);
    if (cb > (int64_t)d.sms * 8) cb = (int64_t)d.sms * 8;
    seg_classify<<<(unsigned)cb, 256, 0, s>>>(a);
    st = check_launch();
    if (st) return st;
    a.long_ctas = (int64_t)d.sms * 2;
  }
  const int64_t groups = cdiv_h(nseg, 32) * outer;
  int64_t sb = cdiv_h(groups, 8);
  if (sb > (int64_t)d.sms * 64) sb = (int64_t)d.sms * 64;
  if (sb < 1) sb = 1;
  foldseg_main<OP, T, PREC, ZIP><<<(unsigned)(a.long_ctas + sb), 256, 0, s>>>(a);
  return check_launch();
}

static bool foldseg_per_segment() {
  static const bool v = getenv("ACC_GB300_FOLDSEG") && strcmp(getenv("ACC_GB300_FOLDSEG"), "segments") == 0;
  return v;
}

// `lengths`: `off` holds the segments' lengths; *taken says whether the call
// was made (one launch scans them too), and nothing else is tried.
int foldseg_dispatch(Workspace *w, int op, int type, int prec, const void *in, const void *off,
                     int off64, void *out, int64_t outer, int64_t inner, int64_t nseg,
                     const void *seed, cudaStream_t s, bool lengths = false, bool *lengths_taken = nullptr) {
  return with_type(type, [&](auto tv) -> int {
    using T = decltype(tv);
    const uint64_t sb = seed_bits<T>(seed);
    return with_op<T>(op, [&](auto opc) -> int {
      constexpr int OP = decltype(opc)::value;
      return with_prec<OP, T>(prec, [&](auto pc) -> int {
        constexpr int P = decltype(pc)::value;
        // Rows of one segmented vector take the tiled single pass unless
        // ACC_GB300_FOLDSEG=segments asks for the per-segment kernels.
        const bool per_segment = foldseg_per_segment();
        if (outer == 1 && !per_segment) {
          bool taken = false;
          const int st = foldseg_tile_typed<OP, T, P>(w, static_cast<const T *>(in), off, off64, lengths,
                                                      static_cast<T *>(out), inner, nseg, seed != nullptr, sb, s,
                                                      &taken);
          if (lengths) *lengths_taken = taken;
          if (taken || st) return st;
        }
        if (lengths) return ACC_OK;
        return foldseg_typed<OP, T, P>(w, static_cast<const T *>(in), off, off64, static_cast<T *>(out),
                                       outer, inner, nseg, seed != nullptr, sb, s);
      });
    });
  });
}

}  // namespace accgb

using namespace accgb;

static int fold_seg_check(int type, int offset_type, const void *in, const void *offsets, void *out,
                          int64_t outer, int64_t inner, int64_t nseg) {
  if (outer < 0 || inner < 0 || nseg < 0) return ACC_ERR_INVALID;
  if (offset_type != ACC_I32 && offset_type != ACC_I64) return ACC_ERR_INVALID;
  if (type < ACC_I32 || type > ACC_F64) return ACC_ERR_INVALID;
  if (outer > 0 && nseg > 0 && (!offsets || !out)) return ACC_ERR_INVALID;
  if (outer > 0 && inner > 0 && nseg > 0 && !in) return ACC_ERR_INVALID;
  return ACC_OK;
}

extern "C" int acc_fold_seg(int op, int type, int prec, const void *in, const void *offsets,
                            int offset_type, void *out, int64_t outer, int64_t inner, int64_t nseg,
                            const void *seed, void *stream) {
  int st = fold_seg_check(type, offset_type, in, offsets, out, outer, inner, nseg);
  if (st) return st;
  if (outer == 0 || nseg == 0) return ACC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Workspace *w = workspace(s, &st);
  if (!w) return st;
  std::lock_guard<std::mutex> lk(w->mu);
  return foldseg_dispatch(w, op, type, prec, in, offsets, offset_type == ACC_I64, out, outer, inner, nseg, seed, s);
}

extern "C" int acc_fold_seg_lengths(int op, int type, int prec, const void *in, const void *lengths,
                                    int length_type, void *out, int64_t outer, int64_t inner,
                                    int64_t nseg, const void *seed, void *stream) {
  int st = fold_seg_check(type, length_type, in, lengths, out, outer, inner, nseg);
  if (st) return st;
  if (outer == 0 || nseg == 0) return ACC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Workspace *w = workspace(s, &st);
  if (!w) return st;
  std::lock_guard<std::mutex> lk(w->mu);
  bool taken = false;
  st = foldseg_dispatch(w, op, type, prec, in, lengths, length_type == ACC_I64, out, outer, inner, nseg, seed, s, true,
                        &taken);
  if (taken || st) return st;
  // The offsets live at the END of the scratch area.  The front part,
  // list_bytes, holds what the fold itself keeps in scratch: the per-segment
  // path's long-segment list (at most inner / LONG_SEG + 1 entries) or the
  // tiled path's slots and tile index (40 bytes per tile of at least 4096
  // values), both within list_bytes, so neither grows (and moves) the
  // scratch under the offsets.
  const size_t esz = length_type == ACC_I64 ? 8 : 4;
  const size_t list_bytes = (size_t)(inner / LONG_SEG + 2) * 3 * sizeof(int64_t) + 512;
  const size_t off_bytes = (size_t)(nseg + 1) * esz;
  st = ws_scratch(w, list_bytes + off_bytes + 256);
  if (st) return st;
  void *offsets = static_cast<char *>(w->scratch) + ((list_bytes + 255) & ~size_t(255));
  st = scan_offsets(w, length_type, lengths, offsets, nseg, s);
  if (st) return st;
  return foldseg_dispatch(w, op, type, prec, in, offsets, length_type == ACC_I64, out, outer, inner, nseg, seed, s);
}

// foldSeg f z (zipWith g xs ys): the reference fuses the producer into the
// segmented fold's kernel (its delayed input, PTX/CodeGen/FoldSeg.hs:56-458
// reading a MIRDelayed array).  Here the tiles of both arrays are zipped in
// shared memory before the walk (short 1-D calls, both 16-byte aligned), or the
// per-segment kernels zip each element as they load it; the zipped array is never
// written.
// f in {+, min, max}, g in {+, *, min, max}, Int32 / Int64 / Float32 /
// Float64, as for the fused fold and scans.
extern "C" int acc_fold_seg_zipwith(int op, int zop, int type, int prec, const void *xs, const void *ys,
                                    const void *offsets, int offset_type, void *out, int64_t outer, int64_t inner,
                                    int64_t nseg, const void *seed, void *stream) {
  int st = fold_seg_check(type, offset_type, xs, offsets, out, outer, inner, nseg);
  if (st) return st;
  if (op < ACC_ADD || op > ACC_XOR || zop < ACC_ADD || zop > ACC_XOR) return ACC_ERR_INVALID;
  if (outer > 0 && inner > 0 && nseg > 0 && !ys) return ACC_ERR_INVALID;
  if (op != ACC_ADD && op != ACC_MIN && op != ACC_MAX) return ACC_ERR_UNSUPPORTED;
  if (zop != ACC_ADD && zop != ACC_MUL && zop != ACC_MIN && zop != ACC_MAX) return ACC_ERR_UNSUPPORTED;
  if (type == ACC_U32) return ACC_ERR_UNSUPPORTED;
  if (outer == 0 || nseg == 0) return ACC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Workspace *w = workspace(s, &st);
  if (!w) return st;
  std::lock_guard<std::mutex> lk(w->mu);
  return with_type(type, [&](auto tv) -> int {
    using T = decltype(tv);
    const uint64_t sb = seed_bits<T>(seed);
    return with_op<T>(op, [&](auto opc) -> int {
      constexpr int OP = decltype(opc)::value;
      if constexpr ((OP != ACC_ADD && OP != ACC_MIN && OP != ACC_MAX) || std::is_same<T, uint32_t>::value) {
        return ACC_ERR_UNSUPPORTED;
      } else {
        return with_prec<OP, T>(prec, [&](auto pc) -> int {
          constexpr int P = decltype(pc)::value;
          if (outer == 1 && !foldseg_per_segment()) {
            bool taken = false;
            const int st2 = foldseg_tile_typed<OP, T, P, true>(
                w, static_cast<const T *>(xs), offsets, offset_type == ACC_I64, false, static_cast<T *>(out), inner, nseg,
                seed != nullptr, sb, s, &taken, static_cast<const T *>(ys), zop);
            if (taken || st2) return st2;
          }
          return foldseg_typed<OP, T, P, true>(w, static_cast<const T *>(xs), offsets, offset_type == ACC_I64,
                                               static_cast<T *>(out), outer, inner, nseg, seed != nullptr, sb, s,
                                               static_cast<const T *>(ys), zop);
        });
      }
    });
  });
}
