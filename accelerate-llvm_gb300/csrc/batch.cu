// batch.cu -- many independent fold / scanl1 requests in ONE persistent launch,
// replayable as a CUDA graph, with tile sizes from the library's autotuner.
//
// The reference launches every skeleton separately, each with host-side
// set-up (PTX/Execute.hs:835-881); thousands of small and medium requests are
// dominated by launch latency.  Here a plan flattens a batch into work items
// (request, tile), each request cut into tiles of NT x IPT elements (scans) or
// up to B_FOLD_STEPS such steps (folds); the autotuner picks the launch shape
// (NT threads per CTA: 128, 256 or 512) and the tile shape (IPT elements per
// thread) per (kind, type, size bucket), and a batch runs with the NT preferred
// by most of its bytes.  One persistent kernel draws items from an atomic
// ticket in table order; its design is at batch_kernel below.
// All scratch is owned by the plan and allocated when the plan is made; a
// launch allocates nothing and takes its look-back epoch from a device word
// that the last CTA advances, so a captured graph replays unchanged.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "common.cuh"

namespace accgb {

constexpr int BT = 256;                    // threads per CTA of untuned launches and of the serving arena
constexpr int B_FOLD_STEPS = 4;            // tiles' worth of elements in one fold item
constexpr int B_BYTES[2] = {16, 64};       // bytes of a tile per thread, the two tile shapes

struct BReq {
  const void *in;
  void *out;
  int64_t n;
  uint64_t seed;
  int64_t first_item;
  int64_t ntiles;
  int32_t kind, type, has_seed, ipt;
};

struct BatchArgs {
  const BReq *reqs;
  const int32_t *item_req;
  int64_t nitems;
  uint64_t *status;      // 2 words per item (scan look-back)
  uint64_t *partials;    // one state per item (fold)
  uint32_t *req_ticket;  // per request, zero between launches
  uint32_t *words;       // [0] error, [1] item ticket, [2] epoch
};

// ---------------------------------------------------------------- device parts
template <class S>
__device__ __forceinline__ void b_publish(uint64_t *status, int64_t t, uint32_t epoch, uint32_t flag, S v) {
  uint64_t b = to_bits(v);
  uint64_t tag = (uint64_t)((epoch << 2) | flag) << 32;
  if constexpr (sizeof(S) == 8) st_relaxed_u64(status + 2 * t + 1, tag | (b >> 32));
  st_relaxed_u64(status + 2 * t, tag | (b & 0xffffffffull));
}
template <class S>
__device__ __forceinline__ uint32_t b_decode(SlotWords s, uint32_t epoch, S &v) {
  const uint32_t tag = (uint32_t)(s.w0 >> 32);
  if ((tag >> 2) != epoch) return 0;
  uint64_t b = s.w0 & 0xffffffffull;
  if constexpr (sizeof(S) == 8) {
    if ((uint32_t)(s.w1 >> 32) != tag) return 0;
    b |= (s.w1 & 0xffffffffull) << 32;
  }
  v = from_bits<S>(b);
  return tag & 3u;
}

enum { BK_FOLD = 0, BK_SCAN = 1 };

// An item as the CTA sees it: its request and its place in it.
struct __align__(16) BDesc {
  BReq q;
  int64_t item;  // -1: no more items
  int32_t r, pad;
};
static_assert(sizeof(BReq) == 64, "a request's descriptor is four 16-byte words");

template <int OP, class T> constexpr int b_prec() {
  return OP == ACC_ADD && std::is_same<T, float>::value ? PREC_COMP : PREC_PLAIN;
}
// f(T{}) for the request's element type (I32, I64, F32, F64)
template <class F> __device__ __forceinline__ void b_with_type(int type, F &&f) {
  switch (type) {
    case ACC_I32: f(int32_t{}); break;
    case ACC_I64: f(int64_t{}); break;
    case ACC_F32: f(float{}); break;
    default: f(double{}); break;
  }
}

// A compute thread's part of a tile, raw: 16 words, of which a tile of 16
// bytes per thread uses four.  A warp's part is 32 x ipt consecutive elements,
// read coalesced: element j * 32 + lane of the part is word(s) j.
struct BRaw { uint32_t w[16]; };

template <class W, int N>
__device__ __forceinline__ void b_load_words(const W *p, int64_t left, BRaw &raw) {
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (j * 32 < left) {
      const W v = p[j * 32];
      memcpy(&raw.w[j * (sizeof(W) / 4)], &v, sizeof(W));
    }
}
// Elements [at, at + 32 ipt) of the request, from lane's first one (at + lane).
__device__ __forceinline__ void b_load(const BReq &q, int64_t at, BRaw &raw) {
  const int64_t left = q.n - at;
  if (q.type == ACC_I32 || q.type == ACC_F32) {
    const uint32_t *p = static_cast<const uint32_t *>(q.in) + at;
    if (q.ipt == 16) b_load_words<uint32_t, 16>(p, left, raw);
    else b_load_words<uint32_t, 4>(p, left, raw);
  } else {
    const uint64_t *p = static_cast<const uint64_t *>(q.in) + at;
    if (q.ipt == 8) b_load_words<uint64_t, 8>(p, left, raw);
    else b_load_words<uint64_t, 2>(p, left, raw);
  }
}
template <class T> __device__ __forceinline__ T b_elem(const BRaw &raw, int j) {
  T x;
  memcpy(&x, &raw.w[j * (sizeof(T) / 4)], sizeof(T));
  return x;
}

// Scan, first pass: the warp turns its part in shared memory into K consecutive
// elements per lane (rows of an odd pitch) and scans the lanes' sums.  Returns
// the state of the lanes before this one; `sum` is the warp's.
template <int OP, class T, int K>
__device__ __forceinline__ uint64_t b_scan_pass1(const BRaw &raw, int64_t left, unsigned char *wbuf, uint64_t &sum) {
  using A = Acc<OP, T, b_prec<OP, T>()>;
  using S = typename A::S;
  const int lane = threadIdx.x & 31;
  T *turn = reinterpret_cast<T *>(wbuf) + (lane / K) * (K + 1) + lane % K;
  const T *row = reinterpret_cast<const T *>(wbuf) + lane * (K + 1);
#pragma unroll
  for (int j = 0; j < K; ++j) turn[j * (32 / K) * (K + 1)] = j * 32 < left ? b_elem<T>(raw, j) : Prim<OP, T>::id();
  __syncwarp();
  S agg = A::lift(row[0]);
#pragma unroll
  for (int j = 1; j < K; ++j) agg = A::push(agg, row[j]);
  const S incl = warp_scan_incl<A>(agg);
  const S up = shfl_up(incl, 1);
  sum = to_bits(shfl_idx(incl, 31));
  return to_bits(lane == 0 ? A::id() : up);
}
// Scan, second pass: rescan from the state before this lane and store.
template <int OP, class T, int K>
__device__ __forceinline__ void b_scan_pass2(const BReq &q, int64_t at, unsigned char *wbuf, uint64_t before) {
  using A = Acc<OP, T, b_prec<OP, T>()>;
  const int lane = threadIdx.x & 31;
  T *row = reinterpret_cast<T *>(wbuf) + lane * (K + 1);
  const T *turn = reinterpret_cast<const T *>(wbuf) + (lane / K) * (K + 1) + lane % K;
  typename A::S run = from_bits<typename A::S>(before);
#pragma unroll
  for (int j = 0; j < K; ++j) {
    run = A::push(run, row[j]);
    row[j] = A::lower(run);
  }
  __syncwarp();
  T *to = static_cast<T *>(q.out) + at;
  const int64_t left = q.n - at;
#pragma unroll
  for (int j = 0; j < K; ++j)
    if (j * 32 < left) to[j * 32] = turn[j * (32 / K) * (K + 1)];
  __syncwarp();
}

// The service warp's look-back: the combination of every earlier tile of the
// request, from the nearest published inclusive prefix on (warp-collective), in
// windows of 32 x B_LOOK tiles whose slots are loaded at once (1000 requests,
// 256 threads: one slot per lane 0.652 ms, two 0.669, four 0.700: a window
// waits for every tile in it up to the prefix).
constexpr int B_LOOK = 1;
template <class A>
__device__ __forceinline__ typename A::S b_lookback(const BatchArgs &a, int64_t item, int64_t tile, uint32_t epoch) {
  using S = typename A::S;
  const int lane = threadIdx.x & 31;
  S acc = A::id();
  int64_t k0 = 0;
  bool gave_up = false;
  while (true) {
    uint32_t fl[B_LOOK];
    S v[B_LOOK];
#pragma unroll
    for (int i = 0; i < B_LOOK; ++i) {
      fl[i] = k0 + lane * B_LOOK + i < tile ? 0u : 2u;  // predecessors of the same request only
      v[i] = A::id();
    }
    uint32_t it = 0;
    uint64_t t_wait = 0;
    bool resolved = false, whole = false;
    int kp = 32;
    while (true) {
      const int kp0 = lb_stop_lane<B_LOOK>(fl);
      SlotWords sw[B_LOOK];
#pragma unroll
      for (int i = 0; i < B_LOOK; ++i) {
        sw[i] = SlotWords{0ull, 0ull};
        if (fl[i] == 0 && lane <= kp0) sw[i] = ld_slot(a.status + 2 * (item - 1 - (k0 + lane * B_LOOK + i)));
      }
#pragma unroll
      for (int i = 0; i < B_LOOK; ++i)
        if (fl[i] == 0 && lane <= kp0) fl[i] = b_decode<S>(sw[i], epoch, v[i]);
      kp = lb_window<B_LOOK>(fl, resolved, whole);
      if (resolved || whole) break;
      ++it;
      if (it == 8) t_wait = global_ns();  // first checked at it == 64
      const bool stop = gave_up || it > SPIN_LIMIT ||
                        ((it & 63u) == 0 && ((ld_relaxed_u32(a.words) & DEV_ERR_TIMEOUT) != 0u ||
                                             global_ns() - t_wait > WAIT_LIMIT_NS));
      if (__any_sync(0xffffffffu, stop)) {
        gave_up = true;
        if (lane == 0) raise_error(a.words, DEV_ERR_TIMEOUT);
#pragma unroll
        for (int i = 0; i < B_LOOK; ++i)
          if (fl[i] == 0) fl[i] = 2u;
        kp = lb_window<B_LOOK>(fl, resolved, whole);
        break;
      }
      __nanosleep(it < 8 ? 32 : 128);
    }
    // lane-local fold from the nearest predecessor outwards, up to the first prefix
    bool seen = false;
    S lv = A::id();
#pragma unroll
    for (int i = 0; i < B_LOOK; ++i) {
      if (!seen) lv = A::comb(v[i], lv);
      seen = seen || fl[i] == 2u;
    }
    if (lane > kp) lv = A::id();
    acc = A::comb(shfl_idx(warp_reduce_rev<A>(lv), 0), acc);
    if (resolved) break;
    k0 += 32 * B_LOOK;
  }
  return acc;
}

// The persistent kernel.  NT compute threads and one service warp per CTA, which
// hand items over through mbarriers:
//   * the service warp draws the next item and fetches its descriptor while the
//     compute warps work on this one, looks back for scan tiles, and finishes
//     folds (one partial per item, the last item of a request folds them in
//     order);
//   * the compute warps keep the next tile's loads in flight in registers while
//     they work on one.  A scan tile takes two passes: its second, from the
//     prefix that the service warp found, runs after the first pass of the
//     CTA's next item, so that a look-back overlaps that.
// An item waits only on items with smaller tickets, which running CTAs hold and
// work through in order, so the smallest unfinished one can always finish.
// Every wait is bounded; a warp whose wait ran out raises DEV_ERR_TIMEOUT and
// returns (so do the others, in turn).
// Bound: the latency of a scan tile's look-back, then issue.  Measured on a
// GB300, 1000 requests of 2^8 .. 2^22 elements, folds and scans of Int32 and
// Float32 (floor 0.347 ms), against one tile at a time per CTA, loaded, scanned,
// looked back for and stored between barriers: 1.20 -> 0.60 ms (512 threads; 256:
// 0.64).  A tile's sum published by the service warp, after the look-back of the
// item before: 2.6 ms.  Tickets drawn five items ahead: 0.90 ms (a CTA's queue
// holds back the tiles that others wait for).  Fold items of 1 / 2 / 4 / 8 steps
// (256 threads): 0.713 / 0.651 / 0.637 / 0.669 ms.
constexpr int B_RING = 8;   // descriptors
constexpr int B_KEEP = 4;   // items whose warp totals and prefixes are kept

// bytes of a warp's buffer (32 rows of 64 bytes and one element), for one tile
__host__ __device__ constexpr int b_wbuf_bytes() { return 32 * (64 + 8); }

template <int OP, int NT>
__global__ void __launch_bounds__(NT + 32, NT == 128 ? 6 : NT == 256 ? 4 : 2) batch_kernel(BatchArgs a) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BDesc s_desc[B_RING];
  __shared__ uint64_t s_warp[B_KEEP][NW];  // states as bits
  __shared__ uint64_t s_sum[B_KEEP], s_prefix[B_KEEP];
  __shared__ uint32_t s_epoch;
  __shared__ int s_warps[B_KEEP];  // compute warps that have an item's sum
  __shared__ uint64_t b_desc[B_RING], b_sum[2], b_done[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int i = 0; i < B_RING; ++i) mbar_init(&b_desc[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&b_sum[i], 1);
      mbar_init(&b_done[i], 1);
    }
    for (int i = 0; i < B_KEEP; ++i) s_warps[i] = 0;
    s_epoch = (ld_relaxed_u32(a.words + 2) & ((1u << 29) - 1)) + 1;
    fence_mbar_init();
  }
  __syncthreads();
  const uint32_t epoch = s_epoch;
  auto wait = [&](uint64_t *bar, int64_t phase) -> bool {  // warp-uniform
    return __all_sync(0xffffffffu, mbar_wait_flagged(bar, (uint32_t)phase & 1u, a.words));
  };

  if (warp == NW) {
    // ---- service warp
    const uint32_t last_ticket = (uint32_t)a.nitems + gridDim.x - 1;
    // Draw the item of index i and hand it to the compute warps.  The holder of
    // the last ticket knows that every CTA has drawn its last one (and read the
    // epoch): it re-arms the ticket and advances the epoch for the next launch or
    // graph replay.
    auto claim = [&](int64_t i) {
      int64_t item = -1;
      if (lane == 0) {
        const uint32_t t = atomicAdd(a.words + 1, 1u);
        if (t == last_ticket) {
          a.words[1] = 0u;
          atomicAdd(a.words + 2, 1u);
        }
        if ((int64_t)t < a.nitems) item = t;
      }
      item = __shfl_sync(0xffffffffu, item, 0);
      BDesc &d = s_desc[i & (B_RING - 1)];
      if (item >= 0) {
        const int32_t r = a.item_req[item];
        if (lane < 4) reinterpret_cast<uint4 *>(&d.q)[lane] = reinterpret_cast<const uint4 *>(a.reqs + r)[lane];
        if (lane == 0) d.r = r;
      }
      if (lane == 0) d.item = item;
      __syncwarp();
      if (lane == 0) mbar_arrive(&b_desc[i & (B_RING - 1)]);
    };
    claim(0);
    for (int64_t i = 0;; ++i) {
      if (s_desc[i & (B_RING - 1)].item < 0) break;
      claim(i + 1);
      if (!wait(&b_sum[i & 1], i >> 1)) return;
      const BDesc &d = s_desc[i & (B_RING - 1)];
      const int64_t item = d.item, tile = item - d.q.first_item;
      const uint64_t sum_bits = s_sum[i & (B_KEEP - 1)];
      b_with_type(d.q.type, [&](auto tv) {
        using T = decltype(tv);
        using A = Acc<OP, T, b_prec<OP, T>()>;
        using S = typename A::S;
        const S sum = from_bits<S>(sum_bits);
        const S z = A::lift(from_bits<T>(d.q.seed));
        if (d.q.kind == BK_SCAN) {
          S prefix = d.q.has_seed ? z : A::id();  // of the request's first tile
          if (tile > 0) prefix = b_lookback<A>(a, item, tile, epoch);
          if (lane == 0) {
            if (tile + 1 < d.q.ntiles) b_publish<S>(a.status, item, epoch, 2u, A::comb(prefix, sum));
            s_prefix[i & (B_KEEP - 1)] = to_bits(prefix);
          }
        } else if (d.q.ntiles == 1) {
          if (lane == 0) *static_cast<T *>(d.q.out) = A::lower(d.q.has_seed ? A::comb(z, sum) : sum);
        } else {
          // One 8-byte slot per item whatever the state's size, so that requests
          // of different types in one batch never share partial slots.
          auto part = [&](int64_t k) { return reinterpret_cast<S *>(a.partials + k); };
          uint32_t prev = 0;
          if (lane == 0) {
            *part(item) = sum;
            __threadfence();
            prev = atomicAdd(a.req_ticket + d.r, 1u);
          }
          if (__shfl_sync(0xffffffffu, prev, 0) == (uint32_t)(d.q.ntiles - 1)) {
            __threadfence();
            const int64_t per = (d.q.ntiles + 31) / 32;
            const int64_t lo = lane * per, hi = lo + per < d.q.ntiles ? lo + per : d.q.ntiles;
            S v = A::id();
            for (int64_t k = lo; k < hi; ++k) v = A::comb(v, ld_state<S>(part(d.q.first_item + k)));
            v = warp_reduce<A>(v);
            if (lane == 0) {
              *static_cast<T *>(d.q.out) = A::lower(d.q.has_seed ? A::comb(z, v) : v);
              a.req_ticket[d.r] = 0u;  // re-arm for the next launch
            }
          }
        }
      });
      __syncwarp();
      if (lane == 0) mbar_arrive(&b_done[i & 1]);
    }
    return;
  }

  // ---- compute warps
  unsigned char *wbufs = smem + warp * (2 * b_wbuf_bytes());
  auto part_of = [&](const BDesc &d) -> int64_t {  // this lane's first element of the item
    const int64_t tile = d.item - d.q.first_item;
    const int64_t ts = (int64_t)d.q.ipt * NT * (d.q.kind == BK_FOLD ? B_FOLD_STEPS : 1);
    return tile * ts + warp * (32 * d.q.ipt) + lane;
  };
  auto pass2 = [&](int64_t i, uint64_t before) -> bool {
    if (!wait(&b_done[i & 1], i >> 1)) return false;
    const BDesc &d = s_desc[i & (B_RING - 1)];
    if (d.q.kind != BK_SCAN) return true;
    unsigned char *wbuf = wbufs + (i & 1) * b_wbuf_bytes();
    const uint64_t *totals = s_warp[i & (B_KEEP - 1)];
    const uint64_t prefix = s_prefix[i & (B_KEEP - 1)];
    const int64_t at = part_of(d);
    b_with_type(d.q.type, [&](auto tv) {
      using T = decltype(tv);
      using A = Acc<OP, T, b_prec<OP, T>()>;
      using S = typename A::S;
      constexpr int KW = 64 / sizeof(T), KN = 16 / sizeof(T);
      S run = from_bits<S>(prefix);
      for (int w = 0; w < warp; ++w) run = A::comb(run, from_bits<S>(totals[w]));
      run = A::comb(run, from_bits<S>(before));
      if (d.q.ipt == KW) b_scan_pass2<OP, T, KW>(d.q, at, wbuf, to_bits(run));
      else b_scan_pass2<OP, T, KN>(d.q, at, wbuf, to_bits(run));
    });
    return true;
  };
  BRaw raw;
  uint64_t before_prev = 0;
  if (!wait(&b_desc[0], 0)) return;
  if (s_desc[0].item < 0) return;
  b_load(s_desc[0].q, part_of(s_desc[0]), raw);
  for (int64_t i = 0;; ++i) {
    const BDesc &d = s_desc[i & (B_RING - 1)], &dn = s_desc[(i + 1) & (B_RING - 1)];
    const int64_t at = part_of(d);
    uint64_t before = 0, sum = 0;
    bool ok = true;
    auto load_next = [&]() {
      ok = wait(&b_desc[(i + 1) & (B_RING - 1)], (i + 1) / B_RING);
      if (ok && dn.item >= 0) b_load(dn.q, part_of(dn), raw);
    };
    if (d.q.kind == BK_SCAN) {
      unsigned char *wbuf = wbufs + (i & 1) * b_wbuf_bytes();
      const int64_t left = d.q.n - at;
      b_with_type(d.q.type, [&](auto tv) {
        using T = decltype(tv);
        constexpr int KW = 64 / sizeof(T), KN = 16 / sizeof(T);
        before = d.q.ipt == KW ? b_scan_pass1<OP, T, KW>(raw, left, wbuf, sum) : b_scan_pass1<OP, T, KN>(raw, left, wbuf, sum);
      });
    } else {
      // the item's steps, the next one's loads in flight
      const int64_t step = (int64_t)d.q.ipt * NT;
      int64_t end = (d.item - d.q.first_item + 1) * step * B_FOLD_STEPS;
      if (end > d.q.n) end = d.q.n;
      b_with_type(d.q.type, [&](auto tv) {
        using T = decltype(tv);
        using A = Acc<OP, T, b_prec<OP, T>()>;
        constexpr int KW = 64 / sizeof(T), KN = 16 / sizeof(T);
        typename A::S acc = A::id();
        for (int64_t e = at;; e += step) {
          const BRaw cur = raw;
          const int64_t left = d.q.n - e;
          // uniform over the warp: whether any lane has elements in the next step
          const bool more = e - lane + step < end;
          if (more) b_load(d.q, e + step, raw);
          if (d.q.ipt == KW) {
#pragma unroll
            for (int j = 0; j < KW; ++j)
              if (j * 32 < left) acc = A::push(acc, b_elem<T>(cur, j));
          } else {
#pragma unroll
            for (int j = 0; j < KN; ++j)
              if (j * 32 < left) acc = A::push(acc, b_elem<T>(cur, j));
          }
          if (!more) break;
        }
        sum = to_bits(warp_reduce<A>(acc));
      });
    }
    // The warp that completes the item's sum hands it to the service warp, and
    // publishes a scan tile's at once: the service warp may still be looking back
    // for the item before, and later tiles must not wait for that.
    int last = 0;
    if (lane == 0) {
      s_warp[i & (B_KEEP - 1)][warp] = sum;
      __threadfence_block();
      last = atomicAdd(&s_warps[i & (B_KEEP - 1)], 1) == NW - 1;
    }
    if (__shfl_sync(0xffffffffu, last, 0)) {
      __threadfence_block();
      b_with_type(d.q.type, [&](auto tv) {
        using T = decltype(tv);
        using A = Acc<OP, T, b_prec<OP, T>()>;
        using S = typename A::S;
        const S v = warp_reduce<A>(lane < NW ? from_bits<S>(s_warp[i & (B_KEEP - 1)][lane]) : A::id());
        if (lane == 0) {
          if (d.q.kind == BK_SCAN && d.item > d.q.first_item) b_publish<S>(a.status, d.item, epoch, 1u, v);
          s_sum[i & (B_KEEP - 1)] = to_bits(v);
          s_warps[i & (B_KEEP - 1)] = 0;
          mbar_arrive(&b_sum[i & 1]);
        }
      });
      __syncwarp();
    }
    load_next();
    if (!ok) return;
    if (i > 0 && !pass2(i - 1, before_prev)) return;
    before_prev = before;
    if (dn.item < 0) {
      pass2(i, before);
      return;
    }
  }
}

// ---------------------------------------------------------------- autotuner table
// Launch and tile shape per (kind, type, log2 size bucket): NT threads per CTA
// and IPT elements per thread (a tile is NT x IPT elements), 16 or 64 bytes'
// worth.  Filled by acc_batch_autotune, persisted as JSON.
constexpr int B_NT[3] = {128, 256, 512};
struct TuneKey {
  int kind, type, bucket;
  bool operator<(const TuneKey &o) const { return std::tie(kind, type, bucket) < std::tie(o.kind, o.type, o.bucket); }
};
struct TuneVal {
  int ipt, nt;
};
static std::mutex g_tune_mu;
static std::map<TuneKey, TuneVal> g_tune;

static bool valid_nt(int nt) { return nt == 128 || nt == 256 || nt == 512; }
static int type_bytes(int type) { return (type == ACC_I64 || type == ACC_F64) ? 8 : 4; }
// Elements per thread as the kernel takes them: 16 or 64 bytes' worth.  32 bytes, which
// tables and other launch shapes ask for, round up (1000 requests of 2^8 .. 2^22
// elements at 512 threads: 654 us with 16 bytes for those below a megabyte, 589 with 64).
static int norm_ipt(int ipt, int type) {
  const int eb = type_bytes(type);
  return B_BYTES[ipt * eb >= 32 ? 1 : 0] / eb;
}
static int bucket_of(int64_t n) {
  int b = 0;
  while (b < 62 && (int64_t(1) << (b + 1)) <= n) ++b;
  return b;
}
// Before tuning: the narrow tile where it holds the whole request.
static int default_ipt(int type, int64_t n, int nt) {
  return B_BYTES[n * type_bytes(type) > nt * B_BYTES[0] ? 1 : 0] / type_bytes(type);
}
// Before tuning, a request's threads per CTA:
//   * 128 up to 8 KB: more requests are in work at once (2000 scans of 2^8 Int32 / Float32
//     elements 11.0 / 13.7 -> 8.2 / 9.5 us of device time, of 2^10 Int64 15.4 -> 10.9; the tiles
//     of 2^12, 16 KB, are faster with 256: 17 and 19);
//   * 512 from a megabyte on: larger tiles, so fewer look-backs (1000 requests of 2^8 ..
//     2^22 elements 627 -> 589 us, one scan of 2^20 Float32 9.1 -> 8.0);
//   * 256 otherwise, and for Float64, whose additions bind it (500 scans of 2^17 545 us
//     with 512, 480 with 256).
static int default_nt(int type, int64_t n) {
  const int64_t bytes = n * type_bytes(type);
  if (bytes <= 8192) return 128;
  return type != ACC_F64 && bytes >= (1 << 20) ? 512 : BT;
}
// The request's entry of the tuning table, if it has one.
static bool tuned(int kind, int type, int64_t n, TuneVal *v) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  auto it = g_tune.find(TuneKey{kind, type, bucket_of(n)});
  if (it == g_tune.end()) return false;
  *v = it->second;
  return true;
}
// A request's elements per thread in a launch of nt threads: its tuned tile
// shape where the tuned launch shape is nt, else the same tile size in
// elements.
static int ipt_for(const acc_request &q, int nt) {
  TuneVal v;
  if (!tuned(q.kind, q.type, q.n, &v)) return default_ipt(q.type, q.n, nt);
  const int ipt = v.nt == nt ? v.ipt : (int)(((int64_t)v.ipt * v.nt) / nt);
  return norm_ipt(ipt, q.type);
}

// Elements of one item of request q in a launch of nt threads.
static int64_t item_elems(const acc_request &q, int ipt, int nt) {
  return (int64_t)ipt * nt * (q.kind == ACC_REQ_FOLD ? B_FOLD_STEPS : 1);
}

// ---------------------------------------------------------------- plan
struct Batch {
  int op;
  int device;
  int64_t count = 0, nitems = 0;
  BReq *d_reqs = nullptr;
  int32_t *d_item_req = nullptr;
  uint64_t *d_status = nullptr;
  uint64_t *d_partials = nullptr;
  uint32_t *d_req_ticket = nullptr;
  uint32_t *d_words = nullptr;
  int grid = 0;
  int nt = BT;  // threads per CTA
  size_t smem = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

template <int OP> static void *batch_kernel_ptr(int nt) {
  if (nt == 128) return reinterpret_cast<void *>(batch_kernel<OP, 128>);
  if (nt == 512) return reinterpret_cast<void *>(batch_kernel<OP, 512>);
  return reinterpret_cast<void *>(batch_kernel<OP, 256>);
}
static void *kernel_for(int op, int nt) {
  return op == ACC_ADD ? batch_kernel_ptr<ACC_ADD>(nt) : op == ACC_MIN ? batch_kernel_ptr<ACC_MIN>(nt)
                                                                       : batch_kernel_ptr<ACC_MAX>(nt);
}

template <int OP> static void launch_op(Batch *b, const BatchArgs &a, cudaStream_t s) {
  if (b->nt == 128) batch_kernel<OP, 128><<<b->grid, 160, b->smem, s>>>(a);
  else if (b->nt == 512) batch_kernel<OP, 512><<<b->grid, 544, b->smem, s>>>(a);
  else batch_kernel<OP, 256><<<b->grid, 288, b->smem, s>>>(a);
}
static int batch_launch_raw(Batch *b, cudaStream_t s) {
  BatchArgs a{b->d_reqs, b->d_item_req, b->nitems, b->d_status, b->d_partials, b->d_req_ticket, b->d_words};
  switch (b->op) {
    case ACC_ADD: launch_op<ACC_ADD>(b, a, s); break;
    case ACC_MIN: launch_op<ACC_MIN>(b, a, s); break;
    default: launch_op<ACC_MAX>(b, a, s); break;
  }
  return check_launch();
}

static void batch_free(Batch *b) {
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  cudaFree(b->d_reqs);
  cudaFree(b->d_item_req);
  cudaFree(b->d_status);
  cudaFree(b->d_partials);
  cudaFree(b->d_req_ticket);
  cudaFree(b->d_words);
  delete b;
}

// nt_override > 0 fixes the launch shape (with ipt_override, the tile
// shapes: the autotuner's trial launches); otherwise the batch takes the
// tuned launch shape that most of its bytes prefer.
static int batch_make(int op, const acc_request *reqs, int64_t count, const int32_t *ipt_override, int nt_override,
                      Batch **out) {
  if (op != ACC_ADD && op != ACC_MIN && op != ACC_MAX) return ACC_ERR_UNSUPPORTED;
  if (count < 0 || (count > 0 && !reqs) || count > (1ll << 31) - 1) return ACC_ERR_INVALID;
  int nt = BT;
  if (nt_override > 0) {
    if (!valid_nt(nt_override)) return ACC_ERR_INVALID;
    nt = nt_override;
  } else {
    double weight[3] = {0.0, 0.0, 0.0}, folds = 0.0;
    int64_t wide_items = 0;  // folds' items at 512 threads
    for (int64_t i = 0; i < count; ++i) {
      const acc_request &q = reqs[i];
      if (q.type != ACC_I32 && q.type != ACC_I64 && q.type != ACC_F32 && q.type != ACC_F64) continue;
      const double bytes = (double)(q.n > 0 ? q.n : 0) * type_bytes(q.type);
      TuneVal v{0, default_nt(q.type, q.n)};
      const bool table = tuned(q.kind, q.type, q.n, &v);
      for (int c = 0; c < 3; ++c)
        if (B_NT[c] == v.nt) weight[c] += bytes;
      if (q.kind == ACC_REQ_FOLD && !table && q.n > 0) {
        folds += bytes;
        wide_items += cdiv_h(q.n, item_elems(q, default_ipt(q.type, q.n, 512), 512));
      }
    }
    if (weight[0] > weight[1] && weight[0] >= weight[2]) nt = B_NT[0];
    else if (weight[2] > weight[1] && weight[2] > weight[0]) nt = B_NT[2];
    // Untuned folds that leave SMs without one of 512 threads' items take 256 (one fold of
    // 2^20 Float32 values 8.4 -> 7.2 us, of 2^18 Float64 12.1 -> 9.3).
    if (nt == B_NT[2] && folds > 0.5 * (weight[0] + weight[1] + weight[2]) && wide_items < device_info().sms) nt = BT;
  }
  std::vector<BReq> h(count);
  std::vector<int32_t> item_req;
  int64_t nitems = 0;
  for (int64_t i = 0; i < count; ++i) {
    const acc_request &q = reqs[i];
    if (q.kind != ACC_REQ_FOLD && q.kind != ACC_REQ_SCAN) return ACC_ERR_INVALID;
    if (q.type != ACC_I32 && q.type != ACC_I64 && q.type != ACC_F32 && q.type != ACC_F64) return ACC_ERR_UNSUPPORTED;
    if (q.n < 0 || (q.n > 0 && (!q.in || !q.out))) return ACC_ERR_INVALID;
    if (q.kind == ACC_REQ_FOLD && !q.out) return ACC_ERR_INVALID;  // fold z [] still writes z
    if (q.kind == ACC_REQ_FOLD && q.n == 0 && !q.has_seed) return ACC_ERR_EMPTY;
    const int ipt = ipt_override ? norm_ipt(ipt_override[i], q.type) : ipt_for(q, nt);
    const int64_t ts = item_elems(q, ipt, nt);
    int64_t ntl = (q.n + ts - 1) / ts;
    if (q.kind == ACC_REQ_FOLD && ntl == 0) ntl = 1;  // fold z [] = z: one (empty) tile writes the seed
    BReq &r = h[i];
    r.in = q.in; r.out = q.out; r.n = q.n; r.seed = q.seed;
    r.kind = q.kind; r.type = q.type; r.has_seed = q.has_seed; r.ipt = ipt;
    r.first_item = nitems; r.ntiles = ntl;
    for (int64_t k = 0; k < ntl; ++k) item_req.push_back((int32_t)i);
    nitems += ntl;
  }
  if (nitems >= (1ll << 31)) return ACC_ERR_TOO_LARGE;
  Batch *b = new Batch();
  b->op = op;
  b->nt = nt;
  cudaGetDevice(&b->device);
  b->count = count;
  b->nitems = nitems;
  b->smem = (size_t)(nt / 32) * 2 * b_wbuf_bytes();
  auto fail = [&](cudaError_t e) { batch_free(b); return cuda_status(e); };
  cudaError_t e;
  if ((e = cudaMalloc(&b->d_reqs, sizeof(BReq) * (count ? count : 1))) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&b->d_item_req, sizeof(int32_t) * (nitems ? nitems : 1))) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&b->d_status, sizeof(uint64_t) * 2 * (nitems ? nitems : 1))) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&b->d_partials, sizeof(uint64_t) * (nitems ? nitems : 1))) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&b->d_req_ticket, sizeof(uint32_t) * (count ? count : 1))) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&b->d_words, sizeof(uint32_t) * 64)) != cudaSuccess) return fail(e);
  if (count) cudaMemcpy(b->d_reqs, h.data(), sizeof(BReq) * count, cudaMemcpyHostToDevice);
  if (nitems) cudaMemcpy(b->d_item_req, item_req.data(), sizeof(int32_t) * nitems, cudaMemcpyHostToDevice);
  cudaMemset(b->d_status, 0, sizeof(uint64_t) * 2 * (nitems ? nitems : 1));
  cudaMemset(b->d_req_ticket, 0, sizeof(uint32_t) * (count ? count : 1));
  cudaMemset(b->d_words, 0, sizeof(uint32_t) * 64);
  void *kern = kernel_for(op, nt);
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b->smem);
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt + 32, b->smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  int64_t grid = (int64_t)device_info().sms * per_sm;
  if (grid > nitems) grid = nitems > 0 ? nitems : 1;
  b->grid = (int)grid;
  if ((e = cudaDeviceSynchronize()) != cudaSuccess) return fail(e);
  *out = b;
  return ACC_OK;
}

// ---------------------------------------------------------------- arena
// A reusable launch area for batches assembled on the fly (the serving
// loop): device arrays sized once for up to cap_reqs requests / cap_items
// tiles, pinned host staging for the descriptors.  A launch copies the new
// descriptors with cudaMemcpyAsync and runs the kernel; it allocates nothing.
// One arena serves one stream at a time: its staging buffers are reused only
// after the previous launch from the arena has completed.
struct BatchArena {
  Batch dev;            // device arrays and launch shape (count/nitems per launch)
  int64_t cap_reqs = 0, cap_items = 0;
  BReq *h_reqs = nullptr;
  int32_t *h_item = nullptr;
};

int arena_create(int op, int64_t cap_reqs, int64_t cap_items, BatchArena **out) {
  if (op != ACC_ADD && op != ACC_MIN && op != ACC_MAX) return ACC_ERR_UNSUPPORTED;
  BatchArena *ar = new BatchArena();
  Batch *b = &ar->dev;
  b->op = op;
  cudaGetDevice(&b->device);
  ar->cap_reqs = cap_reqs;
  ar->cap_items = cap_items;
  cudaError_t e;
  if ((e = cudaMalloc(&b->d_reqs, sizeof(BReq) * cap_reqs)) != cudaSuccess ||
      (e = cudaMalloc(&b->d_item_req, sizeof(int32_t) * cap_items)) != cudaSuccess ||
      (e = cudaMalloc(&b->d_status, sizeof(uint64_t) * 2 * cap_items)) != cudaSuccess ||
      (e = cudaMalloc(&b->d_partials, sizeof(uint64_t) * cap_items)) != cudaSuccess ||
      (e = cudaMalloc(&b->d_req_ticket, sizeof(uint32_t) * cap_reqs)) != cudaSuccess ||
      (e = cudaMalloc(&b->d_words, sizeof(uint32_t) * 64)) != cudaSuccess ||
      (e = cudaMallocHost(&ar->h_reqs, sizeof(BReq) * cap_reqs)) != cudaSuccess ||
      (e = cudaMallocHost(&ar->h_item, sizeof(int32_t) * cap_items)) != cudaSuccess) {
    arena_free(ar);
    return cuda_status(e);
  }
  cudaMemset(b->d_status, 0, sizeof(uint64_t) * 2 * cap_items);
  cudaMemset(b->d_req_ticket, 0, sizeof(uint32_t) * cap_reqs);
  cudaMemset(b->d_words, 0, sizeof(uint32_t) * 64);
  b->smem = (size_t)(BT / 32) * 2 * b_wbuf_bytes();
  b->nt = BT;
  void *kern = kernel_for(op, BT);
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b->smem);
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BT + 32, b->smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  b->grid = device_info().sms * per_sm;
  e = cudaDeviceSynchronize();
  if (e != cudaSuccess) { arena_free(ar); return cuda_status(e); }
  *out = ar;
  return ACC_OK;
}

// Tiles a request will take (0 if it does not fit the batch kernel).
int64_t arena_tiles(const acc_request &q) {
  const int ipt = ipt_for(q, BT);
  const int64_t ts = item_elems(q, ipt, BT);
  const int64_t nt = (q.n + ts - 1) / ts;
  return (q.kind == ACC_REQ_FOLD && nt == 0) ? 1 : nt;
}

int arena_launch(BatchArena *ar, const acc_request *reqs, int64_t count, cudaStream_t s) {
  Batch *b = &ar->dev;
  int64_t nitems = 0;
  for (int64_t i = 0; i < count; ++i) {
    const acc_request &q = reqs[i];
    const int ipt = ipt_for(q, BT);
    const int64_t ts = item_elems(q, ipt, BT);
    int64_t nt = (q.n + ts - 1) / ts;
    if (q.kind == ACC_REQ_FOLD && nt == 0) nt = 1;
    if (i >= ar->cap_reqs || nitems + nt > ar->cap_items) return ACC_ERR_TOO_LARGE;
    BReq &r = ar->h_reqs[i];
    r.in = q.in; r.out = q.out; r.n = q.n; r.seed = q.seed;
    r.kind = q.kind; r.type = q.type; r.has_seed = q.has_seed; r.ipt = ipt;
    r.first_item = nitems; r.ntiles = nt;
    for (int64_t k = 0; k < nt; ++k) ar->h_item[nitems + k] = (int32_t)i;
    nitems += nt;
  }
  if (nitems == 0) return ACC_OK;
  cudaError_t e = cudaMemcpyAsync(b->d_reqs, ar->h_reqs, sizeof(BReq) * count, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(b->d_item_req, ar->h_item, sizeof(int32_t) * nitems, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cuda_status(e);
  b->count = count;
  b->nitems = nitems;
  const int full_grid = b->grid;
  if (b->grid > nitems) b->grid = (int)nitems;
  const int st = batch_launch_raw(b, s);
  b->grid = full_grid;
  return st;
}

void arena_free(BatchArena *ar) {
  if (!ar) return;
  Batch *b = &ar->dev;
  cudaFree(b->d_reqs);
  cudaFree(b->d_item_req);
  cudaFree(b->d_status);
  cudaFree(b->d_partials);
  cudaFree(b->d_req_ticket);
  cudaFree(b->d_words);
  cudaFreeHost(ar->h_reqs);
  cudaFreeHost(ar->h_item);
  delete ar;
}

// ---------------------------------------------------------------- autotune
static int autotune_run(int kind, int type, int bucket, cudaStream_t s, void *buf, size_t buf_bytes, TuneVal *best) {
  const int64_t n = int64_t(1) << bucket;
  const int eb = type_bytes(type);
  // A batch of equal requests of this bucket's size, up to 2^24 elements in all.
  int64_t count = std::max<int64_t>(1, std::min<int64_t>(4096, (int64_t(1) << 24) / n));
  while (count > 1 && (size_t)(count * n * eb * 2 + count * 8) > buf_bytes) count /= 2;
  std::vector<acc_request> reqs(count);
  char *base = static_cast<char *>(buf);
  for (int64_t i = 0; i < count; ++i) {
    acc_request &q = reqs[i];
    q.kind = kind; q.type = type; q.n = n; q.has_seed = 0; q.seed = 0;
    q.in = base;                                  // all requests read the same input
    q.out = base + (size_t)n * eb + (kind == ACC_REQ_SCAN ? (size_t)i * n * eb : (size_t)i * eb);
  }
  float best_ms = 1e30f;
  TuneVal pick{default_ipt(type, n, BT), BT};
  // every launch shape, and for each every tile shape
  for (int nt : B_NT) {
    for (int bytes : B_BYTES) {
      const int ipt = bytes / eb;
      std::vector<int32_t> ov(count, ipt);
      Batch *b = nullptr;
      int st = batch_make(ACC_ADD, reqs.data(), count, ov.data(), nt, &b);
      if (st) return st;
      cudaEvent_t e0, e1;
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      batch_launch_raw(b, s);
      cudaEventRecord(e0, s);
      for (int rep = 0; rep < 3; ++rep) batch_launch_raw(b, s);
      cudaEventRecord(e1, s);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      batch_free(b);
      if (ms < best_ms) { best_ms = ms; pick = TuneVal{ipt, nt}; }
    }
  }
  *best = pick;
  return check_launch();
}

}  // namespace accgb

using namespace accgb;

extern "C" int acc_batch_create(int op, const acc_request *reqs, int64_t count, acc_batch **out) {
  if (!out) return ACC_ERR_INVALID;
  Batch *b = nullptr;
  int st = batch_make(op, reqs, count, nullptr, 0, &b);
  if (st) return st;
  *out = reinterpret_cast<acc_batch *>(b);
  return ACC_OK;
}

extern "C" int acc_batch_launch(acc_batch *batch, void *stream) {
  Batch *b = reinterpret_cast<Batch *>(batch);
  if (!b) return ACC_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (b->nitems == 0) return ACC_OK;
  if (b->exec) return cuda_status(cudaGraphLaunch(b->exec, s));
  return batch_launch_raw(b, s);
}

extern "C" int acc_batch_capture(acc_batch *batch, void *stream) {
  Batch *b = reinterpret_cast<Batch *>(batch);
  if (!b) return ACC_ERR_INVALID;
  if (b->exec || b->nitems == 0) return ACC_OK;
  (void)stream;  // captured on a private stream; replays go to the launch's stream
  cudaStream_t cap = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
  if (e != cudaSuccess) return cuda_status(e);
  e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    batch_launch_raw(b, cap);
    e = cudaStreamEndCapture(cap, &b->graph);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
  cudaStreamDestroy(cap);
  return cuda_status(e);
}

extern "C" int acc_batch_status(acc_batch *batch, void *stream) {
  Batch *b = reinterpret_cast<Batch *>(batch);
  if (!b) return ACC_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e);
  uint32_t err = 0;
  e = cudaMemcpy(&err, b->d_words, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_status(e);
  if (!err) return ACC_OK;
  cudaMemset(b->d_words, 0, sizeof(uint32_t) * 64);
  cudaMemset(b->d_status, 0, sizeof(uint64_t) * 2 * (b->nitems ? b->nitems : 1));
  cudaMemset(b->d_req_ticket, 0, sizeof(uint32_t) * (b->count ? b->count : 1));
  return ACC_ERR_TIMEOUT;
}

extern "C" int acc_batch_destroy(acc_batch *batch) {
  Batch *b = reinterpret_cast<Batch *>(batch);
  if (b) {
    cudaDeviceSynchronize();
    batch_free(b);
  }
  return ACC_OK;
}

extern "C" int acc_batch_autotune(const char *table_path, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t buf_bytes = (size_t)1 << 28;
  void *buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, buf_bytes);
  if (e != cudaSuccess) return cuda_status(e);
  cudaMemset(buf, 0, buf_bytes);
  std::map<TuneKey, TuneVal> table;
  const int kinds[2] = {ACC_REQ_FOLD, ACC_REQ_SCAN};
  const int types[4] = {ACC_I32, ACC_F32, ACC_I64, ACC_F64};
  int st = ACC_OK;
  for (int kind : kinds)
    for (int type : types)
      for (int bucket = 8; bucket <= 22 && st == ACC_OK; ++bucket) {
        TuneVal best{0, BT};
        st = autotune_run(kind, type, bucket, s, buf, buf_bytes, &best);
        if (st == ACC_OK) table[TuneKey{kind, type, bucket}] = best;
      }
  cudaFree(buf);
  if (st) return st;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    for (auto &kv : table) g_tune[kv.first] = kv.second;
  }
  if (table_path) {
    FILE *f = fopen(table_path, "w");
    if (!f) return ACC_ERR_INVALID;
    cudaDeviceProp p;
    cudaGetDeviceProperties(&p, 0);
    // entries: [kind, type, log2 size bucket, elements per thread, threads per CTA]
    fprintf(f, "{\"gpu\": \"%s\", \"entries\": [", p.name);
    bool first = true;
    for (auto &kv : table) {
      fprintf(f, "%s[%d, %d, %d, %d, %d]", first ? "" : ", ", kv.first.kind, kv.first.type, kv.first.bucket,
              kv.second.ipt, kv.second.nt);
      first = false;
    }
    fprintf(f, "]}\n");
    fclose(f);
  }
  return ACC_OK;
}

extern "C" int acc_batch_load_tuning(const char *table_path) {
  if (!table_path) return ACC_ERR_INVALID;
  FILE *f = fopen(table_path, "r");
  if (!f) return ACC_ERR_INVALID;
  std::string text;
  char chunk[4096];
  size_t got;
  while ((got = fread(chunk, 1, sizeof(chunk), f)) > 0) text.append(chunk, got);
  fclose(f);
  const size_t at = text.find("\"entries\"");
  if (at == std::string::npos) return ACC_ERR_INVALID;
  // entries of five numbers, or of four (tables written before the launch
  // shape was tuned: 256 threads per CTA)
  std::map<TuneKey, TuneVal> table;
  const char *p = text.c_str() + at;
  while ((p = strchr(p, '[')) != nullptr) {
    int kind, type, bucket, ipt, nt = BT;
    const int got5 = sscanf(p, "[%d, %d, %d, %d, %d]", &kind, &type, &bucket, &ipt, &nt);
    if (got5 >= 4) {
      if (got5 == 4) nt = BT;
      if (!valid_nt(nt)) return ACC_ERR_INVALID;
      table[TuneKey{kind, type, bucket}] = TuneVal{ipt, nt};
    }
    ++p;
  }
  std::lock_guard<std::mutex> lk(g_tune_mu);
  for (auto &kv : table) g_tune[kv.first] = kv.second;
  return ACC_OK;
}
