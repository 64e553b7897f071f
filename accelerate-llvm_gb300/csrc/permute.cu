// permute.cu -- permute f defaults p xs for the fixed primitives.
//
// The reference's permute_rmw issues one global atomic read-modify-write per
// source element (accelerate-llvm-ptx/src/Data/Array/Accelerate/LLVM/PTX/
// CodeGen/Permute.hs:117-213), so a skewed (Zipf) histogram serialises on the
// few hot bins in L2.  Kernels here:
//   * permute_count32 / permute_count16 -- integer + of a constant (histograms):
//     private counters in shared memory, 32 bits per bin while they fit, else
//     16 bits; the constant multiplies the counts once, at the end;
//   * permute_private -- every other update of a target that fits in shared
//     memory, where there are enough of them: a private copy of the target per
//     CTA, folded into global memory at the end;
//   * permute_cluster -- for 32-bit integer targets beyond that, up to 8 x 48K
//     bins: the target is privatised in the DISTRIBUTED shared memory of a
//     thread-block cluster (each CTA of the cluster holds 1/CL of the bins);
//   * permute_global -- red.global / atom.global RMW per element (any type,
//     any primitive; CAS loops for the primitives without a native atomic).
// Each update is out[j] = f x out[j] with the new value first, the order of
// the reference's combine (Native/CodeGen/Permute.hs:112-116).  Integer
// results do not depend on the update order; Float32/Float64 + does.
#include <cooperative_groups.h>
#include <cstdlib>
#include <cstring>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace accgb {

struct PermArgs {
  const void *src;
  const void *idx;
  void *out;
  int64_t n, m;
  uint64_t cval;
  int has_src;
  int idx64;
  int vec;  // idx and src are 16-byte aligned
  uint32_t *err;
};

// Atomic out[j] = f(x, out[j]) on global or shared (generic address) memory.
template <int OP, class T>
__device__ __forceinline__ void atomic_combine(T *p, T x) {
  if constexpr (std::is_same<T, int32_t>::value || std::is_same<T, uint32_t>::value) {
    if constexpr (OP == ACC_ADD) atomicAdd(p, x);
    else if constexpr (OP == ACC_MIN) atomicMin(p, x);
    else if constexpr (OP == ACC_MAX) atomicMax(p, x);
    else if constexpr (OP == ACC_AND) atomicAnd(p, x);
    else if constexpr (OP == ACC_OR) atomicOr(p, x);
    else if constexpr (OP == ACC_XOR) atomicXor(p, x);
    else {
      unsigned *q = reinterpret_cast<unsigned *>(p);
      unsigned old = *q, assumed;
      do {
        assumed = old;
        T nv = Prim<OP, T>::ap(x, (T)assumed);
        old = atomicCAS(q, assumed, (unsigned)nv);
      } while (old != assumed);
    }
  } else if constexpr (std::is_same<T, int64_t>::value) {
    unsigned long long *q = reinterpret_cast<unsigned long long *>(p);
    if constexpr (OP == ACC_ADD) atomicAdd(q, (unsigned long long)x);
    else if constexpr (OP == ACC_MIN) atomicMin(reinterpret_cast<long long *>(p), (long long)x);
    else if constexpr (OP == ACC_MAX) atomicMax(reinterpret_cast<long long *>(p), (long long)x);
    else if constexpr (OP == ACC_AND) atomicAnd(q, (unsigned long long)x);
    else if constexpr (OP == ACC_OR) atomicOr(q, (unsigned long long)x);
    else if constexpr (OP == ACC_XOR) atomicXor(q, (unsigned long long)x);
    else {
      unsigned long long old = *q, assumed;
      do {
        assumed = old;
        T nv = Prim<OP, T>::ap(x, (T)assumed);
        old = atomicCAS(q, assumed, (unsigned long long)nv);
      } while (old != assumed);
    }
  } else if constexpr (std::is_same<T, float>::value) {
    if constexpr (OP == ACC_ADD) atomicAdd(p, x);
    else {
      unsigned *q = reinterpret_cast<unsigned *>(p);
      unsigned old = *q, assumed;
      do {
        assumed = old;
        float nv = Prim<OP, float>::ap(x, __uint_as_float(assumed));
        if (__float_as_uint(nv) == assumed) break;  // min / max: already there
        old = atomicCAS(q, assumed, __float_as_uint(nv));
      } while (old != assumed);
    }
  } else {
    if constexpr (OP == ACC_ADD) atomicAdd(p, x);
    else {
      unsigned long long *q = reinterpret_cast<unsigned long long *>(p);
      unsigned long long old = *q, assumed;
      do {
        assumed = old;
        double nv = Prim<OP, double>::ap(x, __longlong_as_double((long long)assumed));
        if ((unsigned long long)__double_as_longlong(nv) == assumed) break;
        old = atomicCAS(q, assumed, (unsigned long long)__double_as_longlong(nv));
      } while (old != assumed);
    }
  }
}

__device__ __forceinline__ int64_t perm_idx(const PermArgs &a, int64_t i) {
  return a.idx64 ? static_cast<const int64_t *>(a.idx)[i] : (int64_t) static_cast<const int32_t *>(a.idx)[i];
}

// Four source elements of a round, in registers: their target indices as
// Int32 (negative: Nothing; a 64-bit index at or past m, which the shared
// memory kernels keep below 2^31, becomes m) and their values.  Unit v is the
// four consecutive elements 4v.. read with 16-byte loads, or four single
// elements.  FIXED: the array forms are known at compile time (IDX64, no
// source); otherwise the flags of PermArgs decide, the same for every thread.
template <class T, bool FIXED = false, bool IDX64 = false> struct PermUnit {
  int32_t j[4];
  T x[4];
  __device__ __forceinline__ static bool idx64(const PermArgs &a) { return FIXED ? IDX64 : a.idx64 != 0; }
  __device__ __forceinline__ static bool src(const PermArgs &a) { return FIXED ? false : a.has_src != 0; }
  __device__ __forceinline__ void clear(T c) {
#pragma unroll
    for (int k = 0; k < 4; ++k) { j[k] = -1; x[k] = c; }
  }
  __device__ __forceinline__ static int32_t narrow(int64_t j, int64_t m) {
    return j < 0 ? -1 : (j >= m ? (int32_t)m : (int32_t)j);
  }
  // ip, sp: the unit's first index and value
  __device__ __forceinline__ void load_vec(const PermArgs &a, const char *ip, const char *sp, T c) {
    if (idx64(a)) {
      const uint4 *p = reinterpret_cast<const uint4 *>(ip);
      const uint4 q0 = ld_stream16(p), q1 = ld_stream16(p + 1);
      int64_t w[4];
      memcpy(w, &q0, 16);
      memcpy(w + 2, &q1, 16);
#pragma unroll
      for (int k = 0; k < 4; ++k) j[k] = narrow(w[k], a.m);
    } else {
      const uint4 q = ld_stream16(ip);
      memcpy(j, &q, 16);
    }
    if (src(a)) {
      constexpr int Q = sizeof(T) / 4;
      uint4 q[Q];
#pragma unroll
      for (int k = 0; k < Q; ++k) q[k] = ld_stream16(reinterpret_cast<const uint4 *>(sp) + k);
      memcpy(x, q, sizeof(x));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = c;
    }
  }
  __device__ __forceinline__ void load_el(const PermArgs &a, int k, int64_t e) {
    if (idx64(a)) j[k] = narrow(ld_stream(static_cast<const int64_t *>(a.idx) + e), a.m);
    else j[k] = ld_stream(static_cast<const int32_t *>(a.idx) + e);
    if (src(a)) x[k] = ld_stream(static_cast<const T *>(a.src) + e);
  }
};

// Stream the source once over the whole grid: every thread gets U units per
// round and calls batch(units) convergently (the lanes of a warp run the same
// rounds; what a round lacks holds index -1).  The next round's loads are in
// flight while a round's updates run: an update's returned value is waited
// for, so without that the loads would start only after the last return
// (permute_count16, 2^28 uniform / Zipf indices: 0.205 / 0.220 ms with four
// units and no prefetch, 0.168 / 0.178 with two prefetched units).
// The source is read with 16-byte loads where idx and src are 16-byte aligned
// (a.vec), else element by element, each load coalesced over the warp.
template <class Unit, int U, class T, class F>
__device__ __forceinline__ void perm_stream(const PermArgs &a, T c, F &&batch) {
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  const int64_t nunits = a.n / 4;
  const int64_t per = a.vec ? U * nth : 4 * U * nth;   // units, or elements, per round
  const int64_t whole = a.vec ? nunits / per : 0;      // rounds in which every unit exists
  const int64_t rounds = a.vec ? (nunits + per - 1) / per + ((a.n & 3) ? 1 : 0) : (a.n + per - 1) / per;
  const int64_t ib = Unit::idx64(a) ? 32 : 16, sb = Unit::src(a) ? 4 * (int64_t)sizeof(T) : 0;  // bytes of a unit
  const char *ip = static_cast<const char *>(a.idx) + tid * ib;
  const char *sp = static_cast<const char *>(a.src) + tid * sb;
  auto load_whole = [&](Unit (&q)[U]) {  // the next round, every unit of it
#pragma unroll
    for (int u = 0; u < U; ++u) q[u].load_vec(a, ip + u * nth * ib, sp + u * nth * sb, c);
    ip += per * ib;
    sp += per * sb;
  };
  Unit next[U];
  if (whole > 0) load_whole(next);
  for (int64_t r = 0; r < whole; ++r) {
    Unit q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = next[u];
    if (r + 1 < whole) load_whole(next);
    batch(q);
  }
  for (int64_t r = whole; r < rounds; ++r) {
    Unit q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u].clear(c);
    if (!a.vec) {
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int64_t e = r * per + (u * 4 + k) * nth + tid;
          if (e < a.n) q[u].load_el(a, k, e);
        }
    } else if (r * per < nunits) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if ((r * U + u) * nth + tid < nunits) q[u].load_vec(a, ip + u * nth * ib, sp + u * nth * sb, c);
    } else if (4 * nunits + tid < a.n) {
      q[0].load_el(a, 0, 4 * nunits + tid);  // the last n % 4 elements
    }
    batch(q);
  }
}

template <int OP, class T>
__global__ void __launch_bounds__(256) permute_global(PermArgs a) {
  const T *src = static_cast<const T *>(a.src);
  T *out = static_cast<T *>(a.out);
  const T c = from_bits<T>(a.cval);
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  bool bad = false;
  auto one = [&](int64_t j, T x) {
    if (j < 0) return;  // Nothing: the element is dropped
    if (j >= a.m) { bad = true; return; }
    atomic_combine<OP, T>(out + j, x);
  };
  int64_t e0 = 0;
  if (OP != ACC_MUL && a.vec) {
    // 16-byte loads of four indices and four values.
    for (int64_t v = tid; v < a.n / 4; v += nth) {
      int64_t j[4];
      T x[4];
      if (a.idx64) {
        const uint4 q0 = ld_stream16(static_cast<const uint4 *>(a.idx) + 2 * v);
        const uint4 q1 = ld_stream16(static_cast<const uint4 *>(a.idx) + 2 * v + 1);
        memcpy(j, &q0, 16);
        memcpy(j + 2, &q1, 16);
      } else {
        const uint4 q = ld_stream16(static_cast<const uint4 *>(a.idx) + v);
        int32_t w[4];
        memcpy(w, &q, 16);
#pragma unroll
        for (int k = 0; k < 4; ++k) j[k] = w[k];
      }
      if (a.has_src) {
        constexpr int Q = sizeof(T) / 4;
        uint4 q[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) q[k] = ld_stream16(static_cast<const uint4 *>(a.src) + Q * v + k);
        memcpy(x, q, sizeof(x));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) one(j[k], a.has_src ? x[k] : c);
    }
    e0 = a.n / 4 * 4;
  }
  for (int64_t i = e0 + tid; i < a.n; i += nth) one(perm_idx(a, i), a.has_src ? src[i] : c);
  if (bad) raise_error(a.err, DEV_ERR_INDEX);
}

// ----------------------------------------------------------------- shared-memory counters
// Histograms (integer + of a constant c): bin j counts its updates and the
// target gets c * count once, which is the same wrapping sum.  One CTA of
// 1024 threads per SM holds all the bins.  Measured on a GB300, 2^28 Int32
// indices (floor 158 us): an increment by a constant 1 whose result is not
// used costs no more than reading the counter would (0.158-0.163 ms
// against 0.153-0.161 for a plain load), same-address lanes included, so the
// kernels are bound by reading the indices and by issue, and what an update
// does besides its increment is what counts.
constexpr int PERM_THREADS = 1024;
constexpr int PERM_U = 2;  // units of four elements per thread and round

// A private bin holds the combination of some of the updates without the
// target's own value, which for the floats' + and * may leave the type's range
// where no order that starts from the target does: 3e38 and 2e38 added to a
// target of -3e38, or 1e30 twice with a target of 0.  Such a bin is not folded in;
// its updates are applied to the target one by one instead, from a second read
// of the CTA's share of the source.  For + the bin itself tells: an infinity or
// NaN stays one.  For * a product that is not a normal number (zeros and lost bits
// of subnormals, too) turns the bin into a NaN, which stays.
template <int OP, class T> constexpr bool perm_redoes() { return is_fp<T>() && (OP == ACC_ADD || OP == ACC_MUL); }
template <class T> __device__ __forceinline__ uint32_t exponent_bits(T v) {  // 0: zero, subnormal; all ones: inf, NaN
  if constexpr (sizeof(T) == 4) return (__float_as_uint(v) >> 23) & 0xffu;
  else return (uint32_t)((unsigned long long)__double_as_longlong(v) >> 52) & 0x7ffu;
}
template <class T> constexpr uint32_t exponent_ones() { return sizeof(T) == 4 ? 0xffu : 0x7ffu; }
template <int OP, class T> __device__ __forceinline__ bool perm_redo(T bin) {
  if constexpr (perm_redoes<OP, T>()) return exponent_bits(bin) == exponent_ones<T>();
  else return false;
}

// The updates of the bins that were not folded in, one by one (a call of its
// own: inlined, it cost the kernel around it registers).
template <int OP, class T> __device__ __noinline__ void permute_redo(PermArgs a, const T *bins) {
  const uint32_t m = (uint32_t)a.m;
  T *out = static_cast<T *>(a.out);
  using Unit = PermUnit<T>;
  perm_stream<Unit, PERM_U>(a, from_bits<T>(a.cval), [&](const Unit (&q)[PERM_U]) {
#pragma unroll
    for (int u = 0; u < PERM_U; ++u)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int32_t j = q[u].j[k];
        if ((uint32_t)j < m && perm_redo<OP, T>(bins[j])) atomic_combine<OP, T>(out + j, q[u].x[k]);
      }
  });
}

// 32 bits per bin.  A counter may wrap mod 2^32 only beyond 2^32 updates per
// CTA, where the 32-bit targets wrap as well and a 64-bit target's source
// could not be in memory.
template <class T, bool I64>
__global__ void __launch_bounds__(PERM_THREADS, 1) permute_count32(PermArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t *bins = reinterpret_cast<uint32_t *>(smem_raw);
  const uint32_t m = (uint32_t)a.m;
  for (uint32_t b = threadIdx.x; b < m; b += PERM_THREADS) bins[b] = 0u;
  __syncthreads();
  int32_t top = -1;
  using Unit = PermUnit<uint32_t, true, I64>;
  perm_stream<Unit, PERM_U>(a, 0u, [&](const Unit (&q)[PERM_U]) {
#pragma unroll
    for (int u = 0; u < PERM_U; ++u)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int32_t j = q[u].j[k];
        top = j > top ? j : top;
        if ((uint32_t)j < m) atomicAdd(bins + j, 1u);
      }
  });
  if (top >= (int32_t)m) raise_error(a.err, DEV_ERR_INDEX);
  __syncthreads();
  T *out = static_cast<T *>(a.out);
  const T c = from_bits<T>(a.cval);
  for (uint32_t b = threadIdx.x; b < m; b += PERM_THREADS) {
    const uint32_t n = bins[b];
    if (n) atomic_combine<ACC_ADD, T>(out + b, Prim<ACC_MUL, T>::ap((T)n, c));
  }
}

// 16 bits per bin, two to a word: bin w in the low half of word w and bin
// w + half in its high half, half = ceil(m / 2), so that neighbouring bins,
// which skewed (Zipf-like) indices make hot together, sit in different banks.
// No counter ever wraps: a counter at or above 0x8000 (its guard bit) is
// moved to the target.  Every update returns the word it found; a thread
// tests the OR of its batch of 8 once, and if a guard bit was set it takes
// each still-guarded word of the batch with an exchange and adds both
// counters to the target.  Until the first such exchange after a counter
// reaches 0x8000, a thread can add at most its current batch to it (any
// update after the crossing sees the guard), so the counter stays below
// 0x8000 + 1024 * 8 < 2^16.
// 2^28 Zipf(1.1) indices to 2^16 bins: a wrap test and repair per update took
// 0.257 ms, this 0.202 ms (uniform indices 0.176); a barrier and a sweep of the words every 32 updates
// 0.29 ms; 57,344 32-bit counters with only the remaining bins packed into
// high halves 0.34 ms (two divergent updates per index).
template <class T, bool I64>
__global__ void __launch_bounds__(PERM_THREADS, 1) permute_count16(PermArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t *words = reinterpret_cast<uint32_t *>(smem_raw);
  constexpr uint32_t GUARD = 0x80008000u;
  const uint32_t m = (uint32_t)a.m, half = (m + 1) / 2;
  for (uint32_t b = threadIdx.x; b < half; b += PERM_THREADS) words[b] = 0u;
  __syncthreads();
  T *out = static_cast<T *>(a.out);
  const T c = from_bits<T>(a.cval);
  auto flush = [&](uint32_t w, uint32_t v) {
    if (v & 0xffffu) atomic_combine<ACC_ADD, T>(out + w, Prim<ACC_MUL, T>::ap((T)(v & 0xffffu), c));
    if (v >> 16) atomic_combine<ACC_ADD, T>(out + w + half, Prim<ACC_MUL, T>::ap((T)(v >> 16), c));
  };
  int32_t top = -1;
  using Unit = PermUnit<uint32_t, true, I64>;
  perm_stream<Unit, PERM_U>(a, 0u, [&](const Unit (&q)[PERM_U]) {
    uint32_t seen = 0u;
#pragma unroll
    for (int u = 0; u < PERM_U; ++u)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int32_t j = q[u].j[k];
        top = j > top ? j : top;
        const bool low = (uint32_t)j < half;
        const uint32_t w = low ? (uint32_t)j : (uint32_t)j - half;
        if ((uint32_t)j < m) seen |= atomicAdd(words + w, low ? 1u : 0x10000u);
      }
    if (seen & GUARD) {
#pragma unroll
      for (int u = 0; u < PERM_U; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int32_t j = q[u].j[k];
          if ((uint32_t)j >= m) continue;
          const uint32_t w = (uint32_t)j < half ? (uint32_t)j : (uint32_t)j - half;
          if (*reinterpret_cast<volatile uint32_t *>(words + w) & GUARD) flush(w, atomicExch(words + w, 0u));
        }
    }
  });
  if (top >= (int32_t)m) raise_error(a.err, DEV_ERR_INDEX);
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < half; b += PERM_THREADS) flush(b, words[b]);
}

// ----------------------------------------------------------------- private target
// A private copy of the target in shared memory (identity-filled), one CTA of
// 1024 threads per SM; at the end each CTA folds its touched bins into the
// target.  L2 takes about 0.15 updates/ns whatever the target and one update
// per 1.5 ns on a single address; shared memory takes five times that.
// 2 * 10^7 Float32 values by 5 * 10^4 uniform keys: 0.166 -> 0.050 ms; 6.4 *
// 10^6 Int64 values by 25,000: 0.057 -> 0.029 ms.  Few updates do not pay for the
// filling and the folding: see perm_private_pays.
//
// 64-bit integer bins are kept as two 32-bit words (all low words first), each
// updated by a native 32-bit atomic: + adds the low halves, sees its carry in
// the returned word and adds it with the high halves (0.06 ms for 2 * 10^7
// values against 0.06-0.11 with the 64-bit compare-and-swap that atomicAdd is
// there, and 0.06 against 0.6 ms under Zipf keys); and / or / xor are
// bitwise.  64-bit min / max and the floats are compare-and-swap loops.
template <int OP, class T> constexpr bool split64() {
  return std::is_same<T, int64_t>::value && (OP == ACC_ADD || OP == ACC_AND || OP == ACC_OR || OP == ACC_XOR);
}
// Float + is a compare-and-swap loop that serialises lanes and warps on a hot
// bin: lanes of a warp with the same key are added up first where keys repeat.
template <int OP, class T> constexpr bool perm_aggregates() { return OP == ACC_ADD && is_fp<T>(); }

template <int OP, class T>
__device__ __forceinline__ void private_update(unsigned char *bins, uint32_t m, uint32_t j, T x) {
  if constexpr (split64<OP, T>()) {
    uint32_t *lo = reinterpret_cast<uint32_t *>(bins) + j, *hi = lo + m;
    const uint32_t xl = (uint32_t)(uint64_t)x, xh = (uint32_t)((uint64_t)x >> 32);
    if constexpr (OP == ACC_ADD) {
      const uint32_t old = atomicAdd(lo, xl);
      atomicAdd(hi, xh + (old + xl < xl ? 1u : 0u));
    } else if constexpr (OP == ACC_AND) { atomicAnd(lo, xl); atomicAnd(hi, xh); }
    else if constexpr (OP == ACC_OR) { atomicOr(lo, xl); atomicOr(hi, xh); }
    else { atomicXor(lo, xl); atomicXor(hi, xh); }
  } else if constexpr (OP == ACC_MUL && is_fp<T>()) {
    using U = typename std::conditional<sizeof(T) == 4, unsigned, unsigned long long>::type;
    U *q = reinterpret_cast<U *>(bins) + j;
    U old = *q, assumed;
    do {
      assumed = old;
      T nv = Prim<OP, T>::ap(x, from_bits<T>(assumed));
      const uint32_t e = exponent_bits(nv);
      if (e == 0u || e == exponent_ones<T>()) nv = Prim<ACC_MAX, T>::id();  // NaN
      if ((U)to_bits(nv) == assumed) break;
      old = atomicCAS(q, assumed, (U)to_bits(nv));
    } while (old != assumed);
  } else {
    atomic_combine<OP, T>(reinterpret_cast<T *>(bins) + j, x);
  }
}
template <int OP, class T>
__device__ __forceinline__ T private_bin(const unsigned char *bins, uint32_t m, uint32_t j) {
  if constexpr (split64<OP, T>()) {
    const uint32_t *lo = reinterpret_cast<const uint32_t *>(bins) + j;
    return (T)((uint64_t)lo[0] | ((uint64_t)lo[m] << 32));
  } else {
    return reinterpret_cast<const T *>(bins)[j];
  }
}

template <int OP, class T>
__global__ void __launch_bounds__(PERM_THREADS, 1) permute_private(PermArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t m = (uint32_t)a.m;
  const T idT = Prim<OP, T>::id();
  if constexpr (split64<OP, T>()) {
    // both halves of the identity (0 or all ones) are the same word
    for (uint32_t b = threadIdx.x; b < 2 * m; b += PERM_THREADS)
      reinterpret_cast<uint32_t *>(smem_raw)[b] = (uint32_t)(uint64_t)idT;
  } else {
    for (uint32_t b = threadIdx.x; b < m; b += PERM_THREADS) reinterpret_cast<T *>(smem_raw)[b] = idT;
  }
  __syncthreads();
  const T c = from_bits<T>(a.cval);
  const int lane = threadIdx.x & 31;
  int32_t top = -1;
  uint32_t round = 0;
  bool repeats = false;
  using Unit = PermUnit<T>;
  perm_stream<Unit, PERM_U>(a, c, [&](const Unit (&q)[PERM_U]) {
    if constexpr (perm_aggregates<OP, T>()) {
      // Every 8th round the warp looks at two of its updates: a key that three
      // lanes share turns the aggregation on (uniform keys over 256 bins do
      // that in 15 % of the looks, Zipf(1.1) keys in 85 %).  2 * 10^7 Float32
      // values over 5 * 10^4 bins, when a lane still added its peers one by one:
      // uniform keys always 0.172 ms, never 0.045; Zipf keys never 0.350.
      if ((round++ & 7u) == 0u) {
        const unsigned g0 = __match_any_sync(0xffffffffu, q[0].j[0]), g1 = __match_any_sync(0xffffffffu, q[PERM_U - 1].j[3]);
        const bool three = (q[0].j[0] >= 0 && __popc(g0) > 2) || (q[PERM_U - 1].j[3] >= 0 && __popc(g1) > 2);
        repeats = __any_sync(0xffffffffu, three);
      }
    }
#pragma unroll
    for (int u = 0; u < PERM_U; ++u)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int32_t j = q[u].j[k];
        top = j > top ? j : top;
        T x = q[u].x[k];
        bool mine = (uint32_t)j < m;
        if constexpr (perm_aggregates<OP, T>()) {
          if (repeats) {  // warp-uniform
            // pairwise in the order of the lanes: a key that every lane has
            // takes 5 steps, not 31 (a lane that its partner has taken leaves the
            // group).  2^22 sorted keys over 20,000 bins: Float32 66 -> 25 us,
            // Float64 283 -> 72 (in L2 86); one key, Float32 73 -> 27.
            const unsigned grp = __match_any_sync(0xffffffffu, j);
            const unsigned below = (1u << lane) - 1u;
            unsigned rest = grp & ~below & ~(1u << lane), rank = __popc(grp & below);
            while (__any_sync(0xffffffffu, rest != 0u)) {
              const T o = shfl_idx(x, rest ? __ffs(rest) - 1 : lane);
              if (rest) x = Prim<OP, T>::ap(x, o);
              rest &= __ballot_sync(0xffffffffu, (rank & 1u) == 0u);
              rank >>= 1;
            }
            mine = mine && (__ffs(grp) - 1) == lane;
          }
        }
        if (mine) private_update<OP, T>(smem_raw, m, (uint32_t)j, x);
      }
  });
  if (top >= (int32_t)m) raise_error(a.err, DEV_ERR_INDEX);
  __syncthreads();

  // Fold this CTA's bins into the target; untouched bins hold the identity.
  T *out = static_cast<T *>(a.out);
  bool redo = false;
  uint32_t b0 = 0;
  if constexpr (OP == ACC_ADD && std::is_same<T, float>::value) {
    // Four bins per reduction; an untouched bin takes -0.0, which changes nothing
    // but a target that the reduction would rewrite: a subnormal is flushed, a NaN
    // may lose its payload.  So the targets are read first; no reduction leaves a
    // subnormal, and one that makes a NaN leaves the canonical one, so an earlier
    // value tells as much as the present one.  Where an untouched target is
    // such a number, each touched bin is added by itself (20 M values into 50,021 bins: 63
    // us with the vector form only where all four were touched, 57 so).
    if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
      const uint32_t none = __float_as_uint(idT);
      b0 = m & ~3u;
#pragma unroll 4
      for (uint32_t b = 4 * threadIdx.x; b < b0; b += 4 * PERM_THREADS) {
        const float4 v = *reinterpret_cast<const float4 *>(smem_raw + b * sizeof(T));
        const uint4 t = __ldcg(reinterpret_cast<const uint4 *>(out + b));
        const float f[4] = {v.x, v.y, v.z, v.w};
        const uint32_t old[4] = {t.x, t.y, t.z, t.w};
        bool any = false, apart = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t mag = old[k] & 0x7fffffffu;
          if (perm_redo<OP, T>(f[k])) redo = apart = any = true;
          else if (__float_as_uint(f[k]) != none) any = true;
          else if (mag - 1u < 0x007fffffu || mag > 0x7f800000u) apart = true;
        }
        if (!any) continue;
        if (!apart) {
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                       :: "l"(out + b), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]) : "memory");
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (__float_as_uint(f[k]) != none && !perm_redo<OP, T>(f[k])) atomic_combine<OP, T>(out + b + k, f[k]);
        }
      }
    }
  }
  for (uint32_t b = b0 + threadIdx.x; b < m; b += PERM_THREADS) {
    const T v = private_bin<OP, T>(smem_raw, m, b);
    if (perm_redo<OP, T>(v)) redo = true;
    else if (to_bits(v) != to_bits(idT)) atomic_combine<OP, T>(out + b, v);
  }
  if constexpr (perm_redoes<OP, T>()) {
    if (__syncthreads_or(redo)) permute_redo<OP, T>(a, reinterpret_cast<const T *>(smem_raw));
  }
}

// Privatised permute into cluster-distributed shared memory.  CL CTAs form a
// cluster; bin j is owned by CTA (j & (CL-1)) of the cluster, at local slot
// j >> log2(CL).  An update to an owned bin is a shared-memory atomic, an
// update to a bin of the partner CTA a `red.shared::cluster` on its shared
// memory.  AGG: lanes of a warp that hit the same bin are combined first
// (match.any) so a hot bin costs one atomic per warp instead of one per lane.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
template <int OP, class T>
__device__ __forceinline__ void red_cluster(uint32_t addr, T v) {
  static_assert(sizeof(T) == 4, "32-bit bins");
  if constexpr (OP == ACC_ADD) asm volatile("red.shared::cluster.add.u32 [%0], %1;" :: "r"(addr), "r"((uint32_t)v) : "memory");
  else if constexpr (OP == ACC_AND) asm volatile("red.shared::cluster.and.b32 [%0], %1;" :: "r"(addr), "r"((uint32_t)v) : "memory");
  else if constexpr (OP == ACC_OR) asm volatile("red.shared::cluster.or.b32 [%0], %1;" :: "r"(addr), "r"((uint32_t)v) : "memory");
  else if constexpr (OP == ACC_XOR) asm volatile("red.shared::cluster.xor.b32 [%0], %1;" :: "r"(addr), "r"((uint32_t)v) : "memory");
  else if constexpr (OP == ACC_MIN) {
    if constexpr (std::is_same<T, int32_t>::value) asm volatile("red.shared::cluster.min.s32 [%0], %1;" :: "r"(addr), "r"(v) : "memory");
    else asm volatile("red.shared::cluster.min.u32 [%0], %1;" :: "r"(addr), "r"(v) : "memory");
  } else {
    if constexpr (std::is_same<T, int32_t>::value) asm volatile("red.shared::cluster.max.s32 [%0], %1;" :: "r"(addr), "r"(v) : "memory");
    else asm volatile("red.shared::cluster.max.u32 [%0], %1;" :: "r"(addr), "r"(v) : "memory");
  }
}
// Value that `cnt` equal lanes combine into (AGG): + multiplies, the
// idempotent primitives keep one, xor keeps the parity.
template <int OP, class T> __device__ __forceinline__ T agg_value(T x, int cnt) {
  if constexpr (OP == ACC_ADD) return (T)((uint32_t)x * (uint32_t)cnt);
  else if constexpr (OP == ACC_XOR) return (cnt & 1) ? x : T(0);
  else return x;
}

template <int OP, class T, int LOG_CL, bool AGG>
__global__ void __launch_bounds__(1024, 1) permute_cluster(PermArgs a, int per) {
  constexpr int CL = 1 << LOG_CL;
  static_assert(CL > 1 && CL <= 8, "a portable cluster");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *bins = reinterpret_cast<T *>(smem_raw);
  const uint32_t rank = cg::this_cluster().block_rank();
  const T idT = Prim<OP, T>::id();
  for (int b = threadIdx.x; b < per; b += blockDim.x) bins[b] = idT;
  cg::this_cluster().sync();
  const uint32_t bins_addr = smem_addr(bins);
  uint32_t remote_base[CL];
#pragma unroll
  for (int r = 0; r < CL; ++r) remote_base[r] = mapa_shared(bins_addr, (uint32_t)r);

  const T *src = static_cast<const T *>(a.src);
  const T c = from_bits<T>(a.cval);
  const uint32_t m = (uint32_t)a.m;
  bool bad = false;
  // Lanes call `one` convergently (AGG needs the whole warp); a dropped or
  // out-of-range element passes j < 0 / j >= m and does nothing.
  auto one = [&](int32_t j, T x) {
    const bool ok = j >= 0 && (uint32_t)j < m;
    bad |= (j >= 0 && !ok);
    T v = x;
    bool lead = ok;
    if constexpr (AGG) {
      // Lanes with the same target AND the same value combine into one update.
      uint32_t xb;
      memcpy(&xb, &x, 4);
      const unsigned long long key = ok ? (((unsigned long long)(uint32_t)j << 32) | xb) : ~0ull;
      const unsigned grp = __match_any_sync(0xffffffffu, key);
      lead = ok && (__ffs(grp) - 1) == (int)(threadIdx.x & 31);
      v = agg_value<OP, T>(x, __popc(grp));
    }
    if (!lead) return;
    const uint32_t owner = (uint32_t)j & (CL - 1), slot = (uint32_t)j >> LOG_CL;
    if (owner == rank) atomic_combine<OP, T>(bins + slot, v);
    else red_cluster<OP, T>(remote_base[owner] + slot * 4u, v);
  };
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;
  if (!a.idx64 && !a.has_src && (reinterpret_cast<uintptr_t>(a.idx) & 15u) == 0) {
    // Histogram fast path: Int32 indices, 16 per thread per round, 4 loads in flight.
    const int64_t nv = a.n / 4;
    const uint4 *iv = static_cast<const uint4 *>(a.idx);
    const int64_t rounds = (nv + 4 * nth - 1) / (4 * nth);
    for (int64_t r = 0; r < rounds; ++r) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t v = (r * 4 + u) * nth + tid;
        q[u] = v < nv ? ld_stream16(iv + v) : make_uint4(~0u, ~0u, ~0u, ~0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        one((int32_t)q[u].x, c); one((int32_t)q[u].y, c); one((int32_t)q[u].z, c); one((int32_t)q[u].w, c);
      }
    }
    const int64_t tail = a.n - nv * 4;  // < 4 elements
    one(tid < tail ? static_cast<const int32_t *>(a.idx)[nv * 4 + tid] : -1, c);
  } else {
    const int64_t rounds = (a.n + nth - 1) / nth;
    for (int64_t r = 0; r < rounds; ++r) {
      const int64_t i = r * nth + tid;
      int64_t j = -1;
      T x = c;
      if (i < a.n) {
        j = perm_idx(a, i);
        if (a.has_src) x = src[i];
      }
      // 64-bit indices beyond Int32 range are out of range for a 32-bit bin array.
      if (j >= (int64_t)m) { bad = true; j = -1; }
      one((int32_t)j, x);
    }
  }
  if (bad) raise_error(a.err, DEV_ERR_INDEX);
  cg::this_cluster().sync();

  // Fold this CTA's bins into the target; untouched bins hold the identity.
  T *out = static_cast<T *>(a.out);
  for (int b = threadIdx.x; b < per; b += blockDim.x) {
    const T v = bins[b];
    const int64_t j = ((int64_t)b << LOG_CL) | rank;
    if (v != idT && j < a.m) atomic_combine<OP, T>(out + j, v);
  }
}

// ----------------------------------------------------------------- host side
// Variant choice (tuning knob, default "auto"): ACC_GB300_PERMUTE = auto |
// cluster | global (anything else is auto), ACC_GB300_PERMUTE_AGG = 0 | 1 (the
// cluster kernel's).
static int env_int(const char *name, int dflt) {
  const char *v = getenv(name);
  return v ? atoi(v) : dflt;
}
static const char *env_str(const char *name) {
  const char *v = getenv(name);
  return v ? v : "auto";
}

template <class K, class... Args>
static int launch_cluster(K kern, int CL, unsigned threads, size_t smem, int64_t want_ctas, cudaStream_t s,
                          Args... args) {
  const Device &d = device_info();
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(CL * d.sms);
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters <= 0) {
    cudaGetLastError();
    clusters = d.sms / CL > 0 ? d.sms / CL : 1;
  }
  int64_t grid = (int64_t)clusters * CL;
  const int64_t want = cdiv_h(want_ctas, CL) * CL;
  if (grid > want) grid = want;
  if (grid < CL) grid = CL;
  cfg.gridDim = dim3((unsigned)grid);
  return cuda_status(cudaLaunchKernelEx(&cfg, kern, args...));
}

template <int OP, class T, int LOG_CL>
static int launch_permute_cluster(PermArgs a, bool agg, cudaStream_t s) {
  const int CL = 1 << LOG_CL;
  const int per = (int)cdiv_h(a.m, CL);
  const size_t smem = (size_t)per * sizeof(T);
  const int64_t want = cdiv_h(a.n, 1024 * 16);
  if (agg) return launch_cluster(permute_cluster<OP, T, LOG_CL, true>, CL, 1024, smem, want, s, a, per);
  return launch_cluster(permute_cluster<OP, T, LOG_CL, false>, CL, 1024, smem, want, s, a, per);
}

// One of the shared-memory kernels above on `smem` bytes of bins.  CTAs: one
// per SM, fewer when each would have less than `per_cta` elements to stream,
// since every CTA fills and folds a whole copy of the bins.
template <class K>
static int launch_private(K kern, std::atomic<uint64_t> &attr_done, size_t smem, int64_t per_cta, const PermArgs &a,
                          cudaStream_t s) {
  const Device &d = device_info();
  smem_attrs_once(kern, d.max_smem_optin, attr_done);
  int64_t grid = cdiv_h(a.n, per_cta);
  if (grid > d.sms) grid = d.sms;
  kern<<<(unsigned)grid, PERM_THREADS, smem, s>>>(a);
  return check_launch();
}

template <class T, bool I64>
static int launch_count(const PermArgs &a, bool wide, size_t smem, int64_t per_cta, cudaStream_t s) {
  static std::atomic<uint64_t> done32{0}, done16{0};
  return wide ? launch_private(permute_count32<T, I64>, done32, smem, per_cta, a, s)
              : launch_private(permute_count16<T, I64>, done16, smem, per_cta, a, s);
}

// Whether n updates of m bins go to private bins (which a CTA fills and folds
// however few of its updates meet there) rather than to L2 one by one (where those
// of one bin take 1.5 ns each).  Neither way is the better one for all keys, and the
// keys are not known here; us of device time, private bins / L2:
//   * 32-bit integers but *, one copy with native atomics: always.
//   * 64-bit integers and every *: from 2^15 updates.  2^14 Int64 values into 2^10
//     bins, uniform keys 7.1 / 4.2, Zipf keys 7.4 / 6.8; 2^15 into 2^9 uniform 6.8 /
//     5.4, Zipf 7.3 / 11; 2^17 into 2^12 uniform 7.6 / 5.0, Zipf 7.8 / 29.
//   * Float32 +: from 2^18, with 128 updates per bin from 2^16.  2^17 values into
//     2^12 bins, uniform 9.9 / 6.8, Zipf 18.7 / 29.7; 2^18 into 2^13 10.4 / 6.4 and
//     19.4 / 53; 2^16 into 2^8 13.6 / 17.3 and 17.7 / 21.5.
//   * Float64 +: from 2^20.  2^18 into 2^12, uniform 14.7 / 6.5, Zipf 79 / 66; 2^20
//     into 2^14 18.6 / 13.6 and 84 / 223.
//   * min and max of floats, compare-and-swap loops either way: from 64 (Float64 128)
//     updates per bin.  2^18 Float32 values into 2^13 bins, uniform 21 / 9.1, Zipf
//     22 / 62; into 2^12 18.7 / 11.6 and 18.5 / 67.
template <int OP, class T> static bool perm_private_pays(int64_t n, int64_t m) {
  if constexpr (is_fp<T>() && (OP == ACC_MIN || OP == ACC_MAX)) return n >= (sizeof(T) == 4 ? 64 : 128) * m;
  else if constexpr (is_fp<T>() && OP == ACC_ADD && sizeof(T) == 4) return n >= (1 << 18) || (n >= (1 << 16) && n >= 128 * m);
  else if constexpr (is_fp<T>() && OP == ACC_ADD) return n >= (1 << 20);
  else if constexpr (sizeof(T) == 8 || OP == ACC_MUL) return n >= (1 << 15);
  else return true;
}

template <int OP, class T>
int permute_typed(Workspace *w, PermArgs a, cudaStream_t s) {
  const Device &d = device_info();
  a.err = w->words + W_ERR;
  if (a.n == 0) return ACC_OK;
  const char *variant = env_str("ACC_GB300_PERMUTE");
  const bool agg = env_int("ACC_GB300_PERMUTE_AGG", 0) != 0;
  const bool force_global = strcmp(variant, "global") == 0, force_cluster = strcmp(variant, "cluster") == 0;
  constexpr bool int32ish = std::is_same<T, int32_t>::value || std::is_same<T, uint32_t>::value;
  a.vec = aligned16(a.idx) && (!a.has_src || aligned16(a.src));
  // Private bins in shared memory from four updates per bin on.
  const bool many = a.m > 0 && a.n >= 4 * a.m;
  const int64_t smem_cap = d.max_smem_optin - 1024;
  const int64_t bytes = a.m * (int64_t)sizeof(T);
  const int64_t per_cta = 1024 * 8;
  if (many && !force_global && !force_cluster && perm_private_pays<OP, T>(a.n, a.m)) {
    if constexpr (OP == ACC_ADD && !is_fp<T>()) {
      const bool wide = a.m * 4 <= smem_cap;
      if (!a.has_src && (a.m + 1) / 2 * 4 <= smem_cap) {
        const size_t smem = (size_t)(wide ? a.m : (a.m + 1) / 2) * 4;
        return a.idx64 ? launch_count<T, true>(a, wide, smem, per_cta, s)
                       : launch_count<T, false>(a, wide, smem, per_cta, s);
      }
    }
    if (bytes <= smem_cap) {
      static std::atomic<uint64_t> done{0};
      return launch_private(permute_private<OP, T>, done, (size_t)bytes, per_cta, a, s);
    }
  }
  if constexpr (int32ish && OP != ACC_MUL) {
    const int64_t cap_bytes = d.max_smem_optin > (200 << 10) ? (192 << 10) : (int64_t)d.max_smem_optin - (8 << 10);
    const int64_t cap = cap_bytes / (int64_t)sizeof(T);
    if (!force_global && many) {
      if (a.m <= 2 * cap) return launch_permute_cluster<OP, T, 1>(a, agg, s);
      if (a.m <= 4 * cap) return launch_permute_cluster<OP, T, 2>(a, agg, s);
      if (a.m <= 8 * cap) return launch_permute_cluster<OP, T, 3>(a, agg, s);
    }
  }
  // Four updates per thread from where one each nearly fills the machine; below, more
  // threads are worth more than wider loads.  Compare-and-swap minima and maxima from
  // 2^19 (2^17 Float32 max into 2^15 bins: 15.2 us by four, 7.0 by one; 2^19 into 2^15 15.7 and
  // 21), native atomics from 2^21 (2^20 Int64 sums into 200,000 bins 18.2 and 16.5, 2^22 32.6
  // and 32.8), products, whose retries four at a time add to, never (2^22 Int32 products into
  // 200,000 bins, uniform keys 108 and 96, 2^24 under Zipf keys 5690 and 5050).
  constexpr bool loops = is_fp<T>() && (OP == ACC_MIN || OP == ACC_MAX);
  if (OP == ACC_MUL || a.n < (loops ? 1 << 19 : 1 << 21)) a.vec = 0;
  int64_t blocks = cdiv_h(a.vec ? cdiv_h(a.n, 4) : a.n, 256);
  if (blocks > (int64_t)d.sms * 16) blocks = (int64_t)d.sms * 16;
  permute_global<OP, T><<<(unsigned)blocks, 256, 0, s>>>(a);
  return check_launch();
}

}  // namespace accgb

using namespace accgb;

extern "C" int acc_permute(int op, int type, const void *src, const void *cval, const void *idx,
                           int index_type, void *out, int64_t n, int64_t m, void *stream) {
  if (n < 0 || m < 0) return ACC_ERR_INVALID;
  if (index_type != ACC_I32 && index_type != ACC_I64) return ACC_ERR_INVALID;
  if (!src && !cval) return ACC_ERR_INVALID;
  if (n > 0 && (!idx || !out)) return ACC_ERR_INVALID;
  if (type < ACC_I32 || type > ACC_F64) return ACC_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int st = ACC_OK;
  Workspace *w = workspace(s, &st);
  if (!w) return st;
  std::lock_guard<std::mutex> lk(w->mu);
  return with_type(type, [&](auto tv) -> int {
    using T = decltype(tv);
    PermArgs a{};
    a.src = src; a.idx = idx; a.out = out; a.n = n; a.m = m;
    a.cval = src ? 0 : seed_bits<T>(cval);
    a.has_src = src != nullptr;
    a.idx64 = index_type == ACC_I64;
    return with_op<T>(op, [&](auto opc) -> int {
      constexpr int OP = decltype(opc)::value;
      return permute_typed<OP, T>(w, a, s);
    });
  });
}

extern "C" int acc_permute_clone(int op, int type, const void *defaults, const void *src, const void *cval,
                                 const void *idx, int index_type, void *out, int64_t n, int64_t m,
                                 void *stream) {
  if (m < 0 || (m > 0 && (!defaults || !out))) return ACC_ERR_INVALID;
  static const size_t esz[] = {4, 8, 4, 4, 8};
  if (type < ACC_I32 || type > ACC_F64) return ACC_ERR_INVALID;
  // acc_permute's own argument checks, made before the clone so that a
  // rejected call leaves `out` untouched.
  if (n < 0 || (index_type != ACC_I32 && index_type != ACC_I64) || (!src && !cval) || (n > 0 && !idx))
    return ACC_ERR_INVALID;
  if (op < ACC_ADD || op > ACC_XOR) return ACC_ERR_INVALID;
  if (op >= ACC_AND && (type == ACC_F32 || type == ACC_F64)) return ACC_ERR_UNSUPPORTED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (m > 0) {
    cudaError_t e = cudaMemcpyAsync(out, defaults, (size_t)m * esz[type], cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return cuda_status(e);
  }
  return acc_permute(op, type, src, cval, idx, index_type, out, n, m, stream);
}
