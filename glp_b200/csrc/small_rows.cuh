// small_rows.cuh -- rows staged in shared memory by the warp, up to 32 entries
// a lane (kernels.cuh, k_small and k_pair; batch.cu): where an entry sits, and
// the row's best label by sorting, for a row per lane and a row per two lanes.
#pragma once
#include <type_traits>

#include "device.cuh"

namespace glp {

// Entry i of thread t's row sits in word small_at<R>(t, i): eight lanes storing
// eight entries of four rows, and 32 threads reading entry i of their rows, both
// touch 32 different banks.
template <int R>
__device__ __forceinline__ int small_turn(int t) {
  constexpr int k = 32 / R;
  return 8 * ((t / k) % (k < 4 ? 4 / k : 1)) + (t >> 2);
}
template <int R>
__device__ __forceinline__ int small_at(int t, int i) {
  return t * R + ((i + small_turn<R>(t)) & (R - 1));
}
// The best (score, label) of one row, N >= its degree d: the labels are sorted
// (K: as they are; with weights or volumes to follow, label * 32 + entry), the
// running total of a run never exceeds its last one, and equal scores come in
// ascending label order, so the last best element is the answer.  `own`: the
// thread's first words.
template <int N, int R, bool W, class S, class K>
__device__ __forceinline__ int32_t small_best(const S& score, const uint32_t* slab, int t, int d) {
  constexpr bool kKeyed = W || S::kLV;
  constexpr K kNone = kKeyed ? (K)~(K)0 : (K)INT32_MAX;
  const uint32_t* sw = slab + 32 * R;
  const uint32_t* svol = slab + 32 * R * (W ? 2 : 1);
  K key[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    key[i] = kNone;
    if (i < d) {
      const uint32_t l = slab[small_at<R>(t, i)];
      if (!S::kKeep || (int32_t)l >= 0) key[i] = kKeyed ? (K)((K)l << 5 | (K)i) : (K)l;  // unlabelled: no entry
    }
  }
  sort_keys(key);
  int32_t bl = -1;
  std::conditional_t<S::kPacked, uint32_t, int64_t> bs{};
  uint32_t run = 0;
  constexpr int U = N < 8 ? N : 8;  // global volume lookups in flight
#pragma unroll
  for (int i0 = 0; i0 < N; i0 += U) {
    int32_t vl[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u;
      if (i >= N) break;
      const int32_t l = (int32_t)(kKeyed ? key[i] >> 5 : key[i]);
      vl[u] = 0;
      if (key[i] != kNone) {
        const int at = small_at<R>(t, (int)(key[i] & 31));
        if constexpr (S::kLV) {
          vl[u] = (int32_t)svol[at];
        } else if constexpr (S::kScan) {  // a run is scored at its last element only
          const bool end = i == N - 1 || (kKeyed ? key[i + 1 < N ? i + 1 : i] >> 5 : key[i + 1 < N ? i + 1 : i]) != (K)l;
          if (end) vl[u] = score.vol_of(l);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u;
      if (i >= N) break;
      if (key[i] == kNone) continue;
      const int32_t l = (int32_t)(kKeyed ? key[i] >> 5 : key[i]);
      const bool same = i > 0 && (kKeyed ? key[i ? i - 1 : 0] >> 5 : key[i ? i - 1 : 0]) == (K)l;
      const uint32_t w = W ? sw[small_at<R>(t, (int)(key[i] & 31))] : 1u;
      run = same ? run + w : w;
      if constexpr (S::kScan && !S::kLV) {
        const bool end = i == N - 1 || (kKeyed ? key[i + 1 < N ? i + 1 : i] >> 5 : key[i + 1 < N ? i + 1 : i]) != (K)l;
        if (!end) continue;
      }
      if constexpr (S::kPacked) {
        const uint32_t c = score.key32(run, vl[u]);
        if (bl < 0 || c >= bs) {
          bs = c;
          bl = l;
        }
      } else {
        const int64_t c = score.from_vol(run, vl[u]);
        if (bl < 0 || c >= bs) {
          bs = c;
          bl = l;
        }
      }
    }
  }
  return bl;
}

// The row of thread t, by the network of the warp's largest degree dmax
// (neighbouring vertices of a degree-sorted graph have about the same).
template <int R, bool W, class S, class K>
__device__ __forceinline__ int32_t small_row_best(const S& score, const uint32_t* slab, int t, int d, int dmax) {
  if constexpr (R == 8) {
    return dmax <= 4 ? small_best<4, R, W, S, K>(score, slab, t, d) : small_best<8, R, W, S, K>(score, slab, t, d);
  } else if constexpr (R == 16) {
    return dmax <= 12 ? small_best<12, R, W, S, K>(score, slab, t, d) : small_best<16, R, W, S, K>(score, slab, t, d);
  } else {
    return dmax <= 8    ? small_best<8, R, W, S, K>(score, slab, t, d)  // a small graph's merged tiers
           : dmax <= 16 ? small_best<16, R, W, S, K>(score, slab, t, d)
           : dmax <= 20 ? small_best<20, R, W, S, K>(score, slab, t, d)
           : dmax <= 24 ? small_best<24, R, W, S, K>(score, slab, t, d)
           : dmax <= 28 ? small_best<28, R, W, S, K>(score, slab, t, d)
                        : small_best<32, R, W, S, K>(score, slab, t, d);
  }
}

// Sorts the first N of 32 keys; the others are the largest key already.
template <int N>
__device__ __forceinline__ void sort_first(int32_t (&x)[32]) {
  int32_t y[N];
#pragma unroll
  for (int i = 0; i < N; ++i) y[i] = x[i];
  sort_keys(y);
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = y[i];
}

// The best (key, label) of a row over two lanes (lane, lane ^ 1), as key << 32 |
// label on both; labels alone (no weights or volumes), 0 when none is labelled
// (scores with kKeep).  The lane holds d <= 32 of the entries, dmax = the
// warp's largest d.  Each lane sorts its own, one exchange in opposite order
// leaves the smaller half of all keys on the even lane, five bitonic rounds
// sort each half, and each lane reads the counts off its runs; the odd lane's
// first run goes on from the even lane's last.
template <class S>
__device__ __forceinline__ unsigned long long pair_best(const S& score, const uint32_t* slab, int lane, int d,
                                                        int dmax) {
  static_assert(S::kPacked && !S::kScan, "counts alone");
  int32_t key[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    key[i] = INT32_MAX;
    if (i < d) {
      const int32_t l = (int32_t)slab[small_at<32>(lane, i)];
      if (!S::kKeep || l >= 0) key[i] = l;  // unlabelled: no entry
    }
  }
  if (dmax <= 20) sort_first<20>(key);
  else if (dmax <= 24) sort_first<24>(key);
  else if (dmax <= 28) sort_first<28>(key);
  else sort_first<32>(key);
  const bool low = (lane & 1) == 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int32_t p = __shfl_xor_sync(kFull, key[31 - i], 1), q = __shfl_xor_sync(kFull, key[i], 1);
    key[i] = low ? min(key[i], p) : max(key[i], p);
    key[31 - i] = low ? min(key[31 - i], q) : max(key[31 - i], q);
  }
#pragma unroll
  for (int j = 16; j >= 1; j /= 2)
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if ((i & j) == 0) {
        const int32_t lo = min(key[i], key[i + j]), hi = max(key[i], key[i + j]);
        key[i] = lo;
        key[i + j] = hi;
      }
  // the even lane's last run, where the odd lane's first label continues it
  uint32_t tail = 1;
#pragma unroll
  for (int i = 1; i < 32; ++i) tail = key[i] == key[i - 1] ? tail + 1u : 1u;
  const int32_t before = __shfl_up_sync(kFull, key[31], 1);
  const uint32_t carry = __shfl_up_sync(kFull, tail, 1);
  uint32_t run = !low && key[0] == before ? carry : 0u;
  PackedCand best;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (i > 0 && key[i] != key[i > 0 ? i - 1 : 0]) run = 0;
    ++run;
    const uint32_t c = score.key32(run, 0);
    if (key[i] != INT32_MAX && c >= best.s) {  // labels ascend: equal keys take the later
      best.s = c;
      best.l = (uint32_t)key[i];
    }
  }
  const unsigned long long mine = ((unsigned long long)best.s << 32) | best.l;
  return max(mine, __shfl_xor_sync(kFull, mine, 1));
}

}  // namespace glp
