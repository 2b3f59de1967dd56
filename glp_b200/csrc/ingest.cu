// ingest.cu -- building the int32 CSR of an edge list on the device.
//
// Reference semantics: tools/normalize.cpp:262-348 (degree-descending
// relabel) and header/graph.h:226-258 (edge list -> CSR: self loops dropped,
// both directions stored for an undirected graph).  Here, on the device, with
// b the bits of an id:
//   1. every edge (u,v), u != v, becomes one key: u << b | v, the smaller id
//      first for an undirected graph (both directions are one key until the
//      columns are written: half the keys to sort);
//   2. unless ids are kept, duplicates are dropped through hash buckets (the
//      keys need no order yet: two partition passes instead of a full sort),
//      degrees counted, vertices renumbered by degree descending, ties by the
//      smaller original id (normalize.cpp's order, made deterministic), and
//      the keys rewritten;
//   3. the keys are sorted (stable LSD radix sort, 8-bit digits).  When ids are
//      kept, duplicates are now adjacent and dropped;
//   4. sorted, the keys are the entries (u, v > u) of every row in order.  An
//      undirected graph's other half, the entries (v, u < v), is a stable sort
//      of the same keys by their second id alone; a row is its part of the
//      second list followed by its part of the first.
// The result equals, bit for bit, the host construction the tests and the
// samplers use (symmetrise, drop self loops, sort, dedupe, relabel).
//
// Measured on one B200, 67.1 M R-MAT scale-22 edges in device memory to the
// handle: the kernels take 10.9 ms (33 ms with both directions sorted twice by
// 12 passes of one key per thread and round, 2.1 ms a pass).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "../../include/glp.h"
#include "device.cuh"
#include "smem_attr.h"

namespace glp {
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
int device_sms();
cudaError_t dev_alloc_raw(void** p, size_t bytes);
void dev_free(void* p);
void dev_pool_trim();
int graph_adopt(int32_t* d_off, int32_t* d_cols, int32_t n, int64_t m, uint32_t flags, glp_graph** out);
}  // namespace glp

namespace {

using glp::kFull;

#define ICUDA(call)                                            \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return glp::cuda_fail(e_, #call);   \
  } while (0)

constexpr int kNT = 256;  // threads per block of the streaming kernels
constexpr int kSortNT = 512, kSortItems = 16, kSortTile = kSortNT * kSortItems;  // 8192 keys per tile
constexpr int kSortWarps = kSortNT / 32;
constexpr int kRadix = 256;
constexpr int kScanNT = 256, kScanPer = 8, kScanBlock = kScanNT * kScanPer;
constexpr uint64_t kNoKey = ~0ull;  // no key has its top bits set

int bit_length(uint64_t x) {
  int b = 0;
  while (x) {
    ++b;
    x >>= 1;
  }
  return b;
}

// ------------------------------------------------------------------ scan
// Exclusive scan of uint32 counts, in place, block by block; sums[b] gets
// block b's total.
__global__ void __launch_bounds__(kScanNT) k_scan_blocks(uint32_t* __restrict__ a, int64_t len,
                                                         uint32_t* __restrict__ sums) {
  __shared__ uint32_t wsum[kScanNT / 32];
  const int64_t base = (int64_t)blockIdx.x * kScanBlock + (int64_t)threadIdx.x * kScanPer;
  uint32_t x[kScanPer], run = 0;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    x[i] = base + i < len ? a[base + i] : 0u;
    const uint32_t t = x[i];
    x[i] = run;
    run += t;
  }
  // exclusive scan of the thread totals
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  uint32_t wbase = 0, total = 0;
  for (int w = 0; w < kScanNT / 32; ++w) {
    if (w < warp) wbase += wsum[w];
    total += wsum[w];
  }
  const uint32_t off = wbase + inc - run;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i)
    if (base + i < len) a[base + i] = x[i] + off;
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void k_scan_add(uint32_t* __restrict__ a, int64_t len, const uint32_t* __restrict__ sums) {
  const int64_t b = blockIdx.x;
  const uint32_t add = sums[b];
  for (int64_t i = b * kScanBlock + threadIdx.x; i < std::min(len, (b + 1) * kScanBlock); i += blockDim.x)
    a[i] += add;
}

// Exclusive scan of len counts (total < 2^32).  scratch: >= scan_scratch(len)
// words.
int64_t scan_scratch(int64_t len) {
  int64_t need = 0;
  while (len > 1) {
    len = (len + kScanBlock - 1) / kScanBlock;
    need += len;
  }
  return need + 1;
}

int scan_u32(uint32_t* a, int64_t len, uint32_t* scratch, cudaStream_t s) {
  if (len <= 0) return GLP_OK;
  const int64_t nb = (len + kScanBlock - 1) / kScanBlock;
  k_scan_blocks<<<(unsigned)nb, kScanNT, 0, s>>>(a, len, scratch);
  ICUDA(cudaGetLastError());
  if (nb > 1) {
    int rc = scan_u32(scratch, nb, scratch + nb, s);
    if (rc) return rc;
    k_scan_add<<<(unsigned)nb, 256, 0, s>>>(a, len, scratch);
    ICUDA(cudaGetLastError());
  }
  return GLP_OK;
}

// ------------------------------------------------------------ radix sort
// The digit a pass sorts by: bits of the key, or of its hash.
struct KeyDigit {
  int shift;
  uint32_t mask;
  __device__ __forceinline__ uint32_t operator()(uint64_t key) const { return (uint32_t)(key >> shift) & mask; }
};
struct HashDigit {
  int shift;
  uint32_t mask;
  __device__ __forceinline__ uint32_t operator()(uint64_t key) const {
    return (uint32_t)(glp::mix64(key) >> shift) & mask;
  }
};

// Per tile, the count of each digit: hist[digit * ntiles + tile]
// (digit-major, so one exclusive scan gives every tile's first position of
// every digit).  A thread adds a run of equal digits at once: the high digits
// of a degree-sorted graph's keys are almost all the same, and adds to one
// address would serialise.
template <class D>
__global__ void __launch_bounds__(kNT) k_digit_hist(const uint64_t* __restrict__ keys, int64_t n, D digit,
                                                    uint32_t* __restrict__ hist, int64_t ntiles) {
  __shared__ uint32_t h[kRadix];
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    for (int d = threadIdx.x; d < kRadix; d += kNT) h[d] = 0;
    __syncthreads();
    const int64_t base = t * kSortTile;
    uint32_t cur = 0, run = 0;
#pragma unroll 8
    for (int r = 0; r < kSortTile / kNT; ++r) {
      const int64_t i = base + (int64_t)r * kNT + threadIdx.x;
      if (i >= n) break;
      const uint32_t d = digit(keys[i]);
      if (d != cur) {
        if (run) atomicAdd(&h[cur], run);
        cur = d;
        run = 0;
      }
      ++run;
    }
    if (run) atomicAdd(&h[cur], run);
    __syncthreads();
    for (int d = threadIdx.x; d <= (int)digit.mask; d += kNT) hist[(int64_t)d * ntiles + t] = h[d];
    __syncthreads();
  }
}

struct ScatterShared {
  uint64_t keys[kSortTile];
  uint32_t wcnt[kSortWarps][kRadix];
  uint32_t first[kRadix];  // a digit's first position in the tile
  uint32_t gofs[kRadix];   // what takes a position in the tile to the output
  uint32_t wsum[kRadix / 32];
};

// Stable scatter by one digit, a tile per block: each warp reads 512
// consecutive keys and ranks them against its own counts (lanes holding one
// digit are found with eight ballots); the warps' counts give every key its
// place in the tile, the tile is put in that order in shared memory, and each
// digit's keys leave as one run of consecutive words (32 keys, 256 bytes, on
// average; a key per thread and round wrote 8-byte words all over the output:
// 134 M keys a pass took 2.1 ms, 64 M keys take 0.46 now).  Bound by issue:
// the eight ballots are a third of its instructions.
template <class D>
__global__ void __launch_bounds__(kSortNT, 2) k_digit_scatter(const uint64_t* __restrict__ in,
                                                              uint64_t* __restrict__ out, int64_t n, D digit,
                                                              const uint32_t* __restrict__ offs, int64_t ntiles) {
  extern __shared__ __align__(16) unsigned char sort_smem[];
  ScatterShared& sh = *reinterpret_cast<ScatterShared*>(sort_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = blockIdx.x, base = t * kSortTile;
  const int32_t cnt = (int32_t)(n - base < kSortTile ? n - base : kSortTile);
  for (int x = threadIdx.x; x < kSortWarps * kRadix; x += kSortNT) (&sh.wcnt[0][0])[x] = 0u;
  const int32_t mine = warp * (32 * kSortItems) + lane;
  uint64_t key[kSortItems];
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) key[i] = mine + 32 * i < cnt ? in[base + mine + 32 * i] : 0ull;
  __syncthreads();
  uint32_t rank[kSortItems / 2] = {};  // ranks among the warp's keys of the digit, two to a word
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const bool valid = mine + 32 * i < cnt;
    const uint32_t d = digit(key[i]);
    uint32_t peers = __ballot_sync(kFull, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const bool bit = (d >> b) & 1u;
      const uint32_t m = __ballot_sync(kFull, bit);
      peers &= bit ? m : ~m;
    }
    const uint32_t before = valid ? sh.wcnt[warp][d] : 0u;
    const uint32_t r = __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
    if (valid && r == 0) sh.wcnt[warp][d] = before + __popc(peers);
    __syncwarp();
    rank[i / 2] |= (before + r) << (16 * (i & 1));
  }
  __syncthreads();
  // per digit, the warps' counts become offsets in warp order; the digits'
  // totals become positions in the tile
  uint32_t total = 0, inc = 0;
  if (threadIdx.x < kRadix) {
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t c = sh.wcnt[w][threadIdx.x];
      sh.wcnt[w][threadIdx.x] = total;
      total += c;
    }
    inc = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) sh.wsum[warp] = inc;
  }
  __syncthreads();
  if (threadIdx.x < kRadix) {
    uint32_t first = inc - total;
    for (int w = 0; w < warp; ++w) first += sh.wsum[w];
    sh.first[threadIdx.x] = first;
    sh.gofs[threadIdx.x] = threadIdx.x <= digit.mask ? offs[(int64_t)threadIdx.x * ntiles + t] - first : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const uint32_t d = digit(key[i]), r = (rank[i / 2] >> (16 * (i & 1))) & 0xffffu;
    if (mine + 32 * i < cnt) sh.keys[sh.first[d] + sh.wcnt[warp][d] + r] = key[i];
  }
  __syncthreads();
  for (int32_t i = threadIdx.x; i < cnt; i += kSortNT) {
    const uint64_t k = sh.keys[i];
    out[sh.gofs[digit(k)] + (uint32_t)i] = k;
  }
}

struct Sorter {
  uint32_t* hist = nullptr;     // kRadix counts per tile
  uint32_t* scratch = nullptr;  // scan_scratch of them
};

template <class D>
int radix_pass(const uint64_t* in, uint64_t* out, int64_t n, const D& digit, const Sorter& so, cudaStream_t s) {
  const int64_t ntiles = (n + kSortTile - 1) / kSortTile;
  k_digit_hist<D><<<(unsigned)std::min<int64_t>(ntiles, (int64_t)glp::device_sms() * 8), kNT, 0, s>>>(in, n, digit,
                                                                                                 so.hist, ntiles);
  ICUDA(cudaGetLastError());
  int rc = scan_u32(so.hist, (int64_t)(digit.mask + 1) * ntiles, so.scratch, s);
  if (rc) return rc;
  ICUDA(glp::raise_smem_limit((const void*)k_digit_scatter<D>, sizeof(ScatterShared)));
  k_digit_scatter<D><<<(unsigned)ntiles, kSortNT, sizeof(ScatterShared), s>>>(in, out, n, digit, so.hist, ntiles);
  ICUDA(cudaGetLastError());
  return GLP_OK;
}

// Sorts n keys by bits [lo, lo + width) of the key (or of its hash), digits of
// at most 8 bits and equal width.  The passes write *a and *b in turn from
// `in`, which may be *b and is otherwise left as it is; *a ends as the sorted
// list (`in` itself when there is nothing to do), *b as the other buffer.
template <class D>
int radix_sort(uint64_t* in, uint64_t** a, uint64_t** b, int64_t n, int lo, int width, const Sorter& so,
               cudaStream_t s) {
  const int passes = n > 1 ? (width + 7) / 8 : 0;
  if (passes == 0) {
    if (in == *b) std::swap(*a, *b);
    else *a = in;
    return GLP_OK;
  }
  const uint64_t* src = in;
  for (int p = 0, at = 0; p < passes; ++p) {
    const int w = (width - at + passes - p - 1) / (passes - p);
    if (p) std::swap(*a, *b);
    int rc = radix_pass(src, *a, n, D{lo + at, (1u << w) - 1u}, so, s);
    if (rc) return rc;
    src = *a;
    at += w;
  }
  return GLP_OK;
}

// ------------------------------------------------------------- CSR steps
// Keys of the valid edges, appended in any order: a block packs the keys of
// 2048 edges with one add to the counter (one add per warp serialised on it:
// 1.7 ms for 67 M edges).  Bad ids (outside [0, n)) set bad.
constexpr int kEdgeItems = 8;
__global__ void __launch_bounds__(kNT) k_edge_keys(const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                                                   int64_t count, int32_t n, int both, int idbits,
                                                   uint64_t* __restrict__ keys, unsigned long long* nkeys,
                                                   uint32_t* bad) {
  __shared__ uint32_t wtot[kNT / 32];
  __shared__ unsigned long long sbase;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t i0 = (int64_t)blockIdx.x * (kNT * kEdgeItems); i0 < count;
       i0 += (int64_t)gridDim.x * (kNT * kEdgeItems)) {
    uint64_t key[kEdgeItems];
    uint32_t in_warp = 0, at[kEdgeItems];
#pragma unroll
    for (int q = 0; q < kEdgeItems; ++q) {
      const int64_t i = i0 + q * kNT + threadIdx.x;
      key[q] = kNoKey;
      if (i < count) {
        const int32_t u = __ldcs(src + i), v = __ldcs(dst + i);
        if (u < 0 || u >= n || v < 0 || v >= n) atomicOr(bad, 1u);
        else if (u != v)
          key[q] = both && v < u ? ((uint64_t)(uint32_t)v << idbits) | (uint32_t)u
                                 : ((uint64_t)(uint32_t)u << idbits) | (uint32_t)v;
      }
    }
#pragma unroll
    for (int q = 0; q < kEdgeItems; ++q) {
      const uint32_t m = __ballot_sync(kFull, key[q] != kNoKey);
      at[q] = in_warp + __popc(m & ((1u << lane) - 1u));
      in_warp += __popc(m);
    }
    if (lane == 0) wtot[warp] = in_warp;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t run = 0;
      for (int w = 0; w < kNT / 32; ++w) {
        const uint32_t c = wtot[w];
        wtot[w] = run;
        run += c;
      }
      sbase = run ? atomicAdd(nkeys, (unsigned long long)run) : 0ull;
    }
    __syncthreads();
    const unsigned long long b = sbase + wtot[warp];
#pragma unroll
    for (int q = 0; q < kEdgeItems; ++q)
      if (key[q] != kNoKey) keys[b + at[q]] = key[q];
    __syncthreads();  // wtot and sbase are read no more
  }
}

// start[r], r in [0, rows]: the first key whose row is at least r (the keys
// ascend by row).
struct FirstId {
  int bits;
  __device__ __forceinline__ int64_t operator()(uint64_t key) const { return (int64_t)(key >> bits); }
};
struct SecondId {
  uint64_t mask;
  __device__ __forceinline__ int64_t operator()(uint64_t key) const { return (int64_t)(key & mask); }
};
struct HashBucket {
  int shift;  // 64: one bucket
  __device__ __forceinline__ int64_t operator()(uint64_t key) const {
    return shift == 64 ? 0 : (int64_t)(glp::mix64(key) >> shift);
  }
};
template <class R>
__global__ void k_starts(const uint64_t* __restrict__ keys, int64_t m, int64_t rows, R row,
                         int32_t* __restrict__ start) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r <= rows; r += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = m;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (row(keys[mid]) < r) lo = mid + 1;
      else hi = mid;
    }
    start[r] = (int32_t)lo;
  }
}

// Claims or finds key's slot in a table of kDedupeSlots; false past kProbeMost
// probes.  *fresh grows when this call claimed it.
constexpr int kDedupeSlots = 2048, kDedupeMean = 1024, kProbeMost = 128;
__device__ __forceinline__ bool dedupe_insert(uint64_t* table, uint64_t key, uint64_t hash, uint32_t* fresh) {
  uint32_t slot = (uint32_t)hash & (kDedupeSlots - 1);
  for (int probe = 0; probe < kProbeMost; ++probe) {
    const uint64_t prev = atomicCAS((unsigned long long*)&table[slot], (unsigned long long)kNoKey,
                                    (unsigned long long)key);
    if (prev == kNoKey) ++*fresh;
    if (prev == kNoKey || prev == key) return true;
    slot = (slot + 1) & (kDedupeSlots - 1);
  }
  return false;
}

// A pair that repeats fills its bucket with copies, and a bucket has one block.
// So the tiles of kSortTile keys that lie within one bucket (an ordinary bucket
// holds none) drop their copies first, a block per tile: the distinct keys move
// to the tile's front and left[t] is their number; a tile of too many keeps all.
// A key already in its slot is read there, not claimed: equal claims of a warp
// serialise.  (67 M edges, a quarter of them one pair: 53.3 -> 10.4 ms to the
// handle; all one pair 177 -> 5.8.)
__global__ void __launch_bounds__(kNT) k_thin(uint64_t* __restrict__ keys, HashBucket bucket,
                                              uint32_t* __restrict__ left) {
  __shared__ uint64_t table[kDedupeSlots];
  __shared__ uint32_t cursor;
  uint64_t* tile = keys + (int64_t)blockIdx.x * kSortTile;
  if (bucket(tile[0]) != bucket(tile[kSortTile - 1])) return;  // block-uniform
  for (int s = threadIdx.x; s < kDedupeSlots; s += kNT) table[s] = kNoKey;
  if (threadIdx.x == 0) cursor = 0u;
  __syncthreads();
  uint32_t fresh = 0;
  bool full = false;
#pragma unroll 8
  for (int i = threadIdx.x; i < kSortTile; i += kNT) {
    const uint64_t key = tile[i], h = glp::mix64(key);
    if (*(volatile uint64_t*)&table[(uint32_t)h & (kDedupeSlots - 1)] != key)
      full = !dedupe_insert(table, key, h, &fresh) || full;
  }
  if (__syncthreads_or(full)) {  // block-uniform; every key has been read
    if (threadIdx.x == 0) left[blockIdx.x] = kSortTile;
    return;
  }
  for (int s = threadIdx.x; s < kDedupeSlots; s += kNT)
    if (table[s] != kNoKey) tile[atomicAdd(&cursor, 1u)] = table[s];
  __syncthreads();
  if (threadIdx.x == 0) left[blockIdx.x] = cursor;
}

// Drops duplicate keys.  A block per hash bucket (about 1000 keys) inserts
// them in a shared table and writes the distinct ones, in no order, to `out`,
// counting degrees.  Of the tiles within the bucket it takes the left[t] keys
// that k_thin left.  A bucket whose keys do not fit (a probe past kProbeMost)
// is split by further bits of the hash, as often as it takes: the classes
// (level, low bits) are walked depth first, each written once.
__global__ void __launch_bounds__(kNT) k_dedupe(const uint64_t* __restrict__ keys, const int32_t* __restrict__ start,
                                                const uint32_t* __restrict__ left, int32_t nbuckets, int idbits,
                                                int both, uint64_t* __restrict__ out, unsigned long long* nout,
                                                int32_t* __restrict__ deg) {
  __shared__ uint64_t table[kDedupeSlots];
  __shared__ uint32_t cursor;
  __shared__ unsigned long long sbase;
  const int lane = threadIdx.x & 31;
  const uint64_t idmask = (1ull << idbits) - 1ull;
  for (int32_t bk = blockIdx.x; bk < nbuckets; bk += gridDim.x) {
    const int32_t kb = start[bk], ke = start[bk + 1];
    const int32_t t0 = (kb + kSortTile - 1) / kSortTile, t1 = ke / kSortTile;  // tiles within the bucket
    int level = 0;
    uint64_t cls = 0;  // keys whose (hash >> 11) & (2^level - 1) is cls
    for (bool more = true; more;) {
      for (int s = threadIdx.x; s < kDedupeSlots; s += kNT) table[s] = kNoKey;
      if (threadIdx.x == 0) cursor = 0u;
      __syncthreads();
      uint32_t fresh = 0;
      bool full = false;
      auto put = [&](uint64_t key) {
        const uint64_t h = glp::mix64(key);  // bucket: high bits; slot: low bits; class: the bits above the slot's
        if (((h >> 11) & ((1ull << level) - 1ull)) == cls) full = !dedupe_insert(table, key, h, &fresh) || full;
      };
      for (int32_t i = kb + threadIdx.x; i < (t0 < t1 ? t0 * kSortTile : ke); i += kNT) put(keys[i]);
      for (int32_t t = t0 + (threadIdx.x >> 5); t < t1; t += kNT / 32)
        for (uint32_t i = lane; i < left[t]; i += 32) put(keys[(int64_t)t * kSortTile + i]);
      if (t0 < t1)
        for (int32_t i = t1 * kSortTile + threadIdx.x; i < ke; i += kNT) put(keys[i]);
      // the hash is a bijection: 53 levels would leave each slot one key
      if (__syncthreads_or(full)) {  // block-uniform
        ++level;
        continue;
      }
      fresh = __reduce_add_sync(kFull, fresh);
      if (lane == 0 && fresh) atomicAdd(&cursor, fresh);
      __syncthreads();
      if (threadIdx.x == 0) {
        sbase = cursor ? atomicAdd(nout, (unsigned long long)cursor) : 0ull;
        cursor = 0u;
      }
      __syncthreads();
      for (int s = threadIdx.x; s < kDedupeSlots; s += kNT) {
        const uint64_t key = table[s];
        const uint32_t m = __ballot_sync(kFull, key != kNoKey);
        uint32_t at = 0;
        if (lane == 0 && m) at = atomicAdd(&cursor, (uint32_t)__popc(m));
        at = __shfl_sync(kFull, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (key != kNoKey) {
          out[sbase + at] = key;
          atomicAdd(deg + (key >> idbits), 1);
          if (both) atomicAdd(deg + (key & idmask), 1);
        }
      }
      // the next class: up while this was an upper half, then the sibling
      while (level && (cls >> (level - 1) & 1ull)) {
        cls &= ~(1ull << (level - 1));
        --level;
      }
      more = level != 0;
      if (more) cls |= 1ull << (level - 1);
      __syncthreads();  // the table is read no more
    }
  }
}

// Distinct keys of a sorted list: per tile their number, then (its scan) their
// places.
__global__ void __launch_bounds__(kNT) k_unique_count(const uint64_t* __restrict__ keys, int64_t n,
                                                      uint32_t* __restrict__ counts) {
  __shared__ uint32_t total;
  if (threadIdx.x == 0) total = 0u;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  uint32_t c = 0;
  for (int r = 0; r < kSortTile / kNT; ++r) {
    const int64_t i = base + r * kNT + threadIdx.x;
    if (i < n && (i == 0 || keys[i] != keys[i - 1])) ++c;
  }
  c = __reduce_add_sync(kFull, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}
__global__ void __launch_bounds__(kNT) k_unique_write(const uint64_t* __restrict__ keys, int64_t n,
                                                      const uint32_t* __restrict__ first,
                                                      uint64_t* __restrict__ out, unsigned long long* nout) {
  __shared__ uint32_t wtot[kNT / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  uint32_t at = first[blockIdx.x];
  for (int r = 0; r < kSortTile / kNT; ++r) {  // block-uniform
    const int64_t i = base + r * kNT + threadIdx.x;
    const uint64_t key = i < n ? keys[i] : 0ull;
    const bool keep = i < n && (i == 0 || key != keys[i - 1]);
    const uint32_t m = __ballot_sync(kFull, keep);
    if (lane == 0) wtot[warp] = __popc(m);
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kNT / 32; ++w) {
      before += w < warp ? wtot[w] : 0u;
      all += wtot[w];
    }
    if (keep) out[at + before + __popc(m & ((1u << lane) - 1u))] = key;
    at += all;
    __syncthreads();
  }
  if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) *nout = at;
}

// Relabel keys ((n - degree) << 32 | id); listed by id, so a stable sort of the
// high half alone puts them in order.
__global__ void k_degree_keys(const int32_t* __restrict__ deg, int32_t n, uint64_t* __restrict__ keys) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
    keys[v] = ((uint64_t)((uint32_t)n - (uint32_t)deg[v]) << 32) | (uint32_t)v;
}

// From the sorted relabel keys: old id of each new vertex, new id of each old.
__global__ void k_perm(const uint64_t* __restrict__ keys, int32_t n, int32_t* __restrict__ old_of,
                       int32_t* __restrict__ new_of) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t old = (int32_t)(uint32_t)keys[r];
    old_of[r] = old;
    new_of[old] = (int32_t)r;
  }
}

__global__ void k_remap(uint64_t* __restrict__ keys, int64_t m, int idbits, int both,
                        const int32_t* __restrict__ new_of) {
  const uint64_t idmask = (1ull << idbits) - 1ull;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    uint32_t u = (uint32_t)__ldg(new_of + (k >> idbits)), v = (uint32_t)__ldg(new_of + (k & idmask));
    if (both && v < u) {
      const uint32_t x = u;
      u = v;
      v = x;
    }
    keys[i] = ((uint64_t)u << idbits) | v;
  }
}

__global__ void k_ids(int32_t* __restrict__ a, int32_t n) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
    a[v] = (int32_t)v;
}

// Row v of an undirected graph: its entries below v (from the list sorted by
// second id; they start at low[v]), then those above (list sorted by first id;
// up[v]).  off[v] = low[v] + up[v], so entry i of the first list goes to
// column i + up[its row] and entry i of the second to i + low[its row + 1].
__global__ void k_add_starts(const int32_t* __restrict__ up, const int32_t* __restrict__ low, int32_t n,
                             int32_t* __restrict__ off) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v <= n; v += (int64_t)gridDim.x * blockDim.x)
    off[v] = low[v] + up[v];
}
__global__ void k_columns(const uint64_t* __restrict__ by_first, const uint64_t* __restrict__ by_second, int64_t e,
                          int idbits, const int32_t* __restrict__ up, const int32_t* __restrict__ low,
                          int32_t* __restrict__ cols) {
  const uint64_t idmask = (1ull << idbits) - 1ull;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < e; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t a = __ldcs((const unsigned long long*)by_first + i);
    cols[i + __ldg(low + (a >> idbits) + 1)] = (int32_t)(a & idmask);
    const uint64_t b = __ldcs((const unsigned long long*)by_second + i);
    cols[i + __ldg(up + (b & idmask))] = (int32_t)(b >> idbits);
  }
}
__global__ void k_second_ids(const uint64_t* __restrict__ keys, int64_t m, int idbits, int32_t* __restrict__ cols) {
  const uint64_t idmask = (1ull << idbits) - 1ull;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    cols[i] = (int32_t)(keys[i] & idmask);
}

// Scratch from the pool that graph handles allocate from; the pool's idle
// memory is bounded when the call ends (dev_pool_trim).  cudaMalloc and
// cudaFree of a dozen buffers took as long as the kernels (the whole call with
// a three-step solve 27.9 -> 17.5 ms at R-MAT scale 22).  Freed once the
// stream it was used on is idle.
template <class T>
struct DevBuf {
  cudaStream_t s;
  T* p = nullptr;
  explicit DevBuf(cudaStream_t stream) : s(stream) {}
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() {
    if (!p) return;
    cudaStreamSynchronize(s);
    glp::dev_free(p);
  }
  cudaError_t alloc(int64_t count) {
    return glp::dev_alloc_raw(reinterpret_cast<void**>(&p), sizeof(T) * (size_t)std::max<int64_t>(count, 1));
  }
  T* release() {
    T* r = p;
    p = nullptr;
    return r;
  }
};

}  // namespace

namespace glp {

// Builds the CSR of an edge list on the current device.  *d_off ([n+1]) and
// *d_cols ([m] and four zero entries) come from dev_alloc_raw and are the
// caller's (dev_free, or cudaFree once idle); d_old
// (nullable, device, [n]) receives the original id of each vertex.
int ingest_edges(const int32_t* src, const int32_t* dst, int64_t count, int32_t n, int32_t on_device, uint32_t flags,
                 int32_t** d_off_out, int32_t** d_cols_out, int64_t* m_out, int32_t* d_old, cudaStream_t s) {
  if (n < 1 || count < 0 || count >= (1ll << 30) || (count > 0 && (!src || !dst))) {
    set_error("bad edge list (n >= 1, 0 <= count < 2^30, src and dst given)");
    return GLP_EINVAL;
  }
  const bool both = (flags & GLP_EDGES_DIRECTED) == 0;
  const bool relabel = (flags & GLP_EDGES_KEEP_IDS) == 0;
  const int idb = std::max(1, bit_length((uint64_t)(n - 1)));  // bits of an id: a key has 2 * idb <= 62
  auto blocks = [](int64_t work) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + kNT - 1) / kNT, (int64_t)device_sms() * 32));
  };
  DevBuf<int32_t> in_src(s), in_dst(s);
  const int32_t* s_src = src;
  const int32_t* s_dst = dst;
  if (!on_device && count) {
    ICUDA(in_src.alloc(count));
    ICUDA(in_dst.alloc(count));
    ICUDA(cudaMemcpyAsync(in_src.p, src, sizeof(int32_t) * count, cudaMemcpyHostToDevice, s));
    ICUDA(cudaMemcpyAsync(in_dst.p, dst, sizeof(int32_t) * count, cudaMemcpyHostToDevice, s));
    s_src = in_src.p;
    s_dst = in_dst.p;
  }
  DevBuf<uint64_t> ka(s), kb(s), kc(s);
  DevBuf<uint32_t> hist(s), scratch(s), flags_d(s);
  DevBuf<unsigned long long> nk(s);  // keys, then distinct keys
  ICUDA(ka.alloc(count));
  ICUDA(kb.alloc(count));
  ICUDA(nk.alloc(2));
  ICUDA(flags_d.alloc(1));
  ICUDA(cudaMemsetAsync(nk.p, 0, 2 * sizeof(unsigned long long), s));
  ICUDA(cudaMemsetAsync(flags_d.p, 0, sizeof(uint32_t), s));
  if (count) {
    k_edge_keys<<<blocks((count + kEdgeItems - 1) / kEdgeItems), kNT, 0, s>>>(s_src, s_dst, count, n, both ? 1 : 0,
                                                                             idb, ka.p, nk.p, flags_d.p);
    ICUDA(cudaGetLastError());
  }
  unsigned long long nkeys = 0;
  uint32_t bad = 0;
  ICUDA(cudaMemcpyAsync(&nkeys, nk.p, sizeof nkeys, cudaMemcpyDeviceToHost, s));
  ICUDA(cudaMemcpyAsync(&bad, flags_d.p, sizeof bad, cudaMemcpyDeviceToHost, s));
  ICUDA(cudaStreamSynchronize(s));
  if (bad) {
    set_error("an edge names a vertex outside [0, n)");
    return GLP_EINVAL;
  }
  const int64_t nk0 = (int64_t)nkeys;
  const int64_t ntiles = (std::max<int64_t>(nk0, n) + kSortTile - 1) / kSortTile;
  ICUDA(hist.alloc((int64_t)kRadix * ntiles));
  ICUDA(scratch.alloc(scan_scratch((int64_t)kRadix * ntiles)));
  const Sorter so{hist.p, scratch.p};
  uint64_t* keys = ka.p;
  uint64_t* tmp = kb.p;
  int64_t e = 0;  // distinct keys
  DevBuf<int32_t> new_of(s), old_of(s), deg(s), bstart(s);
  DevBuf<uint64_t> r1(s), r2(s);
  int rc;
  if (relabel) {
    ICUDA(new_of.alloc(n));
    ICUDA(old_of.alloc(n));
    ICUDA(deg.alloc(n));
    ICUDA(r1.alloc(n));
    ICUDA(r2.alloc(n));
    ICUDA(cudaMemsetAsync(deg.p, 0, sizeof(int32_t) * (size_t)n, s));
    if (nk0) {
      const int bits = bit_length((uint64_t)(nk0 / kDedupeMean));
      const int32_t nbuckets = 1 << bits;
      ICUDA(bstart.alloc((int64_t)nbuckets + 1));
      uint64_t *a = kb.p, *b = ka.p;
      if ((rc = radix_sort<HashDigit>(ka.p, &a, &b, nk0, 64 - bits, bits, so, s))) return rc;
      k_starts<<<blocks((int64_t)nbuckets + 1), kNT, 0, s>>>(a, nk0, nbuckets, HashBucket{64 - bits}, bstart.p);
      if (nk0 >= kSortTile) k_thin<<<(unsigned)(nk0 / kSortTile), kNT, 0, s>>>(a, HashBucket{64 - bits}, hist.p);
      k_dedupe<<<(unsigned)std::min<int64_t>(nbuckets, (int64_t)device_sms() * 64), kNT, 0, s>>>(
          a, bstart.p, hist.p, nbuckets, idb, both ? 1 : 0, b, nk.p + 1, deg.p);
      ICUDA(cudaGetLastError());
      keys = b;
      tmp = a;
    }
    k_degree_keys<<<blocks(n), kNT, 0, s>>>(deg.p, n, r1.p);
    uint64_t *order = r2.p, *spare = r1.p;
    if ((rc = radix_sort<KeyDigit>(r1.p, &order, &spare, n, 32, bit_length((uint64_t)n), so, s))) return rc;
    k_perm<<<blocks(n), kNT, 0, s>>>(order, n, old_of.p, new_of.p);
    ICUDA(cudaGetLastError());
    ICUDA(cudaMemcpyAsync(&nkeys, nk.p + 1, sizeof nkeys, cudaMemcpyDeviceToHost, s));
    ICUDA(cudaStreamSynchronize(s));
    e = (int64_t)nkeys;
    if (e) {
      k_remap<<<blocks(e), kNT, 0, s>>>(keys, e, idb, both ? 1 : 0, new_of.p);
      ICUDA(cudaGetLastError());
      uint64_t *a = tmp, *b = keys;
      if ((rc = radix_sort<KeyDigit>(keys, &a, &b, e, 0, 2 * idb, so, s))) return rc;
      keys = a;
      tmp = b;
    }
    if (d_old) ICUDA(cudaMemcpyAsync(d_old, old_of.p, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, s));
  } else {
    if (nk0) {
      uint64_t *a = kb.p, *b = ka.p;
      if ((rc = radix_sort<KeyDigit>(ka.p, &a, &b, nk0, 0, 2 * idb, so, s))) return rc;
      const int64_t tiles = (nk0 + kSortTile - 1) / kSortTile;
      k_unique_count<<<(unsigned)tiles, kNT, 0, s>>>(a, nk0, hist.p);
      if ((rc = scan_u32(hist.p, tiles, scratch.p, s))) return rc;
      k_unique_write<<<(unsigned)tiles, kNT, 0, s>>>(a, nk0, hist.p, b, nk.p + 1);
      ICUDA(cudaGetLastError());
      ICUDA(cudaMemcpyAsync(&nkeys, nk.p + 1, sizeof nkeys, cudaMemcpyDeviceToHost, s));
      ICUDA(cudaStreamSynchronize(s));
      e = (int64_t)nkeys;
      keys = b;
      tmp = a;
    }
    if (d_old) {
      k_ids<<<blocks(n), kNT, 0, s>>>(d_old, n);
      ICUDA(cudaGetLastError());
    }
  }
  const int64_t m = both ? 2 * e : e;
  if (m >= (1ll << 31)) {
    set_error("the graph exceeds an int32 CSR");
    return GLP_EINVAL;
  }
  DevBuf<int32_t> off(s), cols(s);
  ICUDA(off.alloc((int64_t)n + 1));
  ICUDA(cols.alloc(m + 4));
  ICUDA(cudaMemsetAsync(cols.p + m, 0, 4 * sizeof(int32_t), s));
  const unsigned vgrid = blocks((int64_t)n + 1);
  if (both) {
    DevBuf<int32_t> up(s), low(s);
    ICUDA(kc.alloc(e));
    ICUDA(up.alloc((int64_t)n + 1));
    ICUDA(low.alloc((int64_t)n + 1));
    // the same keys by their second id: `keys` itself stays as it is
    uint64_t *a = tmp, *b = kc.p;
    if ((rc = radix_sort<KeyDigit>(keys, &a, &b, e, 0, idb, so, s))) return rc;
    k_starts<<<vgrid, kNT, 0, s>>>(keys, e, n, FirstId{idb}, up.p);
    k_starts<<<vgrid, kNT, 0, s>>>(a, e, n, SecondId{(1ull << idb) - 1ull}, low.p);
    k_add_starts<<<vgrid, kNT, 0, s>>>(up.p, low.p, n, off.p);
    if (e) k_columns<<<blocks(e), kNT, 0, s>>>(keys, a, e, idb, up.p, low.p, cols.p);
    ICUDA(cudaGetLastError());
    ICUDA(cudaStreamSynchronize(s));
  } else {
    k_starts<<<vgrid, kNT, 0, s>>>(keys, e, n, FirstId{idb}, off.p);
    if (e) k_second_ids<<<blocks(e), kNT, 0, s>>>(keys, e, idb, cols.p);
    ICUDA(cudaGetLastError());
    ICUDA(cudaStreamSynchronize(s));
  }
  *d_off_out = off.release();
  *d_cols_out = cols.release();
  *m_out = m;
  return GLP_OK;
}

}  // namespace glp

extern "C" {

int glp_graph_from_edges(const int32_t* src, const int32_t* dst, int64_t count, int32_t n, int32_t on_device,
                         uint32_t flags, int32_t* old_id, glp_graph** out) {
  if (!out) {
    glp::set_error("out is NULL");
    return GLP_EINVAL;
  }
  *out = nullptr;
  int dev_count = 0;
  if (cudaGetDeviceCount(&dev_count) != cudaSuccess || dev_count == 0) {
    cudaGetLastError();
    glp::set_error("no usable CUDA device");
    return GLP_ENODEV;
  }
  cudaStream_t s = nullptr;
  ICUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  int32_t *d_off = nullptr, *d_cols = nullptr, *d_old = nullptr;
  int64_t m = 0;
  int rc = GLP_OK;
  if (old_id) {
    if (on_device) {
      d_old = old_id;
    } else if (glp::dev_alloc_raw((void**)&d_old, sizeof(int32_t) * (size_t)std::max(n, 1)) != cudaSuccess) {
      glp::set_error("no memory for the old ids");
      rc = GLP_ENOMEM;
    }
  }
  if (!rc) rc = glp::ingest_edges(src, dst, count, n, on_device, flags, &d_off, &d_cols, &m, d_old, s);
  if (!rc && old_id && !on_device) {
    if (cudaMemcpyAsync(old_id, d_old, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
      glp::set_error("copying the old ids to the host failed");
      rc = GLP_ECUDA;
    }
  }
  if (!rc)
    rc = glp::graph_adopt(d_off, d_cols, n, m, (flags & GLP_EDGES_DIRECTED) ? 0u : GLP_GRAPH_SYMMETRIC, out);
  else
    for (int32_t* p : {d_off, d_cols}) glp::dev_free(p);
  if (old_id && !on_device) {
    cudaStreamSynchronize(s);
    glp::dev_free(d_old);
  }
  glp::dev_pool_trim();
  cudaStreamDestroy(s);
  return rc;
}

}  // extern "C"
