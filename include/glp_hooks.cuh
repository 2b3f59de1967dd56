/*
 * glp_hooks.cuh -- method 4 of the label-propagation engine as a header-only
 * CUDA template: user-written PickLabel / LoadNeighbor / LabelScore /
 * UpdateVertex hooks run on a graph handle of libglp_b200.so.
 *
 * Reference surface: README.md:72-101 asks users to fill in four __device__
 * functions (stubs at header/kernel.cuh:6071-6085) and run method=4
 * (prop/UserdefinedLprop.cuh, main.cu:96-100).  Here a hook set is any
 * struct with these four __device__ members:
 *
 *   void   pick(int32_t vid)                               PickLabel
 *   void   load(int32_t vid, int32_t sid, int64_t e,
 *               int32_t* label, double* freq)              LoadNeighbor
 *   double score(int32_t vid, int32_t label, double freq)  LabelScore
 *   void   update(int32_t vid, int32_t label, double score) UpdateVertex
 *
 * and glp_hooks::run() drives, per iteration:
 *   1. pick(v) for every vertex (the classic hook set copies Lnext to L);
 *   2. per vertex v, freq(l) = the sum of the freq values LoadNeighbor gives
 *      for the neighbours (CSR entries e of v, neighbour sid) whose label is
 *      l; the winner maximises LabelScore(v, l, freq(l)), ties -> the
 *      largest label; Lnext[v] = winner, then update(v, winner, score).  An
 *      isolated vertex keeps L[v] and gets update(v, L[v], -inf).
 * LabelScore may be any function of the final frequency: every distinct
 * label is scored once its frequency is complete.  Frequencies are summed in
 * a fixed order -- within a chunk of 32 consecutive CSR entries in entry
 * order, chunks in CSR order -- so FP64 results are deterministic and can be
 * restated exactly on the host.
 *
 * Build a hook set into your own shared object or program with nvcc
 * (-gencode arch=compute_100a,code=sm_100a) and link -lglp_b200; the graph
 * stays resident in the library's handle, so nothing is copied.  The hooks
 * get the device view (glp_hooks::State, filled from glp_graph_device_view)
 * through a member of their own, as in the example below.
 *
 *   struct MyHooks {
 *     glp_hooks::State st;
 *     __device__ void pick(int32_t v) const { st.L[v] = st.Lnext[v]; }
 *     __device__ void load(int32_t, int32_t sid, int64_t, int32_t* l, double* f) const {
 *       *l = st.L[sid];
 *       *f = 1.0 / (1.0 + (st.off[sid + 1] - st.off[sid]));
 *     }
 *     __device__ double score(int32_t, int32_t, double f) const { return f; }
 *     __device__ void update(int32_t, int32_t, double) const {}
 *   };
 *   ...
 *   glp_hooks::run(g, [](const glp_hooks::State& s) { return MyHooks{s}; }, niter, labels, 0, nullptr,
 *                  stream);
 */
#ifndef GLP_B200_GLP_HOOKS_CUH
#define GLP_B200_GLP_HOOKS_CUH

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "glp.h"

namespace glp_hooks {

/* What a hook set sees: the resident CSR, the two label buffers (L read,
 * Lnext written by the step) and, for layered-style scores, two volume
 * arrays (vol_r read, vol_w written).  dstar and user are free for the hook
 * set's own use. */
struct State {
  const int32_t* off;
  const int32_t* cols;
  const int32_t* w;  /* NULL when the graph is unweighted */
  int32_t n;
  int32_t* L;
  int32_t* Lnext;
  const int32_t* vol_r;
  int32_t* vol_w;
  double dstar;
  void* user;
};

constexpr uint32_t kFullMask = 0xffffffffu;
constexpr int kSmemCap = 512; /* runs on graphs with a degree above kSmemCap/2 have the spill tables */
constexpr uint32_t kErrProbe = 1u;

constexpr int kPropThreads = 256;     /* k_prop's block size */
constexpr int kPropWarps = kPropThreads / 32;
constexpr int kGroupDegree = 8;       /* eight lanes per vertex up to here */
constexpr int kWarpDegree = 128;      /* a warp per vertex up to here, */
constexpr int kBlockDegree = 2047;    /* a block of k_prop up to here; above, k_prop_hub */
constexpr int kWarpSlots = 2 * kWarpDegree;
constexpr int kHubThreads = 1024;     /* k_prop_hub's block size */
static_assert(2 * kWarpDegree <= kSmemCap, "rows that may need the spill tables have them");

/* Shared memory of a block that counts one row: a table of Slots labels that
 * takes new ones until it holds Close of them (a whole round of new labels
 * then still fits), and Turns buckets, twice, that order the warps' adds (one
 * bit per warp). */
template <int NT, int Slots, int Close, int Turns>
struct RowShared {
  static constexpr int kThreads = NT, kWarps = NT / 32, kTurnBuckets = Turns;
  static constexpr uint32_t kSlots = Slots, kClose = Close;
  static constexpr int kPerWord = 32 / kWarps; /* buckets per word */
  static_assert(Close + NT <= Slots && (Turns & (Turns - 1)) == 0, "table and bucket sizes");
  double vals[Slots];
  double sf[kWarps][32];
  struct {
    double s;
    int32_t l;
  } red[kWarps];
  uint32_t keys[Slots];
  uint32_t turn[2][Turns / kPerWord];
  int32_t list[NT];
  int32_t nlist;
  uint32_t nkeys;
};
using BlockRows = RowShared<kPropThreads, 2560, 2048, 2048>;
using HubRows = RowShared<kHubThreads, 9216, 4608, 8192>;
static_assert(kBlockDegree < (int)BlockRows::kClose, "k_prop's rows never overflow its table");
static_assert(kPropWarps * kWarpSlots <= (int)BlockRows::kSlots, "the warps' tables fit the block's");

/* The 32-bit finaliser of MurmurHash3 (Appleby): slot of a key. */
__device__ __forceinline__ uint32_t slot_hash(uint32_t k) {
  k ^= k >> 16;
  k *= 0x85ebca6bu;
  k ^= k >> 13;
  k *= 0xc2b2ae35u;
  k ^= k >> 16;
  return k;
}

template <class H>
__global__ void __launch_bounds__(256) k_pick(H h, int32_t n) {
  const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) h.pick(v);
}

/* Claims or finds the slot of `key` (not 0) among cap slots; cap when the
 * table is full.  *fresh: whether this call claimed it. */
__device__ __forceinline__ uint32_t claim_slot(uint32_t* keys, uint32_t cap, uint32_t key, bool* fresh = nullptr) {
  uint32_t slot = __umulhi(slot_hash(key), cap);
  for (uint32_t probe = 0; probe < cap; ++probe) {
    const uint32_t prev = atomicCAS(keys + slot, 0u, key);
    if (prev == 0u || prev == key) {
      if (fresh) *fresh = prev == 0u;
      return slot;
    }
    if (++slot == cap) slot = 0u;
  }
  return cap;
}
/* claim_slot in global memory: four slots are read together before a claim,
 * so that a key a few probes from home costs two round trips. */
__device__ __forceinline__ uint32_t claim_spill(uint32_t* keys, uint32_t cap, uint32_t key) {
  uint32_t slot = __umulhi(slot_hash(key), cap);
  for (uint32_t probe = 0; probe < cap;) {
    uint32_t at[4], cur[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      at[i] = slot + i < cap ? slot + i : slot + i - cap; /* cap > 4 */
      cur[i] = __ldcg(keys + at[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (cur[i] == 0u) cur[i] = atomicCAS(keys + at[i], 0u, key);
      if (cur[i] == 0u || cur[i] == key) return at[i];
    }
    probe += 4;
    slot = at[3] + 1u < cap ? at[3] + 1u : 0u;
  }
  return cap;
}
/* The slot that holds `key` in a table no thread is adding keys to; cap when
 * it is not there. */
__device__ __forceinline__ uint32_t find_slot(const uint32_t* keys, uint32_t cap, uint32_t key) {
  uint32_t slot = __umulhi(slot_hash(key), cap);
  for (uint32_t probe = 0; probe < cap; ++probe) {
    const uint32_t cur = keys[slot];
    if (cur == key) return slot;
    if (cur == 0u) return cap;
    if (++slot == cap) slot = 0u;
  }
  return cap;
}

/* A scored label (l < 0: none); the larger score wins, then the larger label. */
struct Scored {
  double s;
  int32_t l;
};
__device__ __forceinline__ void take_better(Scored& b, double s, int32_t l) {
  if (l >= 0 && (b.l < 0 || s > b.s || (s == b.s && l > b.l))) {
    b.s = s;
    b.l = l;
  }
}
template <int G>
__device__ __forceinline__ Scored group_best(Scored b) {
#pragma unroll
  for (int o = G / 2; o >= 1; o >>= 1) {
    const double os = __shfl_xor_sync(kFullMask, b.s, o);
    const int32_t ol = __shfl_xor_sync(kFullMask, b.l, o);
    take_better(b, os, ol);
  }
  return b;
}

/* The frequency of the lane's label within a chunk of 32 entries, summed in
 * entry order; valid on the first lane holding the label (true there).  lab
 * = -1: the lane has no entry.  sf: the warp's 32 words.  Each such lane
 * walks the lanes that hold its label, so a chunk costs as many reads as its
 * most frequent label has entries (one when all differ). */
__device__ __forceinline__ bool chunk_freq(int32_t lab, double f, double* sf, double* sum) {
  const int lane = threadIdx.x & 31;
  __syncwarp(); /* the previous chunk is read no more */
  sf[lane] = f;
  uint32_t m = __match_any_sync(kFullMask, (uint32_t)lab);
  __syncwarp();
  const bool lead = lab != -1 && lane == __ffs(m) - 1;
  double s = 0.0;
  if (lead)
    for (; m; m &= m - 1u) s += sf[__ffs(m) - 1];
  *sum = s;
  return lead;
}

/* Counts row v in the block's table and returns its best label on thread 0.
 * One chunk of 32 entries per warp at a time: every warp sums its chunk, then
 * the adds to a label's frequency go in chunk order -- each leader notes its
 * warp in the turn bucket of its slot and adds after as many barriers as
 * lower warps share the bucket (none when the labels differ).  The value a
 * leader adds to is read before the first of these barriers, which the first
 * in turn may use as it is.  Labels go to the shared table until it closes
 * (decided between rounds, alike for the whole block); a label that is not
 * there by then goes to the row's own spill region, entries
 * [2*off[v], 2*off[v+1]) of gkeys/gvals.  A row's frequent labels come early,
 * so a hot label's serial adds stay in shared memory and the spill table sees
 * the rare ones.  sh.turn is all zero at entry and at exit. */
template <class H, class Sh>
__device__ __forceinline__ Scored count_row(const H& hook, const State& st, int32_t v, Sh& sh, uint32_t* gkeys,
                                            double* gvals, int& par, bool& full) {
  constexpr int NT = Sh::kThreads;
  H h = hook;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int32_t b = st.off[v];
  const uint32_t d = (uint32_t)(st.off[v + 1] - b), gcap = 2u * d;
  const uint32_t cap = gcap < Sh::kSlots ? gcap : Sh::kSlots;
  uint32_t* keys2 = gkeys + 2ll * b;
  double* vals2 = gvals + 2ll * b;
  for (uint32_t s = threadIdx.x; s < cap; s += NT) {
    sh.keys[s] = 0u;
    sh.vals[s] = 0.0;
  }
  if (d >= Sh::kClose)
    for (uint32_t s = threadIdx.x; s < gcap; s += NT) {
      keys2[s] = 0u;
      vals2[s] = 0.0;
    }
  if (threadIdx.x == 0) sh.nkeys = 0u;
  bool open = true;
  __syncthreads();
  for (uint32_t i0 = 0; i0 < d; i0 += 4 * NT) {
    int32_t lab[4];
    double f[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = i0 + q * NT + threadIdx.x;
      lab[q] = -1;
      f[q] = 0.0;
      if (i < d) h.load(v, st.cols[b + i], b + (int64_t)i, &lab[q], &f[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (d - i0 <= q * NT) break; /* block-uniform */
      double s, old = 0.0;
      const bool lead = chunk_freq(lab[q], f[q], sh.sf[warp], &s);
      double* at = nullptr;
      uint32_t* turn = nullptr;
      uint32_t shift = 0;
      if (lead) {
        const uint32_t key = (uint32_t)lab[q] + 1u;
        bool fresh = false;
        uint32_t slot = open ? claim_slot(sh.keys, cap, key, &fresh) : find_slot(sh.keys, cap, key);
        if (fresh && d >= Sh::kClose) atomicAdd(&sh.nkeys, 1u);
        if (slot < cap) at = sh.vals + slot;
        else if (!open && (slot = claim_spill(keys2, gcap, key)) < gcap) at = vals2 + slot;
        else full = true;
        if (at) {
          const uint32_t bucket = slot & (Sh::kTurnBuckets - 1);
          turn = &sh.turn[par][bucket / Sh::kPerWord];
          shift = (bucket % Sh::kPerWord) * Sh::kWarps;
          atomicOr(turn, 1u << (shift + warp));
          old = *at;
        }
      }
      __syncthreads();
      const int rank = at ? __popc((*turn >> shift) & ((1u << warp) - 1u)) : -1;
      if (d >= Sh::kClose) open = sh.nkeys < Sh::kClose; /* no claim before the next barrier */
      if (rank == 0) *at = old + s;
      for (int r = 1; __syncthreads_or(rank >= r); ++r)
        if (rank == r) *at += s;
      if (at) *turn = 0u; /* the next round uses the other buckets */
      par ^= 1;
    }
  }
  Scored best{-INFINITY, -1};
  for (uint32_t s = threadIdx.x; s < cap; s += NT) {
    const uint32_t key = sh.keys[s];
    if (key) take_better(best, h.score(v, (int32_t)(key - 1u), sh.vals[s]), (int32_t)(key - 1u));
  }
  if (!open)
    for (uint32_t s = threadIdx.x; s < gcap; s += NT) {
      const uint32_t key = keys2[s];
      if (key) take_better(best, h.score(v, (int32_t)(key - 1u), vals2[s]), (int32_t)(key - 1u));
    }
  best = group_best<32>(best);
  if (lane == 0) {
    sh.red[warp].s = best.s;
    sh.red[warp].l = best.l;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < Sh::kWarps; ++w) take_better(best, sh.red[w].s, sh.red[w].l);
  return best;
}

/* Counts the block's rows of degree lo..hi: vertices blockIdx.x, blockIdx.x +
 * gridDim.x, ..., so that the neighbouring large rows of a degree-sorted
 * graph land on different SMs.  The offsets are scanned a round of NT
 * vertices at a time (8 bytes a vertex: cheaper than keeping lists in the
 * public state).  Block-uniform; ends in a barrier. */
template <class H, class Sh, class Settle>
__device__ __forceinline__ void count_rows(const H& h, const State& st, int32_t lo, int32_t hi, Sh& sh,
                                           uint32_t* gkeys, double* gvals, bool& full, const Settle& settle) {
  constexpr int NT = Sh::kThreads;
  uint32_t* turn = &sh.turn[0][0];
  for (uint32_t i = threadIdx.x; i < sizeof(sh.turn) / sizeof(uint32_t); i += NT) turn[i] = 0u;
  int par = 0;
  for (int64_t v0 = blockIdx.x; v0 < st.n; v0 += (int64_t)gridDim.x * NT) {
    if (threadIdx.x == 0) sh.nlist = 0;
    __syncthreads();
    const int64_t vt = v0 + (int64_t)threadIdx.x * gridDim.x;
    if (vt < st.n) {
      const int32_t d = st.off[vt + 1] - st.off[vt];
      if (d >= lo && d <= hi) sh.list[atomicAdd(&sh.nlist, 1)] = (int32_t)vt;
    }
    __syncthreads();
    const int32_t nlist = sh.nlist;
    for (int32_t k = 0; k < nlist; ++k) {
      const int32_t v = sh.list[k];
      const Scored best = count_row(h, st, v, sh, gkeys, gvals, par, full);
      if (threadIdx.x == 0) settle(v, best);
    }
    __syncthreads(); /* the list is read no more */
  }
  __syncthreads();
}

/* One propagation step of the rows up to kBlockDegree.  A step reads each
 * neighbour's label (and whatever LoadNeighbor asks for) at random, so it is
 * bound by the latency of those reads and by the ordered FP64 sums; the split
 * keeps every warp loading:
 *   degree 0..8     eight lanes per vertex, four vertices per warp and round,
 *                   two rounds' loads in flight; frequencies by shuffles;
 *   degree 9..32    a warp per vertex, four vertices' entries loaded before
 *                   the first is summed; one chunk holds the whole row, so
 *                   its sums are the final frequencies and need no table;
 *   degree 33..128  a warp per vertex, the whole row loaded first, then a
 *                   per-warp shared table of two slots an entry;
 *   to kBlockDegree a block per vertex (count_rows), four blocks to an SM.
 * Measured on one B200, R-MAT scale 20 (31.4 M entries), degree-normalised
 * votes, ten steps: 13 ms with k_prop_hub; 640 ms with one warp per
 * vertex of any degree, 512 slots cleared and scanned for each and full-warp
 * shuffle sums. */
template <class H>
__global__ void __launch_bounds__(kPropThreads, 4) k_prop(H h, const State st, unsigned long long* changed,
                                                          uint32_t* err) {
  __shared__ BlockRows sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nb = gridDim.x, nw = nb * kPropWarps;
  uint32_t nchanged = 0; /* this thread's */
  bool full = false;
  auto settle = [&](int32_t v, const Scored& b) {
    st.Lnext[v] = b.l;
    h.update(v, b.l, b.s);
    nchanged += b.l != st.L[v] ? 1u : 0u;
  };
  count_rows(h, st, kWarpDegree + 1, kBlockDegree, sh, nullptr, nullptr, full, settle);

  /* 9..kWarpDegree: a warp per vertex */
  uint32_t* wkeys = sh.keys + warp * kWarpSlots;
  double* wvals = sh.vals + warp * kWarpSlots;
  for (int64_t v0 = warp * nb + blockIdx.x; v0 < st.n; v0 += 32 * nw) {
    const int64_t vt = v0 + lane * nw;
    int32_t vb = 0, vd = 0;
    if (vt < st.n) {
      vb = st.off[vt];
      vd = st.off[vt + 1] - vb;
    }
    uint32_t one = __ballot_sync(kFullMask, vd > kGroupDegree && vd <= 32);
    while (one) { /* four rows of one chunk each */
      int32_t v[4], lab[4];
      double f[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int src = one ? __ffs(one) - 1 : 0;
        v[q] = one ? (int32_t)(v0 + src * nw) : -1;
        one &= one - 1u;
        const int32_t b = __shfl_sync(kFullMask, vb, src), d = __shfl_sync(kFullMask, vd, src);
        lab[q] = -1;
        f[q] = 0.0;
        if (v[q] >= 0 && lane < d) h.load(v[q], st.cols[b + lane], b + lane, &lab[q], &f[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (v[q] < 0) break; /* warp-uniform */
        double s;
        Scored best{-INFINITY, -1};
        if (chunk_freq(lab[q], f[q], sh.sf[warp], &s)) take_better(best, h.score(v[q], lab[q], s), lab[q]);
        best = group_best<32>(best);
        if (lane == 0) settle(v[q], best);
      }
    }
    uint32_t many = __ballot_sync(kFullMask, vd > 32 && vd <= kWarpDegree);
    for (; many; many &= many - 1u) {
      const int src = __ffs(many) - 1;
      const int32_t v = (int32_t)(v0 + src * nw);
      const int32_t b = __shfl_sync(kFullMask, vb, src), d = __shfl_sync(kFullMask, vd, src);
      int32_t lab[4];
      double f[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int32_t i = 32 * q + lane;
        lab[q] = -1;
        f[q] = 0.0;
        if (i < d) h.load(v, st.cols[b + i], b + i, &lab[q], &f[q]);
      }
      const uint32_t cap = 2u * (uint32_t)d;
      for (uint32_t s = lane; s < cap; s += 32) {
        wkeys[s] = 0u;
        wvals[s] = 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (32 * q >= d) break; /* warp-uniform */
        double s;
        if (chunk_freq(lab[q], f[q], sh.sf[warp], &s)) { /* its barriers order the chunks' adds */
          const uint32_t slot = claim_slot(wkeys, cap, (uint32_t)lab[q] + 1u);
          if (slot < cap) wvals[slot] += s;
          else full = true;
        }
      }
      __syncwarp();
      Scored best{-INFINITY, -1};
      for (uint32_t s = lane; s < cap; s += 32) {
        const uint32_t key = wkeys[s];
        if (key) {
          const int32_t l = (int32_t)(key - 1u);
          take_better(best, h.score(v, l, wvals[s]), l);
        }
      }
      best = group_best<32>(best);
      if (lane == 0) settle(v, best);
      __syncwarp(); /* the table is cleared for the next vertex */
    }
  }

  /* 0..kGroupDegree: eight lanes per vertex */
  const int gl = lane & 7;
  for (int64_t w0 = (int64_t)blockIdx.x * kPropWarps + warp; w0 * 8 < st.n; w0 += nw) {
    int32_t v[2], lab[2];
    double f[2];
    bool mine[2], row[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int64_t vt = w0 * 8 + 4 * q + (lane >> 3);
      v[q] = (int32_t)vt;
      lab[q] = -1;
      f[q] = 0.0;
      mine[q] = row[q] = false;
      if (vt < st.n) {
        const int32_t b = st.off[vt], d = st.off[vt + 1] - b;
        mine[q] = d <= kGroupDegree;
        row[q] = d > 0;
        if (mine[q] && gl < d) h.load(v[q], st.cols[b + gl], b + gl, &lab[q], &f[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (!__any_sync(kFullMask, mine[q])) continue;
      double s = 0.0;
      bool lead = lab[q] != -1;
#pragma unroll
      for (int k = 0; k < 8; ++k) { /* entry order; the first holder leads */
        const int32_t ol = __shfl_sync(kFullMask, lab[q], k, 8);
        const double of = __shfl_sync(kFullMask, f[q], k, 8);
        if (ol == lab[q]) {
          s += of;
          if (k < gl) lead = false;
        }
      }
      Scored best{-INFINITY, -1};
      if (lead) take_better(best, h.score(v[q], lab[q], s), lab[q]);
      best = group_best<8>(best);
      if (mine[q] && gl == 0) {
        if (!row[q]) best.l = st.L[v[q]]; /* isolated: keeps its label */
        settle(v[q], best);
      }
    }
  }

  nchanged = __reduce_add_sync(kFullMask, nchanged);
  if (lane == 0 && nchanged) atomicAdd(changed, (unsigned long long)nchanged);
  if (full) atomicOr(err, kErrProbe);
  /* launched on top of k_prop_hub: the step ends when both have.  One block
   * waits for it; the others leave their SM to the blocks still to come. */
  if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

/* The rows above kBlockDegree: a 1024-thread block per vertex.  One block owns
 * a row because its sums are ordered, so the step waits for the largest row's
 * serial rounds, which wide blocks keep few.  k_prop is launched on top
 * (programmatic launch, independent vertices) and fills the SMs as they run
 * out of large rows. */
template <class H>
__global__ void __launch_bounds__(kHubThreads, 1) k_prop_hub(H h, const State st, uint32_t* gkeys, double* gvals,
                                                             unsigned long long* changed, uint32_t* err) {
  extern __shared__ __align__(16) unsigned char hub_smem[];
  HubRows& sh = *reinterpret_cast<HubRows*>(hub_smem);
  uint32_t nchanged = 0;
  bool full = false;
  asm volatile("griddepcontrol.launch_dependents;");
  count_rows(h, st, kBlockDegree + 1, INT32_MAX, sh, gkeys, gvals, full, [&](int32_t v, const Scored& b) {
    st.Lnext[v] = b.l;
    h.update(v, b.l, b.s);
    nchanged += b.l != st.L[v] ? 1u : 0u;
  });
  if (nchanged) atomicAdd(changed, (unsigned long long)nchanged);
  if (full) atomicOr(err, kErrProbe);
}

/* Blocks of k_prop for n vertices on `sms` multiprocessors: four are resident
 * on each, and four times as many share the vertices, so that SMs that
 * k_prop_hub leaves late take fewer (R-MAT scale 20, a step: 1.9 ms with
 * resident blocks only); fewer when a warp would have no vertex. */
inline unsigned prop_grid(int32_t n, int32_t sms) {
  const int64_t want = ((int64_t)n + kPropWarps - 1) / kPropWarps, most = 16ll * (sms > 0 ? sms : 1);
  return (unsigned)(want < most ? want : most);
}

/* Launches the propagation step of one iteration on `stream`; gkeys/gvals are
 * needed from a largest degree above kBlockDegree on. */
template <class H>
inline cudaError_t launch_prop(const H& h, const State& st, int32_t max_degree, int32_t sms, uint32_t* gkeys,
                               double* gvals, unsigned long long* changed, uint32_t* err, cudaStream_t stream) {
  cudaLaunchAttribute attr = {};
  cudaLaunchConfig_t cfg = {};
  if (max_degree > kBlockDegree) {
    const cudaError_t e = cudaFuncSetAttribute(k_prop_hub<H>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(HubRows));
    if (e != cudaSuccess) return e;
    k_prop_hub<H><<<(unsigned)(sms > 0 ? sms : 1), kHubThreads, sizeof(HubRows), stream>>>(h, st, gkeys, gvals,
                                                                                          changed, err);
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
  }
  cfg.gridDim = dim3(prop_grid(st.n, sms));
  cfg.blockDim = dim3(kPropThreads);
  cfg.stream = stream;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_prop<H>, h, st, changed, err);
  return e != cudaSuccess ? e : cudaGetLastError();
}

/* Launches one iteration (pick, then the propagation step) on `stream`. */
template <class H>
inline cudaError_t launch_iteration(const H& h, const State& st, const glp_device_view& vw, int32_t iter,
                                    cudaStream_t stream) {
  if (st.n == 0) return cudaSuccess;
  k_pick<H><<<(unsigned)((st.n + 255) / 256), 256, 0, stream>>>(h, st.n);
  return launch_prop(h, st, vw.max_degree, vw.sms, vw.hook_keys, vw.hook_vals, vw.changed + iter, vw.err, stream);
}

/* Runs niter iterations of the hook set that make(state) returns, on the
 * resident graph g, from label = vertex id.  L is labels[0] and Lnext
 * labels[1] in every iteration: PickLabel moves the previous result into L
 * (the classic hooks copy Lnext to L), so the final labels are in Lnext.
 * labels_out receives them (a device pointer when on_device, else host);
 * changed (nullable, host) the number of labels changed per iteration.
 * Returns a GLP_* code.  The call is synchronous. */
template <class Make>
inline int run(glp_graph* g, Make make, int32_t niter, int32_t* labels_out, int32_t on_device, int64_t* changed,
               cudaStream_t stream) {
  if (!g || !labels_out || niter < 0) return GLP_EINVAL;
  glp_device_view vw;
  int rc = glp_graph_device_view(g, niter, &vw);
  if (rc) return rc;
  cudaStream_t s = stream ? stream : (cudaStream_t)vw.stream;
  cudaError_t e = cudaSuccess;
  if (vw.n > 0) {
    const State st{vw.off, vw.cols, vw.w, vw.n, vw.labels[0], vw.labels[1], nullptr, nullptr, 1.0, nullptr};
    const auto h = make(st);
    for (int32_t it = 0; it < niter && e == cudaSuccess; ++it) e = launch_iteration(h, st, vw, it, s);
    const int32_t* fin = vw.labels[1];
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(labels_out, fin, sizeof(int32_t) * (size_t)vw.n,
                          on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess && changed && niter > 0)
    e = cudaMemcpyAsync(changed, vw.changed, sizeof(int64_t) * (size_t)niter, cudaMemcpyDeviceToHost, s);
  uint32_t err = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&err, vw.err, sizeof err, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return GLP_ECUDA;
  return err ? GLP_EKERNEL : GLP_OK;
}

} /* namespace glp_hooks */

#endif /* GLP_B200_GLP_HOOKS_CUH */
