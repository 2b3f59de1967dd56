// seeded.cuh -- seeded (semi-supervised) label propagation, method 5.
//
// Reference: prop/seedLprop.cuh (driver) with the *_seed kernels of
// header/kernel.cuh:914-1031 (huge), :1742-1836 (big), :3224-3331 (medium),
// :5236-5290 (tiny), and initialize_labels_by_seeds (:453-466): seed
// vertices are labelled with their own id and keep it; every other vertex
// starts unlabelled (-1) and takes the mode of its neighbours' labels.
//
// The rule implemented here, for every vertex v in one synchronous step:
//   seed v           : L'(v) = L(v) (its own id);
//   otherwise        : L'(v) = argmax_l k_l(v) over the LABELLED neighbours
//                      (label >= 0; weights summed exactly when the graph is
//                      weighted), ties -> the largest label; with no labelled
//                      neighbour, L'(v) = L(v).
// The reference's tiers disagree on unlabelled neighbours and on a vertex
// with none labelled: its tiny kernel counts the unlabelled ones as a label
// of their own, which can win (kernel.cuh:5253-5269), and its big and huge
// kernels skip them but then give the vertex its own id (:1767-1768); the
// rule above is the hard-clamping label propagation those kernels approach
// (Zhu and Ghahramani, CMU-CALD-02-107, 2002), the same on every tier.
//
// The steps run on the degree tiers of method 1 (kernels.cuh, ScoreSeeded): a
// label of -1 is no entry, a seed is skipped, a row without a candidate keeps
// its label.  Like theirs, the cost is the label gather and the count tables.
// A warp per vertex of any degree, with 512 slots cleared for each and the
// largest rows in global tables, took 44.7 ms for ten steps on R-MAT
// scale 20 (31.4 M entries, 2 % seeds, one B200); the tiers take 2.6 ms.
#pragma once
#include "device.cuh"

namespace glp {

// Labels at the start: a seed gets its id, every other vertex -1.
__global__ void k_seeded_init(const uint8_t* __restrict__ seeds, int32_t* __restrict__ a, int32_t* __restrict__ b,
                              int32_t n) {
  const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) a[v] = b[v] = seeds[v] ? v : -1;
}

}  // namespace glp
