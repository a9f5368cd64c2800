// The tcgen05 projection against lists of pairs (project_tc.cu), used by the
// hierarchical descent (descent.cu).
#pragma once
#include "common.cuh"

namespace ffsk {

constexpr int PAIR_SLOTS = 8;  // pairs a cell's list holds

// A pair of a list and the output slot of its projection.
__host__ __device__ inline int list_entry(int pair, int slot) { return pair | (slot << 24); }

// ||U_p' y_v||^2 of operand rows v against the pairs of a list, each pair's K
// rows of U fetched by its own TMA box (the pairs need not be neighbours).
//   dense  (tiles NULL): every row v < V against list[0 .. n_list); row v's
//          design is tile_design[v / 256] (NULL: 0); proj[slot * V + v].
//   cells: row tiles tiles[i] = (first row, rows <= 128, key, -), i <
//          *n_tiles <= max_tiles, key = design * P + cell, against the cell's
//          list list[cell * PAIR_SLOTS ..], ended by a negative entry or
//          PAIR_SLOTS entries; proj[row * PAIR_SLOTS + slot].
struct PairProject {
  int V, T, K, P, n_designs, ld;
  const uint16_t* hi;
  const uint16_t* lo;      // [V][ld]
  const int* yexp;         // [V]
  const uint16_t* u_hi;
  const uint16_t* u_lo;    // [n_designs * P * K][ld]
  const int* uexp;         // [n_designs * P]
  const int* list;
  int n_list;
  const int* tile_design;
  const int4* tiles;
  const int* n_tiles;
  int max_tiles;
  float* proj;
  int* flag;
};

int project_pairs(const PairProject& a, cudaStream_t stream);

}  // namespace ffsk
