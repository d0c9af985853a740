// assembly_ring.h -- how an assembly by element matrices (fe_kernels.cu) goes through its scratch ring.  Plain host code.
#pragma once

#include <algorithm>
#include <cstddef>

namespace mgb {

// Bytes of the matrices of one element layer of n instances.
inline size_t ring_layer_bytes(int nex, int ney, int n, size_t value_bytes) {
  return (size_t)n * 576 * nex * ney * value_bytes;
}

// Bytes of a ring: two element layers at least (a workspace's slots count them), and beyond that as many as `most` (three
// quarters of the L2) and a tenth of the free memory hold, no more than there are.  More layers mean fewer launches only.
inline size_t ring_bytes(int nez, size_t layer, size_t most, size_t free_bytes) {
  return std::max(2 * layer, std::min({((size_t)nez + 1) * layer, most, free_bytes / 10}));
}

// Element layers that a ring of `bytes` holds, no more than an assembly uses.
inline int ring_layers(int nez, size_t layer, size_t bytes) {
  const size_t fit = bytes / layer;
  return fit < (size_t)nez + 1 ? (int)fit : nez + 1;
}

// Chunks of layers that it takes: a chunk is all of the ring but the layer that the next one still needs.
inline int ring_chunks(int nez, int layers) { return (nez + layers - 2) / (layers - 1); }

// Kernels of one assembly.
inline int assembly_launches(int nex, int ney, int nez, int n, size_t value_bytes, size_t bytes) {
  return 2 * ring_chunks(nez, ring_layers(nez, ring_layer_bytes(nex, ney, n, value_bytes), bytes));
}

}  // namespace mgb
