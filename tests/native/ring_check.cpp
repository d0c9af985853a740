// Checks assembly_ring.h: every element layer is formed once, a chunk's layers and the one before it fit in the ring, and a
// ring never takes more than two layers or a tenth of the free memory.  Test infrastructure
// (tests/test_assembly_ring.py builds and runs it).
#include <cstdio>

#include "assembly_ring.h"

using namespace mgb;

int main() {
  int bad = 0, cases = 0;
  const size_t most = (size_t)96 << 20;
  for (int nex : {1, 2, 9, 60, 128})
    for (int nez : {1, 2, 3, 5, 60})
      for (int n : {1, 4, 33})
        for (size_t value : {4, 8})
          for (size_t free_mb : {0, 40, 200, 100000}) {
            const size_t layer = ring_layer_bytes(nex, nex + 1, n, value), free_b = free_mb << 20;
            const size_t bytes = ring_bytes(nez, layer, most, free_b);
            const int layers = ring_layers(nez, layer, bytes);
            bool ok = layers >= 2 && layers <= nez + 1 && (size_t)layers * layer <= bytes;
            ok = ok && (bytes <= 2 * layer || (bytes <= free_b / 10 && bytes <= most));
            int z = 0, chunks = 0;
            for (int z0 = 0; z0 < nez; z0 += layers - 1, ++chunks) z += (z0 + layers - 1 < nez ? layers - 1 : nez - z0);
            ok = ok && z == nez && chunks == ring_chunks(nez, layers) &&
                 assembly_launches(nex, nex + 1, nez, n, value, bytes) == 2 * chunks;
            if (!ok) std::printf("nex %d nez %d n %d value %zu free %zu: bytes %zu layers %d\n", nex, nez, n, value, free_mb, bytes, layers);
            bad += !ok;
            ++cases;
          }
  std::printf("%d cases, %d bad\n", cases, bad);
  return bad != 0;
}
