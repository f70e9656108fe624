// Host-side check of the tensor-core engine's ring of operand stages, for every block size
// and every launch shape that fits: the producer (and the MMA issuer, which steps alike) counts
// stages one by one, the epilogue finds the stage of a tile's last operands with ring_last.
// Prints one line per shape: K, CTAs per tile, chunks per stage, stages per tile, ring depth,
// the first tile whose stage differs (-1: none). Built and run by tests/test_ring_stage.py.
#include "../../sred_b200/csrc/global_tc.cu"

#include <cstdio>

int main() {
  using namespace sred;
  for (int K = 1; K <= 288; K++)
    for (int ctas : {1, 2})
      for (bool whole : {true, false}) {
        TcPlan p;
        if (!plan_shape(K, ctas, whole, &p)) continue;
        const int nch = (split_layout(K).pitch + kChunk - 1) / kChunk, nst = (nch + p.sc - 1) / p.sc;
        const uint32_t S = (uint32_t)p.stages, back = (uint32_t)(nst - 1) % S;
        uint32_t s = 0, st0 = 0;
        int bad = -1;
        for (int tile = 0; tile < 1000 && bad < 0; tile++) {
          uint32_t last = 0;
          for (int st = 0; st < nst; st++) {  // the producer's loop
            last = s;
            if (++s == S) s = 0;
          }
          if (ring_last(st0, back, S) != last) bad = tile;
          st0 = last + 1 == S ? 0 : last + 1;  // the epilogue's step
        }
        std::printf("%d %d %d %d %d %d\n", K, p.ctas, p.sc, nst, p.stages, bad);
      }
  return 0;
}
