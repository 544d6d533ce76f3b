// Host-side replay of the GEMM work iterator with the partial wave cut into pieces of K (k_chunks): every k-block of every
// tile is covered exactly once, and a tile that several items share is flagged partial in all of them.
#include <cstdio>
#include <vector>

#include "gemm_common.cuh"

extern "C" void* sr_driver_encode_tiled(void) { return nullptr; }   // the host side of the header refers to it

int main() {
  int failures = 0, cases = 0;
  for (int tiles : {1, 3, 48, 74, 75, 88, 200})
    for (int workers : {1, 7, 37, 74})
      for (int num_kb : {1, 2, 8, 47, 128, 1024})
        for (int want = 1; want <= num_kb && want <= 2 * workers; want += (want < 8 ? 1 : 13)) {
          const int len = (num_kb + want - 1) / want;
          if ((num_kb + len - 1) / len != want) continue;
          GemmParams p{};
          p.num_tiles = tiles;
          p.splitk = 1;
          p.k_chunks = want;
          p.tail_split = 1;
          std::vector<int> cover((size_t)tiles * num_kb, 0), items(tiles, 0), flagged(tiles, 0);
          for (int w = 0; w < workers; ++w) {
            WorkIter wi;
            wi.init(p, num_kb, w, workers, 256);
            int tile, kb0, kb1;
            bool partial;
            while (wi.next(tile, kb0, kb1, partial)) {
              if (tile < 0 || tile >= tiles || kb0 < 0 || kb0 >= kb1 || kb1 > num_kb) {
                ++failures;
                break;
              }
              for (int kb = kb0; kb < kb1; ++kb) ++cover[(size_t)tile * num_kb + kb];
              ++items[tile];
              flagged[tile] += partial;
            }
          }
          for (int c : cover) failures += c != 1;
          for (int t = 0; t < tiles; ++t) failures += items[t] > 1 && flagged[t] != items[t];
          ++cases;
        }
  std::printf("%d schedules checked, %d failures\n", cases, failures);
  return failures == 0 ? 0 : 1;
}
