// CTAs as threads: each sums the counts ahead of its tile, the last to arrive overwrites them with offsets.  Built with
// the thread sanitizer, which reports accesses that nothing orders.  Exits with 1 where a sum or an offset is wrong.
#include <cstdint>
#include <cstdio>
#include <thread>
#include <vector>

#include "../cswap_b200/csrc/tile_counts.cuh"

int main() {
  int bad = 0;
  for (uint32_t tiles : {2u, 7u, 32u})
    for (int round = 0; round < 20; round++) {
      std::vector<uint32_t> words(tiles), offsets(tiles + 1, 0u);
      std::vector<int> wrong(tiles, 0);
      for (uint32_t t = 0; t < tiles; t++) {
        words[t] = (t * 2654435761u + (uint32_t)round) % 4097u;
        offsets[t + 1] = offsets[t] + words[t];
      }
      int writers = 0;
      std::vector<std::thread> ctas;
      for (uint32_t t = 0; t < tiles; t++)
        ctas.emplace_back([&, t] {
          uint32_t ahead = 0;
          for (uint32_t i = 0; i < t; i++) ahead += csw::tile_count(&words[i]);
          wrong[t] = ahead != offsets[t];
          if (!csw::last_to_arrive(words.data(), tiles)) return;
          writers++;
          uint32_t at = 0;
          for (uint32_t i = 0; i < tiles; i++) {
            const uint32_t c = csw::tile_count(&words[i]);
            words[i] = at;
            at += c;
          }
        });
      for (std::thread& c : ctas) c.join();
      bad += writers != 1;
      for (uint32_t t = 0; t < tiles; t++) bad += wrong[t] || words[t] != offsets[t];
    }
  if (bad) std::fprintf(stderr, "%d wrong\n", bad);
  return bad != 0;
}
