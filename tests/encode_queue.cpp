// The staged encoder's use of its expansion queue: entries are read one ahead of the expansion at work, so that a step
// never waits for the entry that it begins with, and never beyond the queue.  Exits with 1 otherwise.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../cswap_b200/csrc/zfp_core.cuh"

namespace {
struct Watch {
  uint32_t words[4096 / 32 + csw::STAGE_SPARE_ROWS] = {};
  uint32_t q[csw::QUEUE_SLOTS] = {};
  int behind = -1;  // the last entry read since they were put
  bool putting = false;
  long late = 0, outside = 0, expansions = 0;
  void or_word(int i, uint32_t v) {
    if (putting && behind >= 0) putting = false;
    words[i] |= v;
  }
  void q_put(int s, int, uint32_t v) {
    if (!putting) behind = -1;
    putting = true;
    outside += s < 0 || s >= csw::QUEUE_SLOTS;
    q[s] = v;
    expansions += v != 0;
  }
  uint32_t q_get(int s, int) {
    outside += s < 0 || s >= csw::QUEUE_SLOTS;
    late += !putting && s > 0 && s != behind && s != behind + 1;  // one further, or the same again
    if (!putting && behind == 0) late++;                           // a step begun with the second entry unread
    behind = s;
    return q[s];
  }
};
}  // namespace

int main() {
  std::vector<uint32_t> lut(csw::ENC3_LUT_SIZE);
  for (int i = 0; i < csw::ENC3_LUT_SIZE; i++) lut[i] = csw::enc3_lut_entry((uint32_t)i);
  long late = 0, outside = 0, expansions = 0;
  uint32_t seed = 1;
  for (int kind = 0; kind < 6; kind++)
    for (int maxbits : {9, 64, 256, 512, 1024, 4096})
      for (int block = 0; block < 50; block++) {
        float f[64];
        for (int i = 0; i < 64; i++) {
          seed = seed * 1664525u + 1013904223u;
          const float r = (float)(int32_t)seed / 2147483648.0f;
          f[i] = kind == 0 ? r : kind == 1 ? r + 10.0f : kind == 2 ? std::sin(0.1f * i) + 0.01f * r : kind == 3 ? 0.0f
                 : kind == 4 ? (i == block ? r : 0.0f) : std::ldexp(r, (int)(seed >> 27) - 16);
        }
        Watch st;
        csw::encode_block3_staged(f, maxbits, st, lut.data(), csw::pipe_consts());
        late += st.late;
        outside += st.outside;
        expansions += st.expansions;
      }
  std::printf("%ld expansions, %ld read late, %ld outside\n", expansions, late, outside);
  return late != 0 || outside != 0 || expansions == 0;
}
