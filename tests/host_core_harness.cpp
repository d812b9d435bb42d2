// Host build of the per-block codec core (cswap_b200/csrc/zfp_core.cuh), used
// by the CPU test-suite to check the register-level algorithm (byte-sliced
// plane transposes, table-driven group-test coding) bit for bit against the
// oracle without a GPU.  Test scaffolding: the shipped library never runs
// the codec on the host.
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <algorithm>
#include <functional>
#include <vector>

#include "../cswap_b200/csrc/zfp_field.cuh"

namespace {
struct VecSink {
  uint32_t* w;
  void put(int i, uint32_t v) { w[i] = v; }
};
struct VecSource {
  const uint32_t* w;
  int n;
  uint32_t get(int i) const { return i < n ? w[i] : 0u; }
};
std::vector<uint32_t> enc_lut() {
  std::vector<uint32_t> t(csw::ENC_LUT_SIZE);
  for (int i = 0; i < csw::ENC_LUT_SIZE; i++) t[i] = csw::enc_lut_entry(i);
  return t;
}
std::vector<uint32_t> dec_lut() {
  std::vector<uint32_t> t(csw::DEC_LUT_SIZE);
  for (int i = 0; i < csw::DEC_LUT_SIZE; i++) t[i] = csw::dec_lut_entry(i);
  return t;
}
const std::vector<uint32_t>& enc1_lut() {
  static const std::vector<uint32_t> t = [] {
    std::vector<uint32_t> v(csw::ENC1_LUT_SIZE);
    for (int i = 0; i < csw::ENC1_LUT_SIZE; i++) v[i] = csw::enc1_lut_entry(i);
    return v;
  }();
  return t;
}
const std::vector<uint16_t>& dec1_lut() {
  static const std::vector<uint16_t> t = [] {
    std::vector<uint16_t> v(csw::DEC1_LUT_SIZE);
    for (int i = 0; i < csw::DEC1_LUT_SIZE; i++) v[i] = csw::dec1_lut_entry(i);
    return v;
  }();
  return t;
}

const std::vector<uint32_t>& enc3_lut() {
  static const std::vector<uint32_t> t = [] {
    std::vector<uint32_t> v(csw::ENC3_LUT_SIZE);
    for (int i = 0; i < csw::ENC3_LUT_SIZE; i++) v[i] = csw::enc3_lut_entry((uint32_t)i);
    return v;
  }();
  return t;
}
const std::vector<uint32_t>& dec3_lut() {
  static const std::vector<uint32_t> t = [] {
    std::vector<uint32_t> v(csw::DEC3_LUT_SIZE);
    for (int i = 0; i < csw::DEC3_LUT_SIZE; i++)
      if (i % (2 << csw::DEC3_BITS)) v[i] = csw::dec3_lut_entry(i);
    return v;
  }();
  return t;
}

// a lane's staged words and expansion queue, as the kernels keep them in shared memory
struct HostStage {
  uint32_t* w;
  uint32_t q[csw::QUEUE_SLOTS][csw::QUEUE_FIELDS];
  void or_word(int i, uint32_t v) { w[i] |= v; }
  void q_put(int s, int f, uint32_t v) { q[s][f] = v; }
  uint32_t q_get(int s, int f) const { return q[s][f]; }
};
struct PadSource {
  const uint32_t* w;
  int n;
  uint32_t word(int i) const { return i < n ? w[i] : 0u; }
};

// The coders that the kernels run, block by block.  `out` holds whole 64-bit words, zeroed: a
// block's bits are those of its words up to maxbits.
template <int DIMS>
void encode_field(const csw::FieldGeom& g, const float* in, int maxbits, uint32_t* out) {
  static const std::vector<uint32_t> lut = enc_lut();
  const int nw = (maxbits + 31) / 32;
  std::vector<uint32_t> rows(nw + csw::STAGE_SPARE_ROWS);
  for (size_t b = 0; b < csw::geom_blocks(g); b++) {
    float q[1 << (2 * DIMS)];
    csw::gather_block<DIMS>(g, in, b, q);
    std::fill(rows.begin(), rows.end(), 0u);
    if constexpr (DIMS == 3) {
      HostStage st{rows.data(), {}};
      csw::encode_block3_staged(q, maxbits, st, enc3_lut().data(), csw::pipe_consts());
    } else {
      VecSink s{rows.data()};
      if constexpr (DIMS == 2) csw::encode_block2(q, maxbits, s, lut.data());
      else csw::encode_block1(q, maxbits, s, enc1_lut().data());
    }
    for (int w = 0; w < nw; w++) {
      const int bits = maxbits - 32 * w < 32 ? maxbits - 32 * w : 32;
      const size_t at = b * maxbits + 32 * (size_t)w;
      const uint64_t v = (uint64_t)(rows[w] & csw::low_mask32(bits)) << (at & 31);
      out[at >> 5] |= (uint32_t)v;
      if (v >> 32) out[(at >> 5) + 1] |= (uint32_t)(v >> 32);
    }
  }
}
template <int DIMS>
void decode_field(const csw::FieldGeom& g, const uint32_t* in, int maxbits, float* out) {
  static const std::vector<uint32_t> lut = dec_lut();
  const int nw = (maxbits + 31) / 32;
  const size_t total = csw::stream_bytes(g, maxbits) / 4;
  std::vector<uint32_t> rows(nw);
  for (size_t b = 0; b < csw::geom_blocks(g); b++) {
    for (int w = 0; w < nw; w++) {  // what follows the block's own bits is left in, as the kernels leave it
      const size_t at = b * maxbits + 32 * (size_t)w, i = at >> 5;
      rows[w] = csw::funnel_r(in[i], i + 1 < total ? in[i + 1] : 0u, (int)(at & 31));
    }
    float q[1 << (2 * DIMS)];
    if constexpr (DIMS == 3) {
      PadSource s{rows.data(), nw};
      csw::decode_block3_pos(s, maxbits, q, dec3_lut().data());
    } else {
      VecSource s{rows.data(), nw};
      if constexpr (DIMS == 2) csw::decode_block2(s, maxbits, q, lut.data());
      else csw::decode_block1(s, maxbits, q, dec1_lut().data());
    }
    csw::scatter_block<DIMS>(g, out, b, q);
  }
}

// The 32 lanes of a warp, each on a stack of its own: a lane runs until it votes, and the votes are counted when all 32
// stand at one.  Lanes that part - one returns while another votes, or they stand at different votes - would wait for
// each other for good on a GPU; here the warp is given up and run() says so.
class Warp : public csw::HostWarp {
 public:
  Warp() : stacks_(32 * kStack) {}
  bool run(const std::function<void(int)>& lane) {
    body_ = &lane;
    csw::host_warp = this;
    for (int i = 0; i < 32; i++) {
      getcontext(&lanes_[i]);
      lanes_[i].uc_stack.ss_sp = stacks_.data() + i * kStack;
      lanes_[i].uc_stack.ss_size = kStack;
      lanes_[i].uc_link = &home_;
      at_[i] = kRuns;
      const uintptr_t self = reinterpret_cast<uintptr_t>(this);
      makecontext(&lanes_[i], reinterpret_cast<void (*)()>(&Warp::enter), 3, (unsigned)(self >> 32), (unsigned)self, i);
    }
    bool together = true;
    while (together) {
      for (now_ = 0; now_ < 32; now_++) swapcontext(&home_, &lanes_[now_]);
      for (int i = 1; i < 32; i++) together = together && at_[i] == at_[0];
      if (at_[0] == kDone) break;
      result_ = value_[0];
      for (int i = 1; i < 32; i++) result_ = at_[0] == kAny ? result_ | value_[i] : std::max(result_, value_[i]);
    }
    csw::host_warp = nullptr;
    return together;
  }
  bool any(bool p) override { return vote(kAny, p) != 0; }
  int max(int v) override { return vote(kMax, v); }

 private:
  enum Where { kRuns, kAny, kMax, kDone };
  static constexpr size_t kStack = 1 << 17;
  static void enter(unsigned hi, unsigned lo, int i) {
    Warp* w = reinterpret_cast<Warp*>(((uintptr_t)hi << 32) | lo);
    (*w->body_)(i);
    w->at_[i] = kDone;
  }
  int vote(Where kind, int v) {
    const int i = now_;
    at_[i] = kind;
    value_[i] = v;
    swapcontext(&lanes_[i], &home_);
    return result_;
  }
  const std::function<void(int)>* body_ = nullptr;
  std::vector<char> stacks_;
  ucontext_t home_, lanes_[32];
  Where at_[32];
  int value_[32], result_ = 0, now_ = 0;
};

// What the decoders did with a warp's blocks.
enum Way { kFloatWay, kIntWay, kStartedAgain, kParted, kWays };

// Decodes the 32 blocks from b on as a warp does: lanes behind the last block get an empty one.
template <int DIMS>
Way decode_warp(Warp& warp, const csw::FieldGeom& g, const uint32_t* in, int maxbits, float* out, size_t b) {
  const int nw = (maxbits + 31) / 32;
  const size_t total = csw::stream_bytes(g, maxbits) / 4, blocks = csw::geom_blocks(g);
  static std::vector<uint32_t> rows[32];
  static float q[32][64];
  Way way = kFloatWay;
  for (int l = 0; l < 32; l++) {
    rows[l].assign(nw + csw::DEC_SPARE_ROWS, 0u);
    for (int w = 0; b + l < blocks && w < nw; w++) {
      const size_t at = (b + l) * maxbits + 32 * (size_t)w, i = at >> 5;
      rows[l][w] = csw::funnel_r(in[i], i + 1 < total ? in[i + 1] : 0u, (int)(at & 31));
    }
    if (maxbits & 31) rows[l][nw - 1] &= csw::low_mask32(maxbits & 31);
  }
  const bool together = warp.run([&](int l) {
    const PadSource src{rows[l].data(), nw + csw::DEC_SPARE_ROWS};
    csw::HostPark park;
    if constexpr (DIMS == 3) {
      static const Way ways[] = {kFloatWay, kIntWay, kStartedAgain};
      way = ways[csw::decode_block3_host(src, park, maxbits, q[l], dec3_lut().data())];
    } else {
      float (&f)[16] = reinterpret_cast<float (&)[16]>(q[l]);
      csw::decode_block2(src, park, maxbits, f, dec3_lut().data());
    }
  });
  for (int l = 0; together && l < 32 && b + l < blocks; l++) {
    if constexpr (DIMS == 3) csw::scatter_block<3>(g, out, b + l, q[l]);
    else csw::scatter_block<2>(g, out, b + l, reinterpret_cast<float (&)[16]>(q[l]));
  }
  return together ? way : kParted;
}
}  // namespace

extern "C" {
// As core_decode, 2-D and 3-D, 32 blocks at a time; ways[] counts the warps by what the decoder did.
void core_decode_warps(const uint32_t* in, size_t nx, size_t ny, size_t nz, int maxbits, float* out, int* ways) {
  static Warp warp;
  const csw::FieldGeom g = csw::make_geom(nx, ny, nz, 0, 0, 0);
  std::fill(ways, ways + kWays, 0);
  for (size_t b = 0; b < csw::geom_blocks(g); b += 32)
    ways[g.dims == 3 ? decode_warp<3>(warp, g, in, maxbits, out, b) : decode_warp<2>(warp, g, in, maxbits, out, b)]++;
}
void core_encode(const float* in, size_t nx, size_t ny, size_t nz, int maxbits, uint32_t* out) {
  csw::FieldGeom g = csw::make_geom(nx, ny, nz, 0, 0, 0);
  if (g.dims == 3) encode_field<3>(g, in, maxbits, out);
  else if (g.dims == 2) encode_field<2>(g, in, maxbits, out);
  else encode_field<1>(g, in, maxbits, out);
}
void core_decode(const uint32_t* in, size_t nx, size_t ny, size_t nz, int maxbits, float* out) {
  csw::FieldGeom g = csw::make_geom(nx, ny, nz, 0, 0, 0);
  if (g.dims == 3) decode_field<3>(g, in, maxbits, out);
  else if (g.dims == 2) decode_field<2>(g, in, maxbits, out);
  else decode_field<1>(g, in, maxbits, out);
}
size_t core_stream_bytes(size_t nx, size_t ny, size_t nz, unsigned maxbits) {
  return csw::stream_bytes(csw::make_geom(nx, ny, nz, 0, 0, 0), maxbits);
}
}
