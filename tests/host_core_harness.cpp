// Host build of the per-block codec core (cswap_b200/csrc/zfp_core.cuh), used
// by the CPU test-suite to check the register-level algorithm (byte-sliced
// plane transposes, table-driven group-test coding) bit for bit against the
// oracle without a GPU.  Test scaffolding: the shipped library never runs
// the codec on the host.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <algorithm>
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
      csw::decode_block3_pos(s, maxbits, q, dec3_lut().data(), csw::pipe_consts());
    } else {
      VecSource s{rows.data(), nw};
      if constexpr (DIMS == 2) csw::decode_block2(s, maxbits, q, lut.data());
      else csw::decode_block1(s, maxbits, q, dec1_lut().data());
    }
    csw::scatter_block<DIMS>(g, out, b, q);
  }
}
}  // namespace

extern "C" {
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
