// Block-level arithmetic of the fixed-rate ZFP float32 codec, written for one
// thread holding one whole block in registers (lane = block).
//
// Format follows cuZFP as vendored by CSWAP+ (CSWAP+/zfp/encode.cuh:306-368,
// decode.cuh:127-288, shared.h:176-250, constants.h:8-131): 1 flag bit + 8-bit
// biased block exponent, block-floating-point cast to int32, passes of the
// 4-point lifting transform, sequency reorder + negabinary, then the embedded
// group-tested bit-plane coder cut at `maxbits` bits per block.
//
// What differs from the reference is only how the same bits are produced:
//  * bit planes come from 8x8 bit-matrix transposes of the coefficient bytes
//    (PRMT gathers + 3 masked swap stages), eight planes at a time, instead of
//    a 64-step gather per plane;
//  * the group-test phase of a plane is expanded (encoder) or parsed (decoder)
//    eight to eleven positions / stream bits per step through small tables held in
//    shared memory instead of one stream bit per step;
//  * coded bits are assembled in a 64-bit register window and leave as whole
//    32-bit words - no atomics and no pre-zeroed output.
//
// Everything here is plain scalar code per block, so the same header also
// compiles for the host (tests drive it lane by lane against the CPU oracle).
#pragma once
#include <cstdint>
#include <utility>

#if defined(__CUDACC__)
#define CSW_HD __host__ __device__ __forceinline__
#else
#define CSW_HD inline
#endif

namespace csw {

// ---- portable intrinsics ------------------------------------------------------
CSW_HD uint32_t byte_perm(uint32_t a, uint32_t b, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __byte_perm(a, b, s);
#else
  uint64_t ab = ((uint64_t)b << 32) | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; i++) r |= (uint32_t)((ab >> (8 * ((s >> (4 * i)) & 7))) & 0xff) << (8 * i);
  return r;
#endif
}
CSW_HD int clz32(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
CSW_HD int popc32(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __popc(x);
#else
  return __builtin_popcount(x);
#endif
}
CSW_HD uint32_t f2u(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  union { float f; uint32_t u; } c; c.f = f; return c.u;
#endif
}
CSW_HD float u2f(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  union { float f; uint32_t u; } c; c.u = u; return c.f;
#endif
}
// float -> int32, round toward zero, saturating, NaN -> 0 (cvt.rzi.s32.f32)
CSW_HD int f2i_rz(float f) {
#if defined(__CUDA_ARCH__)
  return __float2int_rz(f);
#else
  if (f != f) return 0;
  if (f >= 2147483648.0f) return 2147483647;
  if (f <= -2147483648.0f) return (int)0x80000000;
  return (int)f;
#endif
}
// true when the predicate holds on every active lane of the warp (host: the one "lane")
CSW_HD bool warp_all(bool p) {
#if defined(__CUDA_ARCH__)
  return __all_sync(__activemask(), p);
#else
  return p;
#endif
}
// smallest value over the lanes of the warp, all of which must call (host: the one "lane")
CSW_HD int warp_min(int v) {
#if defined(__CUDA_ARCH__)
  return __reduce_min_sync(0xffffffffu, v);
#else
  return v;
#endif
}
CSW_HD int ctz32(uint32_t x) {  // x != 0
#if defined(__CUDA_ARCH__)
  return __ffs((int)x) - 1;
#else
  return __builtin_ctz(x);
#endif
}
CSW_HD uint32_t low_mask32(int n) {  // n in 0..32
#if defined(__CUDA_ARCH__)
  uint32_t m;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"(n));
  return m;
#else
  return n >= 32 ? 0xffffffffu : ((1u << n) - 1u);
#endif
}

// low min(max(n, 0), 32) bits set, for any n
CSW_HD uint32_t low_mask_sat(int n) {
  const int k = n > 0 ? n : 0;
#if defined(__CUDA_ARCH__)
  uint32_t m;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"(k));
  return m;
#else
  return k >= 32 ? 0xffffffffu : ((1u << k) - 1u);
#endif
}
// 1 << n, 0 for n outside 0..31
CSW_HD uint32_t bit_or_none(int n) {
#if defined(__CUDA_ARCH__)
  uint32_t m;
  asm("shl.b32 %0, 1, %1;" : "=r"(m) : "r"(n));  // counts above 31, unsigned, shift everything out
  return m;
#else
  return (uint32_t)n < 32u ? 1u << n : 0u;
#endif
}
// (s * a, s * b), one instruction on the device
CSW_HD void mul2(float s, float a, float b, float& x, float& y) {
#if defined(__CUDA_ARCH__)
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %2};\n\tmov.b64 q, {%3, %4};\n\tmul.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
      : "=f"(x), "=f"(y) : "f"(s), "f"(a), "f"(b));
#else
  x = s * a;
  y = s * b;
#endif
}

// ---- sequency order (constants.h:8-131), entries are x + 4y + 16z ---------------
constexpr int perm3(int i) {
  constexpr unsigned char t[64] = {
      0,  1,  4,  16, 20, 17, 5,  2,  8,  32, 21, 6,  18, 24, 9,  33,
      36, 3,  12, 48, 22, 25, 37, 40, 34, 10, 7,  19, 28, 13, 49, 52,
      41, 38, 26, 23, 29, 53, 11, 35, 44, 14, 50, 56, 42, 27, 39, 45,
      30, 54, 57, 60, 51, 15, 43, 46, 58, 61, 55, 31, 62, 59, 47, 63};
  return t[i];
}
constexpr int perm2(int i) {
  constexpr unsigned char t[16] = {0, 1, 4, 5, 2, 8, 6, 9, 3, 12, 10, 7, 13, 11, 14, 15};
  return t[i];
}
template <int DIMS, int I>
struct PermAt {
  static constexpr int v = DIMS == 3 ? perm3(I & 63) : perm2(I & 15);
};

// ---- lifting (encode.cuh:73-99, shared.h:221-250) --------------------------------
// Arithmetic is done on unsigned patterns where C++ would overflow; the GPU
// reference simply wraps.
CSW_HD int wadd(int a, int b) { return (int)((uint32_t)a + (uint32_t)b); }
CSW_HD int wsub(int a, int b) { return (int)((uint32_t)a - (uint32_t)b); }
CSW_HD void fwd_lift(int& x, int& y, int& z, int& w) {
  x = wadd(x, w); x >>= 1; w = wsub(w, x);
  z = wadd(z, y); z >>= 1; y = wsub(y, z);
  x = wadd(x, z); x >>= 1; z = wsub(z, x);
  w = wadd(w, y); w >>= 1; y = wsub(y, w);
  w = wadd(w, y >> 1); y = wsub(y, w >> 1);
}
CSW_HD int twice_minus(int a, int b) { return (int)(((uint32_t)a << 1) - (uint32_t)b); }
CSW_HD void inv_lift(int& x, int& y, int& z, int& w) {
  y = wadd(y, w >> 1); w = wsub(w, y >> 1);
  y = wadd(y, w); w = twice_minus(w, y);
  z = wadd(z, x); x = twice_minus(x, z);
  y = wadd(y, z); z = twice_minus(z, y);
  w = wadd(w, x); x = twice_minus(x, w);
}

CSW_HD void fwd_xform2(int (&v)[16]) {
#pragma unroll
  for (int y = 0; y < 4; y++) fwd_lift(v[4 * y], v[4 * y + 1], v[4 * y + 2], v[4 * y + 3]);
#pragma unroll
  for (int x = 0; x < 4; x++) fwd_lift(v[x], v[x + 4], v[x + 8], v[x + 12]);
}

template <int DIMS>
CSW_HD void inv_xform(int (&v)[1 << (2 * DIMS)]) {
  if constexpr (DIMS == 3) {
#pragma unroll
    for (int i = 0; i < 16; i++) inv_lift(v[i], v[i + 16], v[i + 32], v[i + 48]);
#pragma unroll
    for (int z = 0; z < 4; z++)
#pragma unroll
      for (int x = 0; x < 4; x++)
        inv_lift(v[16 * z + x], v[16 * z + x + 4], v[16 * z + x + 8], v[16 * z + x + 12]);
#pragma unroll
    for (int i = 0; i < 16; i++) inv_lift(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
#pragma unroll
    for (int x = 0; x < 4; x++) inv_lift(v[x], v[x + 4], v[x + 8], v[x + 12]);
#pragma unroll
    for (int y = 0; y < 4; y++) inv_lift(v[4 * y], v[4 * y + 1], v[4 * y + 2], v[4 * y + 3]);
  }
}

// ---- negabinary (shared.h:176-181, decode.cuh:33-37) ------------------------------
CSW_HD uint32_t int2uint(int x) { return ((uint32_t)x + 0xaaaaaaaau) ^ 0xaaaaaaaau; }
CSW_HD int uint2int(uint32_t x) { return (int)((x ^ 0xaaaaaaaau) - 0xaaaaaaaau); }

template <int... I>
CSW_HD void fwd_order2(const int (&v)[16], uint32_t (&u)[16], std::integer_sequence<int, I...>) {
  ((u[I] = int2uint(v[PermAt<2, I>::v])), ...);
}
template <int... I>
CSW_HD void inv_order2(const uint32_t (&u)[16], int (&v)[16], std::integer_sequence<int, I...>) {
  ((v[PermAt<2, I>::v] = uint2int(u[I])), ...);
}

// ---- block exponent and cast (encode.cuh:40-71,120-149) ---------------------------
// Biased exponent field e = emax + 127 (0 for an all-zero block) from the bit
// pattern of max|v|: frexp's exponent of a normal float with exponent field E
// is E - 126, and denormals are floored at -126 (field 1).
CSW_HD uint32_t biased_emax(float maxabs) {
  uint32_t b = f2u(maxabs);
  return b == 0 ? 0u : (b >> 23) + 1u;
}
// 2^(30 - emax) as a float; +inf for emax < -97, exactly what the reference's
// ldexp-then-narrow yields, so with the saturating conversion such
// (denormal-range) blocks code the way the reference codes them on a GPU.
CSW_HD float quant_scale(uint32_t e) {
  int f = 284 - (int)e;  // exponent field of 2^(30-emax), emax = e - 127
  f = f > 255 ? 255 : f;
  return u2f((uint32_t)f << 23);
}
// 2^(emax - 30) (shared.h:197-203, decode.cuh:278); denormal below emax = -96.
CSW_HD float dequant_scale(uint32_t e) {
  int f = (int)e - 30;  // exponent field of 2^(emax-30) = e - 127 - 30 + 127
  if (f >= 1) return u2f((uint32_t)f << 23);
  return f > -23 ? u2f(1u << (22 + f)) : 0.0f;  // denormal results of ldexp
}

// ---- 8-plane slices by bit-matrix transpose ---------------------------------------
// One masked swap of an 8x8 (per byte lane) bit transpose.
template <int S, uint32_t M>
CSW_HD void tswap(uint32_t& a, uint32_t& b) {
  uint32_t na = (a & M) | ((b << S) & ~M);
  uint32_t nb = ((a >> S) & M) | (b & ~M);
  a = na;
  b = nb;
}
// In every byte lane: bit k of word j <-> bit j of word k.  Its own inverse.
CSW_HD void transpose8(uint32_t (&r)[8]) {
#pragma unroll
  for (int j = 0; j < 4; j++) tswap<4, 0x0f0f0f0fu>(r[j], r[j + 4]);
#pragma unroll
  for (int j = 0; j < 8; j += 4) {
    tswap<2, 0x33333333u>(r[j], r[j + 2]);
    tswap<2, 0x33333333u>(r[j + 1], r[j + 3]);
  }
#pragma unroll
  for (int j = 0; j < 8; j += 2) tswap<1, 0x55555555u>(r[j], r[j + 1]);
}

// p[k] (k = 0..7) <- bit (8c + k) of the sixteen coefficients of a 2-D block, coefficient i at
// bit i.  Byte m of gather word j holds coefficient 8m + j, so after the transpose bit 8m + j
// of a plane word is coefficient 8m + j.  sel = c | (4 + c) << 4 picks byte c of both PRMT operands.
CSW_HD void planes_of_byte2(const uint32_t (&u)[16], uint32_t sel, uint32_t (&p)[8]) {
#pragma unroll
  for (int j = 0; j < 8; j++) p[j] = byte_perm(u[j], u[8 + j], sel) & 0xffffu;
  transpose8(p);
}

// Inverse: write byte c of each coefficient from eight plane words.
// sel0 keeps the other three bytes of the destination and takes byte 0 of the
// second PRMT operand into byte c; adding m << 4c takes byte m instead.
template <int G, int N>
CSW_HD void bytes_from_planes(uint32_t (&p)[8], uint32_t sel0, uint32_t step, uint32_t (&u)[N]) {
  transpose8(p);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    if constexpr (N == 64) {
#pragma unroll
      for (int m = 0; m < 4; m++) u[32 * G + 8 * m + j] = byte_perm(u[32 * G + 8 * m + j], p[j], sel0 + m * step);
    } else {
      u[j] = byte_perm(u[j], p[j], sel0);
      u[8 + j] = byte_perm(u[8 + j], p[j], sel0 + step);
    }
  }
}

// ---- coder tables -----------------------------------------------------------------
// Encoder: entry for the eight positions v of a plane word past the already
// significant prefix.  Each 0 position codes as '0'; each 1 position codes as
// '1' followed by the next group-test bit, which is '1' whenever a later set
// bit exists.  bits 0..15: that pattern; bits 16..20: its length 8 + popc(v);
// bits 24..28: length when the byte holds the last set bit of the plane
// (positions up to the top set bit, plus one per set bit; the final group-test
// bit is then the '0' terminator).
constexpr int ENC_LUT_SIZE = 256;
constexpr CSW_HD uint32_t enc_lut_entry(uint32_t v) {
  uint32_t pat = 0;
  int len = 0, top = -1, ones = 0;
  for (int i = 0; i < 8; i++) {
    if ((v >> i) & 1u) {
      pat |= 3u << len;
      len += 2;
      top = i;
      ones++;
    } else {
      len += 1;
    }
  }
  uint32_t lf = top < 0 ? 0u : (uint32_t)(top + 1 + ones);
  return pat | ((uint32_t)len << 16) | (lf << 24);
}

// The same for the eleven positions of the 3-D staged encoder: pattern in bits 0..21, the
// length 11 + popc(v) in 22..26, the length of a last piece in 27..31: no bit is left over.
constexpr int ENC3_BITS = 11, ENC3_LUT_SIZE = 1 << ENC3_BITS;
constexpr CSW_HD uint32_t enc3_lut_entry(uint32_t v) {
  uint32_t pat = 0, len = 0, last = 0;
  for (int i = 0; i < ENC3_BITS; i++) {
    if ((v >> i) & 1u) {
      pat |= 3u << len;
      len += 2;
      last = len;
    } else {
      len += 1;
    }
  }
  return pat | (len << 22) | (last << 27);
}

// Decoder: entry for (limit L in 0..8, state, next stream byte).  Simulates the
// group-test parser of decode.cuh:147-164 over at most L stream bits.
// State 0: expecting a group-test bit; state 1: inside a unary run (expecting
// value bits until a one); state 2: negative group test seen, plane finished.
// L = 0 (no open position left, or the budget is spent) finishes the plane
// without reading: from state 1 the run's final one is implied.
// One field per byte, so that each is a single byte-permute away:
// byte 0: stream bits consumed; byte 1: positions advanced;
// byte 2: plane bits found, relative to the starting position;
// byte 3: state afterwards.
constexpr int DEC_LUT_SIZE = 9 * 2 * 256;
constexpr CSW_HD int dec_lut_index(int L, int state, uint32_t byte) { return (L * 2 + state) * 256 + (int)byte; }
constexpr CSW_HD uint32_t dec_lut_entry(int idx) {
  uint32_t byte = idx & 255;
  int st = (idx >> 8) & 1, L = idx >> 9;
  int c = 0, dn = 0;
  uint32_t pat = 0;
  if (L == 0) {
    if (st == 1) { pat = 1u; dn = 1; }
    st = 2;
  }
  while (c < L) {
    uint32_t bit = (byte >> c) & 1u;
    c++;
    if (st == 0) {
      if (bit) st = 1;
      else { st = 2; break; }
    } else {
      if (bit) { pat |= 1u << dn; st = 0; }
      dn++;
    }
  }
  return (uint32_t)c | ((uint32_t)dn << 8) | (pat << 16) | ((uint32_t)st << 24);
}
CSW_HD int dec_lut_used(uint32_t e) { return (int)(e & 0xffu); }
CSW_HD int dec_lut_advance(uint32_t e) { return (int)byte_perm(e, 0u, 0x4441u); }
CSW_HD uint32_t dec_lut_pattern(uint32_t e) { return byte_perm(e, 0u, 0x4442u); }
CSW_HD int dec_lut_state(uint32_t e) { return (int)(e >> 24); }

// Blocks of four values: a plane is a nibble and its whole code at most eight bits, so one
// entry holds a plane.  Encoder: entry for (n significant so far, nibble): code in bits
// 0..7, its length in 8..11, n afterwards in 16..18.  Decoder: entry for (n, next eight stream
// bits): nibble in bits 0..3, stream bits read in 4..7, n afterwards in 8..10.
constexpr int ENC1_LUT_SIZE = 5 * 16, DEC1_LUT_SIZE = 5 * 256;
constexpr CSW_HD uint32_t enc1_lut_entry(int idx) {
  int n = idx >> 4, len = n;
  uint32_t x = (uint32_t)idx & 15u, code = x & ((1u << n) - 1u);
  x >>= n;
  while (n < 4) {  // encode.cuh:336-343
    code |= (x != 0u ? 1u : 0u) << len++;
    if (x == 0u) break;
    while (n < 3) {
      const uint32_t b = x & 1u;
      code |= b << len++;
      if (b) break;
      x >>= 1;
      n++;
    }
    x >>= 1;
    n++;
  }
  return code | ((uint32_t)len << 8) | ((uint32_t)n << 16);
}
constexpr CSW_HD uint16_t dec1_lut_entry(int idx) {
  int n = idx >> 8, len = n;
  const uint32_t s = (uint32_t)idx & 255u;
  uint32_t x = s & ((1u << n) - 1u);
  while (n < 4) {  // decode.cuh:147-164
    if (!((s >> len++) & 1u)) break;
    while (n < 3 && !((s >> len++) & 1u)) n++;
    x |= 1u << n++;
  }
  return (uint16_t)(x | ((uint32_t)len << 4) | ((uint32_t)n << 8));
}

// The same for up to ten stream bits, for the 3-D decoder: of a row with limit L only the
// first L bits matter, so its entries are the 1 << L ones behind entry (1 << L) of the
// state's half.  Bits 0..9: plane bits found; 16..23: positions advanced; 24..27: stream bits
// consumed; 30..31: state afterwards.
constexpr int DEC3_BITS = 10, DEC3_LUT_SIZE = 2 << (DEC3_BITS + 1);
constexpr CSW_HD uint32_t dec3_lut_entry(int idx) {
  const int half = idx & ((2 << DEC3_BITS) - 1);
  int st = idx >> (DEC3_BITS + 1), L = 0;
  while ((2 << L) <= half) L++;
  const uint32_t bits = (uint32_t)(half - (1 << L));
  int c = 0, dn = 0;
  uint32_t pat = 0;
  if (L == 0) {
    if (st == 1) { pat = 1u; dn = 1; }
    st = 2;
  }
  while (c < L) {
    const uint32_t bit = (bits >> c) & 1u;
    c++;
    if (st == 0) {
      if (bit) st = 1;
      else { st = 2; break; }
    } else {
      if (bit) { pat |= 1u << dn; st = 0; }
      dn++;
    }
  }
  return pat | ((uint32_t)dn << 16) | ((uint32_t)c << 24) | ((uint32_t)st << 30);
}

// ---- bit emitter ------------------------------------------------------------------
// WordSink::put(w, word) receives the block's w-th 32-bit stream word; words
// arrive in increasing w, each once.  Everything is written for predication
// rather than branches: lanes of a warp code different blocks and would
// otherwise diverge on every word boundary.
CSW_HD uint32_t funnel_l(uint32_t lo, uint32_t hi, int s) {  // ((hi:lo) << s) >> 32, s taken mod 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
#endif
}
CSW_HD uint32_t funnel_r(uint32_t lo, uint32_t hi, int s) {  // low word of (hi:lo) >> s, s taken mod 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
#endif
}

template <class WordSink>
struct Emitter {
  uint32_t a0;  // the word being filled; bits at and above `fill` are zero
  int fill;     // 0..31
  int wpos;     // words already handed to the sink
  int nwords;   // ceil(maxbits / 32)
  WordSink& sink;
  CSW_HD Emitter(WordSink& s, int nw) : a0(0), fill(0), wpos(0), nwords(nw), sink(s) {}
  CSW_HD int total() const { return 32 * wpos + fill; }
  CSW_HD void flush_word(uint32_t next) {
    if (wpos < nwords) sink.put(wpos, a0);
    wpos++;
    a0 = next;
  }
  // append the low `len` (0..32) bits of v; bits of v at and above len must be zero
  CSW_HD void emit32(uint32_t v, int len) {
    const uint32_t t1 = funnel_l(v, 0u, fill);
    a0 |= v << fill;
    int nf = fill + len;
    if (nf >= 32) {
      flush_word(t1);
      nf -= 32;
    }
    fill = nf;
  }
  // hand over whatever is buffered and zero-fill the rest of the block
  CSW_HD void finish() {
    while (wpos < nwords) flush_word(0u);
  }
};

// ---- encoder: coefficient-count state ----------------------------------------------
// n coefficients are significant so far; the masks select plane bits below n
// and the single bit at position n (zero when n == 64).
struct SigState {  // by mask and shift instructions that saturate: a dozen fewer per plane than selects
  int n;
  uint32_t mlo, mhi;  // low n bits of a 64-bit plane word
  uint32_t glo, ghi;  // bit n
  CSW_HD void set(int nn) {
    n = nn;
    mlo = low_mask_sat(nn);
    mhi = low_mask_sat(nn - 32);
    glo = bit_or_none(nn);
    ghi = bit_or_none(nn - 32);
  }
};

// ---- encoder: one plane of a small block ---------------------------------------------
// N = 16 coefficients: the whole code of a plane - verbatim prefix, group
// test, expansions - is at most 32 bits (n verbatim bits, one test, two bits for
// each of the N - n positions less the implied end), so it is put together
// without a loop from one table entry per eight positions and appended at once.
// One path and one append for every lane (with n == 16 nothing is left over, r == 0,
// and no group test is coded), but for planes that the whole warp copies.
template <class WordSink>
CSW_HD void encode_plane2(uint32_t x, int& n, Emitter<WordSink>& em, const uint32_t* enc_lut) {
  constexpr int N = 16;
  if (warp_all(n >= N)) {
    em.emit32(x, N);
    return;
  }
  const uint32_t r = x >> n;
  const int top = (int)(x >> (N - 1));  // last position set: its 1 is implied
  const uint32_t e0 = enc_lut[r & 0xffu], e1 = enc_lut[r >> 8];
  const bool two = r > 0xffu;
  const uint32_t last = two ? e1 : e0;           // of the byte with the last set bit
  const int len1 = (int)(last >> 24) - 2 * top;  // meaningless, and not used, when r == 0
  const int len0 = two ? (int)((e0 >> 16) & 0x1fu) : 0;
  const uint32_t code = ((last & low_mask_sat(len1 + top - 1)) << len0) | (two ? e0 & 0xffffu : 0u);
  const uint32_t head = x & low_mask_sat(n);
  const int plain = n + 1 < N ? n + 1 : N;
  em.emit32(r ? head | ((2u * code + 1u) << n) : head, r ? n + 1 + len0 + len1 : plain);
  if (r) n = 32 - clz32(x);
}

// ---- blocks of four values: all planes at once ------------------------------------------
// Bits 4k .. 4k+3 of w[c] <-> bit 8c+k of the four coefficients.  One bit transpose of
// the four words covers all 32 planes: its word k holds plane 8m+k in byte m.
CSW_HD void transpose_bytes4(uint32_t (&w)[4]) {  // byte i of word m <-> byte m of word i
  const uint32_t a = byte_perm(w[0], w[1], 0x5140), b = byte_perm(w[2], w[3], 0x5140);
  const uint32_t c = byte_perm(w[0], w[1], 0x7362), d = byte_perm(w[2], w[3], 0x7362);
  w[0] = byte_perm(a, b, 0x5410);
  w[1] = byte_perm(a, b, 0x7632);
  w[2] = byte_perm(c, d, 0x5410);
  w[3] = byte_perm(c, d, 0x7632);
}
CSW_HD void nibbles_of_planes(const uint32_t (&u)[4], uint32_t (&w)[4]) {
  uint32_t r[8] = {u[0], u[1], u[2], u[3], 0u, 0u, 0u, 0u};
  transpose8(r);
#pragma unroll
  for (int i = 0; i < 4; i++) w[i] = r[2 * i] | (r[2 * i + 1] << 4);
  transpose_bytes4(w);
}
CSW_HD void planes_of_nibbles(uint32_t (&w)[4], uint32_t (&u)[4]) {
  transpose_bytes4(w);
  uint32_t r[8];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    r[2 * i] = w[i] & 0x0f0f0f0fu;
    r[2 * i + 1] = (w[i] >> 4) & 0x0f0f0f0fu;
  }
  transpose8(r);
#pragma unroll
  for (int i = 0; i < 4; i++) u[i] = r[i];
}

template <class WordSink>
CSW_HD void encode_block1(const float (&f)[4], int maxbits, WordSink& sink, const uint32_t* lut) {
  Emitter<WordSink> em(sink, (maxbits + 31) >> 5);
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; i++) m = fmaxf(m, fabsf(f[i]));
  const uint32_t e = biased_emax(m);
  if (e == 0) {  // all-zero block: nothing is coded (encode.cuh:356-357)
    em.finish();
    return;
  }
  int v[4];
  const float s = quant_scale(e);
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = f2i_rz(s * f[i]);
  fwd_lift(v[0], v[1], v[2], v[3]);
  uint32_t u[4], w[4];
#pragma unroll
  for (int i = 0; i < 4; i++) u[i] = int2uint(v[i]);
  nibbles_of_planes(u, w);
  const int lead = clz32(u[0] | u[1] | u[2] | u[3]);  // empty planes: a failed group test each
  em.emit32((2u * e + 1u) & 0x1ffu, 9);
  em.emit32(0u, lead);
  int n = 0;
  for (int c = 3; c >= 0; c--) {
    const uint32_t now = w[3];
    w[3] = w[2]; w[2] = w[1]; w[1] = w[0];
#pragma unroll
    for (int k = 7; k >= 0; k--) {
      if (8 * c + k < 32 - lead && em.total() < maxbits) {
        const uint32_t en = lut[16 * n + ((now >> (4 * k)) & 15u)];
        em.emit32(en & 0xffu, (int)((en >> 8) & 15u));
        n = (int)(en >> 16);
      }
    }
    if (em.total() >= maxbits) break;
  }
  em.finish();
}

// ---- encoder: 2-D block -------------------------------------------------------------
// f: the block's values, x fastest (index x + 4y).  Produces exactly ceil(maxbits/32) words
// through the sink (the last one masked by the caller when maxbits is not a multiple of 32).
template <class WordSink>
CSW_HD void encode_block2(const float (&f)[16], int maxbits, WordSink& sink, const uint32_t* enc_lut) {
  Emitter<WordSink> em(sink, (maxbits + 31) >> 5);
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; i++) m = fmaxf(m, fabsf(f[i]));
  const uint32_t e = biased_emax(m);
  if (e == 0) {  // all-zero block: nothing is coded (encode.cuh:356-357)
    em.finish();
    return;
  }
  em.emit32((2u * e + 1u) & 0x1ffu, 9);
  int v[16];
  {
    const float s = quant_scale(e);
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = f2i_rz(s * f[i]);
  }
  fwd_xform2(v);
  uint32_t u[16];
  fwd_order2(v, u, std::make_integer_sequence<int, 16>{});

  int n = 0;
  for (int c = 3; c >= 0; c--) {  // planes 8c+7 .. 8c
    uint32_t x[8];
    planes_of_byte2(u, (uint32_t)c | ((uint32_t)(4 + c) << 4), x);
#pragma unroll
    for (int k = 7; k >= 0; k--) {
      if (em.total() < maxbits) encode_plane2(x[k], n, em, enc_lut);
    }
    if (em.total() >= maxbits) break;
  }
  em.finish();
}

// ---- staged encoder (3-D blocks, any budget) ----------------------------------------
// The stream of encode.cuh:306-368, produced in a way that suits a warp whose lanes
// code 32 different blocks:
//
//  * every plane's bit offset is known before its bits are made: a plane costs
//    n verbatim bits, one group-test bit and, when new coefficients turn
//    significant in it, (top - n) value bits + one group-test bit per set bit
//    (minus the implied final 1 and its terminator when the plane ends on the
//    last position).  So the verbatim parts are OR-ed into the staged words at
//    their offsets, one plane after the other, by all lanes in step;
//  * the expansions (the data-dependent part) are queued per lane and worked off
//    in one flat loop per eight planes, each lane running through its own queue,
//    so lanes do not wait for each other plane by plane.
//
// On sm_100 shifts, logic and compares issue on the integer ALU pipe at half
// the warp rate while integer multiply-adds go down the (otherwise idle)
// multiply-add pipe at the same rate.  Additions and left shifts are therefore
// written as multiply-adds with multipliers the compiler cannot see (they come
// in as kernel arguments), which moves about half of the lifting and transpose
// work off the ALU pipe.
struct PipeConsts {
  int one, mone;         // 1, -1
  uint32_t p1, p2, p4;   // 1 << 1, 1 << 2, 1 << 4
  uint32_t nb;           // 0xaaaaaaaa, the negabinary mask
};
CSW_HD PipeConsts pipe_consts() { return PipeConsts{1, -1, 2u, 4u, 16u, 0xaaaaaaaau}; }

CSW_HD int imad(int a, int b, int c) {
#if defined(__CUDA_ARCH__)
  int d;
  asm("mad.lo.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
#else
  return (int)((uint32_t)a * (uint32_t)b + (uint32_t)c);
#endif
}
CSW_HD uint32_t umad(uint32_t a, uint32_t b, uint32_t c) { return (uint32_t)imad((int)a, (int)b, (int)c); }

// fwd_lift with eight of its ten additions on the multiply-add pipe
CSW_HD void fwd_lift_bal(int& x, int& y, int& z, int& w, const PipeConsts& k) {
  x = imad(x, k.one, w); x >>= 1; w = imad(x, k.mone, w);
  z = imad(z, k.one, y); z >>= 1; y = imad(z, k.mone, y);
  x = imad(x, k.one, z); x >>= 1; z = imad(x, k.mone, z);
  w = imad(w, k.one, y); w >>= 1; y = imad(w, k.mone, y);
  w = wadd(w, y >> 1); y = wsub(y, w >> 1);
}
CSW_HD void fwd_xform3_bal(int (&v)[64], const PipeConsts& k) {
#pragma unroll
  for (int i = 0; i < 16; i++) fwd_lift_bal(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3], k);
#pragma unroll
  for (int z = 0; z < 4; z++)
#pragma unroll
    for (int x = 0; x < 4; x++)
      fwd_lift_bal(v[16 * z + x], v[16 * z + x + 4], v[16 * z + x + 8], v[16 * z + x + 12], k);
#pragma unroll
  for (int i = 0; i < 16; i++) fwd_lift_bal(v[i], v[i + 16], v[i + 32], v[i + 48], k);
}

template <int S, uint32_t M>
CSW_HD void tswap_bal(uint32_t& a, uint32_t& b, uint32_t pow) {  // pow = 1 << S
  const uint32_t bs = umad(b, pow, 0u);
  const uint32_t na = (a & M) | (bs & ~M);
  const uint32_t nb = ((a >> S) & M) | (b & ~M);
  a = na;
  b = nb;
}
CSW_HD void transpose8_bal(uint32_t (&r)[8], const PipeConsts& k) {
#pragma unroll
  for (int j = 0; j < 4; j++) tswap_bal<4, 0x0f0f0f0fu>(r[j], r[j + 4], k.p4);
#pragma unroll
  for (int j = 0; j < 8; j += 4) {
    tswap_bal<2, 0x33333333u>(r[j], r[j + 2], k.p2);
    tswap_bal<2, 0x33333333u>(r[j + 1], r[j + 3], k.p2);
  }
#pragma unroll
  for (int j = 0; j < 8; j += 2) tswap_bal<1, 0x55555555u>(r[j], r[j + 1], k.p1);
}
// p[k] (k = 0..7) <- bit (8c + k) of coefficients 32G .. 32G+31 of a 3-D block, coefficient
// 32G + i at bit i, gathered as planes_of_byte2 does
template <int G>
CSW_HD void planes_of_byte_bal(const uint32_t (&u)[64], uint32_t sel, uint32_t (&p)[8], const PipeConsts& k) {
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const uint32_t t0 = byte_perm(u[32 * G + j], u[32 * G + 8 + j], sel);
    const uint32_t t1 = byte_perm(u[32 * G + 16 + j], u[32 * G + 24 + j], sel);
    p[j] = byte_perm(t0, t1, 0x5410);
  }
  transpose8_bal(p, k);
  // the coefficients came in as v + 0xaaaaaaaa; the xor half of the negabinary
  // map flips every odd bit, i.e. it complements the odd planes
  p[1] = ~p[1]; p[3] = ~p[3]; p[5] = ~p[5]; p[7] = ~p[7];
}

constexpr int STAGE_SPARE_ROWS = 2;  // words a write may run past the block's last word
constexpr int QUEUE_SLOTS = 8;       // expansions per lane per eight planes
constexpr int QUEUE_FIELDS = 3;

// Stage: or_word(w, v) ORs v into the block's w-th staged word (rows
// 0 .. nwords + STAGE_SPARE_ROWS - 1 exist and rows below nwords start as 0);
// q_put / q_get access the lane's expansion queue.
template <class Stage>
CSW_HD void stage_put64(Stage& st, int off, uint32_t lo, uint32_t hi) {
  const int s = off & 31, w = off >> 5;
  st.or_word(w, lo << s);
  st.or_word(w + 1, funnel_l(lo, hi, s));
  st.or_word(w + 2, funnel_l(hi, 0u, s));
}

template <int... I>
CSW_HD void fwd_order3_add(const int (&v)[64], uint32_t (&u)[64], uint32_t nb, int one,
                           std::integer_sequence<int, I...>) {
  ((u[I] = umad((uint32_t)v[PermAt<3, I>::v], (uint32_t)one, nb)), ...);
}

template <class Stage>
CSW_HD void encode_block3_staged(const float (&f)[64], int maxbits, Stage& st, const uint32_t* enc_lut,
                                 const PipeConsts& kc) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 64; i++) m = fmaxf(m, fabsf(f[i]));
  const uint32_t e = biased_emax(m);
  if (e == 0) return;  // all-zero block: the staged words stay zero
  st.or_word(0, (2u * e + 1u) & 0x1ffu);
  int v[64];
  {
    const float s = quant_scale(e);
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
      float a, b;
      mul2(s, f[i], f[i + 1], a, b);
      v[i] = f2i_rz(a);
      v[i + 1] = f2i_rz(b);
    }
  }
  fwd_xform3_bal(v, kc);
  uint32_t u[64];
  fwd_order3_add(v, u, kc.nb, kc.one, std::make_integer_sequence<int, 64>{});

  SigState sg;
  sg.set(0);
  int off = 9;
  for (int c = 3; c >= 0; c--) {  // planes 8c+7 .. 8c
    const uint32_t sel = (uint32_t)c | ((uint32_t)(4 + c) << 4);
    uint32_t lo[8], hi[8];
    planes_of_byte_bal<0>(u, sel, lo, kc);
    planes_of_byte_bal<1>(u, sel, hi, kc);
    int count = 0;
#pragma unroll
    for (int k = 7; k >= 0; k--) {
      if (off < maxbits) {
        // one path for every lane: with n == 64 the masks select the whole
        // word, no position is left over and no group test is coded
        const int n = sg.n;
        const uint32_t above_lo = lo[k] & ~sg.mlo, above_hi = hi[k] & ~sg.mhi;
        const bool any = (above_lo | above_hi) != 0u;
        stage_put64(st, off, (lo[k] & sg.mlo) | (any ? sg.glo : 0u), (hi[k] & sg.mhi) | (any ? sg.ghi : 0u));
        off += n + 1 < 64 ? n + 1 : 64;
        if (any) {
          const int top = (int)(hi[k] >> 31);
          const int msb = hi[k] ? 64 - clz32(hi[k]) : 32 - clz32(lo[k]);
          if (off < maxbits) {
            const uint32_t fl = funnel_r(lo[k], hi[k], n), sh = hi[k] >> (n & 31);
            st.q_put(count, 0, n < 32 ? fl : sh);
            st.q_put(count, 1, n < 32 ? sh : 0u);
            st.q_put(count, 2, (uint32_t)off | ((uint32_t)top << 31));
            count++;
          }
          off += (msb - n) + popc32(above_lo) + popc32(above_hi) - 2 * top;
          sg.set(msb);
        }
      }
    }
    // work off this lane's expansions
    int slot = 0;
    bool have = count > 0;
    uint32_t xl = 0, xh = 0;
    int boff = 0, top = 0;
    if (have) {
      xl = st.q_get(0, 0);
      xh = st.q_get(0, 1);
      const uint32_t meta = st.q_get(0, 2);
      boff = (int)(meta & 0x7fffffffu);
      top = (int)(meta >> 31);
    }
    while (have) {
      const uint32_t en = enc_lut[xl & (ENC3_LUT_SIZE - 1)];
      xl = funnel_r(xl, xh, ENC3_BITS);
      xh >>= ENC3_BITS;
      const bool more = (xl | xh) != 0u;
      const int lf = (int)(en >> 27);
      const int len = more ? (int)((en >> 22) & 0x1fu) : lf - 2 * top;
      const uint32_t keep = more ? 0x3fffffu : low_mask_sat(lf - 1 - top);
      const uint32_t pat = en & keep;
      const int s = boff & 31, w = boff >> 5;
      st.or_word(w, pat << s);
      st.or_word(w + 1, funnel_l(pat, 0u, s));
      boff += len;
      if (!more || boff >= maxbits) {
        slot++;
        have = slot < count;
        if (have) {
          xl = st.q_get(slot, 0);
          xh = st.q_get(slot, 1);
          const uint32_t meta = st.q_get(slot, 2);
          boff = (int)(meta & 0x7fffffffu);
          top = (int)(meta >> 31);
        }
      }
    }
    if (off >= maxbits) break;
  }
}

// ---- decoder: one plane of a small block ----------------------------------------------
// The code of a plane of 16 coefficients is at most 32 bits: one window
// of the stream, consumed from the bottom, holds all of it.
CSW_HD uint32_t decode_plane2(uint32_t win, int& n, int& left, const uint32_t* dec_lut) {
  constexpr int N = 16;
  const int m = n < left ? n : left;
  uint32_t x = win & low_mask_sat(m);
  win >>= m;
  left -= m;
  if (n < N) {
    int st = 0;
    do {
      const int lim = N - st - n;
      int L = lim < 8 ? lim : 8;
      L = left < L ? left : L;
      const uint32_t e = dec_lut[dec_lut_index(L, st, win & 0xffu)];
      const int used = dec_lut_used(e);
      x |= dec_lut_pattern(e) << n;
      n += dec_lut_advance(e);
      win >>= used;
      left -= used;
      st = dec_lut_state(e);
    } while (st != 2);
  }
  return x;
}

// Leading empty planes of a block whose first two words are given, `budget` bits of which
// follow the header: while no coefficient is significant a plane is a single '0' bit (the
// group test of decode.cuh:147 fails at n = 0), so the zeros that follow the header are
// whole planes.
CSW_HD int leading_empty_planes(uint32_t head, uint32_t second, int budget) {
  const uint32_t first = funnel_r(head, second, 9);  // stream bits 9..40
  const int zeros = first ? ctz32(first) : 32;
  return zeros < budget ? zeros : budget;
}

// ---- decoder: blocks of four values ---------------------------------------------------
// One table entry per plane.  The last plane may be cut by the budget: the entry is
// then read with the missing bits as zeros, which is right (decode.cuh:141-165) but for a
// run of zeros that is cut: its one belongs where the bits ran out, while the entry ran on
// to the last position, where it is implied.
template <class WordSource>
CSW_HD void decode_block1(WordSource& src, int maxbits, float (&f)[4], const uint16_t* lut) {
  const uint32_t head = src.get(0);
  if (!(head & 1u)) {  // zero block (decode.cuh:240-243)
#pragma unroll
    for (int i = 0; i < 4; i++) f[i] = 0.0f;
    return;
  }
  const uint32_t e = (head >> 1) & 0xffu;
  int left = maxbits - 9, n = 0;
  const int lead = leading_empty_planes(head, src.get(1), left);
  left -= lead;
  uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int c = 3; c >= 0; c--) {
#pragma unroll
    for (int k = 7; k >= 0; k--) {
      if (8 * c + k < 32 - lead && left > 0) {
        const int pos = maxbits - left;
        const uint32_t win = funnel_r(src.get(pos >> 5), src.get((pos >> 5) + 1), pos) & low_mask_sat(left < 8 ? left : 8);
        const uint32_t en = lut[256 * n + win];
        const int over = (int)((en >> 4) & 15u) - left;
        uint32_t x = en & 15u;
        if (over > 0 && n < 4 && (en >> 8) == 4u) x = (x & 7u) | (8u >> over);
        w[c] |= x << (4 * k);
        left = -over;
        n = (int)(en >> 8);
      }
    }
    if (left <= 0) break;
  }
  uint32_t u[4];
  planes_of_nibbles(w, u);
  int v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = uint2int(u[i]);
  inv_lift(v[0], v[1], v[2], v[3]);
  const float scale = dequant_scale(e);
#pragma unroll
  for (int i = 0; i < 4; i++) f[i] = scale * (float)v[i];
}

// ---- decoder: 2-D block -------------------------------------------------------------
// WordSource::get(w) returns the block's w-th 32-bit stream word (0 past the end of the block).
template <class WordSource>
CSW_HD void decode_block2(WordSource& src, int maxbits, float (&f)[16], const uint32_t* dec_lut) {
  const uint32_t head = src.get(0);
  if (!(head & 1u)) {  // zero block (decode.cuh:240-243)
#pragma unroll
    for (int i = 0; i < 16; i++) f[i] = 0.0f;
    return;
  }
  const uint32_t e = (head >> 1) & 0xffu;
  uint32_t u[16];
#pragma unroll
  for (int i = 0; i < 16; i++) u[i] = 0;
  int left = maxbits - 9, n = 0;
  const int lead = leading_empty_planes(head, src.get(1), left);
  left -= lead;
  for (int c = 3; c >= 0; c--) {
    uint32_t x[8];
#pragma unroll
    for (int k = 7; k >= 0; k--) {
      x[k] = 0u;
      if (8 * c + k < 32 - lead && left > 0) {
        const int pos = maxbits - left;
        x[k] = decode_plane2(funnel_r(src.get(pos >> 5), src.get((pos >> 5) + 1), pos), n, left, dec_lut);
      }
    }
    bytes_from_planes<0>(x, (0x3210u & ~(0xfu << (4 * c))) | (4u << (4 * c)), 1u << (4 * c), u);
    if (left <= 0) break;
  }
  int v[16];
  inv_order2(u, v, std::make_integer_sequence<int, 16>{});
  inv_xform<2>(v);
  const float w = dequant_scale(e);
#pragma unroll
  for (int i = 0; i < 16; i++) f[i] = w * (float)v[i];
}

// ---- 3-D decoder (any budget) --------------------------------------------------------
// The values of decode.cuh:232-288.  Instead of shifting a 64-bit window along
// the stream (integer-pipe work on every read), the parser keeps one bit
// position and fetches what it needs from the staged words with two or three
// shared-memory loads and a funnel shift; the bit budget is simply
// maxbits - pos.  WordSrc::word(w) returns the block's w-th 32-bit word and 0
// for the two rows past the end.
template <class WordSrc>
CSW_HD uint32_t peek_at(const WordSrc& src, int pos) {
  const int w = pos >> 5;
  return funnel_r(src.word(w), src.word(w + 1), pos);  // the shift uses pos mod 32
}
// (h:l) rotated right by r, r in 0..31
CSW_HD void ror64_small(uint32_t& l, uint32_t& h, int r) {
  const uint32_t t = funnel_r(l, h, r);
  h = funnel_r(h, l, r);
  l = t;
}
// (h:l) rotated left by r, r in 0..63
CSW_HD void rol64(uint32_t& l, uint32_t& h, int r) {
  const uint32_t a = (r & 32) ? h : l, b = (r & 32) ? l : h;  // halves after a rotation by 32
  l = funnel_l(b, a, r);
  h = funnel_l(a, b, r);
}

template <int... I>
CSW_HD void inv_order3_sub(const uint32_t (&u)[64], int (&v)[64], uint32_t nb, int mone,
                           std::integer_sequence<int, I...>) {
  ((v[PermAt<3, I>::v] = imad((int)nb, mone, (int)u[I])), ...);  // u - 0xaaaaaaaa on the multiply-add pipe
}
// Planes 8c+7 .. 8c of one block: (hi[k]:lo[k]) <- plane 8c+k, odd planes
// complemented (the xor half of the inverse negabinary map, applied to planes
// instead of coefficients).  `skip` leading planes of the slice are known to be
// empty and have been stepped over already (warp-uniform).
template <class WordSrc>
CSW_HD void decode_slice3(const WordSrc& src, int maxbits, const uint32_t* dec_lut, int skip, int& pos, int& n,
                          uint32_t (&lo)[8], uint32_t (&hi)[8]) {
#pragma unroll
  for (int k = 7; k >= 0; k--) {
    uint32_t xl = 0u, xh = 0u;
    if (7 - k >= skip && pos < maxbits) {
      // first min(n, budget) bits verbatim (decode.cuh:143-145)
      const int left0 = maxbits - pos;
      const int m = n < left0 ? n : left0;
      const int w = pos >> 5;
      const uint32_t w0 = src.word(w), w1 = src.word(w + 1), w2 = src.word(w + 2);
      xl = funnel_r(w0, w1, pos) & low_mask_sat(m);
      xh = funnel_r(w1, w2, pos) & low_mask_sat(m - 32);
      pos += m;
      // group tests and unary runs (decode.cuh:147-164), up to ten stream
      // bits per step; none once every coefficient is significant.  The bits
      // found are gathered in (ah:al), kept rotated so that position n is bit
      // 0: a step ORs its pattern in at the bottom and rotates by the positions
      // it advanced.
      if (n < 64) {
        uint32_t al = 0u, ah = 0u;
        int st = 0;
        do {
          // stream bits this step may read: up to ten, no further than the
          // last open position (a run's final one is implied, so it stops one
          // short) and no further than the block's budget; none at all ends
          // the plane through the table's L = 0 rows
          const int left = maxbits - pos;
          const int lim = 64 - st - n;
          int L = lim < DEC3_BITS ? lim : DEC3_BITS;
          L = left < L ? left : L;
          const uint32_t mask = low_mask32(L);
          const uint32_t en = dec_lut[(st << (DEC3_BITS + 1)) + (int)mask + 1 + (int)(peek_at(src, pos) & mask)];
          const int dn = (int)byte_perm(en, 0u, 0x4442u);
          al |= en & ((1u << DEC3_BITS) - 1u);
          ror64_small(al, ah, dn);
          n += dn;
          pos += (int)((en >> 24) & 15u);
          st = (int)(en >> 30);
        } while (st != 2);
        rol64(al, ah, n);  // position 0 back to bit 0
        xl |= al;
        xh |= ah;
      }
    }
    lo[k] = (k & 1) ? ~xl : xl;
    hi[k] = (k & 1) ? ~xh : xh;
  }
}

template <class WordSrc>
CSW_HD void decode_block3_pos(const WordSrc& src, int maxbits, float (&f)[64], const uint32_t* dec_lut,
                              const PipeConsts& kc) {
  const uint32_t head = src.word(0);
  // The empty planes common to the warp (at most the first slice) are skipped in one go; a
  // lane's further ones go through the loop like any other.
  int lead = 8;
  if (head & 1u) {
    const int zeros = leading_empty_planes(head, src.word(1), maxbits - 9);
    lead = zeros < lead ? zeros : lead;
  }
  lead = warp_min(lead);  // every lane of the warp is here: the tile test before the call is warp-uniform
  if (!(head & 1u)) {  // zero block
#pragma unroll
    for (int i = 0; i < 64; i++) f[i] = 0.0f;
    return;
  }
  const uint32_t e = (head >> 1) & 0xffu;
  int pos = 9 + lead, n = 0;
  uint32_t u[64], lo[8], hi[8];
  // u holds coefficient ^ 0xaaaaaaaa throughout: planes never decoded are zero, i.e. 0xaa bytes.
  // The first slice is peeled so that these constants are operands of its byte permutes
  // instead of sixty-four register initialisations carried into a loop.
  decode_slice3(src, maxbits, dec_lut, lead, pos, n, lo, hi);
#pragma unroll
  for (int i = 0; i < 64; i++) u[i] = 0xaaaaaaaau;
  bytes_from_planes<0>(lo, 0x4210u, 0x1000u, u);
  bytes_from_planes<1>(hi, 0x4210u, 0x1000u, u);
  for (int c = 2; c >= 0 && pos < maxbits; c--) {
    decode_slice3(src, maxbits, dec_lut, 0, pos, n, lo, hi);
    const uint32_t sel0 = (0x3210u & ~(0xfu << (4 * c))) | (4u << (4 * c));
    const uint32_t step = 1u << (4 * c);
    bytes_from_planes<0>(lo, sel0, step, u);
    bytes_from_planes<1>(hi, sel0, step, u);
  }
  int v[64];
  inv_order3_sub(u, v, kc.nb, kc.mone, std::make_integer_sequence<int, 64>{});
  inv_xform<3>(v);
  const float w = dequant_scale(e);
#pragma unroll
  for (int i = 0; i < 64; i += 2) mul2(w, (float)v[i], (float)v[i + 1], f[i], f[i + 1]);
}

}  // namespace csw
