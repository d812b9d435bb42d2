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
// Votes.  A host build runs one lane at a time, alone or, where the tests give it a warp, among the 32 of one.
#if !defined(__CUDACC__)
struct HostWarp {
  virtual bool any(bool p) = 0;
  virtual int max(int v) = 0;
};
inline HostWarp* host_warp = nullptr;
#endif
// True when the predicate holds on every lane that happens to be converged here, which CUDA leaves open: for hints only,
// where it does not matter that lanes of a warp get different answers.
CSW_HD bool converged_all(bool p) {
#if defined(__CUDA_ARCH__)
  return __all_sync(__activemask(), p);
#else
  return p;
#endif
}
// true when it holds on some lane of the warp, all of which must call
CSW_HD bool warp_any(bool p) {
#if defined(__CUDA_ARCH__)
  return __any_sync(0xffffffffu, p);
#elif !defined(__CUDACC__)
  return host_warp ? host_warp->any(p) : p;
#else
  return p;
#endif
}
// true when it holds on every lane of the warp, all of which must call
CSW_HD bool warp_all(bool p) { return !warp_any(!p); }
// largest value over the lanes of the warp, all of which must call
CSW_HD int warp_max(int v) {
#if defined(__CUDA_ARCH__)
  return __reduce_max_sync(0xffffffffu, v);
#elif !defined(__CUDACC__)
  return host_warp ? host_warp->max(v) : v;
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

// pairs of floats: two operations in one instruction on the device
struct F2 {
  float x, y;
};
CSW_HD float fma1(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}
CSW_HD F2 fma2(F2 a, float s, F2 c) {
#if defined(__CUDA_ARCH__)
  F2 d;
  asm("{\n\t.reg .b64 p, q, r;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tmov.b64 r, {%5, %6};\n\t"
      "fma.rn.f32x2 p, p, q, r;\n\tmov.b64 {%0, %1}, p;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(s), "f"(c.x), "f"(c.y));
  return d;
#else
  return F2{fma1(a.x, s, c.x), fma1(a.y, s, c.y)};
#endif
}
CSW_HD F2 add2(F2 a, F2 b) {
#if defined(__CUDA_ARCH__)
  F2 d;
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\t"
      "add.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
#else
  return F2{a.x + b.x, a.y + b.y};
#endif
}

// largest magnitude of three
CSW_HD float max_abs3(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  float d;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
#else
  return fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c));
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
CSW_HD void inv_lift(int& x, int& y, int& z, int& w) {
  const int a = wadd(y, w >> 1), b = wsub(w, a >> 1), c = wsub(x, z), d = wadd(x, z);
  x = wadd(wsub(c, b), a);
  y = wadd(wadd(d, b), a);
  z = wsub(wsub(d, b), a);
  w = wsub(wadd(c, b), a);
}

CSW_HD void fwd_xform2(int (&v)[16]) {
#pragma unroll
  for (int y = 0; y < 4; y++) fwd_lift(v[4 * y], v[4 * y + 1], v[4 * y + 2], v[4 * y + 3]);
#pragma unroll
  for (int x = 0; x < 4; x++) fwd_lift(v[x], v[x + 4], v[x + 8], v[x + 12]);
}

CSW_HD void inv_xform3(int (&v)[64]) {
#pragma unroll
  for (int i = 0; i < 16; i++) inv_lift(v[i], v[i + 16], v[i + 32], v[i + 48]);
#pragma unroll
  for (int z = 0; z < 4; z++)
#pragma unroll
    for (int x = 0; x < 4; x++)
      inv_lift(v[16 * z + x], v[16 * z + x + 4], v[16 * z + x + 8], v[16 * z + x + 12]);
#pragma unroll
  for (int i = 0; i < 16; i++) inv_lift(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}
CSW_HD void inv_xform2(int (&v)[16]) {
#pragma unroll
  for (int x = 0; x < 4; x++) inv_lift(v[x], v[x + 4], v[x + 8], v[x + 12]);
#pragma unroll
  for (int y = 0; y < 4; y++) inv_lift(v[4 * y], v[4 * y + 1], v[4 * y + 2], v[4 * y + 3]);
}

// ---- negabinary (shared.h:176-181, decode.cuh:33-37) ------------------------------
CSW_HD uint32_t int2uint(int x) { return ((uint32_t)x + 0xaaaaaaaau) ^ 0xaaaaaaaau; }
CSW_HD int uint2int(uint32_t x) { return (int)((x ^ 0xaaaaaaaau) - 0xaaaaaaaau); }

template <int... I>
CSW_HD void fwd_order2(const int (&v)[16], uint32_t (&u)[16], std::integer_sequence<int, I...>) {
  ((u[I] = int2uint(v[PermAt<2, I>::v])), ...);
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

// Decoder of the larger blocks: up to nine stream bits of a plane's group tests and runs
// (decode.cuh:147-164), limited by the open positions alone (its words are zero past the budget).  With L < 9 exactly L positions are open,
// with L = 9 at least as many; a row of limit L has an entry for each value of L stream bits, behind
// entry (1 << L) of the state's half.  A run reads one bit less: the last position's one is implied.
// Bits 0..8: plane bits found; 9: the plane is finished; 10: a run is open (the other half is
// next; the bits from 9 on are never shifted into what was found); 16..23: stream bits consumed;
// 24..31: positions advanced.
constexpr int DEC_BITS = 9, DEC_LUT_SIZE = 2 << (DEC_BITS + 1);
constexpr uint32_t DEC_END = 1u << DEC_BITS, DEC_RUN = 2u << DEC_BITS;
constexpr CSW_HD uint32_t dec_lut_entry(int idx) {
  const int half = idx & ((2 << DEC_BITS) - 1);
  bool run = (idx >> (DEC_BITS + 1)) != 0, end = false;
  int L = 0;
  while ((2 << L) <= half) L++;
  const uint32_t bits = (uint32_t)(half - (1 << L));
  const int last = L < DEC_BITS ? L - 1 : 1000;  // the last open position, where it is known
  const int most = run && L > 0 ? L - 1 : L;      // bits to read
  int c = 0, dn = 0;
  uint32_t pat = 0;
  while (!end) {
    if (dn > last) {
      end = dn > 0;  // no position open at all is no plane: nothing happens
      break;
    } else if (run && dn == last) {
      pat |= 1u << dn++;
      run = false;
    } else if (c == most) {
      break;
    } else {
      const uint32_t bit = (bits >> c++) & 1u;
      if (!run) {
        if (bit) run = true;
        else end = true;
      } else {
        if (bit) {
          pat |= 1u << dn;
          run = false;
        }
        dn++;
      }
    }
  }
  return pat | (end ? DEC_END : 0u) | (run ? DEC_RUN : 0u) | ((uint32_t)c << 16) | ((uint32_t)dn << 24);
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
  if (converged_all(n >= N)) {
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
//    so lanes do not wait for each other plane by plane.  A queue entry is a place, a count of
//    positions and whether the last one is the block's last; the bits themselves lie one
//    expansion behind the other in one word, for a position becomes significant once.
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
constexpr int QUEUE_SLOTS = 10;      // expansions per lane per eight planes, the end mark, and one that is read ahead of it
constexpr int QUEUE_FIELDS = 1;

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

// All lanes of the warp call.
template <class Stage>
CSW_HD void encode_block3_staged(const float (&f)[64], int maxbits, Stage& st, const uint32_t* enc_lut,
                                 const PipeConsts& kc) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 64; i++) m = fmaxf(m, fabsf(f[i]));
  const uint32_t e = biased_emax(m);
  // an all-zero block's staged words stay zero: its lane has nothing to code, but goes along
  st.or_word(0, e ? (2u * e + 1u) & 0x1ffu : 0u);
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
  int off = e ? 9 : maxbits;
  for (int c = 3; c >= 0; c--) {  // planes 8c+7 .. 8c
    const uint32_t sel = (uint32_t)c | ((uint32_t)(4 + c) << 4);
    uint32_t lo[8], hi[8];
    planes_of_byte_bal<0>(u, sel, lo, kc);
    planes_of_byte_bal<1>(u, sel, hi, kc);
    int count = 0;
    const int from = sg.n;
    uint32_t fl = 0u, fh = 0u;  // what the expansions code: a position becomes significant once
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
          fl |= above_lo;
          fh |= above_hi;
          if (off < maxbits) {
            st.q_put(count, 0, (uint32_t)off | ((uint32_t)(msb - n) << 16) | ((uint32_t)top << 31));
            count++;
          }
          off += (msb - n) + popc32(above_lo) + popc32(above_hi) - 2 * top;
          sg.set(msb);
        }
      }
    }
    st.q_put(count, 0, 0u);
    // Work off this lane's expansions, with a vote at every step: left to itself the compiler makes
    // two loops of this one, the inner one an expansion's steps, and the lanes wait at its end.
    if (from & 32) {
      fl = fh;
      fh = 0u;
    }
    fl = funnel_r(fl, fh, from);
    fh >>= from & 31;
    // The entry behind the one at work is in a register: read when it is due, it and the table would be two
    // shared-memory reads in a row every step (64 KiB at 512 bits, where a step's latency counts, 4.39 us
    // against 4.24; 256 MiB 101.3 against 100.1).
    int slot = 1;
    const uint32_t now = st.q_get(0, 0);
    uint32_t ahead = st.q_get(1, 0);
    int boff = (int)(now & 0xffffu), left = (int)((now >> 16) & 0x7fu), top = (int)(now >> 31);
    while (warp_any(left > 0)) {
      const bool last = left <= ENC3_BITS;
      const int take = last ? left : ENC3_BITS;
      const uint32_t en = enc_lut[fl & low_mask32(take)];
      const int lf = (int)(en >> 27);
      const int len = last ? lf - 2 * top : (int)((en >> 22) & 0x1fu);
      const uint32_t pat = en & (last ? low_mask_sat(lf - 1 - top) : 0x3fffffu);
      const int s = boff & 31, w = boff >> 5;
      st.or_word(w, pat << s);
      st.or_word(w + 1, funnel_l(pat, 0u, s));
      fl = funnel_r(fl, fh, take);
      fh >>= take;
      boff += len;
      const bool next = (int)(left > 0) & ((int)last | (int)(boff >= maxbits));
      left -= take;
      boff = next ? (int)(ahead & 0xffffu) : boff;
      left = next ? (int)((ahead >> 16) & 0x7fu) : left;
      top = next ? (int)(ahead >> 31) : top;
      slot += next ? 1 : 0;
      ahead = st.q_get(slot, 0);
    }
    if (!warp_any(off < maxbits)) break;
  }
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

// ---- decoder: 2-D and 3-D blocks (any budget) ------------------------------------------
// The values of decode.cuh:232-288.  A warp's lanes decode 32 different blocks, whose group
// tests lie in different planes and take different numbers of steps, so nothing here goes
// plane by plane for the warp as a whole:
//
//  * Planes are counted from a block's own first one that is not empty (the empty ones ahead
//    of it are one '0' bit each), and taken sixteen at a time.
//  * Of these every lane first runs through the group tests of its own planes, as long as
//    it has coefficients that are not significant, and parks a mark at the end of each: where
//    the next plane begins and how many of its bits are verbatim.  The loop lasts as long as the lane
//    with the most steps, not the sum over planes of the longest (16.2 steps against 33.7 for
//    3-D at 512 bits, 9.9 against 25.2 for 2-D at 128, counted on the CPU over the benchmark's values).  What the tests find
//    needs no slots: a position becomes significant once, so the bits of all planes fit into one word.
//  * Then the planes are put together by all lanes in step - a funnel shift of staged
//    words, the found bits, masks - and transposed, sixteen of 2-D at once and eight of 3-D.
//
// WordSrc::word(w) returns the block's w-th 32-bit word, with zeros for the bits past the
// budget and for DEC_SPARE_ROWS words behind it: a group test that finds no bits ends its plane,
// as it must, and only a run cut by the budget needs a correction (decode_tests).
// Park: mark(j) is the lane's slot j, j < PARK_SLOTS.
constexpr int DEC_SPARE_ROWS = 4, CHUNK3 = 8, CHUNK2 = 16, PARK_SLOTS = 18;

// (h:l) rotated left by r, r in 0..64
CSW_HD void rol64(uint32_t& l, uint32_t& h, int r) {
  const uint32_t a = (r & 32) ? h : l, b = (r & 32) ? l : h;  // halves after a rotation by 32
  l = funnel_l(b, a, r);
  h = funnel_l(a, b, r);
}

// A place in the stream: bit position in the low half, significant coefficients in the high one.
CSW_HD int mark_pos(uint32_t m) { return (int)(m & 0xffffu); }
CSW_HD int mark_n(uint32_t m) { return (int)(m >> 16); }

struct BlockHead {
  uint32_t e;
  int lead, start;  // empty planes, where the others begin
};
template <class WordSrc>
CSW_HD BlockHead block_head(const WordSrc& src, int maxbits) {
  const uint32_t head = src.word(0);
  BlockHead b;
  b.e = (head >> 1) & 0xffu;
  b.lead = leading_empty_planes(head, src.word(1), maxbits - 9);
  b.start = 9 + b.lead;
  if (!(head & 1u) || b.lead > 31) {  // a zero block (decode.cuh:240-243), or no plane holds anything
    b.e = 127;
    b.lead = 0;
    b.start = maxbits;
  }
  return b;
}

// What the group tests of a block have found so far: position p of n is bit 64 - n + p of (hi:lo).
struct Found {
  uint32_t lo, hi;
};

// The group tests and unary runs of up to CHUNK planes of a block of N coefficients from `m` on, up to
// nine stream bits per step.  Returns how many planes had any; m moves behind them.  All lanes of
// the warp go round together, with a vote at every step: left to itself the compiler makes two
// loops of this one, the inner one a plane's steps, and the lanes wait at its end.
template <int N, int CHUNK, class WordSrc, class Park>
CSW_HD int decode_tests(const WordSrc& src, Park& park, int maxbits, const uint32_t* dec_lut, uint32_t& m, Found& found) {
  constexpr uint32_t kDone = (uint32_t)N << 16;  // no open position: steps change nothing
  int j = 0;
  park.put_mark(0, m);
  uint32_t at = m + (m >> 16), run = 0u;
  if (m >= kDone || mark_pos(m) >= maxbits) at = kDone;
  while (warp_any(at < kDone)) {
    const int open = N - (int)(at >> 16);
    const uint32_t mask = low_mask32(open < DEC_BITS ? open : DEC_BITS);
    const int w = mark_pos(at) >> 5;
    const uint32_t win = funnel_r(src.word(w), src.word(w + 1), (int)at);
    const uint32_t en = dec_lut[run + mask + 1u + (win & mask)];
    const int dn = (int)(en >> 24);
    if (N > 32) found.lo = funnel_r(found.lo, found.hi, dn);
    found.hi = funnel_r(found.hi, en, dn);
    at += byte_perm(en, 0u, 0x4342u);
    run = en & DEC_RUN;
    park.put_mark(j + 1, at);  // stays when the plane is finished
    const bool end = (en & DEC_END) != 0u;
    j += end ? 1 : 0;
    uint32_t next = at + (at >> 16);  // behind the verbatim bits
    next = (int)(j == CHUNK) | (int)(mark_pos(at) >= maxbits) ? kDone : next;
    next = at >= kDone ? kDone : next;
    at = end ? next : at;
  }
  m = park.mark(j);
  // A run cut by the budget: its one belongs where the bits ran out, but it ran on through the
  // zeros behind them to the last position, where it is implied.
  const int over = mark_pos(m) - maxbits;
  if (over > 0 && m >= kDone && j > 0) {
    found.hi &= 0x7fffffffu;
    if (over < 32) found.hi |= 0x80000000u >> over;
    else found.lo |= 0x80000000u >> (over - 32);
  }
  return j;
}

// What decode_tests found in planes of a 3-D block, besides the marks: how many had group tests, the place behind them.
struct Tests3 {
  int tests;
  uint32_t m;
  Found found;
};
template <int PLANES, class WordSrc, class Park>
CSW_HD Tests3 tests_from(const WordSrc& src, Park& park, int maxbits, const uint32_t* dec_lut, uint32_t m, Found found) {
  Tests3 t{0, m, found};
  t.tests = decode_tests<64, PLANES>(src, park, maxbits, dec_lut, t.m, t.found);
  return t;
}
// Planes that begin within the budget; many, where more of them have tests than were gone through.
CSW_HD int planes_behind(const Tests3& t, int maxbits) {
  const int rest = maxbits - mark_pos(t.m);
  return t.tests + (rest > 0 ? (mark_n(t.m) == 64 ? (rest + 63) >> 6 : 64) : 0);
}

// Eight planes from the FIRST one behind a call of decode_tests on, transposed: byte b of w[8 * g + i] holds coefficient
// 32g + 8b + i (in sequency order), the first plane in its top bit, odd bits complemented (the xor half of the
// inverse negabinary map).  `at` is the place of the first of them, and moves behind the last; (fh:fl): what was found, position
// p at bit p.  most_tests, most_planes: of the lanes of the warp.  NARROW: the budget up to which to look
// out for warps none of whose coefficients from the 32nd on is significant yet.
template <int FIRST, int NARROW, class WordSrc, class Park>
CSW_HD void decode_rows3(const WordSrc& src, const Park& park, int maxbits, int tests, int most_tests, int most_planes,
                         uint32_t fl, uint32_t fh, uint32_t& at, uint32_t (&w)[16]) {
  const int nwords = (maxbits + 31) >> 5;
  const int warp_tests = most_tests - FIRST, warp_left = most_planes - FIRST;
  uint32_t ml = low_mask_sat(mark_n(at)), mh = low_mask_sat(mark_n(at) - 32);
  if (warp_left == 1 && warp_tests <= 0) {
    // A plane is left, the usual case behind eight or sixteen of a budget of whole values: no transpose.
    int i = mark_pos(at) >> 5;
    i = i < nwords ? i : nwords;
    const uint32_t w0 = src.word(i), w1 = src.word(i + 1), w2 = src.word(i + 2);
    const uint32_t xl = ~funnel_r(w0, w1, (int)at), xh = ~funnel_r(w1, w2, (int)at);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      w[k] = ((xl << (7 - k)) & 0x80808080u) | 0x2a2a2a2au;
      w[8 + k] = ((xh << (7 - k)) & 0x80808080u) | 0x2a2a2a2au;
    }
    at += 64u * CHUNK3;
    return;
  }
  uint32_t lo[8], hi[8];
  if (maxbits <= NARROW && warp_tests > 0 && warp_max(mark_n(park.mark(tests < FIRST + CHUNK3 ? tests : FIRST + CHUNK3))) <= 32) {
#pragma unroll
    for (int j = 0; j < CHUNK3; j++) {
      uint32_t xl = 0u;
      if (j < warp_tests) {
        int i = mark_pos(at) >> 5;
        i = i < nwords ? i : nwords;
        xl = funnel_r(src.word(i), src.word(i + 1), (int)at);
        if (FIRST + j < tests) at = park.mark(FIRST + j + 1);
        xl = (xl & ml) | (fl & ~ml);
        ml = low_mask_sat(mark_n(at));
        xl &= ml;
      }
      lo[7 - j] = (j & 1) ? xl : ~xl;
    }
    transpose8(lo);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      w[i] = lo[i];
      w[8 + i] = 0xaaaaaaaau;
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < CHUNK3; j++) {
    uint32_t xl = 0u, xh = 0u;
    if (j < warp_left) {
      int i = mark_pos(at) >> 5;
      i = i < nwords ? i : nwords;
      const uint32_t w0 = src.word(i), w1 = src.word(i + 1), w2 = src.word(i + 2);
      xl = funnel_r(w0, w1, (int)at);
      xh = funnel_r(w1, w2, (int)at);
      at += 64u;
      if (j < warp_tests) {
        // the first n bits verbatim (decode.cuh:143-145), then those found up to the next n
        if (FIRST + j < tests) at = park.mark(FIRST + j + 1);
        xl = (xl & ml) | (fl & ~ml);
        xh = (xh & mh) | (fh & ~mh);
        ml = low_mask_sat(mark_n(at));
        mh = low_mask_sat(mark_n(at) - 32);
        xl &= ml;
        xh &= mh;
      }
    }
    lo[7 - j] = (j & 1) ? xl : ~xl;
    hi[7 - j] = (j & 1) ? xh : ~xh;
  }
  // behind planes without tests every coefficient is significant, or the budget is spent
  transpose8(lo);
  transpose8(hi);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    w[i] = lo[i];
    w[8 + i] = hi[i];
  }
}
CSW_HD void empty_rows3(uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i++) w[i] = 0xaaaaaaaau;
}

// inv_lift in floating point, where it is exact (decode_block3): ten operations become nine
CSW_HD void inv_lift2(F2& x, F2& y, F2& z, F2& w) {  // two lines at a time
  const F2 y1 = fma2(w, 0.5f, y);
  const F2 a = fma2(y1, 0.5f, w), b = fma2(y1, -1.5f, w);
  const F2 c = fma2(z, -1.0f, x), d = add2(x, z);
  x = fma2(b, -1.0f, c);
  y = add2(d, a);
  z = fma2(a, -1.0f, d);
  w = add2(c, b);
}
CSW_HD void inv_lift1(float& x, float& y, float& z, float& w) {
  const float y1 = fma1(w, 0.5f, y);
  const float a = fma1(y1, 0.5f, w), b = fma1(y1, -1.5f, w);
  const float c = x - z, d = x + z;
  x = c - b;
  y = d + a;
  z = d - a;
  w = c + b;
}
// the lines along z and y, pairs along x
CSW_HD void inv_xform3_zy(F2 (&q)[32]) {
#pragma unroll
  for (int i = 0; i < 8; i++) inv_lift2(q[i], q[i + 8], q[i + 16], q[i + 24]);
#pragma unroll
  for (int z = 0; z < 4; z++)
#pragma unroll
    for (int x = 0; x < 2; x++) inv_lift2(q[8 * z + x], q[8 * z + x + 2], q[8 * z + x + 4], q[8 * z + x + 6]);
}

constexpr int perm3_inverse(int p) {
  int i = 0;
  while (perm3(i) != p) i++;
  return i;
}
template <int P>
struct SequencyAt {
  static constexpr int v = perm3_inverse(P);
};
// q <- h * s + t
template <int... P>
CSW_HD void floats_of3(const float (&h)[64], float s, float t, F2 (&q)[32], std::integer_sequence<int, P...>) {
  ((q[P] = fma2(F2{h[SequencyAt<2 * P>::v], h[SequencyAt<2 * P + 1>::v]}, s, F2{t, t})), ...);
}
template <int... I>
CSW_HD void ints_of3(const uint32_t (&u)[64], int lead, int (&v)[64], std::integer_sequence<int, I...>) {
  // the digits move down by `lead`, zeros follow; where that takes the odd ones to even places all are
  // complemented, and so is the difference: (x ^ 0xaaaaaaaa) - 0xaaaaaaaa or (~x ^ ...) - ...
  const int sign = (lead & 1) ? -1 : 1, from = (lead & 1) ? 0x55555555 : 0x55555556;
  ((v[PermAt<3, I>::v] = imad((int)funnel_r(u[I], 0xaaaaaaaau, lead), sign, from)), ...);
}

// The values of a block.
//
// Counted from its first plane that is not empty, a block's coefficients are (-1/2)^lead times what
// they would be if that plane were the top one, so as long as the arithmetic is exact the empty planes
// are a factor.  It is exact in float32 for most blocks: with K planes read, the lowest of weight
// 2^p, every intermediate is a multiple of 2^(p - 6) (the inverse lifting halves twice a pass), and of
// a magnitude that the results bound, since each is a mean of results with weights whose magnitudes add up
// to one at most (run the lifting backwards).  So when the results stay below 2^(p + 18), 24 bits
// held everything, and when they stay below 2^31 too the integers of decode.cuh:177-288 would not have
// wrapped (their shifts lose nothing with p > 5): the same values, to the bit.  The results are checked
// for that, with a margin for what rounding could have done to larger ones.  The products with the block's
// scale are powers of two, exact within the exponents asked for.
//
// What can fail the check is not tried, as far as the group tests tell: a block's scale leaves room for results of 2^30, so
// p < 12 (planes + lead > 20) is not, and with p > 26 what the planes below would have added is so much that results beyond
// 2^31 are common where values reach the top of a block's range.  Failing costs: the block is decoded again from the start
// (256 MiB at 256 bits, values of +-1 before rounding: 154.7 us with p = 27 tried, 85.8 without).
//
// The integers take every block, and get the budgets at which few or only some fit:
//  * above 832 bits, where p falls below 12.  (256 MiB, normal values: at 896 bits 110.2 us, 100.3 with floats tried up to 1152
//    bits, but at 1024 bits, where half of the warps fit, 122.3 and 127.1, at 1152 127.0 and 131.8.)
//  * below 256 bits, where p is mostly above 26.
enum Way3 { kFloats3, kInts3, kShortInts3 };
CSW_HD Way3 decode3_way(int maxbits) { return maxbits < 256 ? kShortInts3 : maxbits <= 832 ? kFloats3 : kInts3; }

// What became of a warp's blocks, the same for all lanes: for the tests.
enum Taken3 { kByFloats, kByInts, kByIntsAfterAll };

// A 3-D block; all lanes of the warp call.  WAY: decode3_way(maxbits).  sink(values) takes them; rest() decodes a block again
// that the check turned down.
//
// What both decoders need is written once, and so are the two rounds of sixteen planes: a warp in one beside a warp in
// another is the usual case for values that are neither noise nor smooth, and their code together is more than
// the instruction cache holds.  (With the integers out of line, with a code of their own for the planes: normal
// values + 10 at 704 bits, where half of the warps fit, 154.4 us against 127.4, all of them noise 97.4 against 98.3;
// with the second round unrolled smooth values at 512 bits 176.5 against 164.4.)
// kShortInts3 looks out for warps whose planes have few significant coefficients, or fill one byte (smooth values at 64 bits
// 99.6 -> 93.2 us, normal ones 70.3 -> 68.3; at 1024 bits it costs, 121.5 -> 126.6).
template <Way3 WAY, class WordSrc, class Park, class Sink, class Rest>
CSW_HD Taken3 decode_block3(const WordSrc& src, Park& park, int maxbits, const uint32_t* dec_lut, Sink&& sink,
                            Rest&& rest) {
  constexpr int kNarrow = WAY == kShortInts3 ? 255 : 0;
  const BlockHead blk = block_head(src, maxbits);
  bool floats = WAY == kFloats3;
  uint32_t w0[16], w1[16], first0[16], first1[16], at = (uint32_t)blk.start;
  Found found{0u, 0u};
  int planes, most_planes;
  bool second = false;
  // Sixteen planes, and once more for the others.
#pragma unroll 1
  for (;;) {
    const Tests3 t = tests_from<2 * CHUNK3>(src, park, maxbits, dec_lut, at, found);
    planes = planes_behind(t, maxbits);
    if (floats) {
      const int down = planes + blk.lead;
      floats = warp_all(blk.e >= 34 && blk.e <= 225 && planes <= 2 * CHUNK3 && ((uint32_t)(down - 6) <= 14u || planes == 0));
    }
    const int most_tests = warp_max(t.tests);
    most_planes = warp_max(planes);
    found = t.found;
    uint32_t fl = found.lo, fh = found.hi;
    rol64(fl, fh, mark_n(t.m));
    decode_rows3<0, kNarrow>(src, park, maxbits, t.tests, most_tests, most_planes, fl, fh, at, w0);
    if (most_planes > 8) decode_rows3<8, 0>(src, park, maxbits, t.tests, most_tests, most_planes, fl, fh, at, w1);
    else empty_rows3(w1);
    if (floats || second || most_planes <= 16) break;
    second = true;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      first0[i] = w0[i];
      first1[i] = w1[i];
    }
  }
  if (floats) {
    // h: the sixteen planes as an integer, the first one in bit 15, held as a float
    float h[64];
    const int unit = (int)blk.e - 14 - blk.lead;  // exponent field of the weight of 2^0 of h
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t a = byte_perm(w1[i], w0[i], 0x5140), b = byte_perm(w1[i], w0[i], 0x7362);
      const int at = 32 * (i >> 3) + (i & 7);
      h[at] = u2f(byte_perm(a, 0x4b000000u, 0x7610));  // 2^23 + it
      h[at + 8] = u2f(byte_perm(a, 0x4b000000u, 0x7632));
      h[at + 16] = u2f(byte_perm(b, 0x4b000000u, 0x7610));
      h[at + 24] = u2f(byte_perm(b, 0x4b000000u, 0x7632));
    }
    const float s = u2f(((uint32_t)unit << 23) | ((uint32_t)blk.lead << 31));
    F2 q[32];
    floats_of3(h, s, -s * (8388608.0f + 43690.0f), q, std::make_integer_sequence<int, 32>{});
    inv_xform3_zy(q);
    float top = 0.0f, f[64];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      F2 a = q[2 * i], b = q[2 * i + 1];
      inv_lift1(a.x, a.y, b.x, b.y);
      top = max_abs3(top, a.x, a.y);
      top = max_abs3(top, b.x, b.y);
      f[4 * i] = a.x;
      f[4 * i + 1] = a.y;
      f[4 * i + 2] = b.x;
      f[4 * i + 3] = b.y;
    }
    const int room = 34 - planes < 15 + blk.lead ? 34 - planes : 15 + blk.lead;  // 2^(p + 18)
    if (warp_all(top <= u2f(((uint32_t)(unit + room - 1) << 23) | 0x7ff800u))) {
      sink(f);
      return kByFloats;
    }
    rest();
    return kByIntsAfterAll;
  }
  uint32_t u[64];
  if (second) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
      uint32_t b[4] = {w1[i], w0[i], first1[i], first0[i]};
      transpose_bytes4(b);
      const int j = 32 * (i >> 3) + (i & 7);
      u[j] = b[0];
      u[j + 8] = b[1];
      u[j + 16] = b[2];
      u[j + 24] = b[3];
    }
  } else if (WAY == kShortInts3 && most_planes <= 8) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int j = 32 * (i >> 3) + (i & 7);
      u[j] = byte_perm(w0[i], 0xaaaaaaaau, 0x0444);
      u[j + 8] = byte_perm(w0[i], 0xaaaaaaaau, 0x1444);
      u[j + 16] = byte_perm(w0[i], 0xaaaaaaaau, 0x2444);
      u[j + 24] = byte_perm(w0[i], 0xaaaaaaaau, 0x3444);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t a = byte_perm(w1[i], w0[i], 0x5140), b = byte_perm(w1[i], w0[i], 0x7362);
      const int j = 32 * (i >> 3) + (i & 7);
      u[j] = byte_perm(a, 0xaaaaaaaau, 0x1044);
      u[j + 8] = byte_perm(a, 0xaaaaaaaau, 0x3244);
      u[j + 16] = byte_perm(b, 0xaaaaaaaau, 0x1044);
      u[j + 24] = byte_perm(b, 0xaaaaaaaau, 0x3244);
    }
  }
  int v[64];
  ints_of3(u, blk.lead, v, std::make_integer_sequence<int, 64>{});
  inv_xform3(v);
  const float scale = dequant_scale(blk.e);
  float f[64];
#pragma unroll
  for (int i = 0; i < 64; i += 2) mul2(scale, (float)v[i], (float)v[i + 1], f[i], f[i + 1]);
  sink(f);
  return kByInts;
}

// ---- decoder: 2-D block -------------------------------------------------------------
// Sixteen planes of sixteen coefficients: byte b of w[i], b < 2, holds coefficient 8b + i in the first
// eight of them, byte 2 + b in the others; otherwise as decode_rows3.
template <class WordSrc, class Park>
CSW_HD void decode_chunk2(const WordSrc& src, Park& park, int maxbits, const uint32_t* dec_lut, uint32_t& m, Found& found,
                          int& left, uint32_t (&w)[8]) {
  const int nwords = (maxbits + 31) >> 5;
  uint32_t at = m;
  const int tests = decode_tests<16, CHUNK2>(src, park, maxbits, dec_lut, m, found);
  {
    const int rest = maxbits - mark_pos(m);
    left = tests + (rest > 0 ? (mark_n(m) == 16 ? (rest + 15) >> 4 : 1) : 0);
  }
  const int warp_tests = warp_max(tests), warp_left = warp_max(left);
  const uint32_t bits = funnel_l(found.hi, found.hi, mark_n(m));  // position p at bit p
  uint32_t mask = low_mask32(mark_n(at));
  uint32_t x[16];
#pragma unroll
  for (int j = 0; j < CHUNK2; j++) {
    x[j] = 0u;
    if (j < warp_left) {
      int i = mark_pos(at) >> 5;
      i = i < nwords ? i : nwords;
      x[j] = funnel_r(src.word(i), src.word(i + 1), (int)at);
      at += 16u;
      if (j < warp_tests) {
        if (j < tests) at = park.mark(j + 1);
        x[j] = (x[j] & mask) | (bits & ~mask);
        mask = low_mask32(mark_n(at));
        x[j] &= mask;
      }
    }
  }
  m = at;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const uint32_t both = byte_perm(x[j], x[8 + j], 0x5410);
    w[7 - j] = (j & 1) ? both : ~both;
  }
  transpose8(w);
}

constexpr int perm2_inverse(int p) {
  int i = 0;
  while (perm2(i) != p) i++;
  return i;
}
template <int P>
struct SequencyAt2 {
  static constexpr int v = perm2_inverse(P);
};
template <int... P>
CSW_HD void floats_of2(const float (&h)[16], float s, float t, F2 (&q)[8], std::integer_sequence<int, P...>) {
  ((q[P] = fma2(F2{h[SequencyAt2<2 * P>::v], h[SequencyAt2<2 * P + 1>::v]}, s, F2{t, t})), ...);
}
template <int... I>
CSW_HD void ints_of2(const uint32_t (&u)[16], int lead, uint32_t flip, int (&v)[16], std::integer_sequence<int, I...>) {
  ((v[PermAt<2, I>::v] = (int)(((u[I] >> lead) ^ flip) - 0xaaaaaaaau)), ...);
}

// As the 3-D blocks, with two passes: multiples of 2^(p - 4), so results below 2^(p + 20) are exact
// and p >= 10 is tried.  What does not fit is little work and done in integers at once.
template <class WordSrc, class Park>
CSW_HD void decode_block2(const WordSrc& src, Park& park, int maxbits, float (&f)[16], const uint32_t* dec_lut) {
  const BlockHead blk = block_head(src, maxbits);
  uint32_t w0[8], w1[8], m = (uint32_t)blk.start;
  Found found{0u, 0u};
  int planes, left;
  decode_chunk2(src, park, maxbits, dec_lut, m, found, left, w0);
  planes = left;
  const bool two = warp_any(left > CHUNK2);
  if (two) {
    decode_chunk2(src, park, maxbits, dec_lut, m, found, left, w1);
    if (left > 0) planes = CHUNK2 + left;
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) w1[i] = 0xaaaaaaaau;
  }
  if (warp_all(blk.e >= 40 && blk.e <= 225 && planes <= 24 && planes + blk.lead <= 22)) {
    const int unit = (int)blk.e - 14 - blk.lead;
    float h[16], s = u2f(((uint32_t)unit << 23) | ((uint32_t)blk.lead << 31)), offset = 8388608.0f + 43690.0f;
    if (!two) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        h[i] = u2f(byte_perm(w0[i], 0x4b000000u, 0x7602));  // 2^23 + it
        h[8 + i] = u2f(byte_perm(w0[i], 0x4b000000u, 0x7613));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        h[i] = (float)(byte_perm(w0[i], w1[i], 0x0024) & 0xffffffu);
        h[8 + i] = (float)(byte_perm(w0[i], w1[i], 0x1135) & 0xffffffu);
      }
      offset = 11184810.0f;
      s *= 0.00390625f;
    }
    F2 q[8];
    floats_of2(h, s, -s * offset, q, std::make_integer_sequence<int, 8>{});
    inv_lift2(q[0], q[2], q[4], q[6]);
    inv_lift2(q[1], q[3], q[5], q[7]);
    float top = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      F2 a = q[2 * i], b = q[2 * i + 1];
      inv_lift1(a.x, a.y, b.x, b.y);
      top = max_abs3(top, a.x, a.y);
      top = max_abs3(top, b.x, b.y);
      f[4 * i] = a.x;
      f[4 * i + 1] = a.y;
      f[4 * i + 2] = b.x;
      f[4 * i + 3] = b.y;
    }
    const int room = 36 - planes < 15 + blk.lead ? 36 - planes : 15 + blk.lead;  // 2^(p + 20), 2^31 in units of h
    if (warp_all(top <= u2f(((uint32_t)(unit + room - 1) << 23) | 0x7ff800u))) return;
  }
  uint32_t u[16];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    u[i] = byte_perm(w1[i], w0[i], 0x4602);
    u[8 + i] = byte_perm(w1[i], w0[i], 0x5713);
  }
  int v[16];
  ints_of2(u, blk.lead, (0xaaaaaaaau >> blk.lead) ^ 0xaaaaaaaau, v, std::make_integer_sequence<int, 16>{});
  inv_xform2(v);
  const float scale = dequant_scale(blk.e);
#pragma unroll
  for (int i = 0; i < 16; i++) f[i] = scale * (float)v[i];
}

#if !defined(__CUDACC__)
// For host tests: a block given as words, what follows the budget in the last one ignored.
constexpr int DEC3_BITS = DEC_BITS, DEC3_LUT_SIZE = DEC_LUT_SIZE;
inline uint32_t dec3_lut_entry(int i) { return dec_lut_entry(i); }
template <class Get>
struct CutWords {
  const Get& get;
  int maxbits;
  uint32_t word(int w) const { return 32 * w < maxbits ? get(w) & low_mask_sat(maxbits - 32 * w) : 0u; }
};
struct HostPark {
  uint32_t marks[PARK_SLOTS];
  void put_mark(int j, uint32_t m) { marks[j] = m; }
  uint32_t mark(int j) const { return marks[j]; }
};
// the 3-D decoder as the kernels call it
template <class WordSrc>
Taken3 decode_block3_host(const WordSrc& src, HostPark& slots, int maxbits, float (&f)[64], const uint32_t* dec_lut) {
  const Way3 way = decode3_way(maxbits);
  const auto sink = [&](const float (&v)[64]) {
    for (int i = 0; i < 64; i++) f[i] = v[i];
  };
  const auto rest = [&] { decode_block3<kInts3>(src, slots, maxbits, dec_lut, sink, [] {}); };
  return way == kFloats3 ? decode_block3<kFloats3>(src, slots, maxbits, dec_lut, sink, rest)
         : way == kInts3 ? decode_block3<kInts3>(src, slots, maxbits, dec_lut, sink, rest)
                         : decode_block3<kShortInts3>(src, slots, maxbits, dec_lut, sink, rest);
}
template <class WordSrc>
void decode_block3_pos(const WordSrc& src, int maxbits, float (&f)[64], const uint32_t* dec_lut) {
  const auto get = [&](int w) { return src.word(w); };
  CutWords<decltype(get)> cut{get, maxbits};
  HostPark slots;
  decode_block3_host(cut, slots, maxbits, f, dec_lut);
}
template <class WordSource>
void decode_block2(WordSource& src, int maxbits, float (&f)[16], const uint32_t* dec_lut) {
  const auto get = [&](int w) { return src.get(w); };
  CutWords<decltype(get)> cut{get, maxbits};
  HostPark slots;
  decode_block2(cut, slots, maxbits, f, dec_lut);
}
#endif

}  // namespace csw
