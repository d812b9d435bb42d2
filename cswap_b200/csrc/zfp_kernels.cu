// CUDA kernels of the fixed-rate ZFP float32 codec for sm_100a.
//
// Replaces cuZFP::cudaEncode / cudaDecode3 and their launchers
// (CSWAP+/zfp/encode3.cuh:49-186, decode3.cuh:42-178, encode1/2.cuh,
// decode1/2.cuh).  Two families:
//
//  * slab kernels for the swap path's view (nx = ny = 32, contiguous, whole
//    32-bit words per block): one CTA per group of 8 z-slabs (32 KiB, 128
//    blocks; fewer when the tensor is small), four (encoder) or up to six (decoder) CTAs per SM, lane = zfp block
//    held in registers.  A lane moves its block with sixteen 128-bit accesses
//    (eight neighbouring lanes cover one 128-byte row segment, so a warp
//    access touches four whole lines); stream words sit word-major in shared
//    memory (bank = lane, so diverged lanes never conflict) and each lane
//    reads or writes its own 128-bit pieces of the stream.  After the lookup
//    table is in place no warp waits for another.
//    Measured against a persistent variant that pulled each group with a bulk
//    async copy into a shared tile and wrote the stream through a transposing
//    copy-out: the extra shared-memory hop, its barriers and the registers of
//    the persistent loop cost 40 % at 256 MiB (177 against 125 us).  A second
//    persistent encoder, whose lanes fetched their next block with 16-byte
//    asynchronous copies into slots of their own while coding (no barrier),
//    took 168 us (32 KB more shared memory per CTA, 196 bytes of spills, and
//    the CTAs of an SM marching through the same phase together); asking L2
//    for the successor CTA's lines ahead of time cost 3 % in either kernel.
//  * generic kernels, one thread per block with the same coders and staging, for
//    any 1-D/2-D/3-D extents, strides, partial blocks and bit budgets.
//
// No kernel here waits on another CTA, a flag or a copy engine.
#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"
#include "pdl.cuh"
#include "zfp_field.cuh"
#include "zfp_kernels.h"

namespace csw {

namespace {

constexpr int kThreads = 128;                  // zfp blocks (lanes) per CTA
constexpr int kSlabFloats = 1024;              // one 32x32 z-slab
constexpr int kEncCtasPerSm = 4;                // 128 registers per thread: the encoder needs 113; five CTAs
                                                // spill, 256 MiB at 1024 bits 130.6 -> 146.9 us (before the queue was read ahead)
// 3-D decoders: 80 registers are nearly enough (12 bytes of spills in the floating point one); a CTA more hides more of the
// dependent shared-memory reads (256 MiB at 512 bits 91.7 us with five CTAs, 85.9 with six; at 1024 bits 125.6 and 123.4).
// Fields in their own extents need a few registers more and are seldom more than one wave: 31 x 33 x 4096 at 512 bits 11.1 us
// with five, 11.8 with six.
constexpr int kSlabDecCtasPerSm = 6, kDecCtasPerSm = 5;

// ---- word staging: word w of the block owned by thread t lives at [w * kThreads + t] --
// Staged stream words of the 2-D and 3-D decoders and the slots they park marks in: areas of the
// warp's own, again word-major.
struct WarpWords {
  const uint32_t* p;  // of this lane
  __device__ __forceinline__ uint32_t word(int w) const { return p[w * 32]; }
};
struct WarpPark {
  uint32_t* p;  // of this lane
  __device__ __forceinline__ void put_mark(int j, uint32_t m) { p[32 * j] = m; }
  __device__ __forceinline__ uint32_t mark(int j) const { return p[32 * j]; }
};
// words of a warp's areas together; store_rows3 takes 512 of them when the block is decoded
__host__ __device__ constexpr int warp_words(int nwords) { return 32 * (nwords + DEC_SPARE_ROWS + PARK_SLOTS); }

// Staged words and the per-lane expansion queue of the staged encoder, both
// word-major so that a warp's lanes always hit 32 different banks.
struct SmemStage {
  uint32_t* p;  // &stage[threadIdx.x]
  uint32_t* q;  // &queue[threadIdx.x]
  __device__ __forceinline__ void or_word(int w, uint32_t v) { atomicOr(p + w * kThreads, v); }
  __device__ __forceinline__ void q_put(int slot, int field, uint32_t v) {
    q[(slot * QUEUE_FIELDS + field) * kThreads] = v;
  }
  __device__ __forceinline__ uint32_t q_get(int slot, int field) const {
    return q[(slot * QUEUE_FIELDS + field) * kThreads];
  }
};

template <int SIZE>
__device__ __forceinline__ void copy_table(uint32_t* to, const uint32_t* from) {
  static_assert(SIZE % (4 * kThreads) == 0, "table copy assumes whole 128-bit rounds");
#pragma unroll
  for (int i = 0; i < SIZE / (4 * kThreads); i++)
    reinterpret_cast<uint4*>(to)[i * kThreads + threadIdx.x] =
        __ldg(reinterpret_cast<const uint4*>(from) + i * kThreads + threadIdx.x);
}
// The expansion tables, evaluated at compile time: a CTA copies its own to shared
// memory instead of computing the entries per launch.
struct EncTable {
  uint32_t v[ENC_LUT_SIZE];
};
constexpr EncTable make_enc_table() {
  EncTable t{};
  for (int i = 0; i < ENC_LUT_SIZE; i++) t.v[i] = enc_lut_entry((uint32_t)i);
  return t;
}
__device__ const EncTable g_enc_table = make_enc_table();
// 3-D: eleven positions a step where the table of eight takes one.  Steps are what the lanes
// of a warp differ in, so each one saved is saved by the warp: 256 MiB at 512 / 1024 bits
// 110.6 / 145.2 -> 104.7 / 136.3 us.  (Twelve positions do not fit an entry's 32 bits.)
struct alignas(16) Enc3Table {
  uint32_t v[ENC3_LUT_SIZE];
};
constexpr Enc3Table make_enc3_table() {
  Enc3Table t{};
  for (int i = 0; i < ENC3_LUT_SIZE; i++) t.v[i] = enc3_lut_entry((uint32_t)i);
  return t;
}
__device__ const Enc3Table g_enc3_table = make_enc3_table();

// Block of this thread: a warp takes 1 << lsh neighbouring blocks.  With lsh < 5 the lanes
// above do the work of the ones below a second time - the same data, so they cost
// nothing - and store nothing (blocks_per_warp says when).
__device__ __forceinline__ uint64_t block_of_thread(int lsh) {
  const uint64_t warp = (uint64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  return (warp << lsh) + (threadIdx.x & ((1u << lsh) - 1u));
}
__device__ __forceinline__ bool is_copy(int lsh) { return ((threadIdx.x & 31) >> lsh) != 0; }

// z-slab that feeds row z of a block with vz valid slabs (encode.cuh:17-38
// applied along z: a,a,a,a / a,b,b,a / a,b,c,a)
__device__ __forceinline__ int pad_src_z(int z, int vz) { return z < vz ? z : (z == 3 ? 0 : vz - 1); }

}  // namespace

// =====================================================================================
// slab encoder
// =====================================================================================
// One CTA per group of 8 z-slabs (128 blocks, lane = block; blocks_per_warp when the tensor is
// small).  A lane reads its
// 4x4x4 block with sixteen 128-bit loads (eight neighbouring lanes cover one
// 128-byte row segment, so a warp load touches four full lines), codes it into
// its own column of the word-major staging area and writes its own words out:
// after the table is built no warp waits for another.
// Bound by instructions issued (2558 a warp at 512 bits, ALU pipe 66 % busy).  256 MiB at 256 / 512 / 1024
// bits 82.0 / 104.0 / 135.8 -> 79.9 / 100.1 / 129.4 us with the expansions' bits in one word, a vote that holds
// their loop together, and the queue read one entry ahead.
__global__ void __launch_bounds__(kThreads, kEncCtasPerSm)
zfp_encode_slab_kernel(const float* __restrict__ in, uint32_t* __restrict__ out, uint32_t nz, int maxbits, int lsh,
                       const PipeConsts kc) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  const int nwords = maxbits >> 5;
  uint32_t* stage = smem_words;
  uint32_t* queue = stage + (nwords + STAGE_SPARE_ROWS) * kThreads;
  uint32_t* lut = queue + QUEUE_SLOTS * QUEUE_FIELDS * kThreads;

  const int tid = threadIdx.x;
  // my block: (bx, by) of the 8x8 grid of its tile of four slabs
  const uint32_t b = (uint32_t)block_of_thread(lsh);
  const int bx = b & 7, by = (b >> 3) & 7;
  const uint32_t zt = (b >> 6) * 4;  // first slab of my tile
  const int vz = zt >= nz ? 0 : (nz - zt < 4 ? (int)(nz - zt) : 4);
  copy_table<ENC3_LUT_SIZE>(lut, g_enc3_table.v);
  pdl_wait(in);
  float f[64];
  if (vz > 0) {
    const float* my = in + (size_t)zt * kSlabFloats + by * 128 + bx * 4;
#pragma unroll
    for (int z = 0; z < 4; z++) {
      const float* row = my + pad_src_z(z, vz) * kSlabFloats;
#pragma unroll
      for (int y = 0; y < 4; y++) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(row + y * 32));
        f[16 * z + 4 * y + 0] = v.x;
        f[16 * z + 4 * y + 1] = v.y;
        f[16 * z + 4 * y + 2] = v.z;
        f[16 * z + 4 * y + 3] = v.w;
      }
    }
  }
  for (int w = 0; w < nwords; w++) stage[w * kThreads + tid] = 0u;  // coded bits are OR-ed in
  __syncthreads();  // the table is complete
  if (vz == 0) return;

  SmemStage st{stage + tid, queue + tid};
  encode_block3_staged(f, maxbits, st, lut, kc);

  // a lane's words sit in its own column: no barrier before reading them back
  if (is_copy(lsh)) return;
  uint32_t* dst = out + (size_t)b * nwords;
  const uint32_t* col = stage + tid;
  if ((nwords & 3) == 0) {
    for (int w = 0; w < nwords; w += 4)
      *reinterpret_cast<uint4*>(dst + w) = make_uint4(col[w * kThreads], col[(w + 1) * kThreads],
                                                      col[(w + 2) * kThreads], col[(w + 3) * kThreads]);
  } else {
    for (int w = 0; w < nwords; w++) dst[w] = col[w * kThreads];
  }
}

// =====================================================================================
// slab decoder
// =====================================================================================
namespace {
// The parser table, evaluated at compile time: a CTA copies its own to shared memory with
// 128-bit loads instead of rebuilding the entries.
// Up to nine stream bits a step (8 KiB).  A step saved is worth less now that every lane takes its own: 256 MiB at
// 256 / 512 / 1024 bits with nine 83.9 / 94.4 / 125.0 us, with ten 83.6 / 94.2 / 128.4 (16 KiB leave a CTA less at 1024
// bits: 178 against 162 for normal values), with eight, six CTAs 83.6 / 93.1 / 125.4 against 82.3 / 92.4 / 124.4.
struct alignas(16) DecTable {
  uint32_t v[DEC_LUT_SIZE];
};
constexpr DecTable make_dec_table() {
  DecTable t{};
  for (int i = 0; i < DEC_LUT_SIZE; i++)
    if (i & ((2 << DEC_BITS) - 1)) t.v[i] = dec_lut_entry(i);
  return t;
}
__device__ const DecTable g_dec_table = make_dec_table();
}  // namespace

namespace {
// the staged words of this thread's lane behind the table, the slots behind the words
__device__ __forceinline__ uint32_t* decoder_column(int nwords) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  return smem_words + DEC_LUT_SIZE + (threadIdx.x >> 5) * warp_words(nwords) + (threadIdx.x & 31);
}
// eight neighbouring lanes cover one 128-byte row segment, so every store
// instruction of a warp writes four full lines: no staging of the output
__device__ __forceinline__ void store_slab_block(const float (&f)[64], float* out, uint32_t nz, uint32_t b) {
  const int bx = b & 7, by = (b >> 3) & 7;
  const uint32_t zt = (b >> 6) * 4;  // first slab of the block's tile
  const int vz = nz - zt < 4 ? (int)(nz - zt) : 4;
  float* dst = out + (size_t)zt * kSlabFloats + by * 128 + bx * 4;
#pragma unroll
  for (int z = 0; z < 4; z++)
    if (z < vz) {
#pragma unroll
      for (int y = 0; y < 4; y++)
        *reinterpret_cast<float4*>(dst + z * kSlabFloats + y * 32) =
            make_float4(f[16 * z + 4 * y], f[16 * z + 4 * y + 1], f[16 * z + 4 * y + 2], f[16 * z + 4 * y + 3]);
    }
}
template <Way3 WAY>
__device__ __forceinline__ void decode_slab_block(float* out, uint32_t nz, int maxbits, int lsh);
// a block whose results the floating point decoder could not vouch for, from the start
__device__ __noinline__ void decode_slab_again(float* out, uint32_t nz, int maxbits, int lsh) {
  decode_slab_block<kInts3>(out, nz, maxbits, lsh);
}
template <Way3 WAY>
__device__ __forceinline__ void decode_slab_block(float* out, uint32_t nz, int maxbits, int lsh) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  const int nwords = maxbits >> 5;
  uint32_t* col = decoder_column(nwords);
  WarpWords source{col};
  WarpPark park{col + 32 * (nwords + DEC_SPARE_ROWS)};
  decode_block3<WAY>(
      source, park, maxbits, smem_words,
      [&](const float (&f)[64]) {
        if (!is_copy(lsh)) store_slab_block(f, out, nz, (uint32_t)block_of_thread(lsh));
      },
      [&] { decode_slab_again(out, nz, maxbits, lsh); });
}
}  // namespace

// One CTA per group of 8 z-slabs, lane = block, mirror image of the encoder: a
// lane pulls its own compressed words into its column of the word-major staging
// area, parses them by bit position and stores the rebuilt 4x4x4 block with
// sixteen 128-bit stores.  The only barrier is the one after the table copy.
// WAY: decode3_way(maxbits).
// Bound by instructions issued (1895 a warp at 512 bits, ALU pipe 57 % busy); loads and stores alone take 52 of the 86 us.  Against a
// decoder that goes plane by plane with the slowest lane and lifts in integers, 256 MiB at 256 / 512 / 1024 bits:
//   tanh of normal values                 95.7 / 122.5 / 158.3 ->  75.2 /  86.1 / 122.3 us
//   normal values + 10                   117.9 / 133.6 / 167.0 ->  93.2 / 102.3 / 139.0
//   sines over the field with 3 % noise  129.0 / 148.0 / 179.9 ->  98.7 / 108.0 / 144.1
//   sines alone                          141.6 / 177.5 / 213.6 -> 136.8 / 164.9 / 187.7
template <Way3 WAY>
__global__ void __launch_bounds__(kThreads, kSlabDecCtasPerSm)
zfp_decode_slab_kernel(const uint32_t* __restrict__ in, float* __restrict__ out, uint32_t nz, int maxbits, int lsh) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  const int nwords = maxbits >> 5;
  const uint32_t b = (uint32_t)block_of_thread(lsh);
  const uint32_t zt = (b >> 6) * 4;  // first slab of my tile
  uint32_t* col = decoder_column(nwords);
  copy_table<DEC_LUT_SIZE>(smem_words, g_dec_table.v);
  pdl_wait(in);
  if (zt < nz) {
    const uint32_t* src = in + (size_t)b * nwords;
    if ((nwords & 3) == 0) {
      for (int w = 0; w < nwords; w += 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + w));
        col[w * 32] = v.x;
        col[(w + 1) * 32] = v.y;
        col[(w + 2) * 32] = v.z;
        col[(w + 3) * 32] = v.w;
      }
    } else {
      for (int w = 0; w < nwords; w++) col[w * 32] = __ldg(src + w);
    }
  }
#pragma unroll
  for (int w = 0; w < DEC_SPARE_ROWS; w++) col[(nwords + w) * 32] = 0u;
  __syncthreads();  // the table is complete
  if (zt >= nz) return;

  decode_slab_block<WAY>(out, nz, maxbits, lsh);
}

// =====================================================================================
// generic kernels: one thread per block, any extents, strides and budgets
// =====================================================================================
// The same coders and the same word-major staging as the slab kernels; what differs
// is how a lane finds its block and, for budgets that are not whole words, how the
// stream is put together: 128 blocks of any budget are a whole number of words, so a
// CTA's part of the stream is its own and is assembled from the staged columns -
// no atomics, no zeroed stream.  (One thread per block reading and writing global
// memory word by word, with plane-by-plane coders whose lanes wait for each other,
// took 28.7 + 33.4 us a call for 31 x 33 x 4096 at 512 bits and 22.6 + 26.7 us for
// 768 x 4096 at 128; these take 11.8 + 10.7 and 11.9 + 10.3.  They are bound as the
// slab kernels are, by the number of instructions a block costs.)
namespace {

// Where a block lies and how much of it: offsets of its four positions along an
// axis, with the replicate padding of partial blocks (encode.cuh:17-38) folded in.
__device__ __forceinline__ int pad_src(int i, int valid) { return i < valid ? i : (i == 3 ? 0 : valid - 1); }

template <int DIMS>
struct BlockAt {
  int64_t base;
  int vx, vy, vz;
  __device__ __forceinline__ BlockAt(const FieldGeom& g, uint64_t b) {
    uint32_t x, y = 0, z = 0;
    if (DIMS == 1) {
      x = (uint32_t)b;
    } else if (b <= 0xffffffffu) {
      const uint32_t i = (uint32_t)b, r = i / g.bx;
      x = i - r * g.bx;
      z = DIMS == 3 ? r / g.by : 0u;
      y = r - z * (DIMS == 3 ? g.by : 0u);
    } else {
      const uint64_t r = b / g.bx;
      x = (uint32_t)(b - r * g.bx);
      z = DIMS == 3 ? (uint32_t)(r / g.by) : 0u;
      y = (uint32_t)(r - (uint64_t)z * (DIMS == 3 ? g.by : 0u));
    }
    x *= 4; y *= 4; z *= 4;
    vx = g.nx - x < 4 ? (int)(g.nx - x) : 4;
    vy = DIMS >= 2 && g.ny - y < 4 ? (int)(g.ny - y) : 4;
    vz = DIMS >= 3 && g.nz - z < 4 ? (int)(g.nz - z) : 4;
    base = (int64_t)x * g.sx + (int64_t)y * g.sy + (int64_t)z * g.sz;
  }
};

// `vec`: rows of four values that start on a 16-byte boundary (decided for the whole field)
template <int DIMS>
__device__ __forceinline__ void load_block(const FieldGeom& g, const float* in, bool vec, const BlockAt<DIMS>& at,
                                           float (&f)[1 << (2 * DIMS)]) {
  const float* p = in + at.base;
  if (vec && at.vx == 4) {
#pragma unroll
    for (int r = 0; r < (1 << (2 * DIMS)) / 4; r++) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p + (DIMS >= 2 ? pad_src(r & 3, at.vy) * g.sy : 0) +
                                                             (DIMS >= 3 ? pad_src(r >> 2, at.vz) * g.sz : 0)));
      f[4 * r] = v.x;
      f[4 * r + 1] = v.y;
      f[4 * r + 2] = v.z;
      f[4 * r + 3] = v.w;
    }
  } else {
    int64_t ox[4];
#pragma unroll
    for (int x = 0; x < 4; x++) ox[x] = pad_src(x, at.vx) * g.sx;
#pragma unroll
    for (int r = 0; r < (1 << (2 * DIMS)) / 4; r++) {
      const float* row = p + (DIMS >= 2 ? pad_src(r & 3, at.vy) * g.sy : 0) + (DIMS >= 3 ? pad_src(r >> 2, at.vz) * g.sz : 0);
#pragma unroll
      for (int x = 0; x < 4; x++) f[4 * r + x] = __ldg(row + ox[x]);
    }
  }
}
template <int DIMS>
__device__ __forceinline__ void store_block(const FieldGeom& g, float* out, bool vec, const BlockAt<DIMS>& at,
                                            const float (&f)[1 << (2 * DIMS)]) {
  float* p = out + at.base;
#pragma unroll
  for (int r = 0; r < (1 << (2 * DIMS)) / 4; r++) {
    if ((DIMS < 2 || (r & 3) < at.vy) && (DIMS < 3 || (r >> 2) < at.vz)) {
      float* row = p + (DIMS >= 2 ? (r & 3) * g.sy : 0) + (DIMS >= 3 ? (r >> 2) * g.sz : 0);
      if (vec && at.vx == 4) {
        *reinterpret_cast<float4*>(row) = make_float4(f[4 * r], f[4 * r + 1], f[4 * r + 2], f[4 * r + 3]);
      } else {
#pragma unroll
        for (int x = 0; x < 4; x++)
          if (x < at.vx) row[x * g.sx] = f[4 * r + x];
      }
    }
  }
}

// 3-D blocks whose rows do not start on 16-byte boundaries, x contiguous: the rows of a
// warp's 32 blocks go through shared memory so that a store instruction writes 32
// neighbouring values (lanes storing their own values one by one write 4 of every
// 16 bytes: four times the write transactions; 31 x 33 x 4096 at 512 bits 17.9 -> 14.3
// us, 7 x 7 x 65536 21.1 -> 13.5).  `buf`: 512 words of the warp's own;
// every lane of the warp calls.
__device__ __forceinline__ void store_rows3(const FieldGeom& g, float* out, const BlockAt<3>& at, bool valid, float* buf,
                                            const float (&f)[64]) {
  const int lane = threadIdx.x & 31, x = lane & 3;
  const int have = valid ? at.vx | at.vy << 4 | at.vz << 8 : 0;
  float* dst[4];
  int vy[4], vz[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {  // pass q stores value x of block 8q + lane / 4
    const int src = 8 * q + (lane >> 2), h = __shfl_sync(0xffffffffu, have, src);
    dst[q] = out + __shfl_sync(0xffffffffu, at.base, src) + x;
    vy[q] = x < (h & 15) ? h >> 4 & 15 : 0;
    vz[q] = h >> 8;
  }
#pragma unroll
  for (int z = 0; z < 4; z++) {
#pragma unroll
    for (int y = 0; y < 4; y++)
      *reinterpret_cast<float4*>(buf + 128 * y + 4 * lane) =
          make_float4(f[16 * z + 4 * y], f[16 * z + 4 * y + 1], f[16 * z + 4 * y + 2], f[16 * z + 4 * y + 3]);
    __syncwarp();
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (y < vy[q] && z < vz[q]) dst[q][y * g.sy + z * g.sz] = buf[128 * y + 32 * q + lane];
    __syncwarp();
  }
}

// Tables of the 1-D coders.  A plane of four values is one entry, and one bit transpose serves
// all 32 planes: 4 Mi values at 32 bits 26.8 + 37.2 -> 18.9 + 23.9 us against the step tables of
// the larger blocks and a transpose for every eight planes.
struct Enc1Table {
  uint32_t v[ENC1_LUT_SIZE];
};
constexpr Enc1Table make_enc1_table() {
  Enc1Table t{};
  for (int i = 0; i < ENC1_LUT_SIZE; i++) t.v[i] = enc1_lut_entry(i);
  return t;
}
__device__ const Enc1Table g_enc1_table = make_enc1_table();
struct alignas(16) Dec1Table {
  uint16_t v[DEC1_LUT_SIZE];
};
constexpr Dec1Table make_dec1_table() {
  Dec1Table t{};
  for (int i = 0; i < DEC1_LUT_SIZE; i++) t.v[i] = dec1_lut_entry(i);
  return t;
}
__device__ const Dec1Table g_dec1_table = make_dec1_table();

// a lane's column of the staging area as a word sink / source of the small-block coders
struct ColumnSink {
  uint32_t* p;
  __device__ __forceinline__ void put(int w, uint32_t v) { p[w * kThreads] = v; }
};
struct ColumnSource {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t get(int w) const { return p[w * kThreads]; }
};

template <int DIMS>
__global__ void __launch_bounds__(kThreads, DIMS == 3 ? kEncCtasPerSm : 8)
zfp_encode_generic_kernel(const FieldGeom g, const float* __restrict__ in, bool vec, uint32_t* __restrict__ out,
                          int maxbits, uint64_t nblocks, uint64_t total_words, int lsh, const PipeConsts kc) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  const int nwords = (maxbits + 31) >> 5, tid = threadIdx.x;
  uint32_t* stage = smem_words;
  uint32_t* queue = stage + (nwords + STAGE_SPARE_ROWS) * kThreads;
  uint32_t* lut = queue + (DIMS == 3 ? QUEUE_SLOTS * QUEUE_FIELDS * kThreads : 0);
  static_assert(ENC1_LUT_SIZE <= kThreads && ENC_LUT_SIZE == 2 * kThreads, "one or two table words per thread");
  uint32_t lut0 = 0, lut1 = 0;
  if (DIMS == 1) {
    if (tid < ENC1_LUT_SIZE) lut0 = __ldg(g_enc1_table.v + tid);
  } else if (DIMS == 2) {
    lut0 = __ldg(g_enc_table.v + tid);
    lut1 = __ldg(g_enc_table.v + kThreads + tid);
  } else {
    copy_table<ENC3_LUT_SIZE>(lut, g_enc3_table.v);
  }
  const uint32_t per_cta = (kThreads / 32) << lsh;
  const uint64_t b0 = (uint64_t)blockIdx.x * per_cta, b = block_of_thread(lsh);
  pdl_wait(in);
  float f[1 << (2 * DIMS)];
  if (b < nblocks) load_block<DIMS>(g, in, vec, BlockAt<DIMS>(g, b), f);
  if (DIMS < 3) lut[tid] = lut0;
  if (DIMS == 2) lut[kThreads + tid] = lut1;
  uint32_t* col = stage + tid;
  if (DIMS == 3) {
    for (int w = 0; w < nwords; w++) col[w * kThreads] = 0u;  // coded bits are OR-ed in
  }
  __syncthreads();  // the table is complete
  if constexpr (DIMS == 3) {
    if (b >= nblocks) {
#pragma unroll
      for (int i = 0; i < 64; i++) f[i] = 0.0f;
    }
    SmemStage st{col, queue + tid};
    encode_block3_staged(f, maxbits, st, lut, kc);
  } else {
    if (b < nblocks) {
      ColumnSink sink{col};
      if constexpr (DIMS == 2) encode_block2(f, maxbits, sink, lut);
      else encode_block1(f, maxbits, sink, lut);
    }
  }
  if ((maxbits & 31) == 0) {  // whole words per block: every lane writes its own
    if (b < nblocks && !is_copy(lsh)) {
      uint32_t* dst = out + b * nwords;
      if ((nwords & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        for (int w = 0; w < nwords; w += 4)
          *reinterpret_cast<uint4*>(dst + w) = make_uint4(col[w * kThreads], col[(w + 1) * kThreads],
                                                          col[(w + 2) * kThreads], col[(w + 3) * kThreads]);
      } else {
        for (int w = 0; w < nwords; w++) dst[w] = col[w * kThreads];
      }
      // the stream is whole 64-bit words: the last 32 bits may belong to no block
      if (b == nblocks - 1 && nblocks * nwords < total_words) dst[nwords] = 0u;
    }
    return;
  }
  __syncthreads();  // every column is complete
  const uint64_t first = b0 * (uint64_t)maxbits >> 5;  // of this CTA's words; b0 * maxbits is a multiple of 32
  const int here = nblocks - b0 < per_cta ? (int)(nblocks - b0) : (int)per_cta;
  const uint64_t left = total_words - first;
  const int mine = nblocks - b0 <= per_cta ? (int)left : (int)(per_cta / 32) * maxbits;  // the last CTA: to the end
  for (int w = tid; w < mine; w += kThreads) {
    uint32_t v = 0;
    int blk = 32 * w / maxbits, off = 32 * w - blk * maxbits;
    for (int have = 0; have < 32 && blk < here; blk++, off = 0) {
      const int owner = (blk >> lsh) * 32 + (blk & ((1 << lsh) - 1));  // its first thread
      const uint32_t* c = stage + owner + (off >> 5) * kThreads;       // the row behind the last one exists
      const int take = maxbits - off < 32 - have ? maxbits - off : 32 - have;
      v |= (funnel_r(c[0], c[kThreads], off) & low_mask32(take)) << have;
      have += take;
    }
    out[first + w] = v;
  }
}

// a decoded 3-D block, every lane of the warp calls
__device__ __forceinline__ void store_field_block(const FieldGeom& g, float* out, bool vec, uint64_t b, uint64_t nblocks,
                                                  int nwords, int lsh, const float (&f)[64]) {
  const BlockAt<3> at(g, b < nblocks ? b : nblocks - 1);
  const bool valid = b < nblocks && !is_copy(lsh);
  if (!vec && g.sx == 1) {
    __syncwarp();  // every lane is done with its words
    store_rows3(g, out, at, valid, reinterpret_cast<float*>(decoder_column(nwords) - (threadIdx.x & 31)), f);
  } else if (valid) {
    store_block<3>(g, out, vec, at, f);
  }
}
template <Way3 WAY>
__device__ __forceinline__ void decode_field_block(const FieldGeom& g, float* out, bool vec, uint64_t nblocks, int maxbits,
                                                   int lsh);
// the geometry by value: a reference would put it, and the kernel's arguments, on the stack of every call (0.3 us of 6)
__device__ __noinline__ void decode_field_again(const FieldGeom g, float* out, bool vec, uint64_t nblocks, int maxbits,
                                                int lsh) {
  decode_field_block<kInts3>(g, out, vec, nblocks, maxbits, lsh);
}
template <Way3 WAY>
__device__ __forceinline__ void decode_field_block(const FieldGeom& g, float* out, bool vec, uint64_t nblocks, int maxbits,
                                                   int lsh) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  const int nwords = (maxbits + 31) >> 5;
  uint32_t* col = decoder_column(nwords);
  WarpWords source{col};
  WarpPark park{col + 32 * (nwords + DEC_SPARE_ROWS)};
  decode_block3<WAY>(
      source, park, maxbits, smem_words,
      [&](const float (&f)[64]) { store_field_block(g, out, vec, block_of_thread(lsh), nblocks, nwords, lsh, f); },
      [&] { decode_field_again(g, out, vec, nblocks, maxbits, lsh); });
}

// WAY: of 3-D blocks, decode3_way(maxbits)
// 2-D: 768 x 4096 at 64 / 128 / 256 bits 11.0 / 13.8 / 16.6 -> 9.4 / 10.7 / 13.7 us with the lanes at their own pace through
// the group tests, sixteen planes a transpose and the transform in exact float32; 4096 x 4096 48.2 / 63.5 / 79.5 -> 37.3 /
// 43.0 / 53.7 (and one round of blocks a CTA), smooth values at 128 bits 92.6 -> 81.1.
template <int DIMS, Way3 WAY>
__global__ void __launch_bounds__(kThreads, DIMS == 3 ? kDecCtasPerSm : 8)
zfp_decode_generic_kernel(const FieldGeom g, const uint32_t* __restrict__ in, float* __restrict__ out, bool vec,
                          int maxbits, uint64_t nblocks, uint64_t total_words, int lsh) {
  extern __shared__ __align__(16) uint32_t smem_words[];
  const int nwords = (maxbits + 31) >> 5, tid = threadIdx.x;
  constexpr int kRow = DIMS > 1 ? 32 : kThreads;  // a staged word to the next one of the same lane
  constexpr int kSpare = DIMS > 1 ? DEC_SPARE_ROWS : STAGE_SPARE_ROWS;
  uint32_t* lut = smem_words;
  uint32_t* col;
  if (DIMS == 1) {
    for (int i = tid; i < DEC1_LUT_SIZE / 8; i += kThreads)
      reinterpret_cast<uint4*>(lut)[i] = __ldg(reinterpret_cast<const uint4*>(g_dec1_table.v) + i);
    col = lut + DEC1_LUT_SIZE / 2 + tid;
  } else {
    copy_table<DEC_LUT_SIZE>(lut, g_dec_table.v);
    col = decoder_column(nwords);
  }
  // reads just past a block find zeros and need no bounds test
#pragma unroll
  for (int w = 0; w < kSpare; w++) col[(nwords + w) * kRow] = 0u;
  __syncthreads();  // the table is complete
  pdl_wait(in);
  // whole warps go round: the decoders of the larger blocks vote
  const uint64_t mine = block_of_thread(lsh), my_lane = tid & ((1u << lsh) - 1u);
  for (uint64_t wb = mine - my_lane; wb < nblocks; wb += (uint64_t)gridDim.x * kThreads) {
    const uint64_t b = wb + my_lane, bit0 = b * (uint64_t)maxbits, w0 = bit0 >> 5;
    const int s = (int)(bit0 & 31);
    if (b >= nblocks) {
      col[0] = 0u;  // an empty block, not stored
      col[(nwords - 1) * kRow] = 0u;
    } else if ((maxbits & 127) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
      for (int w = 0; w < nwords; w += 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(in + w0 + w));
        col[w * kRow] = v.x;
        col[(w + 1) * kRow] = v.y;
        col[(w + 2) * kRow] = v.z;
        col[(w + 3) * kRow] = v.w;
      }
    } else {
      uint32_t lo = __ldg(in + w0);
      for (int w = 0; w < nwords; w++) {
        const uint32_t hi = w0 + w + 1 < total_words ? __ldg(in + w0 + w + 1) : 0u;
        col[w * kRow] = funnel_r(lo, hi, s);
        lo = hi;
      }
      if (DIMS > 1) col[(nwords - 1) * kRow] &= low_mask32(maxbits - 32 * (nwords - 1));
    }
    float f[1 << (2 * DIMS)];
    if constexpr (DIMS == 3) {
      decode_field_block<WAY>(g, out, vec, nblocks, maxbits, lsh);
      return;  // the launcher gives a 3-D field a warp for every group of blocks
    } else {
      if constexpr (DIMS == 2) {
        WarpWords source{col};
        WarpPark park{col + 32 * (nwords + DEC_SPARE_ROWS)};
        decode_block2(source, park, maxbits, f, lut);
      } else {
        ColumnSource source{col};
        decode_block1(source, maxbits, f, reinterpret_cast<const uint16_t*>(lut));
      }
      if (b < nblocks && !is_copy(lsh)) store_block<DIMS>(g, out, vec, BlockAt<DIMS>(g, b), f);
    }
  }
}

// rows of four values start on 16-byte boundaries
bool vector_rows(const FieldGeom& g, const void* field) {
  return g.sx == 1 && (g.dims < 2 || g.sy % 4 == 0) && (g.dims < 3 || g.sz % 4 == 0) &&
         (reinterpret_cast<uintptr_t>(field) & 15) == 0;
}

}  // namespace

// =====================================================================================
// launchers
// =====================================================================================
constexpr size_t kDefaultDynamicSmem = 40 * 1024;  // asked for without opting in (48 KiB, static memory included, are allowed)
constexpr uint64_t kSchedulersPerSm = 4;
constexpr int kWholeChip = 148;                    // SMs
constexpr int kMostBits = 4096;                    // largest budget the library accepts
static size_t staged_smem_bytes(int maxbits, bool decode, int dims) {
  const size_t rows = ((size_t)maxbits + 31) / 32 + STAGE_SPARE_ROWS;
  if (decode && dims == 1) return rows * kThreads * 4 + DEC1_LUT_SIZE * 2;
  if (decode) return (DEC_LUT_SIZE + kThreads / 32 * (size_t)warp_words((maxbits + 31) / 32)) * 4;
  return (rows + (dims == 3 ? QUEUE_SLOTS * QUEUE_FIELDS : 0)) * kThreads * 4 + (dims == 3 ? ENC3_LUT_SIZE : ENC_LUT_SIZE) * 4;
}
// Only the largest budgets need it; the call costs host time on every launch.
template <class K>
static cudaError_t allow_smem(K* kernel, size_t smem, bool decode, int dims) {
  if (smem <= kDefaultDynamicSmem) return cudaSuccess;
  return taken(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)staged_smem_bytes(kMostBits, decode, dims)));
}

static uint64_t slab_blocks(const FieldGeom& g) { return ((uint64_t)g.nz + 3) / 4 * 64; }
// log2 of the blocks a warp takes.  While every scheduler of the device has at most one
// warp, a call lasts as long as one warp does, and a warp takes the steps of the one of its
// blocks with the most group tests: the fewer blocks, the shorter.  So blocks are spread until there
// is a warp for each of the schedulers, 4 x 148.  64 KiB at 512 bits 4.70 -> 4.39 us (encode) and 4.56 -> 4.26
// (decode), at 1024 bits 5.65 -> 4.95 and 6.33 -> 5.17; 1 MiB at 1024 bits 5.88 -> 5.42 and 6.42 -> 6.47, the decoder's
// tests being no longer most of its time there.  From two warps a scheduler on the copies cost
// more issue slots than they save: 1 MiB at 512 bits with 4 blocks a warp in place of 8 4.67 -> 6.03 and 4.92 -> 5.49, 4 MiB
// with 16 in place of 32 5.05 -> 6.28 and 5.00 -> 5.80.
static int blocks_per_warp(uint64_t nblocks) {
  const uint64_t schedulers = kSchedulersPerSm * (unsigned)sm_count();
  int lsh = 0;
  while (lsh < 5 && (nblocks >> lsh) > schedulers) lsh++;
  return lsh;
}
static unsigned ctas_of(uint64_t nblocks, int lsh) {
  const uint64_t per = (uint64_t)(kThreads / 32) << lsh;
  return (unsigned)((nblocks + per - 1) / per);
}

bool zfp_slab_eligible(const FieldGeom& g, const void* field, const void* stream, int maxbits) {
  return g.dims == 3 && g.nx == 32 && g.ny == 32 && g.sx == 1 && g.sy == 32 && g.sz == 1024 && (maxbits & 31) == 0 &&
         maxbits >= 32 && maxbits <= 2048 && (reinterpret_cast<uintptr_t>(field) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(stream) & 15) == 0;
}

template <int DIMS>
static cudaError_t encode_generic(const FieldGeom& g, const float* in, uint32_t* out, int maxbits, uint64_t nblocks,
                                  cudaStream_t stream) {
  const size_t smem = staged_smem_bytes(maxbits, false, DIMS);
  cudaError_t e = allow_smem(zfp_encode_generic_kernel<DIMS>, smem, false, DIMS);
  if (e != cudaSuccess) return e;
  int lsh = DIMS == 3 ? blocks_per_warp(nblocks) : 5;
  if (maxbits % 32 && lsh < 3) lsh = 3;  // a CTA puts whole words together: 32 blocks at least
  return pdl_launch(zfp_encode_generic_kernel<DIMS>, ctas_of(nblocks, lsh), kThreads, smem, stream, g, in,
                    vector_rows(g, in), out, maxbits, nblocks, (uint64_t)stream_bytes(g, (unsigned)maxbits) / 4, lsh,
                    pipe_consts());
}
template <int DIMS, Way3 WAY>
static cudaError_t decode_generic(const FieldGeom& g, const uint32_t* in, float* out, int maxbits, uint64_t nblocks,
                                  cudaStream_t stream) {
  const size_t smem = staged_smem_bytes(maxbits, true, DIMS);
  cudaError_t e = allow_smem(zfp_decode_generic_kernel<DIMS, WAY>, smem, true, DIMS);
  if (e != cudaSuccess) return e;
  const int lsh = DIMS == 3 ? blocks_per_warp(nblocks) : 5;
  const uint64_t ctas = ctas_of(nblocks, lsh);
  // 128 1-D blocks are 2 KiB of field, and a CTA begins with a table of 2.5: once every SM has its eight CTAs twice
  // over, a CTA takes up to eight rounds of blocks.  With and without rounds, at 32 bits: 64 Mi values 275 / 298 us, 16 Mi
  // 73.9 / 75.8, but 4 Mi 23.3 / 20.7.  2-D fields (8 KiB a CTA) are better off without at every size: 4096 x 4096 at
  // 64 / 128 / 256 bits 43.0 / 49.0 / 62.4 us with rounds and 37.3 / 43.0 / 53.7 without, 8192 x 8192 at 128 bits 165 and 163.
  // That is a whole chip; a part of one, where it could not be measured, goes round as in 1-D.
  const uint64_t full = 8 * (uint64_t)sm_count();
  const bool once = DIMS == 3 || (DIMS == 2 && sm_count() >= kWholeChip);
  const uint64_t rounds = once || ctas < 2 * full ? 1 : ctas / full < 8 ? ctas / full : 8;
  return pdl_launch(zfp_decode_generic_kernel<DIMS, WAY>, (unsigned)((ctas + rounds - 1) / rounds), kThreads, smem, stream,
                    g, in, out, vector_rows(g, out), maxbits, nblocks, (uint64_t)stream_bytes(g, (unsigned)maxbits) / 4, lsh);
}

cudaError_t zfp_encode_launch(const FieldGeom& g, const float* in, void* out, int maxbits, cudaStream_t stream) {
  const uint64_t nblocks = geom_blocks(g);
  if (nblocks == 0) return cudaSuccess;
  uint32_t* o = reinterpret_cast<uint32_t*>(out);
  if (zfp_slab_eligible(g, in, out, maxbits)) {
    const size_t smem = staged_smem_bytes(maxbits, false, 3);
    cudaError_t e = allow_smem(zfp_encode_slab_kernel, smem, false, 3);
    if (e != cudaSuccess) return e;
    const uint64_t blocks = slab_blocks(g);
    const int lsh = blocks_per_warp(blocks);
    return pdl_launch(zfp_encode_slab_kernel, ctas_of(blocks, lsh), kThreads, smem, stream, in, o, g.nz, maxbits, lsh,
                      pipe_consts());
  }
  return g.dims == 3   ? encode_generic<3>(g, in, o, maxbits, nblocks, stream)
         : g.dims == 2 ? encode_generic<2>(g, in, o, maxbits, nblocks, stream)
                       : encode_generic<1>(g, in, o, maxbits, nblocks, stream);
}

template <Way3 WAY>
static cudaError_t decode_slabs(const FieldGeom& g, const uint32_t* in, float* out, int maxbits, cudaStream_t stream) {
  const size_t smem = staged_smem_bytes(maxbits, true, 3);
  cudaError_t e = allow_smem(zfp_decode_slab_kernel<WAY>, smem, true, 3);
  if (e != cudaSuccess) return e;
  const uint64_t blocks = slab_blocks(g);
  const int lsh = blocks_per_warp(blocks);
  return pdl_launch(zfp_decode_slab_kernel<WAY>, ctas_of(blocks, lsh), kThreads, smem, stream, in, out, g.nz, maxbits,
                    lsh);
}

cudaError_t zfp_decode_launch(const FieldGeom& g, const void* in, float* out, int maxbits, cudaStream_t stream) {
  const uint64_t nblocks = geom_blocks(g);
  if (nblocks == 0) return cudaSuccess;
  const uint32_t* i32 = reinterpret_cast<const uint32_t*>(in);
  const Way3 way = decode3_way(maxbits);
  if (zfp_slab_eligible(g, out, in, maxbits))
    return way == kFloats3 ? decode_slabs<kFloats3>(g, i32, out, maxbits, stream)
           : way == kInts3 ? decode_slabs<kInts3>(g, i32, out, maxbits, stream)
                           : decode_slabs<kShortInts3>(g, i32, out, maxbits, stream);
  if (g.dims == 3)
    return way == kFloats3 ? decode_generic<3, kFloats3>(g, i32, out, maxbits, nblocks, stream)
           : way == kInts3 ? decode_generic<3, kInts3>(g, i32, out, maxbits, nblocks, stream)
                           : decode_generic<3, kShortInts3>(g, i32, out, maxbits, nblocks, stream);
  return g.dims == 2 ? decode_generic<2, kInts3>(g, i32, out, maxbits, nblocks, stream)
                     : decode_generic<1, kInts3>(g, i32, out, maxbits, nblocks, stream);
}

}  // namespace csw
