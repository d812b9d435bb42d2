// CUDA kernels of the zero-value ("ZVC") sparse codec for sm_100a.
//
// Replaces PreGPUcompression / PreAcc / GPUcompression / GPUdecompression of
// CSWAP+/zfp/compression.cu:9-19,134-318.  The reference gives each of 16384
// threads a contiguous chunk (stride-`chunk` loads, a one-thread serial scan
// and a blocking 4-byte copy to size the output).  Here:
//
//  native format  - bitmap[ceil(n/32)] in element order built by warp ballots
//                   from coalesced loads, values[nnz] in element order, and an
//                   exclusive per-tile (4096 elements) offset table so that
//                   decompression is independent per tile.  A value is kept
//                   when its BIT PATTERN is non-zero, so -0.0 and NaN payloads
//                   round-trip exactly.
//  count -> scan -> pack, three launches, no inter-CTA waiting; the total is
//                   written to a caller-supplied word (device or mapped host).
//                   16 MiB at 50 % zeros: 16.4 -> 9.2 us a call back to back
//                   (programmatic launches; bitmap out of the counting pass).
//  single pass    - same bitmap and per-tile contents from one read of the
//                   tensor; tiles claim their segments with an atomic add, so
//                   segment order follows the schedule, not the element order.
//                   16 MiB: 8.2 -> 6.3 us, 256 MiB: 65.8 -> 62.7 us.
//  small tensors  - one cluster, one launch: up to 1 MiB in place of the three
//                   launches (12.3 -> 2.4 ... 4.4 us back to back, which is what
//                   launching costs), up to 512 KiB in place of the single pass
//                   (7.5 -> 2.4 ... 3.1; its launcher says why no further).
//  legacy format  - the reference's `begin | bitmap | values` layout with its
//                   P-worker chunking, one warp per worker, behind the
//                   reference's own entry-point names.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "pdl.cuh"
#include "sparse_kernels.h"
#include "tile_counts.cuh"

namespace csw {

namespace {

constexpr int kTile = SPARSE_TILE;        // elements per tile
constexpr int kThreads = 256;             // 8 warps, 512 elements (16 bitmap words) each
constexpr int kCountThreads = 128;         // 1024 elements per warp, eight 128-bit loads per lane
constexpr int kWordsPerWarp = kTile / 32 / (kThreads / 32);  // 16

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ---- ordered compression, pass 1: per-tile counts -------------------------------------
// A pure read of the tensor.  Bitmap and values are written by pass 3, which reads
// the tensor again (from L2 where it fits).
__global__ void __launch_bounds__(kCountThreads)
sparse_count_kernel(const uint32_t* __restrict__ in, uint64_t n, bool vec, uint32_t* __restrict__ tile_cnt) {
  constexpr int kWarpElems = kTile / (kCountThreads / 32);
  __shared__ uint32_t warp_cnt[kCountThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t base = (uint64_t)blockIdx.x * kTile + (uint64_t)warp * kWarpElems;
  pdl_wait(in);
  pdl_trigger();  // behind the wait: what starts on it may read `in` at once
  uint32_t c = 0;
  if (vec && base + kWarpElems <= n) {
    uint4 v[kWarpElems / 128];
#pragma unroll
    for (int j = 0; j < kWarpElems / 128; j++) v[j] = __ldg(reinterpret_cast<const uint4*>(in + base) + j * 32 + lane);
#pragma unroll
    for (int j = 0; j < kWarpElems / 128; j++)
      c += (v[j].x != 0u) + (v[j].y != 0u) + (v[j].z != 0u) + (v[j].w != 0u);
  } else {
    for (int j = 0; j < kWarpElems / 32; j++) {
      const uint64_t i = base + j * 32 + lane;
      c += i < n && __ldg(in + i) != 0u;
    }
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) warp_cnt[warp] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kCountThreads / 32; i++) s += warp_cnt[i];
    tile_cnt[blockIdx.x] = s;
  }
}

// ---- pass 2: exclusive scan of the counts (one CTA) -----------------------------------
// In place: a[i] <- sum of a[0 .. i-1], the total to *total.  A thread takes four
// or sixteen consecutive counts, so 16384 of them (256 MiB of tensor) are one
// round: the kernel is a chain of latencies, and rounds of 1024 cost it 7 us there.
template <class T>
__global__ void __launch_bounds__(1024) block_exclusive_scan_kernel(T* a, uint32_t len, T* __restrict__ total) {
  __shared__ T warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_trigger();  // in front of the wait: what reads early behind it relies on the kernel ahead (pdl.cuh)
  pdl_wait();
  T carry = 0;
  for (uint32_t base = 0; base < len; base += 16384) {
    const int per = len - base <= 4096 ? 4 : 16;
    const uint32_t first = base + threadIdx.x * per;
    T v[16], sum = 0;
#pragma unroll
    for (int q = 0; q < 16; q++) {
      v[q] = q < per && first + q < len ? a[first + q] : T(0);
      sum += v[q];
    }
    T x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    T s = warp_sum[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= d) s += y;
    }
    const T front = __shfl_sync(0xffffffffu, s, warp - 1);  // of the warps in front of mine
    T off = carry + (warp ? front : T(0)) + x - sum;
    carry += __shfl_sync(0xffffffffu, s, 31);
#pragma unroll
    for (int q = 0; q < 16; q++) {
      if (q < per && first + q < len) a[first + q] = off;
      off += v[q];
    }
    __syncthreads();  // warp_sum is free for the next round
  }
  if (threadIdx.x == 0) *total = carry;
}

// ---- pass 3: bitmap and values ---------------------------------------------------------
// The tile is loaded while the scan still runs (past L1, so that nothing a kernel
// before left there can be met) and only its place in `values` is waited for.  This
// relies on the counting kernel of the same call, which let the scan start only when
// the tensor's producer had finished (pdl.cuh).  Tiles are
// taken from the end: what pass 1 read last is what L2 still holds of a tensor larger than
// itself (126 MB).  256 MiB, the whole call: 126 -> 118 us at 50 % zeros, 116 -> 106 at 90 %;
// tensors that fit into L2 take the same time either way.
__global__ void __launch_bounds__(kThreads)
sparse_pack_kernel(const uint32_t* __restrict__ in, uint64_t n, uint32_t* __restrict__ bitmap, const uint32_t* tile_off,
                   uint32_t* __restrict__ values) {
  __shared__ uint32_t warp_cnt[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tile = gridDim.x - 1 - blockIdx.x;
  const uint64_t base = (uint64_t)tile * kTile + (uint64_t)warp * (kWordsPerWarp * 32);
  uint32_t v[kWordsPerWarp], w[kWordsPerWarp];
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    const uint64_t i = base + j * 32 + lane;
    v[j] = i < n ? __ldcg(in + i) : 0u;
  }
  uint32_t mine = 0, cnt = 0;
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    w[j] = __ballot_sync(0xffffffffu, v[j] != 0u);
    cnt += __popc(w[j]);
    if (lane == j) mine = w[j];
  }
  const uint64_t word0 = base >> 5, nwords = (n + 31) >> 5;
  if (lane == 0) warp_cnt[warp] = cnt;
  __syncthreads();
  pdl_wait();
  if (lane < kWordsPerWarp && word0 + lane < nwords) bitmap[word0 + lane] = mine;
  uint32_t off = tile_off[tile];
  for (int i = 0; i < warp; i++) off += warp_cnt[i];
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    if (v[j] != 0u) values[off + __popc(w[j] & lt)] = v[j];
    off += __popc(w[j]);
  }
}

// The same without a scan in between, for kLeastSummed to kMostSummed tiles: a CTA adds up the counts ahead
// of its tile itself, and the last one to have read them turns them into offsets (tile_counts.cuh); no CTA waits
// for another.  A launch less, but a CTA's loads lie in front of its part in the sum: 50 % zeros, with the scan and without, 1 Mi elements
// 5.94 | 5.22 us, 2 Mi 6.64 | 6.24, 4 Mi 7.77 | 9.53, 8 Mi 13.3 | 15.9; 400 000 elements 5.94 | 6.01.  Where the host's
// part of a call is the longer one the launch counts whole, 1 Mi 8.27 | 6.38; in a graph it is nearly free, 4.93 | 5.09.
constexpr uint32_t kLeastSummed = 128, kMostSummed = 512;
__global__ void __launch_bounds__(kThreads, 8)
sparse_pack_sum_kernel(const uint32_t* __restrict__ in, uint64_t n, uint32_t* __restrict__ bitmap, uint32_t* tile_off,
                       uint32_t* __restrict__ values, uint32_t* __restrict__ nnz_out) {
  constexpr int kWarps = kThreads / 32, kPer = (int)kMostSummed / kThreads;
  __shared__ uint32_t warp_cnt[kWarps], warp_sum[kWarps];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tiles = gridDim.x, tile = tiles - 1 - blockIdx.x;
  const uint64_t base = (uint64_t)tile * kTile + (uint64_t)warp * (kWordsPerWarp * 32);
  uint32_t v[kWordsPerWarp], w[kWordsPerWarp];
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    const uint64_t i = base + j * 32 + lane;
    v[j] = i < n ? __ldcg(in + i) : 0u;
  }
  uint32_t mine = 0, cnt = 0;
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    w[j] = __ballot_sync(0xffffffffu, v[j] != 0u);
    cnt += __popc(w[j]);
    if (lane == j) mine = w[j];
  }
  const uint64_t word0 = base >> 5, nwords = (n + 31) >> 5;
  pdl_wait();
  uint32_t ahead = 0;
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const uint32_t i = q * kThreads + threadIdx.x;
    if (i < tile) ahead += tile_count(tile_off + i);
  }
  ahead = __reduce_add_sync(0xffffffffu, ahead);
  if (lane == 0) {
    warp_cnt[warp] = cnt;
    warp_sum[warp] = ahead;
  }
  __syncthreads();  // every count that this CTA needs has been read
  bool arrived_last = false;
  if (threadIdx.x == 0) arrived_last = last_to_arrive(tile_off, tiles);
  if (lane < kWordsPerWarp && word0 + lane < nwords) bitmap[word0 + lane] = mine;
  uint32_t off = 0;
#pragma unroll
  for (int i = 0; i < kWarps; i++) off += warp_sum[i] + (i < warp ? warp_cnt[i] : 0u);
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    if (v[j] != 0u) values[off + __popc(w[j] & lt)] = v[j];
    off += __popc(w[j]);
  }
  if (threadIdx.x == 0) last = arrived_last;
  __syncthreads();
  if (!last) return;
  uint32_t c[kPer], sum = 0;
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const uint32_t i = threadIdx.x * kPer + q;
    c[q] = i < tiles ? tile_count(tile_off + i) : 0u;
    sum += c[q];
  }
  uint32_t x = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();  // the counts have been read by all
  uint32_t at = x - sum, total = 0;
#pragma unroll
  for (int i = 0; i < kWarps; i++) {
    at += i < warp ? warp_sum[i] : 0u;
    total += warp_sum[i];
  }
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const uint32_t i = threadIdx.x * kPer + q;
    if (i < tiles) tile_off[i] = at;
    at += c[q];
  }
  if (threadIdx.x == 0) *nnz_out = total;
}

// ---- small tensors: one cluster --------------------------------------------------------
// Up to kMaxCluster CTAs of TILES tiles compress the whole tensor: bitmap,
// counts, offsets and values from one read and one launch.  The CTAs exchange their
// counts through distributed shared memory; three launches of 2-3 us each are what
// bounds tensors this small otherwise.
constexpr int kSmallThreads = 512, kMaxCluster = 16;
template <int TILES>
__global__ void __launch_bounds__(kSmallThreads)
sparse_small_kernel(const uint32_t* __restrict__ in, uint64_t n, uint32_t* __restrict__ bitmap,
                    uint32_t* __restrict__ tile_off, uint32_t* __restrict__ values, uint32_t* __restrict__ nnz_out) {
  constexpr int W = kSmallThreads / 32, kWords = TILES * kTile / 32 / W;  // bitmap words per warp
  __shared__ uint32_t warp_cnt[W], cta_cnt[kMaxCluster];
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t cta = blockIdx.x;
  const uint64_t base = (uint64_t)cta * (TILES * kTile) + (uint64_t)warp * (kWords * 32);
  cl.barrier_arrive();  // that every CTA of the cluster runs is only needed further down
  pdl_wait(in);
  uint32_t v[kWords], w[kWords];
#pragma unroll
  for (int j = 0; j < kWords; j++) {
    const uint64_t i = base + j * 32 + lane;
    v[j] = i < n ? __ldg(in + i) : 0u;
  }
  uint32_t mine = 0, cnt = 0;
#pragma unroll
  for (int j = 0; j < kWords; j++) {
    w[j] = __ballot_sync(0xffffffffu, v[j] != 0u);
    cnt += __popc(w[j]);
    if (lane == j) mine = w[j];
  }
  const uint64_t word0 = base >> 5, nwords = (n + 31) >> 5;
  if (lane < kWords && word0 + lane < nwords) bitmap[word0 + lane] = mine;
  if (lane == 0) warp_cnt[warp] = cnt;
  __syncthreads();
  uint32_t x = lane < W ? warp_cnt[lane] : 0u;
  const uint32_t c = x;
#pragma unroll
  for (int d = 1; d < W; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, x, W - 1);
  uint32_t off = __shfl_sync(0xffffffffu, x - c, warp);
  cl.barrier_wait();
  if (threadIdx.x < cl.num_blocks()) cl.map_shared_rank(cta_cnt, threadIdx.x)[cta] = total;
  cl.sync();
  uint32_t front = 0;
  for (uint32_t i = 0; i < cta; i++) front += cta_cnt[i];
  off += front;
  constexpr int kWarpsPerTile = W / TILES;
  const uint64_t tile = (uint64_t)cta * TILES + warp / kWarpsPerTile, ntiles = (n + kTile - 1) / kTile;
  if (lane == 0 && warp % kWarpsPerTile == 0 && tile < ntiles) tile_off[tile] = off;
  if (threadIdx.x == 0 && cta == gridDim.x - 1) *nnz_out = front + total;
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int j = 0; j < kWords; j++) {
    if (v[j] != 0u) values[off + __popc(w[j] & lt)] = v[j];
    off += __popc(w[j]);
  }
}

// ---- single pass: tiles claim their value segments from a cursor ---------------------
// Reads the tensor once.  A tile counts its non-zeros, claims that many slots
// with one atomic add on `cursor` (which must be zero at launch and holds the
// total afterwards) and records where its segment starts in tile_off; bitmap
// and per-tile contents are the same as the three-pass result, but segments
// sit in the order the tiles claimed them, so the values array (not what
// decompression returns) can differ from run to run.  No CTA waits for another.
// The tensor is read before the wait: sparse_zero_kernel, directly in front, triggers
// only behind its own (pdl.cuh).
__global__ void sparse_zero_kernel(uint32_t* word) {
  pdl_wait();
  pdl_trigger();  // behind the wait: what starts on it may read its input at once
  *word = 0u;
}
__global__ void __launch_bounds__(kThreads)
sparse_onepass_kernel(const uint32_t* __restrict__ in, uint64_t n, uint32_t* __restrict__ bitmap,
                      uint32_t* __restrict__ tile_off, uint32_t* __restrict__ values, uint32_t* __restrict__ cursor) {
  __shared__ uint32_t warp_cnt[kThreads / 32];
  __shared__ uint32_t tile_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t base = (uint64_t)blockIdx.x * kTile + (uint64_t)warp * (kWordsPerWarp * 32);
  uint32_t v[kWordsPerWarp], w[kWordsPerWarp];
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    const uint64_t i = base + j * 32 + lane;
    v[j] = i < n ? __ldcg(in + i) : 0u;
  }
  uint32_t mine = 0, cnt = 0;
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    w[j] = __ballot_sync(0xffffffffu, v[j] != 0u);
    cnt += __popc(w[j]);
    if (lane == j) mine = w[j];
  }
  const uint64_t word0 = base >> 5, nwords = (n + 31) >> 5;
  if (lane == 0) warp_cnt[warp] = cnt;
  __syncthreads();
  pdl_wait();  // the cursor is zero
  if (lane < kWordsPerWarp && word0 + lane < nwords) bitmap[word0 + lane] = mine;
  if (threadIdx.x == 0) {
    uint32_t total = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; i++) total += warp_cnt[i];
    const uint32_t at = atomicAdd(cursor, total);
    tile_off[blockIdx.x] = at;
    tile_base = at;
  }
  __syncthreads();
  uint32_t off = tile_base;
  for (int i = 0; i < warp; i++) off += warp_cnt[i];
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    if (v[j] != 0u) values[off + __popc(w[j] & lt)] = v[j];
    off += __popc(w[j]);
  }
}

// ---- decompression -----------------------------------------------------------------
// A CTA is a chain of two loads from memory - bitmap word and tile offset, then values -
// and bound by how many of them an SM has in flight.  (With the offset loaded behind the
// barrier, a chain of three: 256 MiB 70.6 -> 69.3 us at 50 % zeros, 63.1 -> 61.1 at 75 %.  One
// set of CTAs that loads the next tile's words ahead is slower, 80 and 73 us: its CTAs march
// through load and store phases together, those of a plain grid are spread over them.)
__global__ void __launch_bounds__(kThreads)
sparse_unpack_kernel(const uint32_t* __restrict__ bitmap, const uint32_t* __restrict__ values,
                     const uint32_t* __restrict__ tile_off, uint64_t n, uint32_t* __restrict__ out) {
  __shared__ uint32_t warp_cnt[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t base = (uint64_t)blockIdx.x * kTile + (uint64_t)warp * (kWordsPerWarp * 32);
  const uint64_t word0 = base >> 5, nwords = (n + 31) >> 5;
  pdl_wait(bitmap);
  asm volatile("" : "+l"(values), "+l"(tile_off));  // read behind the wait as well
  const uint32_t mine = (lane < kWordsPerWarp && word0 + lane < nwords) ? __ldg(bitmap + word0 + lane) : 0u;
  uint32_t off = __ldg(tile_off + blockIdx.x);  // on its way together with the bitmap
  // exclusive prefix of the popcounts of this warp's 16 words
  uint32_t x = __popc(mine);
  const uint32_t c = x;
#pragma unroll
  for (int d = 1; d < kWordsPerWarp; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == kWordsPerWarp - 1) warp_cnt[warp] = x;
  __syncthreads();
  for (int i = 0; i < warp; i++) off += warp_cnt[i];
  const uint32_t my_off = off + x - c;
  const uint32_t lt = lanemask_lt();
  // three separate sweeps so that all sixteen gathers of a thread are in flight
  // together (the warp shuffles would otherwise pin each load to its store)
  uint32_t src[kWordsPerWarp];  // index of my value, or ~0 when my element is zero
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    const uint32_t w = __shfl_sync(0xffffffffu, mine, j);
    const uint32_t o = __shfl_sync(0xffffffffu, my_off, j);
    src[j] = ((w >> lane) & 1u) ? o + __popc(w & lt) : 0xffffffffu;
  }
  uint32_t val[kWordsPerWarp];
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) val[j] = src[j] != 0xffffffffu ? __ldg(values + src[j]) : 0u;
#pragma unroll
  for (int j = 0; j < kWordsPerWarp; j++) {
    const uint64_t i = base + j * 32 + lane;
    if (i < n) out[i] = val[j];
  }
}

// ---- reference layout: one warp per worker ------------------------------------------
// Worker i owns elements [i*chunk, min((i+1)*chunk, n)); non-zero test is the
// float comparison of compression.cu:158,220 (-0.0 dropped, NaN kept).
__device__ __forceinline__ bool legacy_nz(uint32_t bits) { return __uint_as_float(bits) != 0.0f; }

__global__ void __launch_bounds__(kThreads)
legacy_count_kernel(const uint32_t* __restrict__ in, int n, int chunk, int workers, int* __restrict__ count) {
  pdl_wait(in);
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (i >= workers) return;
  const long long lo = (long long)chunk * i;
  if (lo >= n) return;  // compression.cu:149: such workers leave their slot untouched
  const long long hi = lo + chunk < n ? lo + chunk : n;
  int cnt = 0;
  for (long long p = lo; p < hi; p += 32) {
    const bool nz = p + lane < hi && legacy_nz(__ldg(in + p + lane));
    cnt += __popc(__ballot_sync(0xffffffffu, nz));
  }
  if (lane == 0) count[i] = cnt;
}

__global__ void __launch_bounds__(kThreads)
legacy_pack_kernel(const uint32_t* __restrict__ in, int n, int chunk, int workers, uint32_t* __restrict__ values,
                   const int* __restrict__ begin, uint32_t* __restrict__ bitmap) {
  pdl_wait(in);
  asm volatile("" : "+l"(begin));  // read behind the wait as well
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (i >= workers) return;
  const long long lo = (long long)chunk * i;
  if (lo >= n) return;
  const long long hi = lo + chunk < n ? lo + chunk : n;
  const int words_per = (chunk + 31) / 32;
  int off = begin[i];
  uint32_t* bm = bitmap + (long long)i * words_per;
  const uint32_t lt = lanemask_lt();
  for (long long p = lo; p < hi; p += 32, bm++) {
    const uint32_t v = p + lane < hi ? __ldg(in + p + lane) : 0u;
    const bool nz = p + lane < hi && legacy_nz(v);
    const uint32_t w = __ballot_sync(0xffffffffu, nz);
    if (nz) values[off + __popc(w & lt)] = v;
    off += __popc(w);
    if (lane == 0) *bm = w;
  }
}

// compression.cu:241-318: positions after the last set bit of a bitmap word
// are left untouched.
__global__ void __launch_bounds__(kThreads)
legacy_unpack_kernel(const uint32_t* __restrict__ values, uint32_t* __restrict__ out, int n, int chunk, int workers,
                     const uint32_t* __restrict__ bitmap, const int* __restrict__ begin) {
  pdl_wait(values);
  asm volatile("" : "+l"(bitmap), "+l"(begin));  // read behind the wait as well
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (i >= workers) return;
  const long long lo = (long long)chunk * i;
  if (lo >= n) return;
  const int words_per = (chunk + 31) / 32;
  const uint32_t* bm = bitmap + (long long)i * words_per;
  int off = begin[i];
  const uint32_t lt = lanemask_lt();
  for (int k = 0; k < words_per; k++) {
    const uint32_t w = __ldg(bm + k);
    const int written = 32 - __clz((int)w);  // 0 when the word is empty
    const long long p = lo + 32LL * k + lane;
    if (lane < written && p < n) out[p] = ((w >> lane) & 1u) ? __ldg(values + off + __popc(w & lt)) : 0u;
    off += __popc(w);
  }
}

}  // namespace

// =====================================================================================
// launchers
// =====================================================================================
namespace {
constexpr uint64_t kOnepassClusterElems = (uint64_t)kMaxCluster * 2 * kTile;
// One launch for what a cluster can hold.  Sixteen CTAs in a cluster are more than the
// portable eight and need opting in, once per device.
template <int TILES>
cudaError_t small_launch(const uint32_t* in, uint64_t n, uint32_t* bitmap, uint32_t* values, uint32_t* tile_off,
                         uint32_t* nnz_out, cudaStream_t stream) {
  static std::atomic<uint64_t> allowed{0};
  int dev = 0;
  cudaError_t e = taken(cudaGetDevice(&dev));
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
  if (!(allowed.load(std::memory_order_acquire) & bit)) {
    e = taken(cudaFuncSetAttribute(sparse_small_kernel<TILES>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (e != cudaSuccess) return e;
    allowed.fetch_or(bit, std::memory_order_release);
  }
  const uint32_t ctas = n ? (uint32_t)((n + TILES * kTile - 1) / (TILES * kTile)) : 1u;
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return taken(cudaLaunchKernelEx(&cfg, sparse_small_kernel<TILES>, in, n, bitmap, tile_off, values, nnz_out));
}
// true when the tensor is small enough for one cluster and its launch went through.  A cluster needs
// its CTAs' SMs in one GPC, all at a time: a process that has only part of a GPC (a partition, a
// green context) may be refused the launch, and is served by the ordinary ones.
bool small_compress(const uint32_t* in, uint64_t n, uint32_t* bitmap, uint32_t* values, uint32_t* tile_off,
                    uint32_t* nnz_out, cudaStream_t stream) {
  cudaError_t e = cudaErrorNotSupported;
  if (n <= (uint64_t)kMaxCluster * kTile) e = small_launch<1>(in, n, bitmap, values, tile_off, nnz_out, stream);
  else if (n <= (uint64_t)kMaxCluster * 2 * kTile) e = small_launch<2>(in, n, bitmap, values, tile_off, nnz_out, stream);
  else if (n <= (uint64_t)kMaxCluster * 4 * kTile) e = small_launch<4>(in, n, bitmap, values, tile_off, nnz_out, stream);
  return e == cudaSuccess;
}
}  // namespace

cudaError_t sparse_compress_launch(const float* in, uint64_t n, uint32_t* bitmap, float* values, uint32_t* tile_off,
                                   uint32_t* nnz_out, cudaStream_t stream) {
  const uint32_t ntiles = (uint32_t)((n + kTile - 1) / kTile);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(in);
  uint32_t* val = reinterpret_cast<uint32_t*>(values);
  if (small_compress(src, n, bitmap, val, tile_off, nnz_out, stream)) return cudaSuccess;
  const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  cudaError_t e = cudaSuccess;
  if (ntiles) e = pdl_launch(sparse_count_kernel, ntiles, kCountThreads, 0, stream, src, n, vec, tile_off);
  if (e == cudaSuccess && ntiles >= kLeastSummed && ntiles <= kMostSummed)
    return pdl_launch(sparse_pack_sum_kernel, ntiles, kThreads, 0, stream, src, n, bitmap, tile_off, val, nnz_out);
  if (e == cudaSuccess) e = pdl_launch(block_exclusive_scan_kernel<uint32_t>, 1, 1024, 0, stream, tile_off, ntiles, nnz_out);
  if (e == cudaSuccess && ntiles)
    e = pdl_launch(sparse_pack_kernel, ntiles, kThreads, 0, stream, src, n, bitmap, tile_off, val);
  return e;
}

cudaError_t sparse_compress_preload() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, sparse_small_kernel<1>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, sparse_small_kernel<2>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, sparse_small_kernel<4>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, sparse_count_kernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, block_exclusive_scan_kernel<uint32_t>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, sparse_pack_kernel);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, sparse_pack_sum_kernel);
  return taken(e);
}

cudaError_t sparse_compress_onepass_launch(const float* in, uint64_t n, uint32_t* bitmap, float* values,
                                           uint32_t* tile_off, uint32_t* nnz_out, cudaStream_t stream) {
  const uint32_t ntiles = (uint32_t)((n + kTile - 1) / kTile);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(in);
  uint32_t* val = reinterpret_cast<uint32_t*>(values);
  // Not up to 1 MiB as the ordered compressor: with four tiles each the cluster's CTAs (512 threads of 120
  // registers) fit no SM that runs anything else, and the two launches are short.  180000 elements 4.3 us in the
  // cluster, 3.5 in two launches, back to back; 262144 elements 4.4 and 3.3, and beside matrix products of another
  // stream (which is where the swap manager calls) 15.3 us at the median but 300 at the 90th percentile, a
  // product's whole run, against 14.1 and 16.8.  131072 elements 3.1 and 3.4 idle, 15.6 and 13.7 beside products,
  // 13.2 and 13.3 beside a convolution, 41 and 30 beside elementwise kernels that keep every SM full; 16384
  // elements 2.5 and 3.4, 14.0 and 13.3, 11.6 and 12.7, 36 and 28.
  if (n <= kOnepassClusterElems && small_compress(src, n, bitmap, val, tile_off, nnz_out, stream)) return cudaSuccess;
  cudaError_t e = pdl_launch(sparse_zero_kernel, 1, 1, 0, stream, nnz_out);  // the cursor, then the total
  if (e == cudaSuccess && ntiles)
    e = pdl_launch(sparse_onepass_kernel, ntiles, kThreads, 0, stream, src, n, bitmap, tile_off, val, nnz_out);
  return e;
}

cudaError_t sparse_decompress_launch(const uint32_t* bitmap, const float* values, const uint32_t* tile_off, uint64_t n,
                                     float* out, cudaStream_t stream) {
  const uint32_t ntiles = (uint32_t)((n + kTile - 1) / kTile);
  if (!ntiles) return cudaSuccess;
  return pdl_launch(sparse_unpack_kernel, ntiles, kThreads, 0, stream, bitmap, reinterpret_cast<const uint32_t*>(values),
                    tile_off, n, reinterpret_cast<uint32_t*>(out));
}

static int ceil_div_i(int a, int b) { return a % b == 0 ? a / b : a / b + 1; }

cudaError_t legacy_count_launch(int n, int workers, const float* in, int* count, cudaStream_t stream) {
  if (n <= 0 || workers <= 0) return cudaSuccess;
  const int chunk = ceil_div_i(n, workers);
  return pdl_launch(legacy_count_kernel, (workers + 7) / 8, kThreads, 0, stream, reinterpret_cast<const uint32_t*>(in), n,
                    chunk, workers, count);
}
cudaError_t legacy_scan_launch(int* idx, int len, int* num, cudaStream_t stream) {
  if (len <= 0) return cudaSuccess;
  // in-place scan of the first `len` counts, total to num[0] (compression.cu:9-19)
  return pdl_launch(block_exclusive_scan_kernel<int>, 1, 1024, 0, stream, idx, (uint32_t)len, num);
}
cudaError_t legacy_pack_launch(int n, int workers, const float* in, float* values, const int* begin, uint32_t* bitmap,
                               cudaStream_t stream) {
  if (n <= 0 || workers <= 0) return cudaSuccess;
  const int chunk = ceil_div_i(n, workers);
  return pdl_launch(legacy_pack_kernel, (workers + 7) / 8, kThreads, 0, stream, reinterpret_cast<const uint32_t*>(in), n,
                    chunk, workers, reinterpret_cast<uint32_t*>(values), begin, bitmap);
}
cudaError_t legacy_unpack_launch(const float* values, float* out, int n, int workers, const uint32_t* bitmap,
                                 const int* begin, cudaStream_t stream) {
  if (n <= 0 || workers <= 0) return cudaSuccess;
  const int chunk = ceil_div_i(n, workers);
  return pdl_launch(legacy_unpack_kernel, (workers + 7) / 8, kThreads, 0, stream, reinterpret_cast<const uint32_t*>(values),
                    reinterpret_cast<uint32_t*>(out), n, chunk, workers, bitmap, begin);
}

}  // namespace csw
