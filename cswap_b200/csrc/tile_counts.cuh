// The tile counts that the CTAs of one kernel add up while the last one of them to have read them turns them into
// offsets, in place.  Every CTA calls last_to_arrive() once, behind its reads (a barrier of its own in
// between); the one that gets true may overwrite the words, for all reads of the others lie before.  The number of CTAs
// that have arrived is kept above the thirteen bits of the first word's count.
//
// The reads are of words that others add to, so they are relaxed atomic loads, and an arrival releases the reads
// before it, which the last one acquires: without that nothing orders the last CTA's stores behind the other CTAs' loads.  The host build is for tests, which run CTAs as threads under a race detector.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define CSW_COUNTS __device__ __forceinline__
#else
#define CSW_COUNTS inline
#endif

namespace csw {

constexpr int kCountBits = 13;  // a tile's count is 4096 at most
constexpr uint32_t kCountMask = (1u << kCountBits) - 1u;

CSW_COUNTS uint32_t tile_count(const uint32_t* word) {
  uint32_t v;
#if defined(__CUDACC__)
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
#else
  v = __atomic_load_n(word, __ATOMIC_RELAXED);
#endif
  return v & kCountMask;
}

CSW_COUNTS bool last_to_arrive(uint32_t* words, uint32_t ctas) {
  uint32_t before;
#if defined(__CUDACC__)
  asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;"
               : "=r"(before)
               : "l"(words), "r"(1u << kCountBits)
               : "memory");
#else
  before = __atomic_fetch_add(words, 1u << kCountBits, __ATOMIC_RELEASE);
#endif
  if (before >> kCountBits != ctas - 1u) return false;
#if defined(__CUDACC__)
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(before) : "l"(words) : "memory");
#else
  before = __atomic_load_n(words, __ATOMIC_ACQUIRE);
#endif
  return true;
}

}  // namespace csw
