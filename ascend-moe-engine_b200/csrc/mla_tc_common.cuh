// What the two tensor-core decode kernels share: the tile geometry, the bounded mbarrier waits and the issue of one
// slab group of QK instructions.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace b200kv {
namespace mla {

constexpr int kHeads = 64;
constexpr int kLatent = B200KV_LATENT_DIM;
constexpr int kRope = B200KV_ROPE_DIM;
constexpr int kTile = 64;      // tokens per tile / KV stage
constexpr int kStages = 2;
constexpr int kGroups = 4;                              // slab groups of a stage: slabs 2c, 2c+1 (and 8 with the last)
constexpr int kSlabBytes = kTile * 128;                 // one 64-column slab of a tile: kTile rows x 128 B
constexpr int kStageBytes = 9 * kSlabBytes;             // 73,728
constexpr int kQSlabBytes = kHeads * 128;               // 8,192
constexpr int kQBytes = 9 * kQSlabBytes;                // 73,728
constexpr int kSoftmaxThreads = 128;
constexpr int kSoftmaxWarps = kSoftmaxThreads / 32;     // one lane of each arrives on the barriers they signal
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemColS = 256;                     // S buffers at columns 256 and 256 + kTile
constexpr float kRescaleThreshold = 8.0f;               // log2 units: rescale O only when max grows by > 2^8
// Where running maxima start: finite, so that subtracting one from a score of -infinity leaves -infinity, a weight of zero.
constexpr float kLowest = -3.4028234663852886e38f;

__device__ __forceinline__ int TilesOf(int len) { return (len + kTile - 1) / kTile; }

template <typename Misc>
__device__ __forceinline__ bool Aborting(const Misc* misc) {
  return *reinterpret_cast<const volatile int32_t*>(&misc->abort_flag) != 0;
}

template <typename Misc>
__device__ __noinline__ void RaiseTimeout(Misc* misc, int32_t* status, int site, uint32_t parity) {
  *reinterpret_cast<volatile int32_t*>(&misc->abort_flag) = 1;
  RecordError(status, B200KV_DEV_TIMEOUT, site, static_cast<int32_t>(blockIdx.x), static_cast<int32_t>(parity));
}

// `Misc` is the kernel's block of barriers; its abort_flag is raised by the first wait that runs out.
// Bounded mbarrier wait. Returns false when the CTA is aborting or this wait ran out (about one
// second), after recording where.
template <typename Misc>
__device__ __noinline__ bool BoundedWait(uint32_t bar, uint32_t parity, Misc* misc, int32_t* status, int site) {
  uint64_t start = 0;
  for (uint32_t it = 0;; ++it) {
    if (ptx::MbarTryWait(bar, parity)) return true;
    if ((it & 255u) == 255u) {
      if (Aborting(misc)) return false;
      const uint64_t now = ptx::GlobalTimerNs();
      if (start == 0) start = now;
      if (now - start > 1000000000ull) {
        RaiseTimeout(misc, status, site, parity);
        return false;
      }
    }
  }
}

// The same with a non-blocking probe in a tight loop. mbarrier.try_wait parks the thread and, measured here, a
// parked thread resumes some 500 cycles after the phase completes; the producer's waits sit on the path that
// refills a stage, so it spins instead (one thread: the issue slots it takes are few).
template <typename Misc>
__device__ __noinline__ bool BoundedSpin(uint32_t bar, uint32_t parity, Misc* misc, int32_t* status, int site) {
  uint64_t start = 0;
  for (uint32_t it = 0;; ++it) {
    if (ptx::MbarTestWait(bar, parity)) return true;
    if ((it & 1023u) == 1023u) {
      if (Aborting(misc)) return false;
      const uint64_t now = ptx::GlobalTimerNs();
      if (start == 0) start = now;
      if (now - start > 1000000000ull) {
        RaiseTimeout(misc, status, site, parity);
        return false;
      }
    }
  }
}

// A 64-bit shared-memory descriptor whose start address is advanced by adding to the low word.
__device__ __forceinline__ uint64_t DescAt(uint64_t base_desc, uint32_t byte_offset) {
  return base_desc + static_cast<uint64_t>(byte_offset >> 4);
}

// The QK k-steps of kSlabs 64-column slabs (four each) starting at slab kFirstSlab; called by the whole MMA warp.
// kFresh: the group starts an accumulator of its own instead of adding to what the groups before it left.
template <int kFirstSlab, int kSlabs, bool kFresh = false>
__device__ __forceinline__ void IssueQkGroup(uint64_t q_desc, uint64_t kdesc, uint32_t d) {
  constexpr uint32_t kIdescQk = ptx::InstrDescBf16(64, kTile, 0, 0);
#pragma unroll
  for (int i = 0; i < 4 * kSlabs; ++i) {
    const int c = kFirstSlab + (i >> 2), kk = i & 3;
    const uint64_t a = DescAt(q_desc, c * kQSlabBytes + kk * 32);
    const uint64_t b = DescAt(kdesc, c * kSlabBytes + kk * 32);
    if (ptx::ElectOne()) ptx::MmaF16SS(d, a, b, kIdescQk, (kFresh ? i : kFirstSlab + i) > 0 ? 1u : 0u);
  }
}

}  // namespace mla
}  // namespace b200kv
