// internal.h -- host-side launchers shared between the library's translation
// units.  Not part of the public C-ABI (include/astraea_gb300.h).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "astraea_gb300.h"
#include "common.cuh"

namespace astraea_gb300 {

// Programmatic dependent launch: a kernel started by launchChained is prepared
// while the kernel before it in the stream runs, and its blocks are placed as
// soon as that kernel's blocks have ended; chained(), the first statement of
// such a kernel for every thread, returns when everything before is complete and
// visible, so nothing in the body needs care.  A step has some 25 launches: 16k
// 303 -> 266 us, one gravity call at 60k 113 -> 106.  No kernel lets the next one
// in early (griddepcontrol.launch_dependents): blocks then settle where the
// running kernel happens to leave room, and the walks, whose few blocks a small
// scene has no second wave to even out, ran 16k 344 us, gravity at 60k 157.
__device__ __forceinline__ void chained() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Where a kernel is launched: the stream, and whether it is to run beside the
// kernels of another stream.  An SM divides its memory between L1 and shared
// memory anew only when it is empty, so kernels for which the driver chooses
// different splits do not meet on one; those that should meet ask for the same
// one (all shared memory).
struct LaunchAt {
    cudaStream_t stream;
    bool beside;
    LaunchAt(cudaStream_t s, bool b = false) : stream(s), beside(b) {}
};
template <class... P, class... A>
cudaError_t launchChainedSmem(void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, LaunchAt at, A&&... args) {
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = at.stream;
    cfg.attrs = attr;
    cfg.numAttrs = at.beside ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
template <class... P, class... A>
cudaError_t launchChained(void (*kernel)(P...), uint32_t grid, uint32_t block, LaunchAt at, A&&... args) {
    return launchChainedSmem(kernel, grid, block, 0, at, static_cast<A&&>(args)...);
}

// SMs of the GPU the size thresholds below were measured on (permutation, lanes a
// particle, pass 2's records): where one kernel starts to beat another, not
// limits of a launch.
constexpr uint32_t kTunedSms = 152u;

constexpr int kSortThreads = 512;
constexpr int kSortBins = 256;
constexpr int kSortMaxPasses = 8;

// Keys a thread of the tiled passes holds (a tile is 512 times that): small
// tiles put more blocks on the GPU while there are few, large ones amortise a
// tile's fixed chain (sort.cu).
constexpr uint32_t kSortSmallTileMax = 1u << 19, kSortMiddleTileMax = 1u << 22;
constexpr int sortItems(uint32_t n) { return n <= kSortSmallTileMax ? 4 : (n <= kSortMiddleTileMax ? 8 : 12); }
constexpr uint32_t sortTilesOf(uint32_t n) {
    const uint32_t tile = static_cast<uint32_t>(kSortThreads * sortItems(n));
    return n == 0u ? 1u : (n - 1u) / tile + 1u;
}
// The most tiles of any sort of at most n keys (scratch is kept for a
// capacity, and the tile grows with n).
constexpr uint32_t sortTiles(uint32_t n) {
    uint32_t t = sortTilesOf(n);
    if (n > kSortSmallTileMax && sortTilesOf(kSortSmallTileMax) > t) t = sortTilesOf(kSortSmallTileMax);
    if (n > kSortMiddleTileMax && sortTilesOf(kSortMiddleTileMax) > t) t = sortTilesOf(kSortMiddleTileMax);
    return t;
}

// Onesweep scratch layout (32-bit words):
//   [0, kSortHistWords)                              digit histograms, one per pass
//   [kSortHistWords, + kSortCounterWords)            tile counters, one per pass
//   then kSortMaxPasses * tiles * kSortBins          look-back status words
constexpr size_t kSortHistWords = static_cast<size_t>(kSortMaxPasses) * kSortBins;
constexpr size_t kSortCounterWords = 8;
constexpr size_t sortScratchWordsFor(uint32_t n) {
    return kSortHistWords + kSortCounterWords + static_cast<size_t>(kSortMaxPasses) * sortTiles(n) * kSortBins;
}

// Number of 32-bit words of onesweep scratch for n keys.
size_t sortScratchWords(uint32_t n, uint32_t* maxTilesOut);

// Where the keys of the sort come from.
enum class KeySource { Array, MortonFromPositions };

struct MortonSource {
    const float* x;        // either SoA x/y/z ...
    const float* y;
    const float* z;
    const float4* xyz;     // ... or float4 {x, y, z, _} (used when non-null)
    const uint32_t* boundsOrdered;  // 6 ordered-uint words of the scene AABB
    float* boundsFloatOut;          // optional: decoded bounds written by block 0
};

// Stable LSD radix sort of (u64 key, u32 value) over bits [0, endBit).
// Data starts in (keysA, valsA); (keysB, valsB) is the ping-pong partner.
// Returns (through *resultInA) which pair holds the sorted output.
// With src == MortonFromPositions the keys and values (iota) are generated
// from positions in the histogram kernel and written into (keysA, valsA).
cudaError_t radixSortPairs(uint64_t* keysA, uint32_t* valsA, uint64_t* keysB, uint32_t* valsB, uint32_t n,
                           int endBit, uint32_t* scratch, size_t scratchWords, uint32_t maxTiles, DevStatus* status,
                           uint32_t spinLimit, KeySource src, const MortonSource* morton, bool* resultInA,
                           cudaStream_t stream);

// Failure-detection probe of the bounded look-back wait (see sort.cu).
cudaError_t launchLookbackProbe(const uint32_t* neverSet, DevStatus* status, uint32_t spinLimit, uint32_t* result,
                                cudaStream_t stream);

}  // namespace astraea_gb300
