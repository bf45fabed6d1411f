// sort.cu -- onesweep LSD radix sort of (u64 key, u32 value) pairs for sm_103a.
//
// Replaces the cub::DeviceRadixSort::SortPairs call of
// engine/sph_gravity.cu:2028-2046 (stable, bits [0, 63), value = original
// index).  Design (Adinets & Merrill's single-pass "onesweep"):
//   * one up-front kernel builds the histograms of all 8-bit digits in one
//     read of the keys (and, for the Morton path, computes the 63-bit codes
//     from positions on the fly, engine/sph_gravity.cu:151-171 + 335-361);
//   * one kernel per digit: a tile of 2,048 to 6,144 keys is ranked stably in
//     shared memory (warps match equal digits in input order), the tile's bin
//     counts are published, the exclusive prefix over earlier tiles comes from
//     a decoupled look-back, and keys/values are scattered through a
//     shared-memory staging buffer so global writes stay coalesced per bin;
//   * up to 65,536 keys are sorted by one launch of one thread-block cluster
//     instead, the keys staying in its blocks' shared memory for all digits.
// Every look-back spin is bounded; a timeout sets a device status flag and
// the tile proceeds with the prefix gathered so far (an underestimate, so the
// tile's destinations stay inside its bin).  The result is then not sorted,
// and later passes see keys that no longer match the digit histograms, so
// every store is also checked against n.
#include <algorithm>
#include <atomic>

#include "internal.h"

namespace astraea_gb300 {
namespace {

constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1u;

// Scratch layout: internal.h (sortScratchWordsFor).
constexpr size_t kHistWords = kSortHistWords;
constexpr size_t kCounterWords = kSortCounterWords;

__device__ __forceinline__ uint32_t lanemaskLt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t loadVolatile(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void storeRelaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// 63-bit Morton code of one position (engine/sph_gravity.cu:161-171, 347-359);
// the products and sums are separate IEEE operations, as in the reference.
__device__ __forceinline__ uint64_t mortonCode(float x, float y, float z, const float* b6, const float* inv3) {
    const float fx = fminf(fmaxf(__fmul_rn(__fsub_rn(x, b6[0]), inv3[0]), 0.0f), 2097151.0f);
    const float fy = fminf(fmaxf(__fmul_rn(__fsub_rn(y, b6[1]), inv3[1]), 0.0f), 2097151.0f);
    const float fz = fminf(fmaxf(__fmul_rn(__fsub_rn(z, b6[2]), inv3[2]), 0.0f), 2097151.0f);
    const uint64_t ix = static_cast<uint64_t>(static_cast<uint32_t>(fx));
    const uint64_t iy = static_cast<uint64_t>(static_cast<uint32_t>(fy));
    const uint64_t iz = static_cast<uint64_t>(static_cast<uint32_t>(fz));
    return (spreadBits21(ix) << 2) | (spreadBits21(iy) << 1) | spreadBits21(iz);
}

template <bool kMorton>
__global__ void __launch_bounds__(256) histogramKernel(const uint64_t* __restrict__ keysIn, MortonSource ms,
                                                       uint64_t* __restrict__ keysOut, uint32_t* __restrict__ valsOut,
                                                       uint32_t n, int passes, uint32_t* __restrict__ hist) {
    chained();
    __shared__ uint32_t sh[kSortMaxPasses][kSortBins];
    __shared__ float sB[6];
    __shared__ float sInv[3];
    for (int t = threadIdx.x; t < kSortMaxPasses * kSortBins; t += blockDim.x) (&sh[0][0])[t] = 0u;
    if (kMorton && threadIdx.x == 0) {
        for (int k = 0; k < 6; ++k) sB[k] = floatFromOrdered(ms.boundsOrdered[k]);
        for (int k = 0; k < 3; ++k) {
            const float span = sB[3 + k] - sB[k];
            sInv[k] = (span > 1.0e-6f) ? (2097151.0f / span) : 0.0f;   // sph_gravity.cu:350-355
        }
        if (blockIdx.x == 0 && ms.boundsFloatOut != nullptr)
            for (int k = 0; k < 6; ++k) ms.boundsFloatOut[k] = sB[k];
    }
    __syncthreads();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint64_t key;
        if (kMorton) {
            float x, y, z;
            if (ms.xyz != nullptr) {
                const float4 q = ms.xyz[i];
                x = q.x; y = q.y; z = q.z;
            } else {
                x = __ldg(&ms.x[i]); y = __ldg(&ms.y[i]); z = __ldg(&ms.z[i]);
            }
            key = mortonCode(x, y, z, sB, sInv);
            keysOut[i] = key;
            valsOut[i] = i;
        } else {
            key = keysIn[i];
        }
        for (int p = 0; p < passes; ++p) atomicAdd(&sh[p][(key >> (8 * p)) & 0xFFu], 1u);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < passes * kSortBins; t += blockDim.x) {
        const uint32_t c = (&sh[0][0])[t];
        if (c) atomicAdd(&hist[t], c);
    }
}

// Sum, for bin `bin`, the counts of tiles [0, tile) by walking back over the
// published status words until a tile that carries an inclusive prefix.  The
// walk reads sixteen status words per step (independent loads, so one L2 round
// trip per sixteen tiles instead of one per tile) and takes them in order: it
// stops at the first inclusive prefix, and at the first unpublished word it
// polls that word again.  Every poll of an unpublished word counts against
// spinLimit; on running out the walk stops (returns false) with the partial
// sum in *excl, which keeps the caller's destinations inside its bin.
constexpr int kLookbackWindow = 16;

__device__ __forceinline__ bool lookbackExclusive(const uint32_t* lookback, uint32_t tile, int bin,
                                                  uint32_t spinLimit, uint32_t* excl) {
    int64_t j = static_cast<int64_t>(tile) - 1;
    uint32_t spins = 0, sum = 0;
    while (j >= 0) {
        uint32_t v[kLookbackWindow];
#pragma unroll
        for (int q = 0; q < kLookbackWindow; ++q)   // before tile 0: an empty inclusive prefix
            v[q] = (j - q >= 0) ? loadVolatile(lookback + static_cast<size_t>(j - q) * kSortBins + bin) : kFlagPrefix;
        int used = 0;
        bool unpublished = false, prefix = false;
#pragma unroll
        for (int q = 0; q < kLookbackWindow; ++q) {
            if (unpublished || prefix) continue;
            const uint32_t flag = v[q] & ~kValueMask;
            if (flag == 0u) {
                unpublished = true;
            } else {
                sum += v[q] & kValueMask;
                ++used;
                prefix = (flag == kFlagPrefix);
            }
        }
        if (prefix) break;
        j -= used;
        if (unpublished) {
            if (spins >= spinLimit) { *excl = sum; return false; }
            ++spins;
            __nanosleep(32);
        }
    }
    *excl = sum;
    return true;
}

// Failure-detection probe: one thread runs the look-back wait on a status
// word that nothing publishes, so the wait must give up after spinLimit polls
// and report it through the status flags.
__global__ void lookbackProbeKernel(const uint32_t* neverSet, DevStatus* status, uint32_t spinLimit,
                                    uint32_t* result) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    uint32_t excl = 0;
    const bool ok = lookbackExclusive(neverSet, 1u, 0, spinLimit, &excl);
    if (!ok) atomicOr(&status->flags, kFlagLookbackTimeout);
    *result = ok ? 1u : 2u;
}

constexpr int kSortWarps = kSortThreads / 32;

template <int kItems>
struct SortSmem {
    uint64_t keys[kSortThreads * kItems];
    uint32_t vals[kSortThreads * kItems];
    uint32_t warpHist[kSortWarps][kSortBins];
    uint32_t tileExcl[kSortBins];     // exclusive offset of each bin inside this tile
    uint32_t globalBase[kSortBins];   // destination = globalBase[bin] + tile-local slot
    uint32_t scanTmp[8];
    uint32_t tile;
};

// Exclusive scan over the first 256 threads' values (one per bin); every
// thread of the block must call it, the others pass 0 and ignore the result.
__device__ __forceinline__ uint32_t binExclusiveScan(uint32_t v, uint32_t* tmp8) {
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31 && warp < 8) tmp8[warp] = incl;
    __syncthreads();
    uint32_t off = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) off += (w < warp) ? tmp8[w] : 0u;
    __syncthreads();
    return off + incl - v;
}

// Lanes of the warp whose digit (9 bits: 0x100 means no key) equals this
// lane's, from nine ballots.  __match_any_sync takes time with the number of
// different values in the warp, and the low digits of Morton codes are all
// different.
__device__ __forceinline__ uint32_t matchDigit(uint32_t digit) {
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const uint32_t bit = (digit >> b) & 1u;
        peers &= ~(__ballot_sync(0xffffffffu, bit != 0u) ^ (0u - bit));
    }
    return peers;
}

// Stable rank of `digit` among the keys its warp has counted so far in
// wh[256]: the first lane of each group of equal digits adds their number to
// the warp's count and hands out the old value.  The atomics of one warp are
// in program order, so ranks follow (round, lane) order, and the rounds'
// atomics are in flight together.
__device__ __forceinline__ uint32_t warpRank(uint32_t digit, uint32_t* wh) {
    const uint32_t peers = matchDigit(digit);
    const int leader = __ffs(peers) - 1;
    uint32_t before = 0;
    if ((threadIdx.x & 31) == leader && digit < 0x100u) before = atomicAdd(&wh[digit], __popc(peers));
    __syncwarp();
    return __shfl_sync(0xffffffffu, before, leader) + __popc(peers & lanemaskLt());
}

// One digit pass.  What bounds it: a tile's chain (ticket, load, rank, look-back,
// store) while the tiles fit the GPU at once, HBM beyond.  512 threads of 8 keys
// rank in half the serial rounds of 256 threads of 16, and the look-back
// crosses sixteen tiles per L2 round trip: with four, the last of 245 tiles
// (1M keys) spent thirty round trips meeting the front of finished prefixes.
// Keys are matched by ballots: match.any takes a round per different digit.
// Seven passes on random keys, against 256 threads, 4,096-key tiles, match.any
// and a window of four for every size: 150k 102 -> 86 us, 262k 114 -> 87,
// 1M 160 -> 144, 4M 423 -> 386, 16M 1498 -> 1244 (tiles of 4, 8 and 12 keys a
// thread: at 150k 8 keys take 98 us, at 16M 8 keys 1410).
template <int kItems>
__global__ void __launch_bounds__(kSortThreads, kItems <= 4 ? 3 : 2) onesweepKernel(const uint64_t* __restrict__ keysIn,
                                                               const uint32_t* __restrict__ valsIn,
                                                               uint64_t* __restrict__ keysOut,
                                                               uint32_t* __restrict__ valsOut, uint32_t n, int pass,
                                                               const uint32_t* __restrict__ hist,
                                                               uint32_t* __restrict__ tileCounter,
                                                               uint32_t* __restrict__ lookback, DevStatus* status,
                                                               uint32_t spinLimit) {
    chained();
    extern __shared__ __align__(16) unsigned char smemRaw[];
    SortSmem<kItems>& s = *reinterpret_cast<SortSmem<kItems>*>(smemRaw);
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const int shift = 8 * pass;
    constexpr uint32_t kTile = kSortThreads * kItems;
    const bool owner = t < kSortBins;               // thread t owns bin t

    if (t == 0) s.tile = atomicAdd(tileCounter, 1u);
    const uint32_t binCount = owner ? hist[pass * kSortBins + t] : 0u;
    for (int k = t; k < kSortWarps * kSortBins; k += kSortThreads) (&s.warpHist[0][0])[k] = 0u;
    __syncthreads();
    const uint32_t tile = s.tile;
    const uint32_t tileBase = tile * kTile;
    const uint32_t warpBase = tileBase + static_cast<uint32_t>(warp) * (kItems * 32);

    // Load (warp-striped: item k of lane l is element warpBase + 32k + l) and
    // rank stably inside the warp: items are visited in (k, lane) order, which
    // is input order.
    uint64_t key[kItems];
    uint32_t rank[kItems];
    const uint32_t myFirst = warpBase + static_cast<uint32_t>(lane);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t idx = myFirst + 32u * static_cast<uint32_t>(k);
        key[k] = idx < n ? keysIn[idx] : 0ull;
    }
    auto digitOf = [&](int k) {                     // 0x100 behind the end of the input
        return myFirst + 32u * static_cast<uint32_t>(k) < n ? static_cast<uint32_t>(key[k] >> shift) & 0xFFu : 0x100u;
    };
    // global start of every bin for this pass (exclusive scan of the histogram)
    const uint32_t binStart = binExclusiveScan(binCount, s.scanTmp);
#pragma unroll
    for (int k = 0; k < kItems; ++k) rank[k] = warpRank(digitOf(k), s.warpHist[warp]);
    __syncthreads();

    // Per-bin tile totals and per-warp exclusive offsets.
    uint32_t total = 0;
    uint32_t* myStatus = lookback + static_cast<size_t>(tile) * kSortBins + t;
    if (owner) {
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = s.warpHist[w][t];
            s.warpHist[w][t] = total;
            total += c;
        }
        // Publish this tile's aggregate as early as possible.
        storeRelaxed(myStatus, (tile == 0 ? kFlagPrefix : kFlagAggregate) | total);
    }
    const uint32_t tileExcl = binExclusiveScan(total, s.scanTmp);
    if (owner) {
        s.tileExcl[t] = tileExcl;
        // Decoupled look-back over earlier tiles for bin t.
        uint32_t excl = 0;
        if (tile > 0) {
            if (!lookbackExclusive(lookback, tile, t, spinLimit, &excl)) atomicOr(&status->flags, kFlagLookbackTimeout);
            storeRelaxed(myStatus, kFlagPrefix | ((excl + total) & kValueMask));
        }
        s.globalBase[t] = binStart + excl - tileExcl;
    }
    // the values, needed from here on only: their loads overlap the barrier
    uint32_t val[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t idx = myFirst + 32u * static_cast<uint32_t>(k);
        val[k] = idx < n ? valsIn[idx] : 0u;
    }
    __syncthreads();

    // Stage into shared memory in bin order, then write out coalesced.
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t d = digitOf(k);
        if (d < 0x100u) {
            const uint32_t slot = s.tileExcl[d] + s.warpHist[warp][d] + rank[k];
            s.keys[slot] = key[k];
            s.vals[slot] = val[k];
        }
    }
    __syncthreads();
    const uint32_t tileCount = (tileBase < n) ? min(kTile, n - tileBase) : 0u;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t slot = static_cast<uint32_t>(t + k * kSortThreads);
        if (slot >= tileCount) break;
        const uint64_t kk = s.keys[slot];
        const uint32_t d = static_cast<uint32_t>((kk >> shift) & 0xFFu);
        const uint32_t dst = s.globalBase[d] + slot;
        // Always true for a consistent input.  After a look-back timeout in an
        // earlier pass the keys are no longer a permutation of the histogram's,
        // and a bin can overflow its range: the check keeps the writes in [0, n).
        if (dst < n) {
            keysOut[dst] = kk;
            valsOut[dst] = s.vals[slot];
        }
    }
}

// ------------------------------------------------ one cluster, one launch ---
// All passes of a sort of up to kClusterMaxKeys keys in one launch: a cluster
// of 16 blocks holds the keys in its shared memory (block c the c-th sixteenth
// of the current order), and a pass exchanges digit counts and keys through
// distributed shared memory with two cluster barriers.  A pass of the tiled
// sort is a launch whose chain of latencies hardly depends on n below a few
// tiles, eight times; here a pass costs its ranking, one count exchange and
// the scatter.  It uses 16 of the SMs, so the tiled passes over the whole GPU
// win above 4,096 keys a block.  Seven passes on random keys, one launch
// against tiled: 2k 23 / 51 us, 16k 34 / 65, 30k 44 / 66, 60k 62 / 72 (at 100k,
// with 1,024 threads a block, 91 / 83).  Morton codes take five passes and the
// check: sort stage of a 16k step 111 -> 35 us, 30k 114 -> 43.
constexpr int kClusterBlocks = 16;
constexpr uint32_t kClusterMaxKeys = kClusterBlocks * 4096u;

template <int kThreads, int kItems>
struct ClusterSmem {
    static constexpr int kWarps = kThreads / 32;
    static constexpr uint32_t kChunk = kThreads * kItems;   // keys a block at most
    uint64_t keys[2][kChunk];
    uint32_t vals[2][kChunk];
    uint32_t warpHist[kWarps][kSortBins];             // per-warp counts, then offsets inside the block
    uint32_t counts[kClusterBlocks][kSortBins];       // every block's bin totals of this pass
    uint32_t base[kSortBins];                         // global position of this block's first key of a bin
    uint32_t scanTmp[8];
    uint32_t localStart[kSortBins];                   // first slot of a bin in the block's staged order
    uint32_t unordered[kClusterBlocks];               // blocks whose equal top digits need the low ones
    static_assert(kThreads >= kSortBins, "thread t owns bin t");
};
static_assert(sizeof(ClusterSmem<512, 8>) <= 227 * 1024, "shared memory of one block");

__device__ __forceinline__ void clusterBarrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t mapToBlock(const void* smem, uint32_t block) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))), "r"(block));
    return a;
}
__device__ __forceinline__ void storeCluster(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void storeCluster(uint32_t addr, uint64_t v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

__device__ __forceinline__ uint64_t loadCluster64(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}

constexpr uint32_t kClusterRun = 16;   // longest run of equal top digits ordered in place

// chunk: keys a block, ceil(n / 16); magic: ceil(2^32 / chunk), so that
// (dst * magic) >> 32 = dst / chunk (exact: dst < 2^17, chunk < 2^13).
template <bool kMorton, int kThreads, int kItems>
__global__ void __launch_bounds__(kThreads) clusterSortKernel(const uint64_t* keysIn, const uint32_t* valsIn,
                                                              MortonSource ms, uint64_t* keysOut, uint32_t* valsOut,
                                                              uint32_t n, uint32_t chunk, uint32_t magic, int passes) {
    chained();
    using Smem = ClusterSmem<kThreads, kItems>;
    constexpr int kWarps = Smem::kWarps;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    Smem& s = *reinterpret_cast<Smem*>(smemRaw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t me = blockIdx.x;                 // one cluster: the block's rank in it
    const uint32_t first = me * chunk;
    const uint32_t count = first < n ? min(chunk, n - first) : 0u;
    float b6[6], inv3[3];
    if constexpr (kMorton) {
#pragma unroll
        for (int k = 0; k < 6; ++k) b6[k] = floatFromOrdered(ms.boundsOrdered[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float span = b6[3 + k] - b6[k];
            inv3[k] = (span > 1.0e-6f) ? (2097151.0f / span) : 0.0f;   // sph_gravity.cu:350-355
        }
        if (me == 0 && t < 6 && ms.boundsFloatOut != nullptr) ms.boundsFloatOut[t] = floatFromOrdered(ms.boundsOrdered[t]);
    }
    for (uint32_t k = t; k < count; k += kThreads) {
        const uint32_t i = first + k;
        if constexpr (kMorton) {
            float x, y, z;
            if (ms.xyz != nullptr) {
                const float4 q = ms.xyz[i];
                x = q.x; y = q.y; z = q.z;
            } else {
                x = __ldg(&ms.x[i]); y = __ldg(&ms.y[i]); z = __ldg(&ms.z[i]);
            }
            s.keys[0][k] = mortonCode(x, y, z, b6, inv3);
            s.vals[0][k] = i;
        } else {
            s.keys[0][k] = keysIn[i];
            s.vals[0][k] = valsIn[i];
        }
    }
    // warp w ranks the keys [w per, (w + 1) per) of the block, in order
    const uint32_t per = ((count + kWarps - 1) / kWarps + 31u) & ~31u;
    const uint32_t rounds = per >> 5;               // at most kItems
    const uint32_t warpFirst = static_cast<uint32_t>(warp) * per + static_cast<uint32_t>(lane);
    clusterBarrier();                               // every block runs before another one stores into it
    // Morton codes: the top 40 of the 63 bits first (13 an axis); equal ones
    // are rare then, and are put in order below
    int cur = 0, p = (kMorton && passes == 8) ? 3 : 0;
    bool full = p == 0;
    for (;;) {
        const int shift = 8 * p;
        for (int k = t; k < kWarps * kSortBins; k += kThreads) (&s.warpHist[0][0])[k] = 0u;
        __syncthreads();
        uint64_t key[kItems];
        uint32_t digit[kItems], rank[kItems];
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const uint32_t idx = warpFirst + static_cast<uint32_t>(k) * 32u;
            const bool ok = static_cast<uint32_t>(k) < rounds && idx < count;
            key[k] = ok ? s.keys[cur][idx] : 0ull;
            digit[k] = ok ? static_cast<uint32_t>(key[k] >> shift) & 0xFFu : 0x100u;
        }
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            rank[k] = 0u;
            if (static_cast<uint32_t>(k) < rounds) rank[k] = warpRank(digit[k], s.warpHist[warp]);
        }
        __syncthreads();
        if (t < kSortBins) {                        // per-warp offsets; block total to every block
            uint32_t total = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = s.warpHist[w][t];
                s.warpHist[w][t] = total;
                total += c;
            }
#pragma unroll
            for (int q = 0; q < kClusterBlocks; ++q) {     // neighbours first: no two blocks start with the same target
                const uint32_t to = (me + 1u + static_cast<uint32_t>(q)) & (kClusterBlocks - 1);
                storeCluster(mapToBlock(&s.counts[me][t], to), total);
            }
        }
        clusterBarrier();
        uint32_t all = 0, before = 0, own = 0;
        if (t < kSortBins) {
#pragma unroll
            for (int c = 0; c < kClusterBlocks; ++c) {
                const uint32_t v = s.counts[c][t];
                all += v;
                before += (static_cast<uint32_t>(c) < me) ? v : 0u;
                own = (static_cast<uint32_t>(c) == me) ? v : own;
            }
        }
        const uint32_t start = binExclusiveScan(all, s.scanTmp);
        const uint32_t local = binExclusiveScan(own, s.scanTmp);
        if (t < kSortBins) {
            s.localStart[t] = local;
            s.base[t] = start + before - local;     // + slot = destination
        }
        uint32_t val[kItems];
#pragma unroll
        for (int k = 0; k < kItems; ++k)
            if (digit[k] <= 0xFFu) val[k] = s.vals[cur][warpFirst + static_cast<uint32_t>(k) * 32u];
        __syncthreads();                            // keys and values are in registers: the buffer is free
        // stage in bin order, so that the stores below run along the
        // destinations (a store of scattered 8-byte keys is a packet a key)
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const uint32_t d = digit[k];
            if (d > 0xFFu) continue;
            const uint32_t slot = s.localStart[d] + s.warpHist[warp][d] + rank[k];
            s.keys[cur][slot] = key[k];
            s.vals[cur][slot] = val[k];
        }
        __syncthreads();
        const bool last = full && p + 1 == passes;
        for (uint32_t slot = t; slot < count; slot += kThreads) {
            const uint64_t kk = s.keys[cur][slot];
            const uint32_t vv = s.vals[cur][slot];
            const uint32_t dst = s.base[static_cast<uint32_t>(kk >> shift) & 0xFFu] + slot;
            if (last) {
                keysOut[dst] = kk;
                valsOut[dst] = vv;
            } else {
                const uint32_t c = __umulhi(dst, magic), at = dst - c * chunk;
                storeCluster(mapToBlock(&s.keys[cur ^ 1][at], c), kk);
                storeCluster(mapToBlock(&s.vals[cur ^ 1][at], c), vv);
            }
        }
        if (last) return;
        clusterBarrier();
        cur ^= 1;
        ++p;
        if (full || p < passes) continue;
        // Sorted by the top digits, ties in input order.  A short run of equal
        // top digits inside the block is ordered in place by its first
        // thread; a run that is longer or crosses into the next block sends
        // the whole cluster through all digits (from the present order, which
        // keeps equal codes in input order).
        bool hard = false;
        for (uint32_t slot = t; slot < count; slot += kThreads) {
            uint64_t* q = s.keys[cur] + slot;
            const uint64_t top = q[0] >> 24;
            if (slot + 1u == count) {
                if (first + count < n) hard = hard || (loadCluster64(mapToBlock(&s.keys[cur][0], me + 1u)) >> 24) == top;
                continue;
            }
            if ((slot > 0u && (q[-1] >> 24) == top) || (q[1] >> 24) != top) continue;
            uint32_t len = 2u;
            while (len <= kClusterRun && slot + len < count && (q[len] >> 24) == top) ++len;
            if (len > kClusterRun) { hard = true; continue; }
            uint32_t* v = s.vals[cur] + slot;
            for (uint32_t a = 1u; a < len; ++a) {
                const uint64_t kk = q[a];
                const uint32_t vv = v[a];
                uint32_t b = a;
                for (; b > 0u && q[b - 1u] > kk; --b) { q[b] = q[b - 1u]; v[b] = v[b - 1u]; }
                q[b] = kk;
                v[b] = vv;
            }
        }
        const uint32_t mine = __syncthreads_or(hard);
        if (t < kClusterBlocks) storeCluster(mapToBlock(&s.unordered[me], static_cast<uint32_t>(t)), mine);
        clusterBarrier();
        uint32_t any = 0;
#pragma unroll
        for (int c = 0; c < kClusterBlocks; ++c) any |= s.unordered[c];
        if (any == 0u) {
            for (uint32_t slot = t; slot < count; slot += kThreads) {
                keysOut[first + slot] = s.keys[cur][slot];
                valsOut[first + slot] = s.vals[cur][slot];
            }
            return;
        }
        full = true;
        p = 0;
    }
}

// The cluster sort's launch; *done = false where the device cannot place a
// cluster of 16 such blocks (the caller then runs the tiled passes).
template <bool kMorton, int kThreads, int kItems>
cudaError_t launchClusterSort(const uint64_t* keysIn, const uint32_t* valsIn, const MortonSource& ms, uint64_t* keysOut,
                              uint32_t* valsOut, uint32_t n, int passes, int dev, cudaStream_t stream, bool* done) {
    *done = false;
    if (dev < 0 || dev >= 64) return cudaSuccess;
    const auto kernel = clusterSortKernel<kMorton, kThreads, kItems>;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterBlocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;    // see chained()
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kClusterBlocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem<kThreads, kItems>);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    // 0: not asked yet, 1: fits, 2: does not; every thread that asks gets the same answer
    static std::atomic<int> fits[64] = {};
    int f = fits[dev].load(std::memory_order_acquire);
    if (f == 0) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(cfg.dynamicSmemBytes));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        int clusters = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();               // not a failure of the sort: the tiled passes serve it
            clusters = 0;
        }
        f = clusters > 0 ? 1 : 2;
        fits[dev].store(f, std::memory_order_release);
    }
    if (f != 1) return cudaSuccess;
    const uint32_t chunk = (n + kClusterBlocks - 1) / kClusterBlocks;
    const uint32_t magic = static_cast<uint32_t>(((1ull << 32) + chunk - 1) / chunk);
    *done = true;
    return cudaLaunchKernelEx(&cfg, kernel, keysIn, valsIn, ms, keysOut, valsOut, n, chunk, magic, passes);
}

// Block shape by keys a block: few threads keep the per-warp counts short
// while a thread has at most eight keys.
template <bool kMorton>
cudaError_t clusterSort(const uint64_t* keysIn, const uint32_t* valsIn, const MortonSource& ms, uint64_t* keysOut,
                        uint32_t* valsOut, uint32_t n, int passes, int dev, cudaStream_t stream, bool* done) {
    const auto launch = n <= 16u * 2048u ? launchClusterSort<kMorton, 256, 8> : launchClusterSort<kMorton, 512, 8>;
    return launch(keysIn, valsIn, ms, keysOut, valsOut, n, passes, dev, stream, done);
}

}  // namespace

cudaError_t launchLookbackProbe(const uint32_t* neverSet, DevStatus* status, uint32_t spinLimit, uint32_t* result,
                                cudaStream_t stream) {
    lookbackProbeKernel<<<1, 32, 0, stream>>>(neverSet, status, spinLimit, result);
    return cudaGetLastError();
}

size_t sortScratchWords(uint32_t n, uint32_t* maxTilesOut) {
    if (maxTilesOut) *maxTilesOut = sortTiles(n);
    return sortScratchWordsFor(n);
}

cudaError_t radixSortPairs(uint64_t* keysA, uint32_t* valsA, uint64_t* keysB, uint32_t* valsB, uint32_t n,
                           int endBit, uint32_t* scratch, size_t scratchWords, uint32_t maxTiles, DevStatus* status,
                           uint32_t spinLimit, KeySource src, const MortonSource* morton, bool* resultInA,
                           cudaStream_t stream) {
    *resultInA = true;
    if (n == 0) return cudaSuccess;
    const int passes = std::max(1, std::min(kSortMaxPasses, (endBit + 7) / 8));
    const int items = sortItems(n);
    const uint32_t tiles = sortTilesOf(n);
    if (tiles > maxTiles || n > kValueMask) return cudaErrorInvalidValue;
    const size_t need = kHistWords + kCounterWords + static_cast<size_t>(passes) * tiles * kSortBins;
    if (need > scratchWords) return cudaErrorInvalidValue;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    const bool mortonKeys = src == KeySource::MortonFromPositions;
    if (n >= 2u * kClusterBlocks && n <= kClusterMaxKeys) {
        bool done = false;
        uint64_t* ko = (passes & 1) ? keysB : keysA;       // where the tiled passes would leave the result
        uint32_t* vo = (passes & 1) ? valsB : valsA;
        const MortonSource none{};
        const cudaError_t ce =
            mortonKeys ? clusterSort<true>(nullptr, nullptr, *morton, ko, vo, n, passes, dev, stream, &done)
                       : clusterSort<false>(keysA, valsA, none, ko, vo, n, passes, dev, stream, &done);
        if (ce != cudaSuccess) return ce;
        if (done) {
            *resultInA = (passes & 1) == 0;
            return cudaSuccess;
        }
    }
    uint32_t* hist = scratch;
    uint32_t* counters = scratch + kHistWords;
    uint32_t* look = counters + kCounterWords;
    cudaError_t e = cudaMemsetAsync(scratch, 0, need * sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;

    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int hBlocks = static_cast<int>(std::min<uint32_t>((n + 255) / 256, static_cast<uint32_t>(sms) * 4u));
    if (mortonKeys) {
        e = launchChained(histogramKernel<true>, hBlocks, 256, stream, nullptr, *morton, keysA, valsA, n, passes, hist);
    } else {
        MortonSource none{};
        e = launchChained(histogramKernel<false>, hBlocks, 256, stream, keysA, none, nullptr, nullptr, n, passes, hist);
    }
    if (e != cudaSuccess) return e;

    const auto kernel = items == 4 ? onesweepKernel<4> : (items == 8 ? onesweepKernel<8> : onesweepKernel<12>);
    const size_t smem = items == 4 ? sizeof(SortSmem<4>) : (items == 8 ? sizeof(SortSmem<8>) : sizeof(SortSmem<12>));
    // The shared-memory attribute is set once per device and kernel; host
    // threads that sort on the same device at once may both set it (the same
    // value), and the flag is atomic, so neither reads it torn.
    static std::atomic<bool> attrSet[3][64] = {};
    std::atomic<bool>* set = attrSet[items / 4 - 1];
    if (dev < 0 || dev >= 64 || !set[dev].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) set[dev].store(true, std::memory_order_release);
    }
    uint64_t* kin = keysA;
    uint32_t* vin = valsA;
    uint64_t* kout = keysB;
    uint32_t* vout = valsB;
    for (int p = 0; p < passes; ++p) {
        e = launchChainedSmem(kernel, tiles, kSortThreads, smem, stream, kin, vin, kout, vout, n, p, hist, counters + p,
                              look + static_cast<size_t>(p) * tiles * kSortBins, status, spinLimit);
        if (e != cudaSuccess) return e;
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    *resultInA = (kin == keysA);
    return cudaSuccess;
}

}  // namespace astraea_gb300
