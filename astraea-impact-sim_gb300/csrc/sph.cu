// sph.cu -- neighbour lists, SPH pass 1 / pass 2 and the XSPH drift (sm_103a).
//
// Restates sphPass1Kernel (engine/sph_gravity.cu:645-788), sphPass2Kernel
// (:965-1287) and leapfrogDriftKernel (:1376-1489).  The engine walks the
// tree three times per step with one particle per lane; a lane's pair body
// only runs when that lane is in range, so most lanes idle.  Here:
//   * one group walk per step (buildNeighborsKernel) writes, for every
//     particle, the list of j with r_ij < max(Hs_i, Hs_j) -- a superset of the
//     pass-1, pass-2 and next-drift neighbour sets (see common.cuh);
//   * pass 1, pass 2 and the drift work on the lists, re-applying the engine's
//     exact FP32 range test, one thread per particle; in a small scene, whose
//     threads would not fill the GPU, two or four lanes share a particle's list
//     in pass 1 and the drift and add up their sums (lanesFor);
//   * neighbour data is read from packed records (pass 1: position + Hs
//     and velocity + volume m/rho in one 32-byte record; drift: position + H and
//     velocity + density; pass 2: a 96-byte record written by the EOS
//     kernel, read in three 32-byte pieces), one 256-bit load per piece
//     instead of one gather per field;
//   * a particle whose list does not fit its capacity (a lone particle with a
//     large h beside a dense body has thousands of neighbours) gets a list in a
//     shared pool, and whole warps work on those lists in the first blocks of
//     each pass: one thread over such a list holds up the launch.
// Where the pool does not hold all of those lists, each of their particles is
// served by a per-thread depth-first walk with the same superset test.
#include "kernels.h"

namespace astraea_gb300 {
namespace {

constexpr int kNbWarps = 4;
constexpr int kNbStack = 384;   // entries per warp (peak use: 80 at 1M, 88 at 16M; walkWidth keeps any tree's below it)
constexpr int kNbList = 64;
constexpr uint32_t kNbExpand = 32;   // an opened node of at most this many particles is read as its leaf range

// dirMem[k] (k = 4 [sx > 0] + 2 [sy > 0] + [sz > 0], s in {-1, 1}^3, the
// octant diagonals): the member {x, y, z, Hs} with the largest projection
// on direction s (first member on ties); undMin/undMax: the undecided nodes of one walk round
// {box min, node maxHs} / {box max}; the member positions are staged in
// undMin while dirMem is computed.
struct NbWarpSmem {
    int stack[kNbStack];
    // candidate leaves, pair-interleaved for the f32x2 pipes:
    // cand[8k..8k+7] = {xA, xB, yA, yB, zA, zB, HsA, HsB} of entries 2k, 2k+1
    float cand[8 * (kNbList / 2)];
    int candIdx[kNbList];
    float4 dirMem[8];
    float4 undMin[32];
    float4 undMax[32];
};

__device__ __forceinline__ uint32_t laneMaskLt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// One global store, issued only where `pred` holds (a predicated st.global).
__device__ __forceinline__ void storeIf(uint32_t* p, uint32_t v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.u32 [%0], %1;\n\t}"
                 :: "l"(p), "r"(v), "r"(static_cast<uint32_t>(pred)));
}

// Pool words that the long lists ask for (64 bits: their sum can pass 2^32).
__device__ __forceinline__ unsigned long long* poolUsed(const Work& w) {
    return reinterpret_cast<unsigned long long*>(&w.words[kWPoolUsed]);
}
// Lists in the pool: all the long ones, or none where they do not all have a
// place.  Which of them come first is a matter of timing, and a particle's terms
// are added in another order with a list (32 lanes) than without (one thread's
// walk).  Lists for some would gain little: a launch lasts as long as its longest
// walk (20k particles, 1 % at 2.5 times their h, a quarter of them walked 3.25
// ms, all walked 3.20, none 0.51).
__device__ __forceinline__ uint32_t heavyCount(const Work& w) {
    const uint32_t count = __ldg(&w.words[kWHeavyCount]);
    return count <= w.heavyCap && __ldg(poolUsed(w)) <= w.poolCap ? count : 0u;
}

template <int kWarps, int kMinBlocks>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) buildNeighborsKernel(Work w, uint32_t n, uint32_t numGroups,
                                                                    uint32_t* groupCounter) {
    chained();
    __shared__ NbWarpSmem smem[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    NbWarpSmem& S = smem[warp];
    unsigned long long nEntries = 0, nCand = 0;
    bool overflow = false, stackOverflow = false;
    const uint32_t maxNbr = w.maxNbr;

    if (n < 2u) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            w.nbrCount[i] = 0u;
        return;
    }
    const float4 rootR1 = __ldg(&w.node[1]);
    const int rootL = __float_as_int(rootR1.y), rootR = __float_as_int(rootR1.z);

    for (;;) {
        uint32_t g = 0;
        if (lane == 0) g = atomicAdd(groupCounter, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= numGroups) break;
        const uint32_t i = g * 32u + static_cast<uint32_t>(lane);
        const bool active = i < n;
        const int act = static_cast<int>(min(32u, n - g * 32u));
        float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
        float Hs = 0.0f;
        if (active) {
            me = __ldg(&w.leaf[i].a);
            Hs = me.w;
        }
        const float gminx = warpMinF(active ? me.x : 3.0e38f), gmaxx = warpMaxF(active ? me.x : -3.0e38f);
        const float gminy = warpMinF(active ? me.y : 3.0e38f), gmaxy = warpMaxF(active ? me.y : -3.0e38f);
        const float gminz = warpMinF(active ? me.z : 3.0e38f), gmaxz = warpMaxF(active ? me.z : -3.0e38f);
        const float gHs = warpMaxF(Hs);
        // per-direction extreme members (dirMem); member data staged in undMin
        const float cxg = 0.5f * (gminx + gmaxx), cyg = 0.5f * (gminy + gmaxy), czg = 0.5f * (gminz + gmaxz);
        S.undMin[lane] = make_float4(me.x, me.y, me.z, Hs);
        __syncwarp();
        if (lane < 8) {
            const float sx = (lane & 4) ? 1.0f : -1.0f, sy = (lane & 2) ? 1.0f : -1.0f, sz = (lane & 1) ? 1.0f : -1.0f;
            float best = -3.0e38f;
            int bi = 0;
            for (int m = 0; m < act; ++m) {
                const float4 q = S.undMin[m];
                const float pr = sx * (q.x - cxg) + sy * (q.y - cyg) + sz * (q.z - czg);
                if (pr > best) { best = pr; bi = m; }
            }
            S.dirMem[lane] = S.undMin[bi];
        }
        __syncwarp();
        if (lane == 0) { S.stack[0] = rootL; S.stack[1] = rootR; }
        // candidates form a ring of 64 entries: a round appends at most 32
        // behind the pending ones (at most 31), a flush takes the 32 oldest,
        // which start at entry 0 or 32 (cHead toggles) -- nothing is moved
        int sp = 2, cCount = 0, cHead = 0;
        uint32_t cnt = 0, rounds = 0;
        uint32_t* myList = w.nbrList + static_cast<size_t>(g) * maxNbr * 32u + static_cast<uint32_t>(lane);
        __syncwarp();

        auto putCand = [&](int slot, float x, float y, float z, float hs, int j) {
            float* b = S.cand + 8 * (slot >> 1) + (slot & 1);
            b[0] = x; b[2] = y; b[4] = z; b[6] = hs;
            S.candIdx[slot] = j;
        };
        // Superset test r < max(Hs_i, Hs_j) in plain FMA arithmetic, two
        // candidates per instruction: every pass re-tests its own radius
        // exactly, and Hs exceeds those radii by 0.9 %, far more than any
        // rounding difference.  Tests candidates 0 .. 2 pairs - 1 in order.
        const f2 X2 = pack2(me.x, me.x), Y2 = pack2(me.y, me.y), Z2 = pack2(me.z, me.z);
        auto flush = [&](int pairs) {
            if (active) {
                for (int k = cHead >> 1; k < (cHead >> 1) + pairs; ++k) {
                    const float* b = S.cand + 8 * k;
                    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(b);       // (x), (y)
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(b + 4);   // (z), (Hs)
                    const int2 jj = *reinterpret_cast<const int2*>(S.candIdx + 2 * k);
                    const f2 dx = sub2(X2, u.x), dy = sub2(Y2, u.y), dz = sub2(Z2, v.x);
                    float r2a, r2b, ha, hb;
                    unpack2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), r2a, r2b);
                    unpack2(v.y, ha, hb);
                    const float Ra = fmaxf(Hs, ha), Rb = fmaxf(Hs, hb);
                    // appends as predicated stores: no branch per candidate
                    // (a branch per hit cost 6 % of the build at 1M)
                    const bool hA = r2a < Ra * Ra && jj.x != static_cast<int>(i);
                    storeIf(myList + static_cast<size_t>(cnt) * 32u, static_cast<uint32_t>(jj.x), hA && cnt < maxNbr);
                    cnt += hA ? 1u : 0u;
                    const bool hB = r2b < Rb * Rb && jj.y != static_cast<int>(i);
                    storeIf(myList + static_cast<size_t>(cnt) * 32u, static_cast<uint32_t>(jj.y), hB && cnt < maxNbr);
                    cnt += hB ? 1u : 0u;
                }
            }
        };
        while (sp > 0) {
            if (++rounds > 2u * n + 64u) {     // only reachable on a corrupted tree
                stackOverflow = true;
                break;
            }
            const int take = min(sp, walkWidth<kNbStack>(sp));
            const int c = (lane < take) ? S.stack[sp - take + lane] : 0;
            sp -= take;
            __syncwarp();
            const bool has = lane < take && c >= -static_cast<int>(n) && c < static_cast<int>(n) - 1;
            const bool isLeaf = has && c < 0;
            bool open = false;
            int cl = 0, cr = 0;
            bool undecided = false;
            float4 bmin = make_float4(0.f, 0.f, 0.f, 0.f), bmax = bmin;
            float nodeHs = 0.0f;
            if (has && c >= 0) {
                const float4* rec = w.node + 4 * static_cast<size_t>(c);
                const float4 r1 = __ldg(&rec[1]);
                bmin = __ldg(&rec[2]);
                bmax = __ldg(&rec[3]);
                cl = __float_as_int(r1.y);
                cr = __float_as_int(r1.z);
                nodeHs = bmax.w;
                // (1) box-box distance bounds every member's point-box distance
                const float dx = fmaxf(0.0f, fmaxf(bmin.x - gmaxx, gminx - bmax.x));
                const float dy = fmaxf(0.0f, fmaxf(bmin.y - gmaxy, gminy - bmax.y));
                const float dz = fmaxf(0.0f, fmaxf(bmin.z - gmaxz, gminz - bmax.z));
                const float Rg = fmaxf(gHs, nodeHs);
                if (dx * dx + dy * dy + dz * dz <= Rg * Rg * 1.00001f) {
                    // (2) the member furthest towards the node opens it when in range;
                    // (3) otherwise the whole group decides
                    const float ux = 0.5f * (bmin.x + bmax.x) - cxg, uy = 0.5f * (bmin.y + bmax.y) - cyg,
                                uz = 0.5f * (bmin.z + bmax.z) - czg;
                    const float4 dm = S.dirMem[(ux >= 0.0f ? 4 : 0) | (uy >= 0.0f ? 2 : 0) | (uz >= 0.0f ? 1 : 0)];
                    const float R = fmaxf(dm.w, nodeHs);
                    if (pointBoxDist2(dm.x, dm.y, dm.z, bmin.x, bmin.y, bmin.z, bmax.x, bmax.y, bmax.z) <=
                        R * R * 1.00001f)
                        open = true;
                    else
                        undecided = true;
                }
            }
            const unsigned und = __ballot_sync(0xffffffffu, undecided);
            if (und) {
                const int nu = __popc(und);
                const int slot = __popc(und & laneMaskLt());
                if (undecided) {
                    S.undMin[slot] = make_float4(bmin.x, bmin.y, bmin.z, nodeHs);
                    S.undMax[slot] = make_float4(bmax.x, bmax.y, bmax.z, 0.0f);
                }
                __syncwarp();
                unsigned bits = 0u;
                for (int k = 0; k < nu; ++k) {
                    const float4 mn = S.undMin[k], mx = S.undMax[k];
                    const float R = fmaxf(Hs, mn.w);
                    const bool near = active && pointBoxDist2(me.x, me.y, me.z, mn.x, mn.y, mn.z, mx.x, mx.y, mx.z) <=
                                                    R * R * 1.00001f;
                    bits |= (__any_sync(0xffffffffu, near) ? 1u : 0u) << k;
                }
                if (undecided) open = (bits >> slot) & 1u;
                __syncwarp();
            }
            // An opened node of at most 32 particles is not descended: its
            // sorted leaf range is read whole below (one coalesced load).
            uint2 rng = make_uint2(1u, 0u);               // empty unless a small node is expanded
            if (open) {
                const uint2 r = __ldg(&w.nodeRange[c]);
                if (r.x <= r.y && r.y < n && r.y - r.x < kNbExpand) {
                    rng = r;
                    open = false;
                }
            }
            unsigned expandMask = __ballot_sync(0xffffffffu, rng.x <= rng.y);
            unsigned openMask = __ballot_sync(0xffffffffu, open);
            if (sp + 2 * __popc(openMask) > kNbStack) {
                stackOverflow = true;     // only on a corrupted tree (walkWidth)
                openMask = 0u;
                open = false;
            }
            if (open) {
                const int pos = sp + 2 * __popc(openMask & laneMaskLt());
                S.stack[pos] = cl;
                S.stack[pos + 1] = cr;
            }
            sp += 2 * __popc(openMask);
            // A leaf becomes a candidate only if it can reach the group box.
            float4 pm = make_float4(0.f, 0.f, 0.f, 0.f);
            float hsj = 0.0f;
            bool keep = false;
            if (isLeaf) {
                pm = __ldg(&w.leaf[~c].a);
                hsj = pm.w;
                const float dx = fmaxf(0.0f, fmaxf(gminx - pm.x, pm.x - gmaxx));
                const float dy = fmaxf(0.0f, fmaxf(gminy - pm.y, pm.y - gmaxy));
                const float dz = fmaxf(0.0f, fmaxf(gminz - pm.z, pm.z - gmaxz));
                const float R = fmaxf(gHs, hsj);
                keep = dx * dx + dy * dy + dz * dz <= R * R * 1.00001f;
            }
            const unsigned leafMask = __ballot_sync(0xffffffffu, keep);
            if (keep) putCand((cHead + cCount + __popc(leafMask & laneMaskLt())) & 63, pm.x, pm.y, pm.z, hsj, ~c);
            cCount += __popc(leafMask);
            nCand += __popc(leafMask);
            __syncwarp();
            if (cCount >= 32) {
                flush(16);
                __syncwarp();
                cCount -= 32;
                cHead ^= 32;
            }
            while (expandMask) {                // small opened nodes: their particles, lane by lane
                const int src = __ffs(expandMask) - 1;
                expandMask &= expandMask - 1u;
                const uint32_t first = __shfl_sync(0xffffffffu, rng.x, src);
                const uint32_t last = __shfl_sync(0xffffffffu, rng.y, src);
                for (uint32_t base = first; base <= last; base += 32u) {
                const uint32_t j = base + static_cast<uint32_t>(lane);
                bool keepJ = false;
                float4 pj = make_float4(0.f, 0.f, 0.f, 0.f);
                float hj = 0.0f;
                if (j <= last) {
                    pj = __ldg(&w.leaf[j].a);
                    hj = pj.w;
                    const float dx = fmaxf(0.0f, fmaxf(gminx - pj.x, pj.x - gmaxx));
                    const float dy = fmaxf(0.0f, fmaxf(gminy - pj.y, pj.y - gmaxy));
                    const float dz = fmaxf(0.0f, fmaxf(gminz - pj.z, pj.z - gmaxz));
                    const float R = fmaxf(gHs, hj);
                    keepJ = dx * dx + dy * dy + dz * dz <= R * R * 1.00001f;
                }
                const unsigned km = __ballot_sync(0xffffffffu, keepJ);
                if (keepJ) putCand((cHead + cCount + __popc(km & laneMaskLt())) & 63, pj.x, pj.y, pj.z, hj, static_cast<int>(j));
                cCount += __popc(km);
                nCand += __popc(km);
                __syncwarp();
                if (cCount >= 32) {
                    flush(16);
                    __syncwarp();
                    cCount -= 32;
                    cHead ^= 32;
                }
                }
            }
        }
        if (cCount & 1) {                  // odd tail: a pad entry no member can reach
            if (lane == 0) putCand(cHead + cCount, 3.0e38f, 3.0e38f, 3.0e38f, 0.0f, -1);
            __syncwarp();
        }
        flush((cCount + 1) >> 1);
        if (active) {
            w.nbrCount[i] = cnt;
            if (cnt > maxNbr) {                     // poolListsKernel goes on with it
                overflow = true;
                const unsigned long long place = atomicAdd(poolUsed(w), static_cast<unsigned long long>(cnt));
                const uint32_t slot = atomicAdd(&w.words[kWHeavyCount], 1u);
                if (slot < w.heavyCap) w.heavy[slot] = make_uint4(i, static_cast<uint32_t>(place), cnt, 0u);
            }
        }
        nEntries += cnt;
        __syncwarp();
    }
    const unsigned long long tot = __reduce_add_sync(0xffffffffu, static_cast<unsigned>(nEntries & 0xffffffffu));
    const bool anyOver = __any_sync(0xffffffffu, overflow);
    if (lane == 0) {
        atomicAdd(&w.status->counters[kCntNeighborEntries], tot);
        atomicAdd(&w.status->counters[kCntNeighborCandidates], nCand);
        if (anyOver) atomicOr(&w.status->flags, kFlagNeighborOverflow);
        if (stackOverflow) atomicOr(&w.status->flags, kFlagStackOverflow);
    }
}

// Where a list is: the k-th entry at list[k stride].
struct List {
    const uint32_t* list;
    uint32_t stride, count;
};
// Neighbour lists are group-interleaved: entry k of particle i is word
// ((i / 32) maxNbr + k) 32 + i % 32, so the 32 particles of a group read their
// k-th entries as one 128-byte row and a lane's list never shares a sector with
// another lane's.
__device__ __forceinline__ List listOf(const Work& w, uint32_t i, uint32_t count) {
    return List{w.nbrList + static_cast<size_t>(i >> 5) * w.maxNbr * 32u + (i & 31u), 32u, count};
}

// Visit every j with r_ij < max(Hs_i, Hs_j) by a depth-first tree walk: a
// particle without a list.
template <class F>
__device__ __forceinline__ void walkNeighbors(const Work& w, uint32_t i, F&& f) {
    atomicAdd(&w.status->counters[kCntFallbackWalks], 1ull);
    const float4 me = __ldg(&w.leaf[i].a);
    const float Hs = me.w;
    int stack[kTreeStack];
    int sp = 0;
    const float4 rootR1 = __ldg(&w.node[1]);
    stack[sp++] = __float_as_int(rootR1.y);
    stack[sp++] = __float_as_int(rootR1.z);
    const int nInt = static_cast<int>(w.capacity);
    uint32_t iters = 0;
    while (sp > 0) {
        const int c2 = stack[--sp];
        if (++iters > 4u * w.capacity + 64u || c2 < -nInt || c2 >= nInt - 1) {   // corrupted tree only
            atomicOr(&w.status->flags, kFlagStackOverflow);
            break;
        }
        if (c2 < 0) {
            const uint32_t j = static_cast<uint32_t>(~c2);
            if (j == i) continue;
            const float4 q = __ldg(&w.leaf[j].a);
            const float R = fmaxf(Hs, q.w);
            if (len2Engine(__fsub_rn(me.x, q.x), __fsub_rn(me.y, q.y), __fsub_rn(me.z, q.z)) < __fmul_rn(R, R)) f(j);
            continue;
        }
        const float4* rec = w.node + 4 * static_cast<size_t>(c2);
        const float4 r1 = __ldg(&rec[1]);
        const float4 bmin = __ldg(&rec[2]);
        const float4 bmax = __ldg(&rec[3]);
        const float R = fmaxf(Hs, bmax.w);
        if (pointBoxDist2(me.x, me.y, me.z, bmin.x, bmin.y, bmin.z, bmax.x, bmax.y, bmax.z) <= R * R * 1.00001f) {
            if (sp + 2 <= kTreeStack) {
                stack[sp++] = __float_as_int(r1.y);
                stack[sp++] = __float_as_int(r1.z);
            } else {
                atomicOr(&w.status->flags, kFlagStackOverflow);
            }
        }
    }
}

// List words are read once per pass and the lists (308 B per particle) do
// not fit in L1: read them without allocating in L1, which keeps L1 for the
// neighbour records.
__device__ __forceinline__ uint32_t ldWordNoL1(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ldListNoL1(const List& l, uint32_t k) {
    const uint32_t* p = l.list + static_cast<size_t>(k) * l.stride;
    return make_uint4(ldWordNoL1(p), ldWordNoL1(p + l.stride), ldWordNoL1(p + 2u * l.stride), ldWordNoL1(p + 3u * l.stride));
}

// Lane `sub` of the kLanes that share a list visits its fours sub, sub +
// kLanes, ...: each candidate's first record loaded by `load(j)` for four
// entries before any `body(j, rec)` runs, so four independent gathers are in
// flight per thread, and the next four entries loaded before those four
// bodies run.
template <int kLanes, class L, class B>
__device__ __forceinline__ void forEachListed(const List& l, uint32_t sub, L&& load, B&& body) {
    const uint32_t c = l.count;
    uint32_t k = 4u * sub;
    uint4 q = k + 4u <= c ? ldListNoL1(l, k) : make_uint4(0u, 0u, 0u, 0u);
    for (; k + 4u <= c; k += 4u * kLanes) {
        const uint32_t kn = k + 4u * kLanes;
        const uint4 next = (kn + 4u <= c) ? ldListNoL1(l, kn) : q;
        const auto r0 = load(q.x), r1 = load(q.y), r2 = load(q.z), r3 = load(q.w);
        body(q.x, r0); body(q.y, r1); body(q.z, r2); body(q.w, r3);
        q = next;
    }
    for (; k < c; ++k) {                             // the last, shorter four: one lane's
        const uint32_t j = __ldg(l.list + static_cast<size_t>(k) * l.stride);
        body(j, load(j));
    }
}

// Sum over the kLanes lanes of a particle (every lane of the warp calls it).
template <int kLanes>
__device__ __forceinline__ void sumLanes(float& v) {
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
}
template <int kLanes>
__device__ __forceinline__ void sumLanes(uint32_t& v) {
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
}

// The blocks of a pass: the first kHeavyBlocks work on the pool's lists, a warp
// per particle; then kLanes threads per particle.
constexpr uint32_t kHeavyBlocks = 38, kPassThreads = 128;
constexpr uint32_t kHeavyWarps = kHeavyBlocks * kPassThreads / 32;

// Adds a per-thread count to a device counter with one atomic per group of
// threads that reach the call together (the running threads of a warp).
__device__ __forceinline__ void addCount(DevStatus* st, int which, uint32_t v) {
    const unsigned m = __activemask();
    const unsigned tot = __reduce_add_sync(m, v);
    if ((threadIdx.x & 31u) == static_cast<unsigned>(__ffs(m) - 1))
        atomicAdd(&st->counters[which], static_cast<unsigned long long>(tot));
}

// The lists in the pool: a warp per particle walks the tree with its own radius,
// 32 nodes at a time from a stack in shared memory, and appends the particles
// inside, which are those the group walk counted (the node test has the same
// margin); a list that came out longer or was cut is not used.  Latency bound: a walk is some
// twenty rounds of two dependent loads, and there are few of them; almost always
// there is none, and the launch, chained to the kernels around it, costs less than 1 us
// (2.5 to 4 as a plain one).
constexpr int kPoolStack = 1024, kPoolWarps = 4;
__global__ void __launch_bounds__(kPoolWarps * 32) poolListsKernel(Work w, uint32_t n) {
    chained();
    __shared__ int stacks[kPoolWarps][kPoolStack];
    const uint32_t lane = threadIdx.x & 31u, total = heavyCount(w);
    int* stack = stacks[threadIdx.x >> 5];
    for (uint32_t e = blockIdx.x * kPoolWarps + (threadIdx.x >> 5); e < total; e += gridDim.x * kPoolWarps) {
        const uint4 h = w.heavy[e];
        const float4 me = __ldg(&w.leaf[h.x].a);
        uint32_t* list = w.pool + h.y;
        uint32_t cnt = 0u, rounds = 0u;
        bool whole = true;
        int sp = 1;
        if (lane == 0u) stack[0] = 0;
        __syncwarp();
        while (sp > 0) {
            if (++rounds > 2u * n) {                        // only on a corrupted tree
                whole = false;
                break;
            }
            const int take = min(sp, walkWidth<kPoolStack>(sp));
            const int c = static_cast<int>(lane) < take ? stack[sp - take + lane] : static_cast<int>(n);
            sp -= take;
            __syncwarp();
            uint32_t hitJ = 0u;
            bool hit = false, open = false;
            int cl = 0, cr = 0;
            if (c < 0 && c >= -static_cast<int>(n)) {
                hitJ = static_cast<uint32_t>(~c);
                const float4 q = __ldg(&w.leaf[hitJ].a);
                const float dx = me.x - q.x, dy = me.y - q.y, dz = me.z - q.z;
                const float R = fmaxf(me.w, q.w);
                hit = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < R * R && hitJ != h.x;
            } else if (c >= 0 && c < static_cast<int>(n) - 1) {
                const float4* rec = w.node + 4 * static_cast<size_t>(c);
                const float4 r1 = __ldg(&rec[1]), bmin = __ldg(&rec[2]), bmax = __ldg(&rec[3]);
                const float R = fmaxf(me.w, bmax.w);
                open = pointBoxDist2(me.x, me.y, me.z, bmin.x, bmin.y, bmin.z, bmax.x, bmax.y, bmax.z) <=
                       R * R * 1.00001f;
                cl = __float_as_int(r1.y);
                cr = __float_as_int(r1.z);
            }
            const unsigned hits = __ballot_sync(0xffffffffu, hit), opens = __ballot_sync(0xffffffffu, open);
            const uint32_t at = cnt + __popc(hits & laneMaskLt());
            if (hit && at < h.z) list[at] = hitJ;
            cnt += __popc(hits);
            if (sp + 2 * __popc(opens) > kPoolStack) {      // only on a corrupted tree (walkWidth)
                whole = false;
                break;
            }
            if (open) {
                const int pos = sp + 2 * __popc(opens & laneMaskLt());
                stack[pos] = cl;
                stack[pos + 1] = cr;
            }
            sp += 2 * __popc(opens);
            __syncwarp();
        }
        if (lane == 0u) {
            if (whole && cnt <= h.z && cnt != 0u) {
                w.heavy[e].z = cnt;
                w.nbrCount[h.x] = kHeavyMark;
            } else {                                        // its own walk then, as without a pool
                w.heavy[e].z = 0u;
                if (!whole) atomicOr(&w.status->flags, kFlagStackOverflow);
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- pass 1 ---
// One particle's pass 1; called by its kLanes lanes, `sub` their number.
template <int kLanes>
__device__ __forceinline__ void pass1Particle(const AstraeaParticles& p, const Work& w, uint32_t n, uint32_t i,
                                              const List& l, uint32_t sub, bool walk, bool write) {
    const F8 rec = ldg256(&w.leaf[i].a);
    const float4 me = rec.a, vr = rec.b;
    const float mi = __ldg(&p.mass[i]);
    const float hi = fmaxf(__ldg(&p.h[i]), 1.0e-6f);
    const float h0i = fmaxf(__ldg(&p.h0[i]), 1.0e-6f);
    const float rhoI = fmaxf(__ldg(&p.rho[i]), 1.0e-9f);
    const float Hi = 2.0f * hi;
    const float Hi2 = __fmul_rn(Hi, Hi);
    const float w0 = 21.0f / (2.0f * kPiF * Hi * Hi * Hi);
    const float Hi5 = (Hi * Hi) * (Hi * Hi) * Hi;
    const float gNormI = 210.0f / (kPiF * Hi5);
    const float invHi = 1.0f / Hi;
    float shep = (sub == 0u) ? (mi / rhoI) * w0 : 0.0f;
    uint32_t ngb = (sub == 0u) ? 1u : 0u;
    float nsX = 0.f, nsY = 0.f, nsZ = 0.f;
    float gXX = 0.f, gXY = 0.f, gXZ = 0.f, gYX = 0.f, gYY = 0.f, gYZ = 0.f, gZX = 0.f, gZY = 0.f, gZZ = 0.f;
    // one 32-byte record per candidate: {x, y, z, Hs}, {vx, vy, vz, m / max(rho, 1e-9)}
    auto load = [&](uint32_t j) { return ldg256(&w.leaf[j].a); };
    auto body = [&](uint32_t, const F8& rj) {
        const float4 q = rj.a;
        const float dx = __fsub_rn(me.x, q.x), dy = __fsub_rn(me.y, q.y), dz = __fsub_rn(me.z, q.z);
        const float r2 = len2Engine(dx, dy, dz);
        if (!(r2 < Hi2)) return;                       // sph_gravity.cu:713
        ++ngb;
        const float4 vj = rj.b;
        const float r = sqrtf(r2);
        const float volJ = vj.w;
        const float wij = wendlandC2I(r, Hi, invHi, w0);
        shep += volJ * wij;
        nsX -= volJ * dx * wij;
        nsY -= volJ * dy * wij;
        nsZ -= volJ * dz * wij;
        const float gc = wendlandC2GradI(r, Hi, invHi, gNormI);
        const float gx = gc * dx, gy = gc * dy, gz = gc * dz;
        const float dvx = vj.x - vr.x, dvy = vj.y - vr.y, dvz = vj.z - vr.z;
        gXX += volJ * dvx * gx; gXY += volJ * dvx * gy; gXZ += volJ * dvx * gz;
        gYX += volJ * dvy * gx; gYY += volJ * dvy * gy; gYZ += volJ * dvy * gz;
        gZX += volJ * dvz * gx; gZY += volJ * dvz * gy; gZZ += volJ * dvz * gz;
    };
    if (n >= 2u) {
        forEachListed<kLanes>(l, sub, load, body);
        if (walk && sub == 0u) walkNeighbors(w, i, [&](uint32_t j) { body(j, load(j)); });
    }
    if constexpr (kLanes > 1) {
        sumLanes<kLanes>(shep); sumLanes<kLanes>(ngb);
        sumLanes<kLanes>(nsX); sumLanes<kLanes>(nsY); sumLanes<kLanes>(nsZ);
        sumLanes<kLanes>(gXX); sumLanes<kLanes>(gXY); sumLanes<kLanes>(gXZ);
        sumLanes<kLanes>(gYX); sumLanes<kLanes>(gYY); sumLanes<kLanes>(gYZ);
        sumLanes<kLanes>(gZX); sumLanes<kLanes>(gZY); sumLanes<kLanes>(gZZ);
    }
    if (sub != 0u || !write) return;
    addCount(w.status, kCntPass1Pairs, ngb - 1u);
    p.shepardC[i] = shep;                                   // sph_gravity.cu:772-787
    const float normNs = sqrtf(nsX * nsX + nsY * nsY + nsZ * nsZ);
    float fs = fminf(1.0f, fmaxf(0.0f, 1.6f * fmaxf(1.0f - shep, normNs / hi) - 0.15f));
    if (ngb <= 2u) fs = 1.0f;
    p.surfFactor[i] = fs;
    p.divV[i] = gXX + gYY + gZZ;
    p.curlVX[i] = gZY - gYZ;
    p.curlVY[i] = gXZ - gZX;
    p.curlVZ[i] = gYX - gXY;
    const float ratio = 56.0f / static_cast<float>(ngb);
    const float factor = fminf(1.08f, fmaxf(0.92f, cbrtf(ratio)));
    const float hNew = fminf(6.0f * h0i, fmaxf(0.35f * h0i, hi * factor));
    p.h[i] = hNew;
    // records of the next drift (positions and h do not change before it)
    const float Hd = 2.0f * fmaxf(hNew, 1.0e-6f);
    w.drift[i].a = make_float4(me.x, me.y, me.z, Hd);
    w.driftAux[i] = make_float2(mi, 1.0f / Hd);
}

// 7 blocks per SM (72 registers, 4 words spilled): 250 us at 1M, 74 at 262k; 6 blocks (80)
// 267 and 82, 5 (84) 295 at 1M.
template <int kLanes>
__global__ void __launch_bounds__(kPassThreads, 7) pass1Kernel(AstraeaParticles p, Work w, uint32_t n) {
    chained();
    if (blockIdx.x < kHeavyBlocks) {
        const uint32_t lane = threadIdx.x & 31u, total = heavyCount(w);
        for (uint32_t e = blockIdx.x * (kPassThreads / 32u) + (threadIdx.x >> 5); e < total; e += kHeavyWarps) {
            const uint4 h = __ldg(&w.heavy[e]);
            if (h.z != 0u) pass1Particle<32>(p, w, n, h.x, List{w.pool + h.y, 1u, h.z}, lane, false, true);
        }
        return;
    }
    const uint32_t t = (blockIdx.x - kHeavyBlocks) * kPassThreads + threadIdx.x;
    const uint32_t i = min(t / kLanes, n - 1u), c = __ldg(&w.nbrCount[i]);
    if (kLanes == 1 && t >= n) return;
    const bool listed = c <= w.maxNbr;
    pass1Particle<kLanes>(p, w, n, i, listOf(w, i, listed ? c : 0u), t % kLanes,
                          !listed && c != kHeavyMark, t / kLanes < n && c != kHeavyMark);
}

// ---------------------------------------------------------------- pass 2 ---
// Reads the pass-2 records written by the EOS kernel (layout and derived
// values: integrate.cu, writePass2Record): one 256-bit load per 32-byte
// piece, and no per-pair division for quantities of the neighbour alone.
// kWhole: all of a record is loaded with its first piece, before the test.
struct Rec96 { F8 q01, q23, q45; };
template <int kLanes, bool kWhole>
__device__ __forceinline__ void pass2Particle(const AstraeaParticles& p, const Work& w, uint32_t n, uint32_t i,
                                              const List& l, uint32_t sub, bool walk, bool write,
                                              const uint32_t* livingFlags) {
    const float4* R = w.rec2;
    const float4 a0 = __ldg(&R[kRec2Width * static_cast<size_t>(i) + 0]);
    const float4 a1 = __ldg(&R[kRec2Width * static_cast<size_t>(i) + 1]);
    const float4 a2 = __ldg(&R[kRec2Width * static_cast<size_t>(i) + 2]);
    const float4 a4 = __ldg(&R[kRec2Width * static_cast<size_t>(i) + 4]);
    const float4 a5 = __ldg(&R[kRec2Width * static_cast<size_t>(i) + 5]);
    const float xi = a0.x, yi = a0.y, zi = a0.z, hi = a0.w, Hi = 2.0f * hi;
    const float vxi = a1.x, vyi = a1.y, vzi = a1.z, mi = a1.w;
    const float rhoI = a2.x, pOverRho2I = a2.y, csI = a2.z, fBalI = a2.w;
    const float sXXi = __ldg(&p.sXX[i]), sYYi = __ldg(&p.sYY[i]), sZZi = __ldg(&p.sZZ[i]);
    const float sXYi = __ldg(&p.sXY[i]), sXZi = __ldg(&p.sXZ[i]), sYZi = __ldg(&p.sYZ[i]);
    const int matI = __float_as_int(a4.z);
    const float Ri = a4.w;
    const float gradNormI = a5.y, invRhoI2 = a5.z, invHi = a5.w;
    const float sXXr = sXXi * invRhoI2, sYYr = sYYi * invRhoI2, sZZr = sZZi * invRhoI2;
    const float sXYr = sXYi * invRhoI2, sXZr = sXZi * invRhoI2, sYZr = sYZi * invRhoI2;

    float axS = 0.f, ayS = 0.f, azS = 0.f, drC = 0.f, drD = 0.f, duP = 0.f, duAv = 0.f, duT = 0.f, duS = 0.f;
    float gXX = 0.f, gXY = 0.f, gXZ = 0.f, gYX = 0.f, gYY = 0.f, gYZ = 0.f, gZX = 0.f, gZY = 0.f, gZZ = 0.f;
    uint32_t nPairs = 0;
    // records in 32-byte pieces: {q0, q1} for every candidate (one sector),
    // {q2, q3} and {q4, q5} for the candidates in range
    auto first = [&](uint32_t j) {
        const float4* rj = &R[kRec2Width * static_cast<size_t>(j)];
        if constexpr (kWhole)
            return Rec96{ldg256(rj), ldg256(rj + 2), ldg256(rj + 4)};
        else
            return ldg256(rj);
    };
    auto tested = [&](uint32_t j, const auto& rec) {
        F8 q01;
        if constexpr (kWhole) q01 = rec.q01; else q01 = rec;
        const float4 b0 = q01.a;
        const float dx = __fsub_rn(xi, b0.x), dy = __fsub_rn(yi, b0.y), dz = __fsub_rn(zi, b0.z);
        const float r2 = len2Engine(dx, dy, dz);
        const float hj = b0.w, Hj = 2.0f * hj;
        const float Hm = fmaxf(Hi, Hj);
        if (!(r2 < __fmul_rn(Hm, Hm))) return;          // sph_gravity.cu:1071
        ++nPairs;
        F8 q23, q45;
        if constexpr (kWhole) {
            q23 = rec.q23;
            q45 = rec.q45;
        } else {
            q23 = ldg256(&R[kRec2Width * static_cast<size_t>(j) + 2]);
            q45 = ldg256(&R[kRec2Width * static_cast<size_t>(j) + 4]);
        }
        const float4 b1 = q01.b, b2 = q23.a, b3 = q23.b, b4 = q45.a, b5 = q45.b;
        const float mj = b1.w, rhoJ = b2.x, pOverRho2J = b2.y, csJ = b2.z, fBalJ = b2.w;
        const float volJ = b5.x;
        const float dvx = vxi - b1.x, dvy = vyi - b1.y, dvz = vzi - b1.z;
        const float vDotR = dvx * dx + dvy * dy + dvz * dz;
        const float r = sqrtf(r2);
        const float gI = wendlandC2GradI(r, Hi, invHi, gradNormI), gJ = wendlandC2GradI(r, Hj, b5.w, b5.y);
        const float gb = 0.5f * (gI + gJ);
        const float gx = gb * dx, gy = gb * dy, gz = gb * dz;
        const float vDotG = dvx * gx + dvy * gy + dvz * gz;
        drC += volJ * vDotG;                               // continuity (:1114)
        // The delta-SPH and viscosity terms are evaluated for every pair in
        // range and kept by a select (the engine's conditions, the same
        // values): as branches they cost pass 2 11 % at 1M.
        {                                                  // delta-SPH diffusion (:1115-1119)
            const float rDotG = -(dx * gx + dy * gy + dz * gz);
            const float dd = r2 + 0.01f * Hi * Hi;
            const float t = drD + volJ * (2.0f * (rhoJ - rhoI) / dd) * rDotG;
            drD = (__float_as_int(b4.z) == matI) ? t : drD;
        }
        float piIJ;                                        // Monaghan AV x Balsara (:1121-1128)
        {
            const float hB = 0.5f * (hi + hj), cB = 0.5f * (csI + csJ), rB = 0.5f * (rhoI + rhoJ);
            const float muIJ = __fdividef(hB * vDotR, r2 + 0.01f * hB * hB);
            const float t = __fdividef(-1.0f * cB * muIJ + 2.0f * muIJ * muIJ, rB) * (0.5f * (fBalI + fBalJ));
            piIJ = (vDotR < 0.0f) ? t : 0.0f;
        }
        float tens = 0.0f;                                 // tensile correction (:1130-1142)
        const float Rj = b4.w;
        if (Ri + Rj > 0.0f) {
            const float Hb = 0.5f * (Hi + Hj);
            if (r < Hb) {
                const float qb = __fdividef(r, Hb), om = 1.0f - qb, om2 = om * om;
                const float fr = (om2 * om2 * (1.0f + 4.0f * qb)) * (1.0f / 0.6328125f);
                const float fr2 = fr * fr;
                tens = (Ri + Rj) * (fr2 * fr2);
            }
        }
        const float iso = -mj * ((pOverRho2I + pOverRho2J) + piIJ + tens);
        axS += iso * gx; ayS += iso * gy; azS += iso * gz;
        duP += mj * vDotG;
        duAv += 0.5f * mj * piIJ * vDotG;
        duT += 0.5f * mj * tens * vDotG;
        const float tXX = sXXr + b3.x, tYY = sYYr + b3.y, tZZ = sZZr + b3.z, tXY = sXYr + b3.w;
        const float tXZ = sXZr + b4.x, tYZ = sYZr + b4.y;
        axS += mj * (tXX * gx + tXY * gy + tXZ * gz);      // deviatoric stress (:1161-1163)
        ayS += mj * (tXY * gx + tYY * gy + tYZ * gz);
        azS += mj * (tXZ * gx + tYZ * gy + tZZ * gz);
        const float wx = -dvx, wy = -dvy, wz = -dvz;
        duS += mj * ((sXXi * wx + sXYi * wy + sXZi * wz) * gx + (sXYi * wx + sYYi * wy + sYZi * wz) * gy +
                     (sXZi * wx + sYZi * wy + sZZi * wz) * gz);
        const float gxi = gI * dx, gyi = gI * dy, gzi = gI * dz;   // velocity gradient (:1173-1179)
        gXX += volJ * wx * gxi; gXY += volJ * wx * gyi; gXZ += volJ * wx * gzi;
        gYX += volJ * wy * gxi; gYY += volJ * wy * gyi; gYZ += volJ * wy * gzi;
        gZX += volJ * wz * gxi; gZY += volJ * wz * gyi; gZZ += volJ * wz * gzi;
    };
    if (n >= 2u) {
        forEachListed<kLanes>(l, sub, first, tested);
        if (walk && sub == 0u) walkNeighbors(w, i, [&](uint32_t j) { tested(j, first(j)); });
    }
    if constexpr (kLanes > 1) {
        sumLanes<kLanes>(axS); sumLanes<kLanes>(ayS); sumLanes<kLanes>(azS);
        sumLanes<kLanes>(drC); sumLanes<kLanes>(drD);
        sumLanes<kLanes>(duP); sumLanes<kLanes>(duAv); sumLanes<kLanes>(duT); sumLanes<kLanes>(duS);
        sumLanes<kLanes>(gXX); sumLanes<kLanes>(gXY); sumLanes<kLanes>(gXZ);
        sumLanes<kLanes>(gYX); sumLanes<kLanes>(gYY); sumLanes<kLanes>(gYZ);
        sumLanes<kLanes>(gZX); sumLanes<kLanes>(gZY); sumLanes<kLanes>(gZZ);
        sumLanes<kLanes>(nPairs);
    }
    if (sub != 0u || !write) return;
    const float pI = effectivePressure(__ldg(&p.pressure[i]), __ldg(&p.phaseId[i]));   // the record's P_eff
    const float tempI = __ldg(&p.tempK[i]);
    const float damI = __ldg(&p.damage[i]);
    const float fSurf = __ldg(&p.surfFactor[i]);
    addCount(w.status, kCntPass2Pairs, nPairs);
    p.accX[i] += axS;                                          // sph_gravity.cu:1213-1218
    p.accY[i] += ayS;
    p.accZ[i] += azS;
    const float diffMask = (__ldg(&p.shepardC[i]) > 0.85f) ? (1.0f - fSurf) : 0.0f;
    p.drhoDt[i] = rhoI * drC + 0.05f * Hi * csI * diffMask * drD;
    const float duStress = invRhoI2 * duS;

    // Surface radiative cooling (sph_gravity.cu:1222-1235), in FP32: every
    // quantity stays far inside the float range (area <~1e13 m^2, T^4 <~1e20).
    const bool livingIntact = livingFlags[1] != 0u;
    const float tAmb = (livingIntact && __ldg(&p.bodyId[i]) == 0u && damI < 0.8f) ? 255.0f : 3.0f;
    const float mSi = fmaxf(mi * 1.0e24f, 1.0f);
    const float rhoSi = fmaxf(rhoI * 1.0e6f, 1.0e-3f);
    const float rP = cbrtf((3.0f * mSi) / (4.0f * kPiF * rhoSi));
    const float area = kPiF * rP * rP;
    const float T4 = tempI * tempI * tempI * tempI;
    const float Ta4 = tAmb * tAmb * tAmb * tAmb;
    const float dT4 = fmaxf(0.0f, T4 - Ta4);
    const float pRad = fSurf * 0.9f * 5.670374419e-8f * area * dT4;
    p.radPowerW[i] = pRad;
    const float duRad = -pRad / (fmaxf(mi, 1.0e-30f) * 1.0e27f);
    p.duDt[i] = pOverRho2I * duP + duAv + duT + duStress + duRad;

    // Jaumann stress rate + Grady-Kipp damage (sph_gravity.cu:1239-1286).
    const MatConst& st = c_mat[matIndex(static_cast<uint8_t>(matI))];
    if (st.muShear <= 0.0f || st.tMelt <= 0.0f) {
        p.dSXX[i] = 0.f; p.dSYY[i] = 0.f; p.dSZZ[i] = 0.f; p.dSXY[i] = 0.f; p.dSXZ[i] = 0.f; p.dSYZ[i] = 0.f;
        p.dDamageCbrtDt[i] = 0.0f;
        return;
    }
    const float tNorm = tempI / st.tMelt;
    const float soft = fmaxf(0.0f, 1.0f - tNorm * tNorm);
    const float muEff = (1.0f - damI) * st.muShear * soft;
    const float tr3 = (gXX + gYY + gZZ) * (1.0f / 3.0f);
    const float eXX = gXX - tr3, eYY = gYY - tr3, eZZ = gZZ - tr3;
    const float eXY = 0.5f * (gXY + gYX), eXZ = 0.5f * (gXZ + gZX), eYZ = 0.5f * (gYZ + gZY);
    const float rXY = 0.5f * (gXY - gYX), rXZ = 0.5f * (gXZ - gZX), rYZ = 0.5f * (gYZ - gZY);
    const float rYX = -rXY, rZX = -rXZ, rZY = -rYZ;
    p.dSXX[i] = 2.0f * muEff * eXX + 2.0f * (sXYi * rXY + sXZi * rXZ);
    p.dSYY[i] = 2.0f * muEff * eYY + 2.0f * (sXYi * rYX + sYZi * rYZ);
    p.dSZZ[i] = 2.0f * muEff * eZZ + 2.0f * (sXZi * rZX + sYZi * rZY);
    p.dSXY[i] = 2.0f * muEff * eXY + sXXi * rYX + sXZi * rYZ + sYYi * rXY + sYZi * rXZ;
    p.dSXZ[i] = 2.0f * muEff * eXZ + sXXi * rZX + sXYi * rZY + sZZi * rXZ + sYZi * rXY;
    p.dSYZ[i] = 2.0f * muEff * eYZ + sXYi * rZX + sYYi * rZY + sXZi * rYX + sZZi * rYZ;
    if (tempI < st.tMelt && damI < 1.0f) {
        const float sigmaMax = maxPrincipalStress(pI, sXXi, sYYi, sZZi, sXYi, sXZi, sYZi);
        const float stiff = fmaxf(st.bulkK + (4.0f / 3.0f) * st.muShear, 1.0e-12f);
        const float epsT = fmaxf(0.0f, sigmaMax) / stiff;
        const float epsF = fmaxf(__ldg(&p.epsFail[i]), 1.0e-8f);
        const float cCrack = fmaxf(csI, sqrtf((st.bulkK + (4.0f / 3.0f) * st.muShear) / rhoI));
        p.dDamageCbrtDt[i] = (epsT > epsF) ? (0.4f * cCrack / hi) : 0.0f;
    } else {
        p.dDamageCbrtDt[i] = 0.0f;
    }
}

// A thread a particle at every size, the terms added in list order: a warp's
// lanes sharing a list (as in pass 1 and the drift) made it 27 instead of 45 us
// at 16k, but the other order of the sums moves du/dt and drho/dt by 1e-6 of
// their norm, and the strength of iron just below its melting point amplifies an
// ulp of rho a thousandfold.  While two blocks per SM hold the scene there are
// registers to load whole records ahead (kBlocks 2, 180 registers): 16k 45.6 -> 43.0
// us, 30k 48.6 -> 45.1; beyond, four blocks (70k: 61 us, two 81).
template <int kBlocks>
__global__ void __launch_bounds__(kPassThreads, kBlocks) pass2Kernel(AstraeaParticles p, Work w, uint32_t n,
                                                              const uint32_t* livingFlags) {
    chained();
    if (blockIdx.x < kHeavyBlocks) {
        const uint32_t lane = threadIdx.x & 31u, total = heavyCount(w);
        for (uint32_t e = blockIdx.x * (kPassThreads / 32u) + (threadIdx.x >> 5); e < total; e += kHeavyWarps) {
            const uint4 h = __ldg(&w.heavy[e]);
            if (h.z != 0u) pass2Particle<32, false>(p, w, n, h.x, List{w.pool + h.y, 1u, h.z}, lane, false, true, livingFlags);
        }
        return;
    }
    const uint32_t i = (blockIdx.x - kHeavyBlocks) * kPassThreads + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = __ldg(&w.nbrCount[i]);
    const bool listed = c <= w.maxNbr;
    pass2Particle<1, kBlocks == 2>(p, w, n, i, listOf(w, i, listed ? c : 0u), 0u, !listed && c != kHeavyMark, c != kHeavyMark, livingFlags);
}

// ----------------------------------------------------------------- drift ---
// XSPH position update (sph_gravity.cu:1376-1489).  Neighbour positions come
// from the drift records (the positions before this drift), so no thread reads
// a position another thread is moving.  The position add is done in FP64.
struct DriftArgs {
    const float* dtDev;
    float dtHost;
    bool useList, toScratch;
};
template <int kLanes>
__device__ __forceinline__ void driftParticle(const AstraeaParticles& p, const Work& w, uint32_t n, uint32_t i,
                                              const List& l, uint32_t sub, bool walk, bool write, const DriftArgs& a,
                                              float (&at)[3]) {
    const float dt = (a.dtDev != nullptr) ? *a.dtDev : a.dtHost;
    const F8 rec = ldg256(&w.drift[i].a);
    const float4 me = rec.a, vr = rec.b;               // {x, y, z, H}, {vx, vy, vz, rho}
    const float Hi = me.w;
    const float invHi = __ldg(&w.driftAux[i]).y;
    const float normI = wendlandNorm(Hi);
    const float rhoI = fmaxf(vr.w, 1.0e-9f);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    uint32_t nPairs = 0;
    // one 32-byte record per candidate: {x, y, z, H}, {vx, vy, vz, rho}, and {m, 1 / H} beside it
    struct Rec { F8 r; float2 aux; };
    auto load = [&](uint32_t j) { return Rec{ldg256(&w.drift[j].a), __ldg(&w.driftAux[j])}; };
    auto body = [&](uint32_t, const Rec& both) {
        const F8& rj = both.r;
        const float4 q = rj.a;
        const float dx = __fsub_rn(me.x, q.x), dy = __fsub_rn(me.y, q.y), dz = __fsub_rn(me.z, q.z);
        const float r2 = len2Engine(dx, dy, dz);
        const float Hm = fmaxf(Hi, q.w);
        if (!(r2 < __fmul_rn(Hm, Hm))) return;
        ++nPairs;
        const float2 aj = both.aux;
        const float4 vj = rj.b;
        const float r = sqrtf(r2);
        const float normJ = (aj.y * aj.y) * (aj.y * (21.0f / (2.0f * kPiF)));
        const float wb = 0.5f * (wendlandC2I(r, Hi, invHi, normI) + wendlandC2I(r, q.w, aj.y, normJ));
        const float rb = 0.5f * (rhoI + fmaxf(vj.w, 1.0e-9f));
        const float co = __fdividef(aj.x, rb) * wb;
        sx += co * (vj.x - vr.x);
        sy += co * (vj.y - vr.y);
        sz += co * (vj.z - vr.z);
    };
    if (a.useList && n >= 2u) {
        forEachListed<kLanes>(l, sub, load, body);
        if (walk && sub == 0u) walkNeighbors(w, i, [&](uint32_t j) { body(j, load(j)); });
    }
    if constexpr (kLanes > 1) {
        sumLanes<kLanes>(sx); sumLanes<kLanes>(sy); sumLanes<kLanes>(sz); sumLanes<kLanes>(nPairs);
    }
    if (sub != 0u || !write) return;
    addCount(w.status, kCntDriftPairs, nPairs);
    const double d = static_cast<double>(dt);
    const float nx = static_cast<float>(static_cast<double>(me.x) + d * (static_cast<double>(vr.x) + 0.25 * static_cast<double>(sx)));
    const float ny = static_cast<float>(static_cast<double>(me.y) + d * (static_cast<double>(vr.y) + 0.25 * static_cast<double>(sy)));
    const float nz = static_cast<float>(static_cast<double>(me.z) + d * (static_cast<double>(vr.z) + 0.25 * static_cast<double>(sz)));
    if (a.toScratch) {
        w.driftPos[i] = make_float4(nx, ny, nz, 0.0f);
    } else {
        p.posX[i] = nx; p.posY[i] = ny; p.posZ[i] = nz;
    }
    at[0] = nx; at[1] = ny; at[2] = nz;
}

// 7 blocks per SM (72 registers, 3 words spilled): 295 us at 1M, 6 blocks 319, 8 blocks
// (64 registers, more spilled) 340.  The {m, 1 / H} pair is loaded with the
// record, before it is known whether the candidate is in range: loaded after the
// test, its latency stood in every pair (354).  With 1 / H there instead of the
// norm of H, a division less per pair.
template <int kLanes>
__global__ void __launch_bounds__(kPassThreads, 7) driftKernel(AstraeaParticles p, Work w, uint32_t n, DriftArgs a,
                                                           uint32_t* boundsWords) {
    chained();
    if (blockIdx.x < kHeavyBlocks) {
        const uint32_t lane = threadIdx.x & 31u, total = a.useList ? heavyCount(w) : 0u;
        for (uint32_t e = blockIdx.x * (kPassThreads / 32u) + (threadIdx.x >> 5); e < total; e += kHeavyWarps) {
            const uint4 h = __ldg(&w.heavy[e]);
            float at[3];
            if (h.z != 0u) driftParticle<32>(p, w, n, h.x, List{w.pool + h.y, 1u, h.z}, lane, false, true, a, at);
            if (h.z != 0u && lane == 0u && boundsWords != nullptr)
                for (int k = 0; k < 3; ++k) {
                    atomicMin(&boundsWords[kWBounds + k], orderedFromFloat(fminf(at[k], 1.0e30f)));
                    atomicMax(&boundsWords[kWBounds + 3 + k], orderedFromFloat(fmaxf(at[k], -1.0e30f)));
                }
        }
        return;
    }
    const uint32_t t = (blockIdx.x - kHeavyBlocks) * kPassThreads + threadIdx.x;
    const uint32_t i = min(t / kLanes, n - 1u), c = a.useList ? __ldg(&w.nbrCount[i]) : 0u;
    const bool listed = c <= w.maxNbr, write = t / kLanes < n && c != kHeavyMark;
    float at[3];
    if (kLanes > 1 || t < n)
        driftParticle<kLanes>(p, w, n, i, listOf(w, i, listed ? c : 0u), t % kLanes, !listed && c != kHeavyMark, write, a, at);
    if (boundsWords == nullptr) return;
    const bool own = write && t % kLanes == 0u;          // `at` was set
    const float mn[3] = {own ? at[0] : 1.0e30f, own ? at[1] : 1.0e30f, own ? at[2] : 1.0e30f};
    const float mx[3] = {own ? at[0] : -1.0e30f, own ? at[1] : -1.0e30f, own ? at[2] : -1.0e30f};
    blockBoundsToWords(mn, mx, boundsWords);
}

inline unsigned gridFor(uint32_t n, int block) { return static_cast<unsigned>((n + block - 1) / block); }

}  // namespace

// Registers of the group walk: 64 (kMinBlocks for 32 warps per SM) while there are few
// groups, 56 (36 warps) above.  Pass-1 stage call, 56 / 64 registers: 30k 107 /
// 102 us, 60k 135 / 129, 262k 305 / 300, 400k 428 / 422, 600k 599 / 599, 800k 768 / 769;
// build alone at 1M 639 / 652.
constexpr uint32_t kRoomyMax = 1u << 19;

cudaError_t launchBuildNeighbors(const Work& w, uint32_t n, int sms, LaunchAt st, int warps, bool armed) {
    if (n == 0) return cudaSuccess;
    const uint32_t groups = (n + 31u) / 32u;
    uint32_t* counter = w.words + kWNbrCounter;          // with the pool's words behind it
    cudaError_t e = armed ? cudaSuccess : cudaMemsetAsync(counter, 0, 4 * sizeof(uint32_t), st.stream);
    if (e != cudaSuccess) return e;
    using NbFn = void (*)(Work, uint32_t, uint32_t, uint32_t*);
    const int wps = (warps == 2 || warps == 8) ? warps : kNbWarps;
    const bool few = n <= kRoomyMax;
    const NbFn kernel = (wps == 2)   ? (few ? buildNeighborsKernel<2, 16> : buildNeighborsKernel<2, 0>)
                        : (wps == 8) ? (few ? buildNeighborsKernel<8, 4> : buildNeighborsKernel<8, 0>)
                                     : (few ? buildNeighborsKernel<kNbWarps, 8> : buildNeighborsKernel<kNbWarps, 0>);
    int perSm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, wps * 32, 0);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>(static_cast<uint32_t>(std::max(1, perSm) * sms),
                                               (groups + wps - 1) / wps);
    e = launchChained(kernel, blocks, static_cast<uint32_t>(wps * 32), st, w, n, groups, counter);
    if (e != cudaSuccess) return e;
    return launchChained(poolListsKernel, static_cast<uint32_t>(std::max(1, sms)), kPoolWarps * 32, st, w, n);
}

// Lanes per particle of pass 1 and the drift: as many as keep all of the launch's
// threads resident at once (the lines lie at 6 blocks an SM, where they were
// measured; the kernels have had 7 since).  Below that a
// launch lasts as long as one thread's list; above it a lane more per particle
// only adds sums and partial last fours.  Drift / pass 1 with 1, 2, 4 lanes, us:
// n = 16k 41.6 / 26.6, 25.9 / 18.4, 19.4 / 15.4 (8 lanes: 24.6 / 18.4); 32k
// 39.4 / 27.1, 27.7 / 20.5, 31.8 / 23.1; 50k 40.0 / 28.7, 30.8 / 25.1, 36.9 /
// 28.7; 70k 44.2 / 31.7, 47.9 / 34.8; 200k 87.6 / 63.0, 95.0 / 70.1.
constexpr uint32_t kPass2Wave = 2u * 128u * kTunedSms;   // threads of two blocks per SM (pass2Kernel)
constexpr uint32_t kPassWave = 6u * 128u * kTunedSms;
static uint32_t passBlocks(uint32_t n, int lanes) { return kHeavyBlocks + gridFor(n, static_cast<int>(kPassThreads) / lanes); }
static int lanesFor(uint32_t n) { return n <= kPassWave / 4u ? 4 : (n <= kPassWave / 2u ? 2 : 1); }

cudaError_t launchPass1(const AstraeaParticles& p, const Work& w, uint32_t n, LaunchAt st) {
    if (n == 0) return cudaSuccess;
    const int lanes = lanesFor(n);
    const auto kernel = lanes == 4 ? pass1Kernel<4> : (lanes == 2 ? pass1Kernel<2> : pass1Kernel<1>);
    return launchChained(kernel, passBlocks(n, lanes), kPassThreads, st, p, w, n);
}

cudaError_t launchPass2(const AstraeaParticles& p, const Work& w, uint32_t n, const uint32_t* livingFlags,
                        cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const auto kernel = n <= kPass2Wave ? pass2Kernel<2> : pass2Kernel<4>;
    return launchChained(kernel, passBlocks(n, 1), kPassThreads, st, p, w, n, livingFlags);
}

cudaError_t launchDrift(const AstraeaParticles& p, const Work& w, uint32_t n, const float* dtDev, float dtHost,
                        bool useList, bool toScratch, uint32_t* boundsWords, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int lanes = lanesFor(n);
    const auto kernel = lanes == 4 ? driftKernel<4> : (lanes == 2 ? driftKernel<2> : driftKernel<1>);
    return launchChained(kernel, passBlocks(n, lanes), kPassThreads, st, p, w, n,
                         DriftArgs{dtDev, dtHost, useList, toScratch}, boundsWords);
}

}  // namespace astraea_gb300
