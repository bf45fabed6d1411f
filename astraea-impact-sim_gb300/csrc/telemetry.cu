// telemetry.cu -- the O(N) loops of the engine's per-frame telemetry on the GPU.
//
// Replaces the host loops of Simulation::Impl::computeTelemetryFromDevice
// (engine/simulation.cpp:948-1285) and sumDeviceRadPowerW (:567-582), which
// copy 17 particle arrays to the host and walk them seven times.  Here every
// loop is a device pass that sums in FP64 and decides as the engine's FP64
// arithmetic does (see Cost), and the scalar state between passes (COMs, the
// remnant estimate) stays on the device:
//
//   pass A   totals: mass, COMs and mean velocities per body (body 0 vs the
//            rest), kinetic / potential / internal energy, momentum, angular
//            momentum, max T, max P, max damage, radiated power, and the
//            particle of lowest potential (the remnant seed)      :982-1047, 1183
//   pass B   living-body spin sums (lSpinY, I_yy)                  :1092-1111
//            + remnant iteration 0                                 :1131-1174
//   pass C   remnant iterations 1..4 (skipped once one finds nothing bound)
//   pass D   bound-planet / disk / ejecta / bound-impactor masses  :1176-1230
//
// Cost.  This GPU executes about two FP64 operations a clock on an SM (128
// FP32 ones), so the passes are bound by the number of FP64 instructions a
// particle costs, not by the 28-57 bytes it reads: at 1M, one FP64
// instruction a particle is 1.6 us.  What is in FP64 is what is summed;
// everything else avoids it:
//   * float -> double is exact on the integer pipes (toDouble);
//   * the decisions (bound? disk? inside the spin radius?) are taken in FP32
//     with a margin of 1e-5 of the compared magnitudes, some fifty times the
//     FP32 rounding of these expressions; a particle inside the margin, or
//     whose FP32 values are not finite, takes the engine's FP64 expression,
//     so every decision is the FP64 one;
//   * sums that are sums of others (totals over the bodies, momentum) are
//     formed once at the end, halves and unit factors are applied there;
//   * a warp reduces its K sums in about K FP64 adds a lane (each exchange
//     halves the values a lane carries) instead of 5 K;
//   * the last block sums the blocks' partials with a warp per slot and does
//     the divisions of the results on separate lanes.
// Sum of the seven kernels: 1M particles 959 -> 303 us, 30k 200 -> 106 us (there
// each pass is one wave of latency: loads, the reduction, the last block).
//
// Determinism: each pass is a grid-stride loop over a fixed grid, a block
// reduction in a fixed order, per-block partials in global memory, and a final
// sum over the blocks by the last block to finish (an atomic ticket; nothing
// waits), also in a fixed order: every 32nd block in a lane, then over the
// lanes.  Results are identical run to run; against
// the engine's serial loops they differ only by FP64 summation order.
//
// Scratch (partials, pass state, result) is file-scope device memory: the
// call allocates nothing, and calls must not overlap on the GPU.
#include "kernels.h"

namespace astraea_gb300 {
namespace {

constexpr int kTelThreads = 256;
constexpr int kTelMaxBlocks = 512;
constexpr int kTelSlots = 32;
constexpr double kGPsu = 6.67430e-11 * 1.0e24 * 1.0e3 * 1.0e3 / (1.0e6 * 1.0e6 * 1.0e6);   // engine/units.hpp:27

// Pass A slot layout: seven sums of body 0, the same seven of the rest, then
// 2 KE, 2 PE, IE, L and the radiated power.
enum SlotA {
    kM0 = 0, kX0, kY0, kZ0, kVx0, kVy0, kVz0,
    kM1, kX1, kY1, kZ1, kVx1, kVy1, kVz1,
    kKe2, kPe2, kIe, kLx, kLy, kLz, kRad,
    kSlotsA
};
// Remnant-pass slot layout (passes B and C); B adds two spin slots at the end.
enum SlotR { kRM = 0, kRX, kRY, kRZ, kRVx, kRVy, kRVz, kRMR2, kSpinL, kSpinI, kSlotsB };
enum SlotD { kBound = 0, kDisk, kEjecta, kImpBound, kSlotsD };

// (double)f on the integer pipes, exact for every float: a normal number's
// exponent is rebiased (127 -> 1023) and its fraction moved up 29 bits;
// subnormals are scaled by 2^24 first; infinities and NaNs take the top exponent.
__device__ __forceinline__ double toDouble(float f) {
    const uint32_t raw = __float_as_uint(f);
    const bool sub = (raw & 0x7f800000u) == 0u;
    const uint32_t u = sub ? __float_as_uint(f * 16777216.0f) : raw;     // zero stays zero
    const uint32_t mag = u & 0x7fffffffu;
    uint32_t hi = (mag >> 3) + (sub ? 0x38000000u - (24u << 20) : 0x38000000u);
    if (mag >= 0x7f800000u) hi = (mag >> 3) | 0x7ff00000u;
    if (mag == 0u) hi = 0u;
    return __hiloint2double(static_cast<int>(hi | (u & 0x80000000u)), static_cast<int>(u << 29));
}

// A double as two floats (hi + lo), so a float minus it loses nothing that
// FP32 can hold.
struct F2 { float hi, lo; };
__device__ __forceinline__ F2 split(double d) {
    const float h = static_cast<float>(d);
    return F2{h, static_cast<float>(d - toDouble(h))};
}
__device__ __forceinline__ float minus(float a, F2 b) { return (a - b.hi) - b.lo; }

// The remnant as the FP32 decisions read it, formed once by the block that
// finds it (FP64 splits in every thread would cost more than the decisions).
struct Remnant {
    F2 x, y, z, vx, vy, vz;
    float gm, rSoft, radius;
};

struct TelState {
    uint32_t ticket;            // last-block detection, reset by the last block
    uint32_t stop;              // a remnant iteration found nothing bound
    double remX, remY, remZ, remVx, remVy, remVz, remMass, remRadius;
    double x0, y0, z0, vx0, vy0, vz0;   // body-0 COM and mean velocity
    double rSoft;               // softening of the remnant's potential
    Remnant q;                  // the remnant in FP32
    F2 bx, by, bz;              // body-0 COM in FP32
};

__device__ double g_partials[kTelMaxBlocks * kTelSlots];
__device__ float g_maxA[kTelMaxBlocks * 3];         // max T, max P, max damage per block
__device__ unsigned long long g_minKey[kTelMaxBlocks];   // lowest finite potential: {ordered phi, index}
__device__ TelState g_state;
__device__ AstraeaTelemetry g_out;

// Warp sums of kCnt values: each exchange sends one half of the values a
// lane carries and adds the other half, so after five of them lane l carries
// the warp's total of value `slot` (valid says whether it carries one).
template <int kCnt, int kOff>
struct WarpSums {
    static __device__ __forceinline__ void run(double* v, int have, int& slot, bool& valid, double& out) {
        constexpr int kHalf = (kCnt + 1) / 2;
        const bool up = (threadIdx.x & kOff) != 0;
#pragma unroll
        for (int k = 0; k < kHalf; ++k) {
            const double a = v[k], b = (k + kHalf < kCnt) ? v[k + kHalf] : 0.0;
            const double other = __shfl_xor_sync(0xffffffffu, up ? a : b, kOff);
            v[k] = (up ? b : a) + other;
        }
        if (up) slot += kHalf;
        WarpSums<kHalf, kOff / 2>::run(v, up ? have - kHalf : min(have, kHalf), slot, valid, out);
    }
};
template <int kCnt>
struct WarpSums<kCnt, 0> {
    static __device__ __forceinline__ void run(double* v, int have, int&, bool& valid, double& out) {
        valid = have >= 1;
        out = v[0];
    }
};

// Sums kCnt per-thread values over the block (fixed order) and stores them
// as this block's partials.
template <int kCnt>
__device__ __forceinline__ void blockPartials(double (&v)[kCnt]) {
    static_assert(kCnt <= 32, "one value a lane after the exchanges");
    __shared__ double red[kTelThreads / 32][kCnt];
    int slot = 0;
    bool valid = false;
    double s = 0.0;
    WarpSums<kCnt, 16>::run(v, kCnt, slot, valid, s);
    if (valid) red[threadIdx.x >> 5][slot] = s;
    __syncthreads();
    if (threadIdx.x < kCnt) {
        double t = red[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < kTelThreads / 32; ++w) t += red[w][threadIdx.x];
        g_partials[blockIdx.x * kTelSlots + threadIdx.x] = t;
    }
}

// True in every thread of the block that finished last (after its partials
// are visible); that block then resets the ticket.
__device__ __forceinline__ bool lastBlock() {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&g_state.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) {
        __threadfence();
        if (threadIdx.x == 0) g_state.ticket = 0u;
    }
    return last;
}

// The blocks' partials summed per slot into tot (shared): a warp per slot,
// lane l over the blocks l, l + 32, ..., then over the lanes.
template <int kCnt>
__device__ __forceinline__ void gridTotals(double* tot) {
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < kCnt; k += kTelThreads / 32) {
        double s = 0.0;
        for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) s += __ldcg(&g_partials[b * kTelSlots + k]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) tot[k] = s;
    }
    __syncthreads();
}

// The derived members of the state, from the remnant the caller has stored
// (after a barrier): a lane each.
__device__ __forceinline__ void finishRemnant(TelState& s) {
    const int t = threadIdx.x;
    if (t < 6) (&s.q.x)[t] = split((&s.remX)[t]);
    if (t == 6) s.q.gm = static_cast<float>(kGPsu * s.remMass);
    if (t == 7) {
        s.rSoft = fmax(0.5 * s.remRadius, 0.1);
        s.q.rSoft = static_cast<float>(s.rSoft);
        s.q.radius = static_cast<float>(s.remRadius);
    }
    if (t >= 8 && t < 11) (&s.bx)[t - 8] = split((&s.x0)[t - 8]);
}

__global__ void __launch_bounds__(kTelThreads) passA(AstraeaParticles p, uint32_t n, double targetRadius) {
    chained();
    double v[kSlotsA];
#pragma unroll
    for (int k = 0; k < kSlotsA; ++k) v[k] = 0.0;
    float maxT = 0.0f, maxP = 0.0f, maxD = 0.0f;
    unsigned long long minKey = ~0ull;
    for (uint32_t i = blockIdx.x * kTelThreads + threadIdx.x; i < n; i += gridDim.x * kTelThreads) {
        const float fphi = __ldg(&p.phiGrav[i]), temp = __ldg(&p.tempK[i]), pres = __ldg(&p.pressure[i]);
        const float fw = __ldg(&p.radPowerW[i]);
        const double m = toDouble(__ldg(&p.mass[i]));
        const double x = toDouble(__ldg(&p.posX[i])), y = toDouble(__ldg(&p.posY[i])), z = toDouble(__ldg(&p.posZ[i]));
        const double vx = toDouble(__ldg(&p.velX[i])), vy = toDouble(__ldg(&p.velY[i])), vz = toDouble(__ldg(&p.velZ[i]));
        if (__ldg(&p.bodyId[i]) == 0u) {
            v[kM0] += m;
            v[kX0] += m * x; v[kY0] += m * y; v[kZ0] += m * z;
            v[kVx0] += m * vx; v[kVy0] += m * vy; v[kVz0] += m * vz;
        } else {
            v[kM1] += m;
            v[kX1] += m * x; v[kY1] += m * y; v[kZ1] += m * z;
            v[kVx1] += m * vx; v[kVy1] += m * vy; v[kVz1] += m * vz;
        }
        v[kKe2] += m * (vx * vx + vy * vy + vz * vz);
        v[kPe2] += m * toDouble(fphi);
        v[kIe] += m * toDouble(__ldg(&p.u[i]));
        v[kLx] += m * (y * vz - z * vy);
        v[kLy] += m * (z * vx - x * vz);
        v[kLz] += m * (x * vy - y * vx);
        if (isfinite(fw) && fw > 0.0f) v[kRad] += toDouble(fw);
        if (isfinite(temp)) maxT = fmaxf(maxT, temp);
        if (isfinite(pres)) maxP = fmaxf(maxP, pres);
        maxD = fmaxf(maxD, __ldg(&p.damage[i]));
        if (isfinite(fphi)) {                        // + 0: the two zeros compare equal
            const unsigned long long key = (static_cast<unsigned long long>(orderedFromFloat(fphi + 0.0f)) << 32) | i;
            minKey = key < minKey ? key : minKey;
        }
    }
    blockPartials<kSlotsA>(v);
    // maxima and the first index of the lowest potential, by warp then block
    __shared__ float smax[3][kTelThreads / 32];
    __shared__ unsigned long long skey[kTelThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    maxT = warpMaxF(maxT); maxP = warpMaxF(maxP); maxD = warpMaxF(maxD);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long k = __shfl_xor_sync(0xffffffffu, minKey, o);
        minKey = k < minKey ? k : minKey;
    }
    if (lane == 0) { smax[0][warp] = maxT; smax[1][warp] = maxP; smax[2][warp] = maxD; skey[warp] = minKey; }
    __syncthreads();
    if (threadIdx.x < 3) {
        float a = 0.0f;
#pragma unroll
        for (int k = 0; k < kTelThreads / 32; ++k) a = fmaxf(a, smax[threadIdx.x][k]);
        g_maxA[3 * blockIdx.x + threadIdx.x] = a;
    } else if (threadIdx.x == 32) {
        unsigned long long k0 = ~0ull;
#pragma unroll
        for (int k = 0; k < kTelThreads / 32; ++k) k0 = skey[k] < k0 ? skey[k] : k0;
        g_minKey[blockIdx.x] = k0;
    }
    if (!lastBlock()) return;
    __shared__ double tot[kSlotsA];
    __shared__ float sMaxAll[3];
    __shared__ uint32_t sSeed;
    gridTotals<kSlotsA>(tot);
    if (warp < 3) {
        float a = 0.0f;
        for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) a = fmaxf(a, __ldcg(&g_maxA[3 * b + warp]));
        a = warpMaxF(a);
        if (lane == 0) sMaxAll[warp] = a;
    } else if (warp == 3) {
        unsigned long long k0 = ~0ull;
        for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) {
            const unsigned long long k = __ldcg(&g_minKey[b]);
            k0 = k < k0 ? k : k0;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long k = __shfl_xor_sync(0xffffffffu, k0, o);
            k0 = k < k0 ? k : k0;
        }
        if (lane == 0) sSeed = (k0 == ~0ull) ? 0u : static_cast<uint32_t>(k0);   // :999 (no finite potential)
    }
    __syncthreads();
    AstraeaTelemetry& o = g_out;
    TelState& s = g_state;
    const double M = tot[kM0] + tot[kM1];
    // one division a lane: lanes 0..5 body 0's COM and mean velocity, 6..11
    // the rest's, 12..14 the system's COM (:1049-1074)
    __shared__ double com[15];
    if (threadIdx.x < 15) {
        const int k = threadIdx.x;
        const double num = k < 6 ? tot[kX0 + k] : (k < 12 ? tot[kX1 + k - 6] : tot[kX0 + k - 12] + tot[kX1 + k - 12]);
        const double den = k < 6 ? tot[kM0] : (k < 12 ? tot[kM1] : M);
        com[k] = den > 0.0 ? num / den : (k < 12 ? num : 0.0);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
    const uint32_t seed = sSeed;
    o.totalMassPsu = M;
    o.kineticPsu = 0.5 * tot[kKe2]; o.potentialPsu = 0.5 * tot[kPe2]; o.internalPsu = tot[kIe];
    o.angularMomentumPsu[0] = tot[kLx]; o.angularMomentumPsu[1] = tot[kLy]; o.angularMomentumPsu[2] = tot[kLz];
    o.maxTempK = sMaxAll[0]; o.maxPressureGPa = static_cast<double>(sMaxAll[1]) * 1000.0; o.maxDamage = sMaxAll[2];
    o.radiatedPowerW = tot[kRad];
    o.remnantSeedIndex = seed;
    o.massBody0Psu = tot[kM0];
    o.massOtherPsu = tot[kM1];
    for (int k = 0; k < 3; ++k) {
        o.momentumPsu[k] = tot[kVx0 + k] + tot[kVx1 + k];
        o.sysComPsu[k] = com[12 + k];
        o.comBody0Psu[k] = com[k]; o.velBody0Psu[k] = com[3 + k];
        o.comOtherPsu[k] = com[6 + k]; o.velOtherPsu[k] = com[9 + k];
        o.livingComPsu[k] = tot[kM0] > 0.0 ? com[k] : com[12 + k];
    }
    s.x0 = com[0]; s.y0 = com[1]; s.z0 = com[2]; s.vx0 = com[3]; s.vy0 = com[4]; s.vz0 = com[5];
    // remnant seed, :1121-1128
    s.remX = p.posX[seed]; s.remY = p.posY[seed]; s.remZ = p.posZ[seed];
    s.remVx = p.velX[seed]; s.remVy = p.velY[seed]; s.remVz = p.velZ[seed];
    s.remMass = fmax(tot[kM0], M * 0.5);
    s.remRadius = fmax(targetRadius, 0.25);
    s.stop = 0u;
    o.spinLPsu = 0.0;
    o.spinIPsu = 0.0;
    o.remnantIterations = 0;
    }
    __syncthreads();
    finishRemnant(s);
}

// Decisions taken in FP32 where the two sides differ by more than kMargin of
// their magnitudes (kTiny: an absolute floor far above FP32 underflow).
constexpr float kMargin = 1.0e-5f, kTiny = 1.0e-28f;
enum Verdict { kNo = 0, kYes = 1, kUnsure = 2 };
__device__ __forceinline__ Verdict less(float a, float b, float scale) {   // a < b?
    const float d = a - b, t = kMargin * scale + kTiny;
    return d < -t ? kYes : (d > t ? kNo : kUnsure);        // a NaN or infinity compares false twice
}

struct Rel { float dx, dy, dz, dvx, dvy, dvz, r2, v2, r; };
__device__ __forceinline__ Rel relative(const Remnant& q, float x, float y, float z, float vx, float vy, float vz) {
    Rel o;
    o.dx = minus(x, q.x); o.dy = minus(y, q.y); o.dz = minus(z, q.z);
    o.dvx = minus(vx, q.vx); o.dvy = minus(vy, q.vy); o.dvz = minus(vz, q.vz);
    o.r2 = o.dx * o.dx + o.dy * o.dy + o.dz * o.dz;
    o.v2 = o.dvx * o.dvx + o.dvy * o.dvy + o.dvz * o.dvz;
    o.r = sqrtf(o.r2);
    return o;
}
// v^2 / 2 < G M / max(r, rSoft), multiplied out.
__device__ __forceinline__ Verdict boundTest(const Remnant& q, const Rel& d) {
    const float lhs = 0.5f * d.v2 * fmaxf(d.r, q.rSoft);
    return less(lhs, q.gm, lhs + q.gm);
}

// The engine's FP64 specific energy (:1144-1151, :1190-1196).
static __device__ __noinline__ double energyF64(const TelState& s, double rSoft, float x, float y, float z, float vx,
                                             float vy, float vz) {
    const double dx = x - s.remX, dy = y - s.remY, dz = z - s.remZ;
    const double dvx = vx - s.remVx, dvy = vy - s.remVy, dvz = vz - s.remVz;
    const double r = sqrt(dx * dx + dy * dy + dz * dz);
    return 0.5 * (dvx * dvx + dvy * dvy + dvz * dvz) + (-kGPsu * s.remMass / fmax(r, rSoft));
}

// What a remnant pass reads of a particle; the loops load the next particle
// before they work on the current one.
struct TelIn { float x, y, z, vx, vy, vz, m; uint32_t body; };
template <bool kBody>
__device__ __forceinline__ TelIn telLoad(const AstraeaParticles& p, uint32_t i) {
    return TelIn{__ldg(&p.posX[i]), __ldg(&p.posY[i]), __ldg(&p.posZ[i]), __ldg(&p.velX[i]), __ldg(&p.velY[i]),
                 __ldg(&p.velZ[i]), __ldg(&p.mass[i]), kBody ? static_cast<uint32_t>(__ldg(&p.bodyId[i])) : 0u};
}

// Remnant iteration (:1131-1174), plus the living-body spin sums in pass B.
template <bool kWithSpin>
__global__ void __launch_bounds__(kTelThreads) passRemnant(AstraeaParticles p, uint32_t n, double targetRadius,
                                                           int living) {
    chained();
    const TelState s = g_state;                                  // written by the previous launch
    if (s.stop) return;
    constexpr int kCnt = kWithSpin ? kSlotsB : kRMR2 + 1;
    double v[kCnt];
#pragma unroll
    for (int k = 0; k < kCnt; ++k) v[k] = 0.0;
    const double rSoft = s.rSoft;
    const Remnant q = s.q;
    const double rLimSq = (1.5 * targetRadius) * (1.5 * targetRadius);
    const F2 bx = s.bx, by = s.by, bz = s.bz;
    const uint32_t stride = gridDim.x * kTelThreads, i0 = blockIdx.x * kTelThreads + threadIdx.x;
    TelIn next{};
    if (i0 < n) next = telLoad<kWithSpin>(p, i0);
    for (uint32_t i = i0; i < n; i += stride) {
        const TelIn in = next;
        if (n - i > stride) next = telLoad<kWithSpin>(p, i + stride);
        const float fx = in.x, fy = in.y, fz = in.z, fvx = in.vx, fvy = in.vy, fvz = in.vz, fm = in.m;
        bool spin = kWithSpin && living && in.body == 0u;
        const Verdict b = boundTest(q, relative(q, fx, fy, fz, fvx, fvy, fvz));
        const bool bound = b == kUnsure ? energyF64(s, rSoft, fx, fy, fz, fvx, fvy, fvz) < 0.0 : b == kYes;
        if constexpr (kWithSpin) {
            if (spin) {                                          // :1097-1111
                const float gx = minus(fx, bx), gy = minus(fy, by), gz = minus(fz, bz);
                const float g2 = gx * gx + gy * gy + gz * gz, lim = static_cast<float>(rLimSq);
                const Verdict near = less(g2, lim, g2 + lim);
                if (near == kUnsure) {
                    const double ex = fx - s.x0, ey = fy - s.y0, ez = fz - s.z0;
                    spin = ex * ex + ey * ey + ez * ez <= rLimSq;
                } else {
                    spin = near == kYes;
                }
            }
        }
        if (bound || spin) {
            const double m = toDouble(fm), x = toDouble(fx), y = toDouble(fy), z = toDouble(fz);
            const double vx = toDouble(fvx), vy = toDouble(fvy), vz = toDouble(fvz);
            if (bound) {
                const double dx = x - s.remX, dy = y - s.remY, dz = z - s.remZ;
                v[kRM] += m;
                v[kRX] += m * x; v[kRY] += m * y; v[kRZ] += m * z;
                v[kRVx] += m * vx; v[kRVy] += m * vy; v[kRVz] += m * vz;
                v[kRMR2] += m * (dx * dx + dy * dy + dz * dz);
            }
            if constexpr (kWithSpin) {
                if (spin) {
                    const double ex = x - s.x0, ez = z - s.z0, evx = vx - s.vx0, evz = vz - s.vz0;
                    v[kSpinL] += m * (ez * evx - ex * evz);
                    v[kSpinI] += m * (ex * ex + ez * ez);
                }
            }
        }
    }
    blockPartials<kCnt>(v);
    if (!lastBlock()) return;
    __shared__ double tot[kCnt];
    gridTotals<kCnt>(tot);
    if constexpr (kWithSpin) {
        if (threadIdx.x == 32) {
            g_out.spinLPsu = tot[kSpinL];
            g_out.spinIPsu = tot[kSpinI];
        }
    }
    const double nm = tot[kRM];
    if (nm > 0.0) {                                              // :1162-1173
        if (threadIdx.x < 6) (&g_state.remX)[threadIdx.x] = tot[kRX + threadIdx.x] / nm;
        if (threadIdx.x == 6) {
            g_state.remMass = nm;
            g_state.remRadius = fmax(0.5 * targetRadius, sqrt(5.0 / 3.0) * sqrt(tot[kRMR2] / nm));
            g_out.remnantIterations += 1;
        }
        __syncthreads();
        finishRemnant(g_state);
    } else if (threadIdx.x == 0) {
        g_state.stop = 1u;
    }
}

// The engine's FP64 disk test of a bound particle (:1201-1216).
static __device__ __noinline__ bool diskF64(const TelState& s, double rSoft, float x, float y, float z, float vx,
                                            float vy, float vz) {
    const double mu = kGPsu * s.remMass;
    const double dx = x - s.remX, dy = y - s.remY, dz = z - s.remZ;
    const double dvx = vx - s.remVx, dvy = vy - s.remVy, dvz = vz - s.remVz;
    const double r = sqrt(dx * dx + dy * dy + dz * dz);
    if (!(r > s.remRadius && mu > 0.0)) return false;
    const double eSpec = 0.5 * (dvx * dvx + dvy * dvy + dvz * dvz) + (-mu / fmax(r, rSoft));
    const double jx = dy * dvz - dz * dvy, jy = dz * dvx - dx * dvz, jz = dx * dvy - dy * dvx;
    const double j2 = jx * jx + jy * jy + jz * jz;
    const double ecc = sqrt(fmax(0.0, 1.0 + (2.0 * eSpec * j2) / (mu * mu)));
    return j2 / (mu * (1.0 + ecc)) > s.remRadius;
}

// The same test in FP32.  With p = j^2 / mu the engine's condition
// p / (1 + e) > R, e^2 = max(0, 1 + 2 E p / mu), squares to
// j^2 > mu R and j^2 > 2 mu R + 2 E R^2 (E the specific energy): no root, no
// division by a difference.
__device__ __forceinline__ Verdict diskTest(const Remnant& q, const Rel& d) {
    const float R = q.radius;
    if (!(q.gm > kTiny)) return kUnsure;
    const Verdict out = less(R, d.r, R + d.r);
    if (out != kYes) return out;
    const float jx = d.dy * d.dvz - d.dz * d.dvy, jy = d.dz * d.dvx - d.dx * d.dvz, jz = d.dx * d.dvy - d.dy * d.dvx;
    const float j2 = jx * jx + jy * jy + jz * jz;
    const float pot = q.gm / fmaxf(d.r, q.rSoft), R2 = R * R, muR = q.gm * R;
    const float scale = d.r2 * d.v2 + R2 * (d.v2 + 2.0f * pot) + 2.0f * muR;
    const Verdict a = less(muR, j2, scale);
    const Verdict b = less(2.0f * muR + R2 * (d.v2 - 2.0f * pot), j2, scale);
    if (a == kNo || b == kNo) return kNo;
    return (a == kYes && b == kYes) ? kYes : kUnsure;
}

// Final classification (:1176-1230).
__global__ void __launch_bounds__(kTelThreads) passClassify(AstraeaParticles p, uint32_t n) {
    chained();
    const TelState s = g_state;
    double v[kSlotsD] = {0.0, 0.0, 0.0, 0.0};
    const double rSoft = s.rSoft;
    const Remnant q = s.q;
    const uint32_t stride = gridDim.x * kTelThreads, i0 = blockIdx.x * kTelThreads + threadIdx.x;
    TelIn next{};
    if (i0 < n) next = telLoad<true>(p, i0);
    for (uint32_t i = i0; i < n; i += stride) {
        const TelIn in = next;
        if (n - i > stride) next = telLoad<true>(p, i + stride);
        const float fx = in.x, fy = in.y, fz = in.z, fvx = in.vx, fvy = in.vy, fvz = in.vz;
        const double m = toDouble(in.m);
        const Rel d = relative(q, fx, fy, fz, fvx, fvy, fvz);
        const Verdict e = boundTest(q, d);
        // a NaN energy counts as bound here and as unbound above, as in the engine
        const bool bound = e == kUnsure ? !(energyF64(s, rSoft, fx, fy, fz, fvx, fvy, fvz) >= 0.0) : e == kYes;
        bool disk = false;
        if (bound) {
            const Verdict k = diskTest(q, d);
            disk = k == kUnsure ? diskF64(s, rSoft, fx, fy, fz, fvx, fvy, fvz) : k == kYes;
        }
        if (!bound) {
            v[kEjecta] += m;
        } else {
            if (in.body != 0u) v[kImpBound] += m;
            if (disk) v[kDisk] += m;
            else v[kBound] += m;
        }
    }
    blockPartials<kSlotsD>(v);
    if (!lastBlock()) return;
    __shared__ double tot[kSlotsD];
    gridTotals<kSlotsD>(tot);
    if (threadIdx.x != 0) return;
    AstraeaTelemetry& o = g_out;
    o.boundPlanetMassPsu = tot[kBound];
    o.diskMassPsu = tot[kDisk];
    o.ejectaMassPsu = tot[kEjecta];
    o.impactorBoundMassPsu = tot[kImpBound];
    o.remnantPsu[0] = s.remX; o.remnantPsu[1] = s.remY; o.remnantPsu[2] = s.remZ;
    o.remnantVelPsu[0] = s.remVx; o.remnantVelPsu[1] = s.remVy; o.remnantVelPsu[2] = s.remVz;
    o.remnantMassPsu = s.remMass;
    o.remnantRadiusPsu = s.remRadius;
}

}  // namespace

cudaError_t launchTelemetry(const AstraeaParticles& p, uint32_t n, double targetRadiusPsu, int livingBodyPresent,
                            int sms, AstraeaTelemetry* hostOut, cudaStream_t st) {
    void* state = nullptr;                     // a ticket left by an aborted call must not survive
    cudaError_t e = cudaGetSymbolAddress(&state, g_state);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(state, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::max<uint32_t>(
        1u, std::min<uint32_t>(static_cast<uint32_t>(std::min(2 * sms, kTelMaxBlocks)),
                               (n + kTelThreads - 1) / kTelThreads));
    e = launchChained(passA, blocks, kTelThreads, st, p, n, targetRadiusPsu);
    if (e == cudaSuccess) e = launchChained(passRemnant<true>, blocks, kTelThreads, st, p, n, targetRadiusPsu, livingBodyPresent);
    for (int it = 1; it < 5 && e == cudaSuccess; ++it)
        e = launchChained(passRemnant<false>, blocks, kTelThreads, st, p, n, targetRadiusPsu, 0);
    if (e == cudaSuccess) e = launchChained(passClassify, blocks, kTelThreads, st, p, n);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyFromSymbolAsync(hostOut, g_out, sizeof(AstraeaTelemetry), 0, cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

}  // namespace astraea_gb300
