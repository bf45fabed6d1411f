// gravity.cu -- Barnes-Hut monopole gravity for sm_103a.
//
// Same interaction set as the engine kernel gravityBarnesHutKernel
// (engine/sph_gravity.cu:810-961): particles are taken in groups of 32
// consecutive sorted particles (one engine warp); every internal node reached
// is accepted as a monopole for the whole group iff every active member has
// dNode^2 < theta^2 r^2 and r^2 > 1e-20 (and, when theta^2 > 1/3, lies outside
// the node box), otherwise the group descends; leaves are evaluated
// particle-particle with eps_ij = (eps_i + eps_j)/2, monopoles with eps_i.
//
// GB300 restructuring (same sets, different schedule).  The kernel is bound by
// instruction issue (78 % of the issue slots at 262k, DRAM idle), and most
// instructions are the walk's, so the walk is built to decide a node in few:
//   * what a walk reads of a node is its two children, side by side in one
//     64-byte record of its own (pairNodesKernel): one lane opens one node and
//     has both children's COM, mass, size and reference in two loads, already
//     in the register pairs of the packed FP32 pipes; a leaf child brings its
//     particle, so a leaf is never loaded again.  32 opened nodes (64
//     children) are taken a round (the monopole walk, gravityOrderedKernel: 16
//     nodes, a child a lane), and the stack holds opened nodes only;
//   * a child is accepted when a sound lower bound on every member's distance
//     to its COM (the larger of the group-box distance and the distance to the
//     supporting plane of the group in the octant diagonal the COM lies in)
//     passes the test, and opened when the exact test of the member that lies
//     furthest in that diagonal fails; the members and planes of the eight
//     diagonals are found once a group;
//   * children neither decides wait in a ring in shared memory; 32 of them at
//     a time, one a lane, are tested exactly against every member (the monopole
//     walk: in their round, a member a lane);
//   * accepted monopoles and reached leaves are appended to two per-warp
//     interaction lists in shared memory; every 32 entries the warp evaluates
//     them with each lane summing its own particle's force from broadcast
//     shared-memory reads, two entries per instruction on the packed FP32
//     pipes (add/mul/fma.rn.f32x2) plus one rsqrt per pair;
//   * a persistent grid pulls groups from an atomic counter.
// 1M impact, theta 0.5, per group of 32: 1,600 opened nodes, 2,940 tested
// children of which 295 wait for the exact test, 51,254 interactions; the
// evaluation, at the FP32 pipes' rate, is about half of the instructions.  Launch at 1M: monopole,
// theta 0.5, 1.69 -> 1.37 ms; quadrupole, theta 0.7, 1.63 -> 1.35; 4M Plummer
// sphere, quadrupole, 9.5 -> 7.9; 60k spheres, monopole, 139 -> 120 us; of which the
// records of the children cost 0.04 ms at 1M.
#include <type_traits>

#include "kernels.h"

namespace astraea_gb300 {
namespace {

constexpr int kGravWarps = 4;
// Opened nodes per warp.  Peak use of gravityOrderedKernel / gravityKernel: 1M impact,
// theta 0.5, 133 / 156; 4M Plummer sphere, theta 0.5, 208 / 282, theta 0.1, full / 359.
// gravityKernel takes smaller rounds as it fills (walkWidth).  Without that it ran
// out at small angles, so opened nodes became monopoles: rms force error 0.62 at
// theta 0.2 on the 4M sphere, 0.023 at theta 0.1 on one of 1M (now 1.5e-5, 5.9e-6).
// It costs 30.3 -> 31.8 ms (1M) and 150 -> 163 (4M) at theta 0.2, nothing from 0.5 up.
constexpr int kGravStack = 448;
// Ring lists: a round appends up to 64 entries behind at most 31 pending ones.
// The quadrupole's monopole entries are 40 bytes: its list (and mode 3's far
// list) is emptied between a round's two halves instead.
constexpr int kGravList = 128, kGravListQ = 64;
constexpr int kGravCounts = 6;            // interactions, tests, undecided, rounds, group evaluations, bucket leaves

// Interaction lists are stored field by field (x, y, z, -G m; with the
// quadrupole, far-field mode 1, also G Q_xx, G Q_yy, G Q_zz, G Q_xy, G Q_xz,
// G Q_yz of the traceless Q = 3 S - tr(S) I; particles: x, y, z, -G m, eps / 2),
// so one 16-byte shared load yields a field of four entries as two packed
// operands, and an append computes one address.  The lists are rings: a flush
// evaluates the 32 oldest entries, which start at a multiple of 32 (the head
// advances by 32), so no entry is ever moved and the evaluation order is the
// append order.
// und is the ring of undecided children (2 parent + side in the child
// records).  memXY / memZ are the members' positions, pair-interleaved
// ({xA, xB, yA, yB}, {zA, zB}; a short group repeats its first member).
// dirPos[k] (k = 4 [x < 0] + 2 [y < 0] + [z < 0]): the member with the largest
// projection on that octant's unit diagonal (first member on ties) and, in
// .w, that projection measured from the box centre plus the margin of the
// plane test.
template <bool kQuad, bool kExpand, bool kLearned>
struct __align__(16) GravWarpSmem {
    int stack[kGravStack];
    float mlist[(kQuad ? 10 * kGravListQ : 4 * kGravList)];
    float plist[5 * kGravList];
    uint32_t und[kGravList];
    unsigned long long counts[kGravCounts];   // the warp's device counters, added up at the end
    float4 memXY[16];
    float2 memZ[16];
    float4 dirPos[8];
    float farDir[kLearned ? 28 : 4];    // mode 2's far test: the group's extent in 26 directions
    // far-field mode 3 only; last, and whole float4s, so the arrays above
    // keep the 16-byte alignment of their vector loads in every variant
    float4 flist4[kExpand ? 10 * kGravListQ / 4 : 1];    // far nodes of the group expansion (mlist layout)
    float4 facc4[kExpand ? 5 : 1];                      // the group's expansion coefficients (see farTaylor)
};
// the vector loads of the lists and members (16 bytes)
template <bool kQuad, bool kExpand, bool kLearned>
constexpr bool gravSmemAligned() {
    using S = GravWarpSmem<kQuad, kExpand, kLearned>;
    return offsetof(S, mlist) % 16 == 0 && offsetof(S, plist) % 16 == 0 && offsetof(S, memXY) % 16 == 0 && offsetof(S, memZ) % 8 == 0 &&
           offsetof(S, dirPos) % 16 == 0 &&
           offsetof(S, flist4) % 16 == 0 && offsetof(S, facc4) % 16 == 0 && sizeof(S) % 16 == 0;
}
static_assert(gravSmemAligned<false, false, false>() && gravSmemAligned<true, false, false>() &&
              gravSmemAligned<true, true, false>() && gravSmemAligned<false, false, true>(),
              "gravity shared-memory layout must keep 16-byte alignment");

__device__ __forceinline__ uint32_t laneMaskLt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// rsqrtf for arguments that are not subnormal (softened square distances are
// at least 6.4e-13): the same values without its scaling of subnormals, three
// instructions more each.
__device__ __forceinline__ float rsqrtNormal(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ f2 rsqrt2(f2 v) {
    float a, b;
    unpack2(v, a, b);
    return pack2(rsqrtNormal(a), rsqrtNormal(b));
}

struct Accum2 {
    f2 ax, ay, az, phi;   // two partial sums each (even / odd entries)
};

// Monopole terms: f = -G m / (r^2 + eps_i^2 + 1e-20)^(3/2) (sph_gravity.cu:935-942)
// of entries first .. first + count - 1 (a multiple of four) of a list of
// kRing-entry fields, two entries per instruction.  E2 = packed
// eps_i^2 + 1e-20 (eps >= 8e-7, so 1e-20 is below half an ulp of eps^2).
// kQuad adds the quadrupole field of the node, r = x_i - COM, with the same
// softened 1/r:  a += G [Q r / r^5 - 5/2 (r.Q.r) r / r^7],
//                phi -= G (r.Q.r) / (2 r^5).
// kLast: the softening is added to the complete r^2 (gravityOrderedKernel).
template <bool kQuad, int kRing, bool kLast = false>
__device__ __forceinline__ void evalMonopoles2(const float* list, int first, int count, f2 X, f2 Y, f2 Z, f2 E2,
                                               Accum2& a) {
    const f2 kHalfNeg = pack2(-0.5f, -0.5f), kFiveHalvesNeg = pack2(-2.5f, -2.5f);
    auto field = [&](int k, int i) { return *reinterpret_cast<const ulonglong2*>(list + kRing * k + i); };
#pragma unroll 1
    for (int i = first; i < first + count; i += 4) {
        const ulonglong2 x = field(0, i), y = field(1, i), z = field(2, i), g = field(3, i);
        ulonglong2 q[6];
        if constexpr (kQuad) {
#pragma unroll
            for (int k = 0; k < 6; ++k) q[k] = field(4 + k, i);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            auto half = [&](const ulonglong2& v) { return h == 0 ? v.x : v.y; };
            const f2 gm = half(g);
            const f2 dx = sub2(X, half(x)), dy = sub2(Y, half(y)), dz = sub2(Z, half(z));
            const f2 inv = kLast ? rsqrt2(add2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), E2))
                                 : rsqrt2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, E2))));
            const f2 inv2 = mul2(inv, inv);
            const f2 inv3 = mul2(inv2, inv);
            const f2 f = mul2(gm, inv3);
            a.ax = fma2(f, dx, a.ax);
            a.ay = fma2(f, dy, a.ay);
            a.az = fma2(f, dz, a.az);
            a.phi = fma2(gm, inv, a.phi);
            if constexpr (kQuad) {
                const f2 xx = half(q[0]), yy = half(q[1]), zz = half(q[2]), xy = half(q[3]), xz = half(q[4]),
                         yz = half(q[5]);
                const f2 qr0 = fma2(xz, dz, fma2(xy, dy, mul2(xx, dx)));
                const f2 qr1 = fma2(yz, dz, fma2(yy, dy, mul2(xy, dx)));
                const f2 qr2 = fma2(zz, dz, fma2(yz, dy, mul2(xz, dx)));
                const f2 rqr = fma2(dz, qr2, fma2(dy, qr1, mul2(dx, qr0)));
                const f2 i5 = mul2(inv3, inv2);
                const f2 t = mul2(mul2(rqr, mul2(i5, inv2)), kFiveHalvesNeg);
                a.ax = fma2(t, dx, fma2(qr0, i5, a.ax));
                a.ay = fma2(t, dy, fma2(qr1, i5, a.ay));
                a.az = fma2(t, dz, fma2(qr2, i5, a.az));
                a.phi = fma2(mul2(rqr, i5), kHalfNeg, a.phi);
            }
        }
    }
}

// Particle-particle terms with eps_ij = (eps_i + eps_j)/2 (sph_gravity.cu:875-889).
// The list includes the particle itself; its term adds exactly zero force
// (dx = dy = dz = 0) and a potential the caller subtracts again.
template <int kRing = kGravList, bool kLast = false>
__device__ __forceinline__ void evalParticles2(const float* list, int first, int count, f2 X, f2 Y, f2 Z, f2 HE,
                                               Accum2& a) {
    auto field = [&](int k, int i) { return *reinterpret_cast<const ulonglong2*>(list + kRing * k + i); };
#pragma unroll 1
    for (int i = first; i < first + count; i += 4) {
        const ulonglong2 x = field(0, i), y = field(1, i), z = field(2, i), g = field(3, i), e = field(4, i);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            auto half = [&](const ulonglong2& v) { return h == 0 ? v.x : v.y; };
            const f2 gm = half(g);
            const f2 dx = sub2(X, half(x)), dy = sub2(Y, half(y)), dz = sub2(Z, half(z));
            const f2 eij = add2(HE, half(e));
            const f2 inv = kLast ? rsqrt2(fma2(eij, eij, fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)))))
                                 : rsqrt2(fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, mul2(eij, eij)))));
            const f2 f = mul2(gm, mul2(inv, mul2(inv, inv)));
            a.ax = fma2(f, dx, a.ax);
            a.ay = fma2(f, dy, a.ay);
            a.az = fma2(f, dz, a.az);
            a.phi = fma2(gm, inv, a.phi);
        }
    }
}

// Store entry `slot` of a particle list.
template <int kRing = kGravList>
__device__ __forceinline__ void putParticle(float* list, int slot, float x, float y, float z, float gm, float halfEps) {
    float* b = list + slot;
    b[0] = x; b[kRing] = y; b[2 * kRing] = z; b[3 * kRing] = gm; b[4 * kRing] = halfEps;
}

// Monopole entry of a list; with kQuad also its six quadrupole terms.
template <bool kQuad, int kRing>
__device__ __forceinline__ void putMono(float* list, int slot, const float (&e)[10]) {
    float* b = list + slot;
#pragma unroll
    for (int k = 0; k < (kQuad ? 10 : 4); ++k) b[kRing * k] = e[k];
}
template <bool kQuad, int kRing>
__device__ __forceinline__ void getMono(const float* list, int slot, float (&e)[10]) {
    const float* b = list + slot;
#pragma unroll
    for (int k = 0; k < (kQuad ? 10 : 4); ++k) e[k] = b[kRing * k];
}

// Far-field mode 3: the field of a far node about the group centre c, to
// second order in d = x_i - c.  With r = c - COM, s^2 = r^2 + eps_g^2 (Plummer
// softening with the group's mean eps^2), GM = G m:
//   phi(c) = -GM/s - (r.Q.r)/(2 s^5),   a(c) = -GM r/s^3 + [Q r/s^5 - 5/2 (r.Q.r) r/s^7]
// (monopole + quadrupole, Q = G (3S - tr S I), the expression of the member
// evaluation), and the monopole's derivatives
//   J_ij = da_i/dx_j = -GM (d_ij/s^3 - 3 r_i r_j/s^5)
//   H_ijk = dJ_ij/dx_k = -GM (-3 (d_ij r_k + d_ik r_j + d_jk r_i)/s^5 + 15 r_i r_j r_k/s^7).
// Coefficients (20): phi, a (3), J xx yy zz xy xz yz (6), H xxx yyy zzz xxy
// xxz xyy yyz xzz yzz xyz (10).  A member then takes
//   a_i = a + J d + 1/2 H:dd,   phi_i = phi - a.d - 1/2 d.J.d.
__device__ __forceinline__ void farTaylor(const float (&e)[10], float cx, float cy, float cz, float epsG2,
                                          float (&t)[20]) {
    const float rx = cx - e[0], ry = cy - e[1], rz = cz - e[2];
    const float s2 = rx * rx + ry * ry + rz * rz + epsG2;
    const float is = rsqrtNormal(s2), is2 = is * is, is3 = is * is2, is5 = is3 * is2, is7 = is5 * is2;
    const float gm = -e[3];                       // e[3] = -G m
    // quadrupole part of phi and a
    const float q0 = e[4] * rx + e[7] * ry + e[8] * rz;
    const float q1 = e[7] * rx + e[5] * ry + e[9] * rz;
    const float q2 = e[8] * rx + e[9] * ry + e[6] * rz;
    const float rqr = rx * q0 + ry * q1 + rz * q2;
    const float tq = -2.5f * rqr * is7;
    t[0] = -gm * is - 0.5f * rqr * is5;
    t[1] = -gm * is3 * rx + q0 * is5 + tq * rx;
    t[2] = -gm * is3 * ry + q1 * is5 + tq * ry;
    t[3] = -gm * is3 * rz + q2 * is5 + tq * rz;
    const float a3 = -gm * is3, b5 = 3.0f * gm * is5;   // J = a3 I + b5 r r^T
    t[4] = a3 + b5 * rx * rx; t[5] = a3 + b5 * ry * ry; t[6] = a3 + b5 * rz * rz;
    t[7] = b5 * rx * ry; t[8] = b5 * rx * rz; t[9] = b5 * ry * rz;
    const float c5 = 3.0f * gm * is5, c7 = -15.0f * gm * is7;   // H = c5 (sym d r) + c7 r r r
    t[10] = 3.0f * c5 * rx + c7 * rx * rx * rx;          // xxx
    t[11] = 3.0f * c5 * ry + c7 * ry * ry * ry;          // yyy
    t[12] = 3.0f * c5 * rz + c7 * rz * rz * rz;          // zzz
    t[13] = c5 * ry + c7 * rx * rx * ry;                  // xxy
    t[14] = c5 * rz + c7 * rx * rx * rz;                  // xxz
    t[15] = c5 * rx + c7 * rx * ry * ry;                  // xyy
    t[16] = c5 * rz + c7 * ry * ry * rz;                  // yyz
    t[17] = c5 * rx + c7 * rx * rz * rz;                  // xzz
    t[18] = c5 * ry + c7 * ry * rz * rz;                  // yzz
    t[19] = c7 * rx * ry * rz;                            // xyz
}

// 1 / |s| for a direction s in {-1, 0, 1}^3 with nz non-zero components.
__device__ __forceinline__ float invDirNorm(int nz) { return nz == 3 ? 0.57735027f : (nz == 2 ? 0.70710678f : 1.0f); }

// Extreme member of each octant diagonal (GravWarpSmem::dirPos): lanes 4 k ..
// 4 k + 3 search diagonal k, every fourth member each.
__device__ __forceinline__ void extremeMembers(float4* dirPos, float xi, float yi, float zi, float cx, float cy, float cz,
                                               float slack, int act, int lane) {
    const int k = lane >> 2;
    const float sx = (k & 4) ? -1.0f : 1.0f, sy = (k & 2) ? -1.0f : 1.0f, sz = (k & 1) ? -1.0f : 1.0f;
    float best = -3.0e38f;
    int bi = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int m = 4 * q + (lane & 3);
        const float px = __shfl_sync(0xffffffffu, xi, m), py = __shfl_sync(0xffffffffu, yi, m),
                    pz = __shfl_sync(0xffffffffu, zi, m);
        const float pr = (sx * (px - cx) + sy * (py - cy) + sz * (pz - cz)) * 0.57735027f;
        if (m < act && pr > best) { best = pr; bi = m; }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    const float px = __shfl_sync(0xffffffffu, xi, bi), py = __shfl_sync(0xffffffffu, yi, bi),
                pz = __shfl_sync(0xffffffffu, zi, bi);
    if ((lane & 3) == 0) dirPos[k] = make_float4(px, py, pz, best + slack);
}

// One child: COM, -G m, dNode and index of an internal node; position, -G m,
// half the softening length and ~j of leaf j (mode 3: the particle count, and
// whether it is a right child).
struct Child { float x, y, z, gm, w; int ref; uint32_t cnt = 1u; bool right = false; };

// A node's children (layout: pairNodesKernel) as packed operands.
struct PairRec { f2 x, y, z, gm, w; int refA, refB; float farA, farB; uint32_t cntA, cntB; };
template <bool kFar>                     // with the box and count fields
__device__ __forceinline__ PairRec loadPair(const float4* p) {
    PairRec r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.x), "=l"(r.y), "=l"(r.z), "=l"(r.gm) : "l"(p));
    f2 refs, fars = 0ull, cnts = 0ull;
    if (kFar)
        asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.w), "=l"(refs), "=l"(fars), "=l"(cnts) : "l"(p + 2));
    else
        asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(r.w), "=l"(refs) : "l"(p + 2));
    float a, b;
    unpack2(refs, a, b);
    r.refA = __float_as_int(a);
    r.refB = __float_as_int(b);
    unpack2(fars, r.farA, r.farB);
    unpack2(cnts, a, b);
    r.cntA = __float_as_uint(a);
    r.cntB = __float_as_uint(b);
    return r;
}

// The pair record of every internal node p: {xA, xB, yA, yB} {zA, zB, gmA, gmB}
// {wA, wB, refA, refB} {far^2 A, B, count A, B}, A the left and B the right
// child: COM, -G m, dNode and the reference of an internal child, position,
// -G m, half the softening length and ~j of a leaf j; far^2 (furthest corner
// of the box) and the particle count of an internal child, which for the left
// child c ends at sorted particle c, for the right child begins there.
// dNode is the root of the refit's rounded
// square, so dNode * dNode rounds to that square again.  Written by every
// gravity call from the node and leaf records it finds.  Bound by the memory
// system: ~180 bytes read and written a node, most of it still in L2 from the
// refit; 38 us at 1M, where it saves the gravity walk 350.
__global__ void __launch_bounds__(256) pairNodesKernel(Work w, uint32_t n) {
    chained();
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0u) w.words[kWGroupCounter] = 0u;
    if (p + 1u >= n) return;
    const float4 r1 = __ldg(&w.node[4 * static_cast<size_t>(p) + 1]);
    float v[2][5], farC[2] = {0.0f, 0.0f};
    uint32_t cnt[2] = {1u, 1u};
    int ref[2] = {__float_as_int(r1.y), __float_as_int(r1.z)};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int c = ref[s];
        if (c >= 0 && c < static_cast<int>(n) - 1) {
            const float4 a = __ldg(&w.node[4 * static_cast<size_t>(c)]);
            const float4 b = __ldg(&w.node[4 * static_cast<size_t>(c) + 1]);
            v[s][0] = a.x; v[s][1] = a.y; v[s][2] = a.z; v[s][3] = -kGPsuF * a.w; v[s][4] = __fsqrt_rn(b.x);
            farC[s] = b.w;
            const uint2 r = __ldg(&w.nodeRange[c]);
            cnt[s] = r.y - r.x + 1u;
        } else {                                    // a leaf; out of range only in a corrupted tree
            const uint32_t j = min(static_cast<uint32_t>(~c), n - 1u);
            const float4 a = __ldg(&w.leaf[j].a);
            const float4 b = __ldg(&w.leafAux[j]);
            v[s][0] = a.x; v[s][1] = a.y; v[s][2] = a.z; v[s][3] = -kGPsuF * b.w; v[s][4] = 0.5f * b.y;
            ref[s] = ~static_cast<int>(j);
        }
    }
    float4* o = w.pair + 4 * static_cast<size_t>(p);
    o[0] = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
    o[1] = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
    o[2] = make_float4(v[0][4], v[1][4], __int_as_float(ref[0]), __int_as_float(ref[1]));
    o[3] = make_float4(farC[0], farC[1], __uint_as_float(cnt[0]), __uint_as_float(cnt[1]));
}

// kWarpsPerSm: the resident warps the registers are bounded for (72, 80 and 96
// registers).  At 1M: quadrupole, theta 0.7, 24 warps 1.36 ms, 20 1.44 (4M Plummer
// sphere 7.94, 28 with spills 8.08); expansion, theta 0.7, 20 warps 1.32, 16 1.46, 24
// (spills) 1.37; learned, the walk alone, 28 warps 1.37, 24 1.42, 20 1.42, 32 1.46.
template <bool kQuad, bool kExpand>
constexpr int kWarpsPerSm = kExpand ? 20 : (kQuad ? 24 : 28);
template <int kWarps, bool kInside, bool kQuad, bool kLearned, bool kExpand = false>
__global__ void __launch_bounds__(kWarps * 32, kWarpsPerSm<kQuad, kExpand> / kWarps) gravityKernel(AstraeaParticles p, Work w, uint32_t n,
                                                                 float theta2, uint32_t numGroups,
                                                                 uint32_t* groupCounter, FarCapture ff) {
    chained();
    static_assert(!kExpand || kQuad, "the group expansion is a quadrupole mode");
    constexpr int kMRing = kQuad ? kGravListQ : kGravList;
    __shared__ GravWarpSmem<kQuad, kExpand, kLearned> smem[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    GravWarpSmem<kQuad, kExpand, kLearned>& S = smem[warp];
    int spPeak = 0;
    bool overflowed = false;
    if (lane < kGravCounts) S.counts[lane] = 0ull;

    if (w.runIf != nullptr && *w.runIf == 0u) return;   // the gate of the learned mode passed
    if (n == 1u) {                                   // sph_gravity.cu:824-832
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            p.accX[0] = 0.0f; p.accY[0] = 0.0f; p.accZ[0] = 0.0f; p.phiGrav[0] = 0.0f;
        }
        return;
    }
    for (;;) {
        uint32_t g = 0;
        if (lane == 0) g = atomicAdd(groupCounter, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= numGroups) break;
        const uint32_t i = g * 32u + static_cast<uint32_t>(lane);
        const bool active = i < n;                  // active members are lanes 0 .. act-1
        const int act = static_cast<int>(min(32u, n - g * 32u));
        float4 me = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float epsI = 0.8e-6f;
        if (active) {
            me = __ldg(&w.leaf[i].a);
            const float4 aux = __ldg(&w.leafAux[i]);
            epsI = aux.y;
            me.w = aux.w;                                // the mass
        }
        const float xi = me.x, yi = me.y, zi = me.z;
        const float epsI2 = epsI * epsI + 1.0e-20f;
        const float gminx = warpMinF(active ? xi : 3.0e38f), gmaxx = warpMaxF(active ? xi : -3.0e38f);
        const float gminy = warpMinF(active ? yi : 3.0e38f), gmaxy = warpMaxF(active ? yi : -3.0e38f);
        const float gminz = warpMinF(active ? zi : 3.0e38f), gmaxz = warpMaxF(active ? zi : -3.0e38f);
        const float gExt = (gmaxx - gminx) + (gmaxy - gminy) + (gmaxz - gminz);
        // c: the box centre; hx, hy, hz: its half sides.  Rounding of the box
        // term max(|u| - h, 0): relative 1.2e-5 of it at most where |u| is
        // under a hundred times |u| - h, else under 1.3e-7 of h; the sides
        // carry 1e-6 of the group's extent and the squared bound 1e-4.
        const float cx = 0.5f * (gminx + gmaxx), cy = 0.5f * (gminy + gmaxy), cz = 0.5f * (gminz + gmaxz);
        const float slack = 1.0e-6f * gExt;
        const float hx = fmaxf(gmaxx - cx, cx - gminx) + slack, hy = fmaxf(gmaxy - cy, cy - gminy) + slack,
                    hz = fmaxf(gmaxz - cz, cz - gminz) + slack;
        const f2 CX = pack2(cx, cx), CY = pack2(cy, cy), CZ = pack2(cz, cz);
        const bool emitFar = kLearned && (g % ff.groupStride) == 0u;
        if (kLearned && lane == 0) ff.groups[g] = make_float4(cx, cy, cz, gExt);

        extremeMembers(S.dirPos, xi, yi, zi, cx, cy, cz, slack, act, lane);
        {
            // every lane shuffles (also those that keep their own position)
            const float fx = __shfl_sync(0xffffffffu, xi, 0), fy = __shfl_sync(0xffffffffu, yi, 0),
                        fz = __shfl_sync(0xffffffffu, zi, 0);
            float* xy = reinterpret_cast<float*>(&S.memXY[lane >> 1]) + (lane & 1);
            xy[0] = active ? xi : fx;
            xy[2] = active ? yi : fy;
            reinterpret_cast<float*>(&S.memZ[lane >> 1])[lane & 1] = active ? zi : fz;
        }
        if (kLearned) {                          // projections on s / |s|, s in {-1, 0, 1}^3
            const float sx = static_cast<float>(lane / 9 - 1), sy = static_cast<float>((lane / 3) % 3 - 1),
                        sz = static_cast<float>(lane % 3 - 1);
            const float inv = invDirNorm(static_cast<int>(fabsf(sx) + fabsf(sy) + fabsf(sz)));
            float best = -3.0e38f;
            for (int m = 0; m < act; ++m) {
                const float px = __shfl_sync(0xffffffffu, xi, m), py = __shfl_sync(0xffffffffu, yi, m),
                            pz = __shfl_sync(0xffffffffu, zi, m);
                best = fmaxf(best, (sx * (px - cx) + sy * (py - cy) + sz * (pz - cz)) * inv);
            }
            if (lane < 27) S.farDir[lane] = best;
        }
        if (lane == 0) S.stack[0] = 0;   // the root is opened by every group
        int sp = 1, mCount = 0, pCount = 0, uCount = 0, fCount = 0;
        int mHead = 0, pHead = 0, uHead = 0;   // first pending entry of each ring
        uint32_t rounds = 0, entries = 0, tests = 0, undecidedTests = 0, groupEvals = 0, bucketLeaves = 0;
        // group expansion: the group's radius about its box centre (IEEE
        // operations, so the far decision is reproducible) and mean eps^2
        float rg2 = 0.0f, epsG2 = 0.0f;
        if (kExpand) {
            rg2 = warpMaxF(active ? len2Exact(__fsub_rn(xi, cx), __fsub_rn(yi, cy), __fsub_rn(zi, cz)) : 0.0f);
            epsG2 = warpSumF(active ? epsI * epsI : 0.0f) / static_cast<float>(act);
            if (lane < 20) reinterpret_cast<float*>(S.facc4)[lane] = 0.0f;
        }
        const f2 X = pack2(xi, xi), Y = pack2(yi, yi), Z = pack2(zi, zi);
        const f2 E2 = pack2(epsI2, epsI2), HE = pack2(0.5f * epsI, 0.5f * epsI);
        Accum2 acc{0ull, 0ull, 0ull, 0ull};
        const uint32_t base = g * 32u;
        unsigned selfSeen = 0u;   // bit l: member l met its own leaf
        // far list -> the group's expansion coefficients: lane l takes entry l
        // of the first `cnt`, the 20 coefficients are summed over the warp
        auto flushFar = [&](int cnt) {
            if constexpr (!kExpand) return;
            float t[20];
            if (lane < cnt) {
                float e[10];
                getMono<true, kGravListQ>(reinterpret_cast<const float*>(S.flist4), lane, e);
                farTaylor(e, cx, cy, cz, epsG2, t);
            } else {
#pragma unroll
                for (int k = 0; k < 20; ++k) t[k] = 0.0f;
            }
            float mine = 0.0f;
#pragma unroll
            for (int k = 0; k < 20; ++k) {
                const float v = warpSumF(t[k]);
                if (lane == k) mine = v;
            }
            if (lane < 20) reinterpret_cast<float*>(S.facc4)[lane] += mine;
            __syncwarp();
        };
        auto flushP = [&]() {                 // evaluate the 32 entries from pHead
            if (active) evalParticles2(S.plist, pHead, 32, X, Y, Z, HE, acc);
            entries += 32u;
            __syncwarp();
            pCount -= 32;
            pHead = (pHead + 32) & (kGravList - 1);
        };
        __syncwarp();

        auto flushM = [&]() {                 // evaluate the 32 entries from mHead
            if (active) evalMonopoles2<kQuad, kMRing>(S.mlist, mHead, 32, X, Y, Z, E2, acc);
            entries += 32u;
            __syncwarp();
            mCount -= 32;
            mHead = (mHead + 32) & (kMRing - 1);
        };
        // An accepted node of each lane that has one, into the monopole list
        // (mode 3: or into the group's expansion, where the node is far against
        // the group: group radius <= gamma |c - COM|).
        auto putAccepted = [&](bool accept, const Child& c) {
            bool far = false;
            if (kExpand && accept) {
                const float R2 = len2Exact(__fsub_rn(cx, c.x), __fsub_rn(cy, c.y), __fsub_rn(cz, c.z));
                far = rg2 <= __fmul_rn(w.expandGamma2, R2);
            }
            const unsigned accMask = __ballot_sync(0xffffffffu, accept && !far);
            const unsigned farMask = kExpand ? __ballot_sync(0xffffffffu, far) : 0u;
            if (accept) {
                float e[10] = {c.x, c.y, c.z, c.gm, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (kQuad) {
                    const float4 s0 = __ldg(&w.nodeQuad[2 * static_cast<size_t>(c.ref)]);      // Sxx Syy Szz Sxy
                    const float4 s1 = __ldg(&w.nodeQuad[2 * static_cast<size_t>(c.ref) + 1]);  // Sxz Syz
                    const float tr = s0.x + s0.y + s0.z;
                    e[4] = kGPsuF * (3.0f * s0.x - tr);
                    e[5] = kGPsuF * (3.0f * s0.y - tr);
                    e[6] = kGPsuF * (3.0f * s0.z - tr);
                    e[7] = kGPsuF * 3.0f * s0.w;
                    e[8] = kGPsuF * 3.0f * s1.x;
                    e[9] = kGPsuF * 3.0f * s1.y;
                }
                const int slot = (mHead + mCount + __popc(accMask & laneMaskLt())) & (kMRing - 1);
                if constexpr (kExpand) {
                    if (far)
                        putMono<true, kGravListQ>(reinterpret_cast<float*>(S.flist4), fCount + __popc(farMask & laneMaskLt()), e);
                    else
                        putMono<kQuad, kMRing>(S.mlist, slot, e);
                } else {
                    putMono<kQuad, kMRing>(S.mlist, slot, e);
                }
            }
            mCount += __popc(accMask);
            if (kExpand) {
                fCount += __popc(farMask);
                groupEvals += static_cast<uint32_t>(__popc(farMask));
                __syncwarp();
                if (fCount >= 32) {
                    flushFar(32);
                    fCount -= 32;
                    if (lane < fCount) {
                        float e2[10];
                        getMono<true, kGravListQ>(reinterpret_cast<const float*>(S.flist4), 32 + lane, e2);
                        putMono<true, kGravListQ>(reinterpret_cast<float*>(S.flist4), lane, e2);
                    }
                    __syncwarp();
                }
            }
            if (kQuad) {
                __syncwarp();
                if (mCount >= 32) flushM();
            }
        };
        // mode 3: an opened node of at most leafBucket particles is not
        // descended; its sorted leaf range is evaluated particle-particle
        auto bucketOf = [&](bool& open, const Child& c) {
            uint2 brng = make_uint2(1u, 0u);
            if (kExpand && open && c.cnt <= w.leafBucket) {
                const uint32_t first = static_cast<uint32_t>(c.ref) - (c.right ? 0u : c.cnt - 1u);
                if (c.cnt - 1u < 32u && first < n && n - first >= c.cnt) {   // always, for a valid tree
                    brng = make_uint2(first, first + c.cnt - 1u);
                    open = false;
                }
            }
            return brng;
        };
        auto putBuckets = [&](uint2 brng) {   // each range (at most 32 sorted particles) by the warp at once
            unsigned bucketMask = __ballot_sync(0xffffffffu, brng.x <= brng.y);
            while (bucketMask) {
                const int src = __ffs(bucketMask) - 1;
                bucketMask &= bucketMask - 1u;
                const uint32_t first = __shfl_sync(0xffffffffu, brng.x, src);
                const uint32_t last = __shfl_sync(0xffffffffu, brng.y, src);
                const uint32_t j = first + static_cast<uint32_t>(lane);
                const bool has = j <= last;
                const unsigned hm = __ballot_sync(0xffffffffu, has);
                unsigned sb = 0u;
                if (has) {
                    const float4 pm = __ldg(&w.leaf[j].a);
                    const float4 aux = __ldg(&w.leafAux[j]);
                    const int slot = (pHead + pCount + __popc(hm & laneMaskLt())) & (kGravList - 1);
                    putParticle(S.plist, slot, pm.x, pm.y, pm.z, -kGPsuF * aux.w, 0.5f * aux.y);
                    const uint32_t rel = j - base;
                    if (rel < 32u) sb = 1u << rel;
                }
                const unsigned selfHere = __reduce_or_sync(0xffffffffu, sb);
                selfSeen |= selfHere;
                pCount += __popc(hm);
                bucketLeaves += static_cast<uint32_t>(act * __popc(hm) - __popc(selfHere));
                __syncwarp();
                if (pCount >= 32) flushP();
            }
        };
        // Puts the decided nodes among up to two children a lane (kTwo) where
        // they belong: opened ones on the stack, accepted ones into the lists.
        // The group expansion calls it from one place, and its evaluations stand in
        // loops over the two sides, to keep the code small: with four copies of
        // them that walk waited 4 of its 10.8 cycles an instruction for
        // instructions (1M, theta 0.75, buckets of 8, 1.49 ms; now 1.16).  The other
        // modes' evaluations are short enough: there one copy costs 3 %.
        auto place = [&](auto two, bool openA, bool accA, const Child& A, bool openB, bool accB, const Child& B) {
            constexpr bool kTwo = decltype(two)::value;
            const uint2 brA = bucketOf(openA, A), brB = kTwo ? bucketOf(openB, B) : make_uint2(1u, 0u);
            unsigned mA = __ballot_sync(0xffffffffu, openA), mB = kTwo ? __ballot_sync(0xffffffffu, openB) : 0u;
            if (sp + __popc(mA) + __popc(mB) > kGravStack) {
                // Out of stack, only on a corrupted tree (walkWidth): the group takes
                // these nodes as monopoles, the rule of the engine kernel when its
                // stack is full (:933).
                accA = accA || openA;
                accB = accB || openB;
                openA = openB = false;
                mA = mB = 0u;
                overflowed = true;
            }
            if (openA) S.stack[sp + __popc(mA & laneMaskLt())] = A.ref;
            sp += __popc(mA);
            if (kTwo && openB) S.stack[sp + __popc(mB & laneMaskLt())] = B.ref;
            sp += __popc(mB);
            if constexpr (kExpand) {
#pragma unroll 1
                for (int side = 0; side < 2; ++side) {
                    const bool acc = side != 0 ? accB : accA;
                    if (__any_sync(0xffffffffu, acc)) putAccepted(acc, side != 0 ? B : A);
                }
                __syncwarp();
#pragma unroll 1
                for (int side = 0; side < 2; ++side) putBuckets(side != 0 ? brB : brA);
            } else {
                putAccepted(accA, A);
                if (kTwo) putAccepted(accB, B);
                __syncwarp();
                if (!kQuad)
                    while (mCount >= 32) flushM();
            }
        };
        // The cheap tests of one child (u = COM - c): accepted by the bound,
        // opened by the extreme member, or left undecided.
        auto decide = [&](bool isNode, float x, float y, float z, float dd, float ux, float uy, float uz, int ref,
                          float far2, bool& accept, bool& open, bool& undecided) {
            const float ax = fabsf(ux), ay = fabsf(uy), az = fabsf(uz);
            const float bx = fmaxf(ax - hx, 0.0f), by = fmaxf(ay - hy, 0.0f), bz = fmaxf(az - hz, 0.0f);
            const float D2 = bx * bx + by * by + bz * bz;
            const float4 dp = S.dirPos[((__float_as_uint(ux) >> 29) & 4u) | ((__float_as_uint(uy) >> 30) & 2u) |
                                       (__float_as_uint(uz) >> 31)];
            // distance to the octant's supporting plane, |u|_1 with its 1e-6 margin
            const float L = (ax + ay + az) * (0.57735027f - 1.0e-6f) - dp.w;
            const float Lb2 = fmaxf(D2, L * fabsf(L)) * 0.9999f;
            const float r2 = len2Engine(__fsub_rn(dp.x, x), __fsub_rn(dp.y, y), __fsub_rn(dp.z, z));
            bool boundAccepts = Lb2 > 2.0e-20f && dd < theta2 * Lb2;
            bool extreme = dd < __fmul_rn(theta2, r2) && r2 > 1.0e-20f;     // the engine's test, without its box
            auto apart = [&](const float4& bmin, const float4& bmax) {    // the group's box from the node's
                return bmax.x < gminx || bmin.x > gmaxx || bmax.y < gminy || bmin.y > gmaxy || bmax.z < gminz ||
                       bmin.z > gmaxz;
            };
            // the box is only looked at where the members in question may be as
            // near the COM as its furthest corner
            if (kInside && isNode && ((boundAccepts && !(Lb2 > far2)) || (extreme && !(r2 > far2)))) {
                const float4 bmin = __ldg(&w.node[4 * static_cast<size_t>(ref) + 2]);
                const float4 bmax = __ldg(&w.node[4 * static_cast<size_t>(ref) + 3]);
                boundAccepts = boundAccepts && apart(bmin, bmax);
                if (dp.x >= bmin.x && dp.x <= bmax.x && dp.y >= bmin.y && dp.y <= bmax.y && dp.z >= bmin.z &&
                    dp.z <= bmax.z)
                    extreme = false;
            }
            accept = isNode && boundAccepts;
            undecided = isNode && !boundAccepts && extreme;
            open = isNode && !boundAccepts && !extreme;
            if (kLearned) {
                // far test of mode 2 on the nodes the theta test may open: every
                // member passes theta_far (by a sound bound: the box distance or
                // the supporting plane of the nearest of 26 directions) and the
                // node is far against the group's size.  Such a node is decided here: a
                // monopole plus the learned correction of this (group, node),
                // unless every member accepts it anyway.
                const float gx = fmaxf(0.0f, fmaxf(gminx - x, x - gmaxx)), gy = fmaxf(0.0f, fmaxf(gminy - y, y - gmaxy)),
                            gz = fmaxf(0.0f, fmaxf(gminz - z, z - gmaxz));
                const float t = 0.41421356f * fmaxf(ax, fmaxf(ay, az));
                const int sx = (ux >= t) - (ux <= -t), sy = (uy >= t) - (uy <= -t), sz = (uz >= t) - (uz <= -t);
                const float Lf = (static_cast<float>(sx) * ux + static_cast<float>(sy) * uy + static_cast<float>(sz) * uz) *
                                     invDirNorm(abs(sx) + abs(sy) + abs(sz)) -
                                 S.farDir[13 + 9 * sx + 3 * sy + sz] - 1.0e-6f * (ax + ay + az + gExt);
                const float Fb2 = fmaxf(gx * gx + gy * gy + gz * gz, Lf > 0.0f ? Lf * Lf : 0.0f);
                bool farOk = !accept && isNode && emitFar && Fb2 > 2.0e-20f && dd < ff.thetaFar2 * Fb2 * 0.99999f &&
                             gExt * gExt <= ff.gamma2 * (ux * ux + uy * uy + uz * uz);
                if (farOk)                       // and the boxes are apart
                    farOk = apart(__ldg(&w.node[4 * static_cast<size_t>(ref) + 2]), __ldg(&w.node[4 * static_cast<size_t>(ref) + 3]));
                // only an undecided one needs the exact test of every member here (a
                // box of such a node holds no member)
                bool all = false;
                unsigned todo = __ballot_sync(0xffffffffu, farOk && undecided);
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    const float qx = __shfl_sync(0xffffffffu, x, src), qy = __shfl_sync(0xffffffffu, y, src),
                                qz = __shfl_sync(0xffffffffu, z, src), qd = __shfl_sync(0xffffffffu, dd, src);
                    const float m2 = len2Engine(__fsub_rn(xi, qx), __fsub_rn(yi, qy), __fsub_rn(zi, qz));
                    const bool each = __all_sync(0xffffffffu, !active || (qd < __fmul_rn(theta2, m2) && m2 > 1.0e-20f));
                    if (lane == src) all = each;
                }
                const unsigned take = __ballot_sync(0xffffffffu, farOk && !all);
                if (take) {
                    uint32_t first = 0;
                    if (lane == 0) first = atomicAdd(ff.count, static_cast<uint32_t>(__popc(take)));
                    first = __shfl_sync(0xffffffffu, first, 0);
                    const uint32_t slot = first + static_cast<uint32_t>(__popc(take & laneMaskLt()));
                    if (farOk && !all && slot < ff.cap) {           // full buffer: the node is opened
                        ff.pairs[slot] = make_uint2(g, static_cast<uint32_t>(ref));
                        all = true;
                    }
                }
                if (farOk) {
                    accept = all;
                    open = !all;
                    undecided = false;
                }
            }
        };
        while (sp > 0 || uCount > 0) {
            if (++rounds > 4u * n + 64u) {     // only reachable on a corrupted tree
                overflowed = true;
                break;
            }
            // every undecided child may still be opened
            const int width = walkWidth<kGravStack>(sp + uCount);
            Child A, B;
            bool accA = false, openA = false, accB = false, openB = false;
            if (uCount >= 32 || sp == 0 || (width == 1 && uCount > 0)) {
                // The oldest undecided children, up to 32, one a lane, against every
                // member: the engine's member test (sph_gravity.cu:914-929) with
                // the engine's rounding of r^2 (len2Engine's operations, packed).
                // fl(theta^2 r^2) grows with r^2, so all members accept when the
                // smallest r^2 does.
                const int take = min(uCount, 32);
                const bool has = lane < take;
                undecidedTests += static_cast<uint32_t>(take);
                Child c;
                float far2 = 0.0f;
                {
                    const uint32_t id = has ? S.und[uHead + lane] : 0u;
                    const float* r = reinterpret_cast<const float*>(w.pair + 4 * static_cast<size_t>(id >> 1)) + (id & 1u);
                    c.x = __ldg(r); c.y = __ldg(r + 2); c.z = __ldg(r + 4); c.gm = __ldg(r + 6); c.w = __ldg(r + 8);
                    c.ref = __float_as_int(__ldg(r + 10));
                    if (kInside) far2 = __ldg(r + 12);
                    if (kExpand) c.cnt = __float_as_uint(__ldg(r + 14));
                    c.right = (id & 1u) != 0u;
                }
                uCount -= take;
                uHead = (uHead + 32) & (kGravList - 1);   // take < 32 empties the ring: any head will do
                const f2 NX = pack2(c.x, c.x), NY = pack2(c.y, c.y), NZ = pack2(c.z, c.z);
                float rmin = 3.4e38f;
#pragma unroll 4
                for (int k = 0; k < 16; ++k) {
                    const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(&S.memXY[k]);
                    const f2 dx = sub2(xy.x, NX), dy = sub2(xy.y, NY),
                             dz = sub2(*reinterpret_cast<const f2*>(&S.memZ[k]), NZ);
                    float ra, rb;
                    unpack2(fma2(dz, dz, fma2(dx, dx, mul2(dy, dy))), ra, rb);
                    rmin = fminf(rmin, fminf(ra, rb));
                }
                bool all = __fmul_rn(c.w, c.w) < __fmul_rn(theta2, rmin) && rmin > 1.0e-20f;
                if (kInside) {                  // nor may a member lie in the node's box
                    float4 bmin = make_float4(0.f, 0.f, 0.f, 0.f), bmax = bmin;
                    bool near = has && all && rmin <= far2;
                    if (near) {
                        bmin = __ldg(&w.node[4 * static_cast<size_t>(c.ref) + 2]);
                        bmax = __ldg(&w.node[4 * static_cast<size_t>(c.ref) + 3]);
                        near = !(bmax.x < gminx || bmin.x > gmaxx || bmax.y < gminy || bmin.y > gmaxy ||
                                 bmax.z < gminz || bmin.z > gmaxz);
                    }
                    if (__any_sync(0xffffffffu, near)) {
                        for (int k = 0; k < 16; ++k) {
                            const float4 xy = S.memXY[k];
                            const float2 zz = S.memZ[k];
                            if (near && ((xy.x >= bmin.x && xy.x <= bmax.x && xy.z >= bmin.y && xy.z <= bmax.y &&
                                          zz.x >= bmin.z && zz.x <= bmax.z) ||
                                         (xy.y >= bmin.x && xy.y <= bmax.x && xy.w >= bmin.y && xy.w <= bmax.y &&
                                          zz.y >= bmin.z && zz.y <= bmax.z)))
                                all = false;
                        }
                    }
                }
                if constexpr (!kExpand) {
                    place(std::false_type{}, has && !all, has && all, c, false, false, c);
                    continue;
                }
                A = B = c;
                openA = has && !all;
                accA = has && all;
            } else {
                // open up to 32 nodes: both children of each
                spPeak = max(spPeak, sp);
                const int take = min(sp, width);
                sp -= take;
                int node = (lane < take) ? S.stack[sp + lane] : 0;
                __syncwarp();
                // indices outside [0, n-2] cannot come from a valid tree
                const bool has = lane < take && static_cast<uint32_t>(node) < n - 1u;
                node = has ? node : 0;
                const PairRec rec = loadPair<kInside || kExpand>(w.pair + 4 * static_cast<size_t>(node));
                const f2 du = sub2(rec.x, CX), dv = sub2(rec.y, CY), dw = sub2(rec.z, CZ), dd = mul2(rec.w, rec.w);
                tests += 2u * static_cast<uint32_t>(take);
                unpack2(rec.x, A.x, B.x);
                unpack2(rec.y, A.y, B.y);
                unpack2(rec.z, A.z, B.z);
                unpack2(rec.gm, A.gm, B.gm);
                unpack2(rec.w, A.w, B.w);
                A.ref = rec.refA;
                B.ref = rec.refB;
                A.cnt = rec.cntA;
                B.cnt = rec.cntB;
                A.right = false;
                B.right = true;
                float uxA, uxB, uyA, uyB, uzA, uzB, ddA, ddB;
                unpack2(du, uxA, uxB);
                unpack2(dv, uyA, uyB);
                unpack2(dw, uzA, uzB);
                unpack2(dd, ddA, ddB);
                bool undA, undB;
                decide(has && A.ref >= 0, A.x, A.y, A.z, ddA, uxA, uyA, uzA, A.ref, rec.farA, accA, openA, undA);
                decide(has && B.ref >= 0, B.x, B.y, B.z, ddB, uxB, uyB, uzB, B.ref, rec.farB, accB, openB, undB);
                // undecided children of both sides
                const unsigned uA = __ballot_sync(0xffffffffu, undA), uB = __ballot_sync(0xffffffffu, undB);
                if (uA | uB) {
                    const int s0 = uHead + uCount + __popc(uA & laneMaskLt());
                    if (undA) S.und[s0 & (kGravList - 1)] = 2u * static_cast<uint32_t>(node);
                    const int s1 = uHead + uCount + __popc(uA) + __popc(uB & laneMaskLt());
                    if (undB) S.und[s1 & (kGravList - 1)] = 2u * static_cast<uint32_t>(node) + 1u;
                    uCount += __popc(uA) + __popc(uB);
                }
                // leaves of both sides
                const bool leafA = has && A.ref < 0, leafB = has && B.ref < 0;
                const unsigned lA = __ballot_sync(0xffffffffu, leafA), lB = __ballot_sync(0xffffffffu, leafB);
                if (lA | lB) {
                    unsigned selfBit = 0u;
                    auto putLeaf = [&](const Child& c, int slot) {
                        putParticle(S.plist, slot, c.x, c.y, c.z, c.gm, c.w);
                        const uint32_t rel = static_cast<uint32_t>(~c.ref) - base;
                        if (rel < 32u) selfBit |= 1u << rel;
                    };
                    if (leafA) putLeaf(A, (pHead + pCount + __popc(lA & laneMaskLt())) & (kGravList - 1));
                    if (leafB) putLeaf(B, (pHead + pCount + __popc(lA) + __popc(lB & laneMaskLt())) & (kGravList - 1));
                    selfSeen |= __reduce_or_sync(0xffffffffu, selfBit);
                    const int cnt = __popc(lA) + __popc(lB);
                    pCount += cnt;
                    tests -= static_cast<uint32_t>(cnt);
                    __syncwarp();
                    while (pCount >= 32) flushP();
                }
            }
            place(std::true_type{}, openA, accA, A, openB, accB, B);
        }
        if (kExpand && fCount > 0) flushFar(fCount);
        // tails: pad to fours with massless entries (they add exactly zero)
        if (lane < 3) {
            if (lane < ((4 - mCount) & 3)) {
                const float zero[10] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                putMono<kQuad, kMRing>(S.mlist, mHead + mCount + lane, zero);
            }
            if (lane < ((4 - pCount) & 3)) putParticle(S.plist, pHead + pCount + lane, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncwarp();
        if (active) {
            evalMonopoles2<kQuad, kMRing>(S.mlist, mHead, (mCount + 3) & ~3, X, Y, Z, E2, acc);
            evalParticles2(S.plist, pHead, (pCount + 3) & ~3, X, Y, Z, HE, acc);
            float a0, a1, b0, b1, c0, c1, d0, d1;
            unpack2(acc.ax, a0, a1);
            unpack2(acc.ay, b0, b1);
            unpack2(acc.az, c0, c1);
            unpack2(acc.phi, d0, d1);
            float phi = d0 + d1;
            if (selfSeen & (1u << lane)) {
                // the self term added to phi: -G m_i / sqrt(eps_i^2), exactly as evaluated
                phi -= (-kGPsuF * me.w) * rsqrtNormal(__fmul_rn(epsI, epsI));
            }
            float ax = a0 + a1, ay = b0 + b1, az = c0 + c1;
            if (kExpand) {                     // the group's far field at this member (farTaylor)
                const float* t = reinterpret_cast<const float*>(S.facc4);
                const float dx = xi - cx, dy = yi - cy, dz = zi - cz;
                const float jx = t[4] * dx + t[7] * dy + t[8] * dz;      // J d
                const float jy = t[7] * dx + t[5] * dy + t[9] * dz;
                const float jz = t[8] * dx + t[9] * dy + t[6] * dz;
                const float xx = dx * dx, yy = dy * dy, zz = dz * dz, xy = dx * dy, xz = dx * dz, yz = dy * dz;
                const float hx = t[10] * xx + t[15] * yy + t[17] * zz + 2.0f * (t[13] * xy + t[14] * xz + t[19] * yz);
                const float hy = t[13] * xx + t[11] * yy + t[18] * zz + 2.0f * (t[15] * xy + t[19] * xz + t[16] * yz);
                const float hz = t[14] * xx + t[16] * yy + t[12] * zz + 2.0f * (t[19] * xy + t[17] * xz + t[18] * yz);
                ax += t[1] + jx + 0.5f * hx;
                ay += t[2] + jy + 0.5f * hy;
                az += t[3] + jz + 0.5f * hz;
                phi += t[0] - (t[1] * dx + t[2] * dy + t[3] * dz) - 0.5f * (jx * dx + jy * dy + jz * dz);
            }
            p.accX[i] = ax;
            p.accY[i] = ay;
            p.accZ[i] = az;
            p.phiGrav[i] = phi;
        }
        if (lane == 0) {
            const unsigned long long inter = static_cast<unsigned long long>(act) *
                                                 (entries + static_cast<unsigned>(mCount + pCount)) -
                                             static_cast<unsigned long long>(__popc(selfSeen));
            S.counts[0] += inter;
            S.counts[1] += tests;
            S.counts[2] += undecidedTests;
            S.counts[3] += rounds;
            if (kExpand) {
                S.counts[4] += groupEvals;
                S.counts[5] += bucketLeaves;
            }
        }
        __syncwarp();
    }
    if (lane == 0) {
        DevStatus* st = reinterpret_cast<DevStatus*>(w.status);
        atomicAdd(&st->counters[kCntGravityInteractions], S.counts[0]);
        atomicAdd(&st->counters[kCntGravityNodeTests], S.counts[1]);
        atomicAdd(&st->counters[kCntGravityUndecided], S.counts[2]);
        if (kExpand) {
            atomicAdd(&st->counters[kCntGravityGroupEvals], S.counts[4]);
            atomicAdd(&st->counters[kCntGravityBucketLeaves], S.counts[5]);
        }
        atomicAdd(&st->counters[kCntGravityRounds], S.counts[3]);
        atomicMax(&st->counters[kCntGravityStackPeak], static_cast<unsigned long long>(spPeak));
        if (overflowed) atomicOr(&st->flags, kFlagStackOverflow);
    }
}

// The monopole walk: the same sets, with the terms of a particle added in one
// fixed order -- rounds of 32 children (16 opened nodes), accepted nodes and leaves
// appended in the children's order, undecided children settled within their round,
// each list evaluated when it holds 32 -- the order in which the library's results have always
// been added up.  gravityKernel's order (64 children a round, undecided ones
// later) changes the last bit of a third of the accelerations (at 1M it takes the
// same time, at 60k 106 instead of 120 us), and a step amplifies that: in a
// gas giant impact at 32 km/s the velocities' last bits move strain rates by up to
// 1e-3 of their rms, and iron just below its melting point turns an ulp of rho
// into 1e-4 of its strength.  Bound, like that kernel, by instruction issue; it
// shares the child records, the octant planes and the list layout.  Against the walk over
// nodes before it (one node a lane, leaves loaded again): 1M 1.69 -> 1.37 ms, 60k
// 139 -> 120 us.  Resident warps per SM the registers are bounded for, 1M: theta 0.5
// 28 1.54, 32 1.50, 36 1.40, 40 (spills) 1.42 ms; theta 0.7, whose box test needs more
// registers, 24 1.07, 28 0.99, 32 1.01, 36 (spills) 1.04.  Those boxes are loaded only where
// a member may be as near as the furthest corner: loaded for every undecided child, a
// dependent trip each, a call at theta 0.6 took 97 instead of 77 us at 16k, 136
// instead of 110 at 60k, 1146 instead of 977 at 1M.
constexpr int kOrdRing = 64;
struct __align__(16) OrderedSmem {
    int stack[kGravStack];
    float mlist[4 * kOrdRing];
    float plist[5 * kOrdRing];
    float4 und[32];                    // undecided children: COM, dNode^2
    int undRef[32];
    float undFar[32];
    float4 dirPos[8];                  // see GravWarpSmem
};
static_assert(offsetof(OrderedSmem, mlist) % 16 == 0 && offsetof(OrderedSmem, plist) % 16 == 0 &&
              offsetof(OrderedSmem, und) % 16 == 0 && offsetof(OrderedSmem, dirPos) % 16 == 0, "vector loads");
// kDebug: the variant that serves the debugging calls (per-group interaction
// counts, the trace of one group's accepted nodes and leaves in walk order); their
// checks are kept out of the production variants.
template <int kWarps, bool kInside, bool kDebug = false>
__global__ void __launch_bounds__(kWarps * 32, (kInside ? 28 : 36) / kWarps) gravityOrderedKernel(AstraeaParticles p, Work w, uint32_t n,
                                                                                float theta2, uint32_t numGroups,
                                                                                uint32_t* groupCounter, FarCapture) {
    chained();
    __shared__ OrderedSmem smem[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    OrderedSmem& S = smem[warp];
    unsigned long long nInter = 0;
    uint32_t nTests = 0, nUndecided = 0, nRounds = 0;
    int spPeak = 0;
    bool overflowed = false;
    if (w.runIf != nullptr && *w.runIf == 0u) return;   // the gate of the learned mode passed
    if (n == 1u) {                                   // sph_gravity.cu:824-832
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            p.accX[0] = 0.0f; p.accY[0] = 0.0f; p.accZ[0] = 0.0f; p.phiGrav[0] = 0.0f;
        }
        return;
    }
    for (;;) {
        uint32_t g = 0;
        if (lane == 0) g = atomicAdd(groupCounter, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= numGroups) break;
        const uint32_t i = g * 32u + static_cast<uint32_t>(lane);
        const bool active = i < n;
        const int act = static_cast<int>(min(32u, n - g * 32u));
        float4 me = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float epsI = 0.8e-6f;
        if (active) {
            me = __ldg(&w.leaf[i].a);
            const float4 aux = __ldg(&w.leafAux[i]);
            epsI = aux.y;
            me.w = aux.w;                                // the mass
        }
        const float xi = me.x, yi = me.y, zi = me.z;
        const float epsI2 = epsI * epsI + 1.0e-20f;
        const float gminx = warpMinF(active ? xi : 3.0e38f), gmaxx = warpMaxF(active ? xi : -3.0e38f);
        const float gminy = warpMinF(active ? yi : 3.0e38f), gmaxy = warpMaxF(active ? yi : -3.0e38f);
        const float gminz = warpMinF(active ? zi : 3.0e38f), gmaxz = warpMaxF(active ? zi : -3.0e38f);
        const float gExt = (gmaxx - gminx) + (gmaxy - gminy) + (gmaxz - gminz);
        // box centre, half sides and margins: as in gravityKernel
        const float cx = 0.5f * (gminx + gmaxx), cy = 0.5f * (gminy + gmaxy), cz = 0.5f * (gminz + gmaxz);
        const float slack = 1.0e-6f * gExt;
        const float hx = fmaxf(gmaxx - cx, cx - gminx) + slack, hy = fmaxf(gmaxy - cy, cy - gminy) + slack,
                    hz = fmaxf(gmaxz - cz, cz - gminz) + slack;
        extremeMembers(S.dirPos, xi, yi, zi, cx, cy, cz, slack, act, lane);
        if (lane == 0) S.stack[0] = 0;   // the root is opened by every group
        int sp = 1, mCount = 0, pCount = 0, mHead = 0, pHead = 0;
        uint32_t rounds = 0, traced = 0;
        [[maybe_unused]] const unsigned long long interBefore = nInter;
        const f2 X = pack2(xi, xi), Y = pack2(yi, yi), Z = pack2(zi, zi);
        const f2 E2 = pack2(epsI2, epsI2), HE = pack2(0.5f * epsI, 0.5f * epsI);
        Accum2 acc{0ull, 0ull, 0ull, 0ull};
        const uint32_t base = g * 32u;
        unsigned selfSeen = 0u;   // bit l: member l met its own leaf
        __syncwarp();
        while (sp > 0) {
            if (++rounds > 4u * n + 64u) {     // only reachable on a corrupted tree
                overflowed = true;
                break;
            }
            spPeak = max(spPeak, sp);
            const int take = min(sp, 16);
            sp -= take;
            // lane 2 k: the left child of opened node k, lane 2 k + 1: the right one
            int node = (lane >> 1) < take ? S.stack[sp + (lane >> 1)] : 0;
            __syncwarp();
            const bool has = (lane >> 1) < take && static_cast<uint32_t>(node) < n - 1u;
            node = has ? node : 0;
            const float4* rec = w.pair + 4 * static_cast<size_t>(node);
            const float4 q0 = __ldg(rec), q1 = __ldg(rec + 1), q2 = __ldg(rec + 2);
            const bool right = (lane & 1) != 0;
            const float x = right ? q0.y : q0.x, y = right ? q0.w : q0.z, z = right ? q1.y : q1.x,
                        gm = right ? q1.w : q1.z, wc = right ? q2.y : q2.x;
            const int ref = __float_as_int(right ? q2.w : q2.z);
            const bool isLeaf = has && ref < 0, isNode = has && ref >= 0;
            const float dd = __fmul_rn(wc, wc);
            const float ux = x - cx, uy = y - cy, uz = z - cz;
            const float ax = fabsf(ux), ay = fabsf(uy), az = fabsf(uz);
            const float bx = fmaxf(ax - hx, 0.0f), by = fmaxf(ay - hy, 0.0f), bz = fmaxf(az - hz, 0.0f);
            const float D2 = bx * bx + by * by + bz * bz;
            const float4 dp = S.dirPos[((__float_as_uint(ux) >> 29) & 4u) | ((__float_as_uint(uy) >> 30) & 2u) |
                                       (__float_as_uint(uz) >> 31)];
            const float L = (ax + ay + az) * (0.57735027f - 1.0e-6f) - dp.w;
            const float Lb2 = fmaxf(D2, L * fabsf(L)) * 0.9999f;
            const float r2 = len2Engine(__fsub_rn(dp.x, x), __fsub_rn(dp.y, y), __fsub_rn(dp.z, z));
            bool boundAccepts = Lb2 > 2.0e-20f && dd < theta2 * Lb2;
            bool extreme = dd < __fmul_rn(theta2, r2) && r2 > 1.0e-20f;
            const float far2 = kInside ? __ldg(reinterpret_cast<const float*>(rec + 3) + (lane & 1)) : 0.0f;
            if (kInside) {
                if (isNode && ((boundAccepts && !(Lb2 > far2)) || (extreme && !(r2 > far2)))) {
                    const float4 bmin = __ldg(&w.node[4 * static_cast<size_t>(ref) + 2]);
                    const float4 bmax = __ldg(&w.node[4 * static_cast<size_t>(ref) + 3]);
                    boundAccepts = boundAccepts && (bmax.x < gminx || bmin.x > gmaxx || bmax.y < gminy || bmin.y > gmaxy ||
                                                    bmax.z < gminz || bmin.z > gmaxz);
                    if (dp.x >= bmin.x && dp.x <= bmax.x && dp.y >= bmin.y && dp.y <= bmax.y && dp.z >= bmin.z &&
                        dp.z <= bmax.z)
                        extreme = false;
                }
            }
            bool accept = isNode && boundAccepts;
            const bool undecided = isNode && !boundAccepts && extreme;
            const unsigned und = __ballot_sync(0xffffffffu, undecided);
            if (und) {                          // by all members at once, the engine's test and rounding
                const int nu = __popc(und), slot = __popc(und & laneMaskLt());
                nUndecided += static_cast<uint32_t>(nu);
                if (undecided) {
                    S.und[slot] = make_float4(x, y, z, dd);
                    if (kInside) {
                        S.undRef[slot] = ref;
                        S.undFar[slot] = far2;
                    }
                }
                __syncwarp();
                unsigned bits = 0u;
                auto settle = [&](int k) {
                    const float4 q = S.und[k];
                    const float m2 = len2Engine(__fsub_rn(xi, q.x), __fsub_rn(yi, q.y), __fsub_rn(zi, q.z));
                    const bool ok = q.w < __fmul_rn(theta2, m2) && m2 > 1.0e-20f;
                    bool all = __all_sync(0xffffffffu, !active || ok);
                    if (kInside && all && __any_sync(0xffffffffu, active && !(m2 > S.undFar[k]))) {
                        const float4 mn = __ldg(&w.node[4 * static_cast<size_t>(S.undRef[k]) + 2]);
                        const float4 mx = __ldg(&w.node[4 * static_cast<size_t>(S.undRef[k]) + 3]);
                        all = __all_sync(0xffffffffu, !active || !(xi >= mn.x && xi <= mx.x && yi >= mn.y && yi <= mx.y &&
                                                                   zi >= mn.z && zi <= mx.z));
                    }
                    bits |= (all ? 1u : 0u) << k;
                };
                if constexpr (kInside) {
#pragma unroll 2
                    for (int k = 0; k < nu; ++k) settle(k);
                } else {                         // the compiler's choice: 1M 1.37 ms, 60k 120 us; not unrolled 1.41, 134
                    for (int k = 0; k < nu; ++k) settle(k);
                }
                if (undecided) accept = (bits >> slot) & 1u;
                __syncwarp();
            }
            bool open = isNode && !accept;
            unsigned openMask = __ballot_sync(0xffffffffu, open);
            if (sp + __popc(openMask) > kGravStack) {
                // Out of stack: the group takes these nodes as monopoles, the
                // rule of the engine kernel when its stack is full (:933).
                if (open) { open = false; accept = true; }
                openMask = 0u;
                overflowed = true;
            }
            if (open) S.stack[sp + __popc(openMask & laneMaskLt())] = ref;
            sp += __popc(openMask);
            const unsigned accMask = __ballot_sync(0xffffffffu, accept), leafMask = __ballot_sync(0xffffffffu, isLeaf);
            if (kDebug && w.traceList != nullptr && g == w.traceGroup) {
                const unsigned both = accMask | leafMask;
                const uint32_t k = traced + static_cast<uint32_t>(__popc(both & laneMaskLt()));
                if ((accept || isLeaf) && k < w.traceCap) w.traceList[1 + k] = ref;
                traced += static_cast<uint32_t>(__popc(both));
                if (lane == 0) w.traceList[0] = static_cast<int>(traced);
            }
            if (accept) {
                const float e[10] = {x, y, z, gm, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                putMono<false, kOrdRing>(S.mlist, (mHead + mCount + __popc(accMask & laneMaskLt())) & (kOrdRing - 1), e);
            }
            mCount += __popc(accMask);
            if (leafMask) {
                unsigned selfBit = 0u;
                if (isLeaf) {
                    putParticle<kOrdRing>(S.plist, (pHead + pCount + __popc(leafMask & laneMaskLt())) & (kOrdRing - 1), x, y, z,
                                          gm, wc);
                    const uint32_t rel = static_cast<uint32_t>(~ref) - base;
                    if (rel < 32u) selfBit = 1u << rel;
                }
                selfSeen |= __reduce_or_sync(0xffffffffu, selfBit);
                pCount += __popc(leafMask);
            }
            nTests += 2u * static_cast<uint32_t>(take) - static_cast<uint32_t>(__popc(leafMask));
            __syncwarp();
            if (mCount >= 32) {
                if (active) evalMonopoles2<false, kOrdRing, true>(S.mlist, mHead, 32, X, Y, Z, E2, acc);
                nInter += static_cast<unsigned long long>(act) * 32u;
                __syncwarp();
                mCount -= 32;
                mHead ^= 32;
            }
            if (pCount >= 32) {
                if (active) evalParticles2<kOrdRing, true>(S.plist, pHead, 32, X, Y, Z, HE, acc);
                nInter += static_cast<unsigned long long>(act) * 32u;
                __syncwarp();
                pCount -= 32;
                pHead ^= 32;
            }
        }
        // tails: pad to fours with massless entries (they add exactly zero)
        if (lane < 3) {
            if (lane < ((4 - mCount) & 3)) {
                const float zero[10] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                putMono<false, kOrdRing>(S.mlist, mHead + mCount + lane, zero);
            }
            if (lane < ((4 - pCount) & 3)) putParticle<kOrdRing>(S.plist, pHead + pCount + lane, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncwarp();
        if (active) {
            evalMonopoles2<false, kOrdRing, true>(S.mlist, mHead, (mCount + 3) & ~3, X, Y, Z, E2, acc);
            evalParticles2<kOrdRing, true>(S.plist, pHead, (pCount + 3) & ~3, X, Y, Z, HE, acc);
            float a0, a1, b0, b1, c0, c1, d0, d1;
            unpack2(acc.ax, a0, a1);
            unpack2(acc.ay, b0, b1);
            unpack2(acc.az, c0, c1);
            unpack2(acc.phi, d0, d1);
            float phi = d0 + d1;
            if (selfSeen & (1u << lane)) phi -= (-kGPsuF * me.w) * rsqrtNormal(__fmul_rn(epsI, epsI));   // the self term
            p.accX[i] = a0 + a1;
            p.accY[i] = b0 + b1;
            p.accZ[i] = c0 + c1;
            p.phiGrav[i] = phi;
        }
        nInter += static_cast<unsigned long long>(act) * static_cast<unsigned>(mCount + pCount) -
                  static_cast<unsigned long long>(__popc(selfSeen));
        if (kDebug && w.groupCounts != nullptr && lane == 0) w.groupCounts[g] = static_cast<uint32_t>(nInter - interBefore);
        nRounds += rounds;
        __syncwarp();
    }
    if (lane == 0) {
        DevStatus* st = reinterpret_cast<DevStatus*>(w.status);
        atomicAdd(&st->counters[kCntGravityInteractions], nInter);
        atomicAdd(&st->counters[kCntGravityNodeTests], static_cast<unsigned long long>(nTests));
        atomicAdd(&st->counters[kCntGravityUndecided], static_cast<unsigned long long>(nUndecided));
        atomicAdd(&st->counters[kCntGravityRounds], static_cast<unsigned long long>(nRounds));
        atomicMax(&st->counters[kCntGravityStackPeak], static_cast<unsigned long long>(spPeak));
        if (overflowed) atomicOr(&st->flags, kFlagStackOverflow);
    }
}

}  // namespace

cudaError_t launchGravity(const AstraeaParticles& p, const Work& w, uint32_t n, float theta, bool quadrupole, int sms,
                          LaunchAt st, const FarCapture* far, int warps, bool expansion) {
    if (n == 0) return cudaSuccess;
    const float th = fmaxf(0.0f, theta);
    const float theta2 = th * th;
    const bool checkInside = theta2 > 0.333333f;
    const uint32_t groups = (n + 31u) / 32u;
    uint32_t* counter = w.words + kWGroupCounter;
    // The pair kernel also clears the counter.  (The learned mode's fallback,
    // runIf, walks the records its first walk wrote.)
    cudaError_t e = n >= 2u && w.runIf == nullptr ? launchChained(pairNodesKernel, (n - 1u + 255u) / 256u, 256, st, w, n)
                                                  : cudaMemsetAsync(counter, 0, sizeof(uint32_t), st.stream);
    if (e != cudaSuccess) return e;
    FarCapture ff{};
    using GravFn = void (*)(AstraeaParticles, Work, uint32_t, float, uint32_t, uint32_t*, FarCapture);
    GravFn kernel = nullptr;
    int wps = kGravWarps;
    if (w.traceList != nullptr || w.groupCounts != nullptr) {
        // the debugging calls (monopole walk, 4-warp blocks)
        kernel = checkInside ? gravityOrderedKernel<kGravWarps, true, true> : gravityOrderedKernel<kGravWarps, false, true>;
    } else if (expansion && quadrupole && far == nullptr) {
        if (warps == 2) {
            kernel = checkInside ? gravityKernel<2, true, true, false, true> : gravityKernel<2, false, true, false, true>;
            wps = 2;
        } else {
            kernel = checkInside ? gravityKernel<kGravWarps, true, true, false, true>
                                 : gravityKernel<kGravWarps, false, true, false, true>;
        }
    } else if (far != nullptr) {
        ff = *far;
        if (ff.groupStride == 0u) ff.groupStride = 1u;
        kernel = checkInside ? gravityKernel<kGravWarps, true, false, true> : gravityKernel<kGravWarps, false, false, true>;
    } else if (quadrupole && warps == 2) {
        kernel = checkInside ? gravityKernel<2, true, true, false> : gravityKernel<2, false, true, false>;
        wps = 2;
    } else if (quadrupole && warps == 8) {
        kernel = checkInside ? gravityKernel<8, true, true, false> : gravityKernel<8, false, true, false>;
        wps = 8;
    } else if (quadrupole) {
        kernel = checkInside ? gravityKernel<kGravWarps, true, true, false> : gravityKernel<kGravWarps, false, true, false>;
    } else if (warps == 2) {
        kernel = checkInside ? gravityOrderedKernel<2, true> : gravityOrderedKernel<2, false>;
        wps = 2;
    } else if (warps == 8) {
        kernel = checkInside ? gravityOrderedKernel<8, true> : gravityOrderedKernel<8, false>;
        wps = 8;
    } else {
        kernel = checkInside ? gravityOrderedKernel<kGravWarps, true> : gravityOrderedKernel<kGravWarps, false>;
    }
    int perSm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, wps * 32, 0);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>(static_cast<uint32_t>(std::max(1, perSm) * sms),
                                               (groups + wps - 1) / wps);
    return launchChained(kernel, blocks, static_cast<uint32_t>(wps * 32), st, p, w, n, theta2, groups, counter, ff);
}

}  // namespace astraea_gb300
