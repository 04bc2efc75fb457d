// Contact-to-constraint setup, Jacobi contact/friction solver with velocity
// averaging, and transform integration, for sm_100a.
//
// Solver semantics are btPgsJacobiSolver with usePgs = false
// (P2/btPgsJacobiSolver.cpp:35), as solveContacts configures it (:171-191):
// 10 iterations, splitImpulse off, erp 0.2, linearSlop 0, solver mode
// WARMSTARTING | SIMD | USE_2_FRICTION_DIRECTIONS (btContactSolverInfo.h:72-90
// defaults plus :180), which means
//   * one solver-body copy per (manifold, dynamic body); a static body is a
//     single shared solver body with zero inverse mass (getOrInitSolverBody
//     :689-722); m_bodyCount[b] = number of manifolds touching b (:1105-1129)
//   * per point (skipped if depth + 0.01 > 0.02, :124-155 and :961):
//     normal row (setupContactConstraint :725-888) with Baumgarte rhs and the
//     count-scaled denominator relaxation/(d0*countA + d1*countB), then two
//     friction rows, direction 2 first, along the relative tangential velocity
//     when its squared length exceeds FLT_EPSILON, else btPlaneSpace1(n)
//     (convertContact :933-1080, setupFrictionConstraint :505-592)
//   * inverse inertia used by the rows is the body's local diagonal inverse
//     inertia (getInvInertiaTensorWorld returns m_initInvInertia, :51-66)
//   * each iteration: all normal rows (lower limit 0), averageVelocities,
//     all friction rows clamped to +-mu*lambda_n (skipped while lambda_n <= 0),
//     averageVelocities (solveSingleIteration :1372-1614,
//     solveGroupCacheFriendlyIterations :1656-1681, averageVelocities :1683-1720)
//   * finish: every copy of a dynamic body adds sum/count to the body
//     velocity (solveGroupCacheFriendlyFinish :1790-1803), so a body with k
//     copies receives k times the averaged delta.
// Impulses reach every solver body (the SIMD row solvers used by this
// solver mode have no per-body guard).
//
// B200 mapping: rows within a copy are Gauss-Seidel, copies are independent, so a
// manifold is solved by one thread (k_jacobi_pass, k_jacobi_worlds) or by two
// lanes, one per body (k_jacobi), its rows in order, the copies' delta velocities
// in registers. The per-body average is a deterministic segmented sum over the
// body's copies in manifold order (the copy list is a stable radix sort of (body,
// copy) entries). All phases of all iterations run in one persistent cooperative
// kernel, separated by a grid barrier whose wait is bounded. Rows are stored
// structure-of-arrays (row slot major): k_jacobi keeps those of a lane pair's first
// manifolds in shared memory, otherwise each phase streams them with coalesced
// float4 loads.
#include "solver_common.cuh"

#include <algorithm>
#include <cfloat>

using namespace b3m;
using namespace b3solver;

namespace {

// ---------------------------------------------------------------------------
// Manifold compaction: manifold index = exclusive scan of per-pair flags.
// ---------------------------------------------------------------------------
__global__ void k_manifold_emit(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ scan,
                                const int32_t* __restrict__ numPairsDev,
                                const b3Contact4* __restrict__ contacts, const float* __restrict__ invMass,
                                int numBodies, int* __restrict__ manifoldPair,
                                uint32_t* __restrict__ incKeys, uint32_t* __restrict__ incVals,
                                int32_t* __restrict__ scalars, b3Counters* __restrict__ counters) {
    const int np = *numPairsDev;
    const int M = scalars[b3::S_NUM_MANIFOLDS];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        scalars[b3::S_NUM_INC] = 2 * M;
        counters->numManifolds = M;
    }
    int pts = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
        if (!flag[p]) continue;
        const int m = (int)scan[p];
        manifoldPair[m] = p;
        const b3Contact4& c = contacts[p];
        const int a = abs(c.bodyAPtrAndSignBit), b = abs(c.bodyBPtrAndSignBit);
        // copies exist for dynamic bodies only; static ones get the
        // out-of-range key numBodies and sort past every body
        incKeys[2 * m] = invMass[a] != 0.f ? (uint32_t)a : (uint32_t)numBodies;
        incVals[2 * m] = 2u * m;
        incKeys[2 * m + 1] = invMass[b] != 0.f ? (uint32_t)b : (uint32_t)numBodies;
        incVals[2 * m + 1] = 2u * m + 1u;
        pts += (int)c.worldNormal[3];
    }
    if (pts) atomicAdd(&counters->numContactPoints, pts);
}

// Ranges of the sorted copy list per body, and where each manifold's copies
// lie in it (a static side's place is past every body's range).
__global__ void k_body_ranges(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                              const int32_t* __restrict__ nDev, uint32_t* __restrict__ start,
                              uint32_t* __restrict__ end, uint32_t* __restrict__ incPos, int numBodies,
                              unsigned long long* __restrict__ sortBarrier) {
    const int n = *nDev;
    if (blockIdx.x == 0 && threadIdx.x == 0) *sortBarrier = 0ull;  // for the next sort
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        incPos[vals[i]] = (uint32_t)i;
        if (k >= (uint32_t)numBodies) continue;
        if (i == 0 || keys[i - 1] != k) start[k] = (uint32_t)i;
        if (i == n - 1 || keys[i + 1] != k) end[k] = (uint32_t)(i + 1);
    }
}

// ---------------------------------------------------------------------------
// Constraint setup (one thread per manifold). The contact is read where it lies:
// a copy of its 96 bytes, indexed by the point, went through local memory
// (1,048,576 cubes, 2.85 M manifolds: 602 -> 541 us; the 96 bytes read and 432
// written of each take 230 at 6.55 TB/s).
// ---------------------------------------------------------------------------
struct SetupParams {
    float dt;
    float erp;
    float contactProcessing;
    float slopOffset;
};

// Friction row along dir: (dir, rhs) to its stream, 1/diag returned.
__device__ __forceinline__ float setup_friction_row(const SolverView& V, int slot, int m, float3 dir, float3 r1,
                                                    float3 r2, float imA, float imB, float3 iiA, float3 iiB,
                                                    float cA, float cB, float3 vA, float3 wA, float3 vB, float3 wB) {
    const float3 t1 = cross(r1, dir);
    const float3 t2 = cross(r2, -dir);
    const float3 angA = mulv(iiA, t1);
    const float3 angB = mulv(iiB, t2);
    const float d0 = imA + dot(dir, cross(angA, r1));
    const float d1 = imB + dot(dir, cross(-angB, r2));
    const float denom = 1.f / (d0 + d1);
    const float scaled = 1.f / (d0 * cA + d1 * cB);
    const float relv = (dot(dir, vA) + dot(t1, wA)) + (-dot(dir, vB) + dot(t2, wB));
    const float rhs = (0.f - relv) * scaled;
    R(V, slot, m) = make_float4(dir.x, dir.y, dir.z, rhs);
    return denom;
}

__global__ void k_setup_rows(b3::BodiesDev Bd, SolverView V, const int* __restrict__ manifoldPair,
                             const b3Contact4* __restrict__ contacts, SetupParams SP,
                             unsigned long long* __restrict__ barrier) {
    const int M = *V.numManifolds;
    if (blockIdx.x == 0 && threadIdx.x == 0) *barrier = 0ull;  // of the solve that follows
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const b3Contact4& c = contacts[manifoldPair[m]];
        const int A = abs(c.bodyAPtrAndSignBit), B = abs(c.bodyBPtrAndSignBit);
        const float imA = Bd.invMass[A], imB = Bd.invMass[B];
        const bool dynA = imA != 0.f, dynB = imB != 0.f;
        const uint32_t sA = dynA ? V.incStart[A] : 0u, eA = dynA ? V.incEnd[A] : 0u;
        const uint32_t sB = dynB ? V.incStart[B] : 0u, eB = dynB ? V.incEnd[B] : 0u;
        const float kA = dynA ? (float)(eA - sA) : 1.f;
        const float kB = dynB ? (float)(eB - sB) : 1.f;
        const float3 iiA = dynA ? f3(Bd.invInertia[A]) : make_float3(0.f, 0.f, 0.f);
        const float3 iiB = dynB ? f3(Bd.invInertia[B]) : make_float3(0.f, 0.f, 0.f);
        const float3 pA = f3(Bd.pos[A]), pB = f3(Bd.pos[B]);
        // solver body velocities (static bodies contribute zero)
        const float3 vA = dynA ? f3(Bd.linVel[A]) : make_float3(0.f, 0.f, 0.f);
        const float3 wA = dynA ? f3(Bd.angVel[A]) : make_float3(0.f, 0.f, 0.f);
        const float3 vB = dynB ? f3(Bd.linVel[B]) : make_float3(0.f, 0.f, 0.f);
        const float3 wB = dynB ? f3(Bd.angVel[B]) : make_float3(0.f, 0.f, 0.f);
        const float restitution = Bd.restitution[A] * Bd.restitution[B];
        const float mu = c.friction;
        int nRows = 0;
        float fjac[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const int npts = (int)c.worldNormal[3];
        const bool solve = dynA || dynB;
        float3 n = normalize(make_float3(-c.worldNormal[0], -c.worldNormal[1], -c.worldNormal[2]));
        for (int j = 0; j < npts && solve; ++j) {
            const float4 wp = *reinterpret_cast<const float4*>(&c.worldPos[j][0]);
            const float depth = wp.w;
            const float dist = depth + SP.slopOffset;
            if (!(dist <= SP.contactProcessing)) continue;
            const float3 posB = f3(wp);
            const float3 posA = posB + n * dist;
            const float3 r1 = posA - pA;
            const float3 r2 = posB - pB;
            const float3 t0 = cross(r1, n);
            const float3 t1 = cross(r2, n);
            const float3 angA = mulv(iiA, t0);
            const float3 angB = mulv(iiB, -t1);
            const float d0 = imA + dot(n, cross(angA, r1));
            const float d1 = imB + dot(n, cross(-angB, r2));
            const float denom = 1.f / (d0 + d1);
            const float scaled = 1.f / (d0 * kA + d1 * kB);
            const float penetration = dist;  // + linearSlop (0)
            const float3 vel1 = vA + cross(wA, r1);
            const float3 vel2 = vB + cross(wB, r2);
            const float3 vel = vel1 - vel2;
            const float relv0 = dot(n, vel);
            float rest = restitution * -relv0;
            if (rest <= 0.f) rest = 0.f;
            const float v1n = dot(n, vA) + dot(t0, wA);
            const float v2n = -dot(n, vB) + dot(-t1, wB);
            const float relv = v1n + v2n;
            float posErr = 0.f;
            float velErr = rest - relv;
            if (penetration > 0.f) {
                velErr -= penetration / SP.dt;
            } else {
                posErr = -penetration * SP.erp / SP.dt;
            }
            const float rhs = posErr * scaled + velErr * scaled;
            const int s = kPoint0 + 4 * nRows;
            R(V, s + 0, m) = make_float4(r1.x, r1.y, r1.z, rhs);
            R(V, s + 1, m) = make_float4(r2.x, r2.y, r2.z, denom);
            // friction directions (convertContact :1015-1049)
            float3 d1v = vel - n * relv0;
            const float lat = dot(d1v, d1v);
            float3 d2v;
            if (lat > FLT_EPSILON) {
                d1v = d1v * (1.f / sqrtf(lat));
                d2v = normalize(cross(d1v, n));
            } else {
                plane_space(n, d1v, d2v);
            }
            const float q2 = setup_friction_row(V, s + 2, m, d2v, r1, r2, imA, imB, iiA, iiB, kA, kB, vA, wA, vB, wB);
            const float q1 = setup_friction_row(V, s + 3, m, d1v, r1, r2, imA, imB, iiA, iiB, kA, kB, vA, wA, vB, wB);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q == nRows) {
                    fjac[2 * q] = q2;
                    fjac[2 * q + 1] = q1;
                }
            ++nRows;
        }
        const int dyn = (dynA ? 1 : 0) | (dynB ? 2 : 0);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        R(V, kHead0, m) = make_float4(__uint_as_float(sA), __uint_as_float(eA), __uint_as_float(V.incPos[2 * m]),
                                      __uint_as_float(sB));
        R(V, kHead1, m) = make_float4(__uint_as_float(eB), __uint_as_float(V.incPos[2 * m + 1]),
                                      __int_as_float(nRows | dyn << 16), mu);
        R(V, kNorm, m) = f4(n, imA);
        R(V, kInA, m) = f4(iiA, imB);
        R(V, kInB, m) = f4(iiB);
        R(V, kIds, m) = make_float4(__int_as_float(A), __int_as_float(B), kA, kB);
        R(V, kFJac, m) = make_float4(fjac[0], fjac[1], fjac[2], fjac[3]);
        R(V, kFJac + 1, m) = make_float4(fjac[4], fjac[5], fjac[6], fjac[7]);
        R(V, kLamN, m) = zero;
        R(V, kLamF, m) = zero;
        R(V, kLamF + 1, m) = zero;
    }
}

// ---------------------------------------------------------------------------
// Persistent Jacobi kernels
// ---------------------------------------------------------------------------
// Both bodies' averages as the pass over the bodies left them, in the first
// record of each body's range.
__device__ __forceinline__ void read_averages(const float4* __restrict__ copies, const Heads& H, float3& vA, float3& wA,
                                              float3& vB, float3& wB) {
    if (H.dyn & 1) {
        vA = f3(__ldcg(&copies[2 * (size_t)H.sA]));
        wA = f3(__ldcg(&copies[2 * (size_t)H.sA + 1]));
    }
    if (H.dyn & 2) {
        vB = f3(__ldcg(&copies[2 * (size_t)H.sB]));
        wB = f3(__ldcg(&copies[2 * (size_t)H.sB + 1]));
    }
}

// The normal rows of one manifold in order, from the copies' velocities at
// the phase's start; the impulses go back to their stream.
template <bool TAPE, class Rows>
__device__ __forceinline__ void normal_rows(const Rows& S, int nRows, float3& dvA, float3& dwA, float3& dvB,
                                            float3& dwB, float4* tape) {
    const float4 nn = S(kNorm), ia = S(kInA), ib = S(kInB), l4 = S(kLamN);
    float4 a[4], b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // past the last point: that one again
        const int k = kPoint0 + 4 * min(j, nRows - 1);
        a[j] = S(k);
        b[j] = S(k + 1);
    }
    float lam[4] = {l4.x, l4.y, l4.z, l4.w};
    const float3 n = f3(nn);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (j < nRows)
            solve_row(n, arm(f3(a[j]), n), arm_neg(f3(b[j]), n), a[j].w, b[j].w, lam[j], 0.f, 1e10f, nn.w, ia.w, f3(ia),
                      f3(ib), dvA, dwA, dvB, dwB);
    const float4 r = make_float4(lam[0], lam[1], lam[2], lam[3]);
    S(kLamN) = r;
    if (TAPE) *tape = r;
}

// The friction rows, two per point that carries a normal impulse. Points are
// fetched one ahead of the one being solved, and only where they carry one
// (1,048,576 cubes 5.59 -> 5.46 ms).
template <bool TAPE, class Rows>
__device__ __forceinline__ void friction_rows(const Rows& S, int nRows, float mu, float3& dvA, float3& dwA,
                                              float3& dvB, float3& dwB, float4* tape, size_t cap) {
    const float4 n4 = S(kLamN), ia = S(kInA), ib = S(kInB);
    const float imA = S(kNorm).w;
    const float ln[4] = {n4.x, n4.y, n4.z, n4.w};
    float4 l4[2] = {S(kLamF), S(kLamF + 1)};
    const float4 q4[2] = {S(kFJac), S(kFJac + 1)};
    float4 a, b, d2, d1;
    auto fetch = [&](int j) {
        const int k = kPoint0 + 4 * j;
        a = S(k);
        b = S(k + 1);
        d2 = S(k + 2);
        d1 = S(k + 3);
    };
    a = b = d2 = d1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ln[0] > 0.f) fetch(0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j < nRows) {
            const float4 ca = a, cb = b, c2 = d2, c1 = d1;
            if (j < 3 && ln[j < 3 ? j + 1 : 3] > 0.f) fetch(j + 1);
            if (ln[j] > 0.f) {
                const float lim = mu * ln[j];
                const float3 r1 = f3(ca), r2 = f3(cb);
                float& m2 = (j & 1) ? l4[j >> 1].z : l4[j >> 1].x;
                float& m1 = (j & 1) ? l4[j >> 1].w : l4[j >> 1].y;
                const float j2 = (j & 1) ? q4[j >> 1].z : q4[j >> 1].x, j1 = (j & 1) ? q4[j >> 1].w : q4[j >> 1].y;
                solve_row(f3(c2), arm(r1, f3(c2)), arm_rev(r2, f3(c2)), c2.w, j2, m2, -lim, lim, imA, ia.w, f3(ia), f3(ib),
                          dvA, dwA, dvB, dwB);
                solve_row(f3(c1), arm(r1, f3(c1)), arm_rev(r2, f3(c1)), c1.w, j1, m1, -lim, lim, imA, ia.w, f3(ia), f3(ib),
                          dvA, dwA, dvB, dwB);
            }
        }
    }
    S(kLamF) = l4[0];
    S(kLamF + 1) = l4[1];
    if (TAPE) {
        tape[0] = l4[0];
        tape[cap] = l4[1];
    }
}

// One phase for one manifold: start each copy from its body's average of the
// previous phase (zero in the first phase), solve the manifold's normal or
// friction rows in order, store both copies in `out`. A copy of a manifold
// without rows keeps the average, as in the reference. PASS: the averages were
// formed by a pass over the bodies; otherwise each side gathers its body's
// copies here.
template <bool TAPE, bool PASS, class Rows>
__device__ __forceinline__ void solve_manifold(const Rows& S, bool friction, bool first, const float4* __restrict__ in,
                                               float4* __restrict__ out, int m, size_t cap, const b3::JacobiTape& T,
                                               int phase) {
    const Heads H = load_heads(S);
    float3 dvA = make_float3(0.f, 0.f, 0.f), dwA = dvA, dvB = dvA, dwB = dvA;
    if (!first) {
        if (PASS) read_averages(in, H, dvA, dwA, dvB, dwB);
        else gather_averages<4>(in, H, dvA, dwA, dvB, dwB);
    }
    float4* tn = TAPE ? T.lamN + (size_t)(phase >> 1) * cap + m : nullptr;
    float4* tf = TAPE ? T.lamF + (size_t)(phase & ~1) * cap + m : nullptr;
    float4* const tape = TAPE ? T.in + (size_t)phase * 4 * cap + m : nullptr;
    if (TAPE) {
        tape[0] = f4(dvA);
        tape[cap] = f4(dwA);
        tape[2 * cap] = f4(dvB);
        tape[3 * cap] = f4(dwB);
    }
    if (H.nRows > 0) {
        if (!friction) normal_rows<TAPE>(S, H.nRows, dvA, dwA, dvB, dwB, tn);
        else friction_rows<TAPE>(S, H.nRows, H.mu, dvA, dwA, dvB, dwB, tf, cap);
    } else if (TAPE) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!friction) *tn = zero;
        else tf[0] = tf[cap] = zero;
    }
    if (H.dyn & 1) {
        __stcg(&out[2 * (size_t)H.pA], f4(dvA));
        __stcg(&out[2 * (size_t)H.pA + 1], f4(dwA));
    }
    if (H.dyn & 2) {
        __stcg(&out[2 * (size_t)H.pB], f4(dvB));
        __stcg(&out[2 * (size_t)H.pB + 1], f4(dwB));
    }
}

__device__ __forceinline__ float4* copy_buffer(const SolverView& V, int buf) {
    return V.copies + (size_t)buf * 4 * V.cap;
}

// test of the give-up path: block 0 arrives late (bounded sleep)
__device__ __forceinline__ void hold_back(const SolverView& V, unsigned block) {
    if (V.holdMicros > 0 && block == 0 && threadIdx.x == 0)
        for (int i = 0; i < V.holdMicros; ++i) __nanosleep(1000);
}

// Phases p = 0 .. 2*iterations-1 alternate normal (even) and friction (odd)
// rows; the averaging of the reference happens at the start of the next
// phase from the double-buffered copies, so phases are separated by one
// bounded grid barrier each.
//
// k_jacobi, small scenes: what counts is the chain of a phase (barrier, copies
// in, rows, copies out). Two lanes share a manifold, one per body: each gathers
// its body's copies, forms its half of a row's J dv and takes the other's by a
// shuffle, so that a row is half the instructions in one warp. The first
// `resident` manifolds of a pair of lanes stay in shared memory for all phases,
// their rows with the angular parts formed. Of a phase's 3.5 us on 1,000 cubes a
// third each is the barrier, the way of the copies through L2 and the rows. 20
// phases, a lane per manifold -> two: 4,096 cubes (10,550 manifolds) 106 -> 90 us,
// 20,011 spheres (12,361) 113 -> 74, 33,000 falling bodies (9,400) 123 -> 71; with
// every row streamed in every phase 219, 162 and 211.
//
// Lane slots (float4 per lane): angular part and 1/diag of normal row j at j, of
// friction row r at 4 + r, then (inverse mass, inverse inertia) and (s, e, p,
// rows | dynamic << 16). Pair slots (float4 per manifold): (n, mu), rhs of the
// normal rows, (axis, rhs) of each friction row, impulses.
constexpr int kLaneBody = 12, kLaneHead = 13, kLaneSlots = 14;
constexpr int kPairNorm = 0, kPairRhs = 1, kPairFric = 2, kPairLam = 10, kPairSlots = 13;

struct LaneSide {
    uint32_t s, e, p;
    int nRows;
    bool dyn;
    float im;
    float3 ii;
};

// One manifold's rows as a lane sees them: in shared memory, or formed from the
// streams (manifolds beyond the resident ones).
struct KeptRows {
    static constexpr bool kKept = true;
    float4 *lane, *pair;  // strides tb and tb / 2
    int tb;
    __device__ __forceinline__ float4& at(int k) const { return pair[k * (tb / 2)]; }
    __device__ __forceinline__ float4 normal(int j, float3, bool) const { return lane[j * tb]; }
    __device__ __forceinline__ void point(int, bool, float4&) const {}
    __device__ __forceinline__ float4 friction(int r, const float4&, float3, bool, const float4*) const {
        return lane[(4 + r) * tb];
    }
    __device__ __forceinline__ LaneSide side(bool) const {
        const float4 b = lane[kLaneBody * tb], h = lane[kLaneHead * tb];
        const int f = __float_as_int(h.w);
        return LaneSide{__float_as_uint(h.x), __float_as_uint(h.y), __float_as_uint(h.z), f & 0xffff, (f >> 16) != 0,
                        b.x, make_float3(b.y, b.z, b.w)};
    }
    __device__ __forceinline__ float4 jac(int) const { return make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ float4 norm() const { return at(kPairNorm); }
    __device__ __forceinline__ float4 rhs() const { return at(kPairRhs); }
    __device__ __forceinline__ float4 axis(int r) const { return at(kPairFric + r); }
    __device__ __forceinline__ float4& lam(int k) const { return at(kPairLam + k); }
};
struct StreamRows {
    static constexpr bool kKept = false;
    SolverView V;
    int m;
    __device__ __forceinline__ float4 normal(int j, float3 n, bool isB) const {
        const float4 a = R(V, kPoint0 + 4 * j, m), b = R(V, kPoint0 + 4 * j + 1, m);
        return f4(isB ? arm_neg(f3(b), n) : arm(f3(a), n), b.w);
    }
    __device__ __forceinline__ void point(int j, bool isB, float4& r) const { r = R(V, kPoint0 + 4 * j + (isB ? 1 : 0), m); }
    __device__ __forceinline__ float4 friction(int r, const float4& arm0, float3 d, bool isB, const float4* jac) const {
        const float4 q = jac[r >> 2];
        const float j = (r & 3) == 0 ? q.x : (r & 3) == 1 ? q.y : (r & 3) == 2 ? q.z : q.w;
        return f4(isB ? arm_rev(f3(arm0), d) : arm(f3(arm0), d), j);
    }
    __device__ __forceinline__ LaneSide side(bool isB) const {
        const Heads H = load_heads(GlobalRows{V.rows + m, (size_t)V.cap});
        const float4 nn = R(V, kNorm, m), ia = R(V, kInA, m), ib = R(V, kInB, m);
        return isB ? LaneSide{H.sB, H.eB, H.pB, H.nRows, (H.dyn & 2) != 0, ia.w, f3(ib)}
                   : LaneSide{H.sA, H.eA, H.pA, H.nRows, (H.dyn & 1) != 0, nn.w, f3(ia)};
    }
    __device__ __forceinline__ float4 jac(int k) const { return R(V, kFJac + k, m); }
    __device__ __forceinline__ float4 norm() const {
        const float4 n = R(V, kNorm, m);
        return make_float4(n.x, n.y, n.z, R(V, kHead1, m).w);
    }
    __device__ __forceinline__ float4 rhs() const {
        return make_float4(R(V, kPoint0, m).w, R(V, kPoint0 + 4, m).w, R(V, kPoint0 + 8, m).w, R(V, kPoint0 + 12, m).w);
    }
    __device__ __forceinline__ float4 axis(int r) const { return R(V, kPoint0 + 4 * (r >> 1) + 2 + (r & 1), m); }
    __device__ __forceinline__ float4& lam(int k) const { return R(V, k == 0 ? kLamN : kLamF + k - 1, m); }
};

// A row by its two lanes: solve_row with each side's products in its own lane.
__device__ __forceinline__ void half_row(float3 n, const float4& t, float rhs, float& lam, float lo, float hi, bool on,
                                         bool isB, const LaneSide& L, float3& v, float3& w) {
    const float x = dot_fma(n, v), y = dot_fma(f3(t), w);
    const float own = __fadd_rn(y, isB ? -x : x);
    const float other = __shfl_xor_sync(0xffffffffu, own, 1);
    float delta = __fmaf_rn(-(isB ? other : own), t.w, rhs);
    delta = __fmaf_rn(-(isB ? own : other), t.w, delta);
    const float sum = lam + delta;
    const float na = sum < lo ? lo : sum > hi ? hi : sum;
    delta = sum < lo || sum > hi ? na - lam : delta;
    delta = on ? delta : 0.f;  // a row that is not solved changes nothing
    lam = on ? na : lam;
    // A: v + n (im delta); B: v + (-n im) delta
    v = fma3(n * (isB ? -L.im : 1.f), (isB ? 1.f : L.im) * delta, v);
    w = fma3(mulv(L.ii, f3(t)), delta, w);
}

// The lane's body's average over its copies, the first K in flight at once.
template <int K>
__device__ __forceinline__ void gather_side(const float4* copies, const LaneSide& L, float3& v, float3& w) {
    float3 sl = make_float3(0.f, 0.f, 0.f), sa = sl;
    for (uint32_t i0 = L.s; i0 < L.e; i0 += K) {
        float4 l[K], a[K];
#pragma unroll
        for (int u = 0; u < K; ++u) {
            const float4* r = copies + 2 * (size_t)min(i0 + u, L.e - 1u);
            l[u] = __ldcg(r);
            a[u] = __ldcg(r + 1);
        }
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (i0 + u < L.e) {
                sl += f3(l[u]);
                sa += f3(a[u]);
            }
    }
    if (L.dyn) {
        const float f = 1.f / (float)(L.e - L.s);
        v = scaled(sl, f);
        w = scaled(sa, f);
    }
}

// A phase of one manifold by two lanes (a warp's lanes go through it together;
// on: the manifold exists).
template <bool TAPE, class Rows>
__device__ __forceinline__ void pair_phase(const Rows& S, bool isB, bool on, bool friction, bool first, const float4* in,
                                           float4* out, int m, size_t cap, const b3::JacobiTape& T, int phase) {
    LaneSide L = Rows::kKept || on ? S.side(isB) : LaneSide{0u, 0u, 0u, 0, false, 0.f, make_float3(0.f, 0.f, 0.f)};
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float3 v = make_float3(0.f, 0.f, 0.f), w = v;
    if (!first) gather_side<4>(in, L, v, w);
    if (TAPE && on) {
        float4* tape = T.in + ((size_t)phase * 4 + (isB ? 2 : 0)) * cap + m;
        tape[0] = f4(v);
        tape[cap] = f4(w);
    }
    const int most = __reduce_max_sync(0xffffffffu, L.nRows);
    const float4 l4 = Rows::kKept || on ? S.lam(0) : zero;
    float ln[4] = {l4.x, l4.y, l4.z, l4.w};
    if (!friction) {
        const float4 n4 = Rows::kKept || on ? S.norm() : zero, r4 = Rows::kKept || on ? S.rhs() : zero;
        const float rhs[4] = {r4.x, r4.y, r4.z, r4.w};
        const float3 n = f3(n4);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < most) {
                const bool row = j < L.nRows;
                half_row(n, Rows::kKept || row ? S.normal(j, n, isB) : zero, rhs[j], ln[j], 0.f, 1e10f, row, isB, L, v, w);
            }
        const float4 r = make_float4(ln[0], ln[1], ln[2], ln[3]);
        if ((Rows::kKept || on) && !isB) {
            S.lam(0) = r;
            if (TAPE && on) T.lamN[(size_t)(phase >> 1) * cap + m] = r;
        }
    } else {
        const float mu = Rows::kKept || on ? S.norm().w : 0.f;
        float4 f0 = Rows::kKept || on ? S.lam(1) : zero, f1 = Rows::kKept || on ? S.lam(2) : zero;
        float lam[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
        float4 jac[2] = {zero, zero}, arm0 = zero;
        if (!Rows::kKept && on) {
            jac[0] = S.jac(0);
            jac[1] = S.jac(1);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < most) {
                const bool row = j < L.nRows, solve = row && ln[j] > 0.f;
                const float lim = mu * ln[j];
                if (row) S.point(j, isB, arm0);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int r = 2 * j + q;
                    const float4 d = Rows::kKept || row ? S.axis(r) : zero;
                    half_row(f3(d), Rows::kKept || row ? S.friction(r, arm0, f3(d), isB, jac) : zero, d.w, lam[r], -lim, lim, solve, isB,
                             L, v, w);
                }
            }
        f0 = make_float4(lam[0], lam[1], lam[2], lam[3]);
        f1 = make_float4(lam[4], lam[5], lam[6], lam[7]);
        if ((Rows::kKept || on) && !isB) {
            S.lam(1) = f0;
            S.lam(2) = f1;
            if (TAPE && on) {
                float4* tf = T.lamF + (size_t)(phase & ~1) * cap + m;
                tf[0] = f0;
                tf[cap] = f1;
            }
        }
    }
    if (L.dyn) {
        __stcg(&out[2 * (size_t)L.p], f4(v));
        __stcg(&out[2 * (size_t)L.p + 1], f4(w));
    }
    __syncwarp();  // the impulses one lane writes, both read
}

// Blocks without a manifold leave: the barriers are among the others.
template <bool TAPE>
__global__ void __launch_bounds__(256, 1)
k_jacobi(SolverView V, int iterations, int resident, int most, uint32_t* bar, int32_t* err, b3Counters* counters,
         b3::JacobiTape T) {
    extern __shared__ float4 kept[];  // [resident]([kLaneSlots][blockDim], [kPairSlots][blockDim / 2])
    const int M = *V.numManifolds;
    if (M > most) return;  // the pass over the bodies takes them
    const int phases = 2 * iterations;
    const int tb = (int)blockDim.x, tid = (int)threadIdx.x;
    const unsigned busy = min(gridDim.x, (unsigned)(M + tb / 2 - 1) / (unsigned)(tb / 2));
    // from the last block of the grid on: the first ones of a cooperative grid come
    // several to an SM
    const unsigned block = gridDim.x - 1 - blockIdx.x;
    if (block >= busy) return;
    GridBarrier barrier(bar, err, counters, V.spinLimit, true, busy);
    const bool isB = tid & 1;
    const int m0 = (block * tb + tid) >> 1, warp0 = (block * tb + (tid & ~31)) >> 1;
    const int stride = (gridDim.x * tb) >> 1;
    const int each = kLaneSlots * tb + kPairSlots * (tb / 2);
    auto rows = [&](int k) {
        float4* at = kept + (size_t)k * each;
        return KeptRows{at + tid, at + kLaneSlots * tb + (tid >> 1), tb};
    };
    for (int k = 0; k < resident; ++k) {
        const int m = m0 + k * stride;
        const KeptRows K = rows(k);
        if (m >= M) {  // no manifold: nothing to solve, no copies
            for (int q = 0; q < kLaneSlots; ++q) K.lane[q * tb] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int q = 0; q < kPairSlots && !isB; ++q) K.at(q) = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const StreamRows S{V, m};
        const LaneSide L = S.side(isB);
        const float4 n = S.norm();
        const float4 jac[2] = {S.jac(0), S.jac(1)};
        K.lane[kLaneBody * tb] = make_float4(L.im, L.ii.x, L.ii.y, L.ii.z);
        K.lane[kLaneHead * tb] = make_float4(__uint_as_float(L.s), __uint_as_float(L.e), __uint_as_float(L.p),
                                             __int_as_float(L.nRows | (L.dyn ? 1 << 16 : 0)));
        if (!isB) {
            K.at(kPairNorm) = n;
            K.at(kPairRhs) = S.rhs();
#pragma unroll
            for (int q = 0; q < 3; ++q) K.lam(q) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // rows past the last one stay zero: a warp goes through as many as any of
        // its manifolds has
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = L.nRows; j < 4; ++j) {
            K.lane[j * tb] = K.lane[(4 + 2 * j) * tb] = K.lane[(5 + 2 * j) * tb] = zero;
            if (!isB) K.at(kPairFric + 2 * j) = K.at(kPairFric + 2 * j + 1) = zero;
        }
        for (int j = 0; j < L.nRows; ++j) {
            float4 arm0;
            S.point(j, isB, arm0);
            K.lane[j * tb] = S.normal(j, f3(n), isB);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float4 d = S.axis(2 * j + q);
                K.lane[(4 + 2 * j + q) * tb] = S.friction(2 * j + q, arm0, f3(d), isB, jac);
                if (!isB) K.at(kPairFric + 2 * j + q) = d;
            }
        }
    }
    __syncwarp();
    for (int p = 0; p < phases; ++p) {
        if (p == 1) hold_back(V, block);
        if (p > 0 && !barrier.wait()) return;
        const bool friction = (p & 1) != 0, first = p == 0;
        const float4* in = copy_buffer(V, (p - 1) & 1);
        float4* out = copy_buffer(V, p & 1);
        int m = m0, k = 0;
        for (int base = warp0; base < M; base += stride, m += stride, ++k) {
            if (k < resident)
                pair_phase<TAPE>(rows(k), isB, m < M, friction, first, in, out, m, V.cap, T, p);
            else
                pair_phase<TAPE>(StreamRows{V, min(m, M - 1)}, isB, m < M, friction, first, in, out, m, V.cap, T, p);
        }
    }
}

// k_jacobi_pass, large scenes: what counts is the bytes of a phase. A body's
// copies are read once, by a pass over the bodies between two barriers that
// leaves the average in the first record of the body's range, instead of once
// per manifold of the body (at 5.4 copies a body, 64 B instead of 350 B of L2
// reads per manifold and phase); the extra barrier is a few microseconds.
// 1,048,576 cubes (2.85 M manifolds): 7.22 -> 5.46 ms, of which the streams
// and copies take 4.4 ms at 6.55 TB/s; 131,072 mixed bodies (395 K): 1.26 -> 0.90 ms.
template <bool TAPE>
__global__ void __launch_bounds__(256, 2)
k_jacobi_pass(SolverView V, int iterations, int above, uint32_t* bar, int32_t* err, b3Counters* counters,
              b3::JacobiTape T) {
    const int M = *V.numManifolds;
    if (M <= above) return;  // k_jacobi took them
    GridBarrier barrier(bar, err, counters, V.spinLimit, true);
    const int phases = 2 * iterations;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    for (int p = 0; p < phases; ++p) {
        if (p == 1) hold_back(V, blockIdx.x);
        const float4* in = copy_buffer(V, (p - 1) & 1);
        if (p > 0) {
            if (!barrier.wait()) return;
            float4* mean = copy_buffer(V, (p - 1) & 1);
            for (int b = t0; b < V.numBodies; b += stride) {
                const uint32_t s = V.incStart[b], e = V.incEnd[b];
                if (e <= s + 1) continue;  // no copies, or its own average
                float3 l, a;
                copy_average<4>(in, s, e, l, a);
                __stcg(&mean[2 * (size_t)s], f4(l));
                __stcg(&mean[2 * (size_t)s + 1], f4(a));
            }
            if (!barrier.wait()) return;
        }
        for (int m = t0; m < M; m += stride)
            solve_manifold<TAPE, true>(GlobalRows{V.rows + m, (size_t)V.cap}, (p & 1) != 0, p == 0, in,
                                                 copy_buffer(V, p & 1), m, V.cap, T, p);
    }
}

// Batched worlds: the manifolds of one world are contiguous (the pair list
// follows the world-major cell keys) and touch only that world's bodies, so
// a block can run all phases of a world by itself with block barriers in
// place of grid barriers. Same per-manifold arithmetic and averaging order
// as k_jacobi, hence bit-identical results.
// Span [start, end) of each world's manifolds. When a world's manifolds are
// not contiguous (pairs between two large bodies come after the tiles) the
// span covers foreign manifolds, which k_jacobi_worlds skips: every
// manifold is still solved by its own world's block only.
__global__ void k_world_ranges(SolverView V, const int* __restrict__ worldId, int* __restrict__ start,
                               int* __restrict__ end) {
    const int M = *V.numManifolds;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const int w = worldId[__float_as_int(R(V, kIds, m).x)];
        if (m == 0 || worldId[__float_as_int(R(V, kIds, m - 1).x)] != w) atomicMin(&start[w], m);
        if (m == M - 1 || worldId[__float_as_int(R(V, kIds, m + 1).x)] != w) atomicMax(&end[w], m + 1);
    }
}

template <bool TAPE>
__global__ void __launch_bounds__(256)
k_jacobi_worlds(SolverView V, int iterations, const int* __restrict__ start, const int* __restrict__ end,
                int numWorlds, const int* __restrict__ worldId, b3::JacobiTape T) {
    const int phases = 2 * iterations;
    for (int w = blockIdx.x; w < numWorlds; w += gridDim.x) {
        const int s = start[w], e = end[w];
        if (s >= e) continue;
        for (int p = 0; p < phases; ++p) {
            if (p > 0) __syncthreads();
            for (int m = s + (int)threadIdx.x; m < e; m += blockDim.x)
                if (worldId[__float_as_int(R(V, kIds, m).x)] == w)
                    solve_manifold<TAPE, false>(GlobalRows{V.rows + m, (size_t)V.cap}, (p & 1) != 0, p == 0,
                                                          copy_buffer(V, (p - 1) & 1), copy_buffer(V, p & 1), m, V.cap,
                                                          T, p);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Integration (copyVelocitiesKernel + integrateTransformsKernel2)
// ---------------------------------------------------------------------------
struct IntegrateParams {
    float dt;
    float damping;
    float threshold;  // BT_GPU_ANGULAR_MOTION_THRESHOLD = 0.25 * pi
};

__global__ void k_integrate(b3::BodiesDev Bd, SolverView V, int finalBuf, IntegrateParams P, int applySolve) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Bd.n) return;
    if (Bd.invMass[i] == 0.f) return;
    float4 v = Bd.linVel[i];
    float4 w = Bd.angVel[i];
    // solveGroupCacheFriendlyFinish (:1790-1803): each of the k copies adds
    // sum/k of the last averaging to the body velocity
    if (applySolve && V.incEnd[i] > V.incStart[i]) {
        const uint32_t k = V.incEnd[i] - V.incStart[i];
        float3 sl, sa;
        copy_average<4>(copy_buffer(V, finalBuf), V.incStart[i], V.incEnd[i], sl, sa);
        for (uint32_t c = 0; c < k; ++c) {
            v.x += sl.x; v.y += sl.y; v.z += sl.z;
            w.x += sa.x; w.y += sa.y; w.z += sa.z;
        }
    }
    v.w = 0.f;
    w.x *= P.damping;
    w.y *= P.damping;
    w.z *= P.damping;
    w.w = 0.f;
    float fAngle = sqrtf(w.x * w.x + w.y * w.y + w.z * w.z);
    if (fAngle * P.dt > P.threshold) fAngle = P.threshold / P.dt;
    float s;
    if (fAngle < 0.001f) {
        s = 0.5f * P.dt - (P.dt * P.dt * P.dt) * 0.020833333333f * fAngle * fAngle;
    } else {
        s = sinf(0.5f * fAngle * P.dt) / fAngle;
    }
    const float4 dorn = make_float4(w.x * s, w.y * s, w.z * s, cosf(fAngle * P.dt * 0.5f));
    const float4 q0 = Bd.quat[i];
    float4 q = quat_mult(dorn, q0);
    const float len = sqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
    if (len > 0.f) {
        const float il = 1.f / len;
        q.x *= il; q.y *= il; q.z *= il; q.w *= il;
    } else {
        q = make_float4(0.f, 0.f, 0.f, 1.f);
    }
    float4 p = Bd.pos[i];
    p.x += v.x * P.dt;
    p.y += v.y * P.dt;
    p.z += v.z * P.dt;
    Bd.pos[i] = p;
    Bd.quat[i] = q;
    Bd.linVel[i] = v;
    Bd.angVel[i] = w;
}

}  // namespace

SolverView b3solver::solver_view(b3World_t* w) {
    SolverView V;
    V.rows = w->d.rows;
    V.cap = w->cfg.maxPairs;
    V.copies = w->d.copies;
    V.incPos = w->d.incPos;
    V.incStart = w->d.bodyIncStart;
    V.incEnd = w->d.bodyIncEnd;
    V.numManifolds = w->d.scalars + b3::S_NUM_MANIFOLDS;
    V.numBodies = (int)w->bodies.size();
    V.spinLimit = w->waitSpinLimit;
    V.holdMicros = w->waitHoldMicros;
    return V;
}

namespace b3 {

int launch_manifolds(b3World_t* w, cudaStream_t st) {
    const int N = (int)w->bodies.size();
    const int cap = w->cfg.maxPairs;
    if (cap == 0 || N == 0) {
        B3_CUDA(cudaMemsetAsync(w->d.scalars + S_NUM_MANIFOLDS, 0, sizeof(int32_t) * 2, st));
        if (N > 0) B3_CUDA(cudaMemsetAsync(w->d.bodyIncStart, 0, 2 * sizeof(uint32_t) * (size_t)w->capBodies, st));
        return B3_OK;
    }
    // the scan's words and the bodies' ranges in one
    B3_CUDA(cudaMemsetAsync(w->d.manifoldZero, 0, w->d.manifoldScanBytes + 2 * sizeof(uint32_t) * (size_t)w->capBodies,
                            st));
    // manifold slots: the pairs', then (compound and mesh worlds) the sub-pairs'
    const int32_t* slots = w->d.scalars + (w->hasSubPairs() ? S_NUM_SLOTS : S_NUM_PAIRS);
    B3_TRY(exclusive_scan_u32(w->d.manifoldFlag, w->d.manifoldScan, slots, cap,
                              (uint32_t*)(w->d.scalars + S_NUM_MANIFOLDS), w->d.manifoldZero,
                              w->d.manifoldScanBytes, w->d.scalars + S_ERR, st, w->ctx->numSMs, true));
    const int g = w->ctx->numSMs * 8;
    k_manifold_emit<<<g, 256, 0, st>>>(w->d.manifoldFlag, w->d.manifoldScan, slots,
                                      w->d.contacts, w->d.invMass, N, w->d.manifoldPair, w->d.incKeys,
                                      w->d.incVals, w->d.scalars, w->d.counters);
    B3_CHECK_LAUNCH();
    if (w->gs) return B3_OK;  // body incidences serve the Jacobi averaging only
    bool alt = false;
    B3_TRY(radix_sort_pairs(w->d.incKeys, w->d.incVals, w->d.incKeysAlt, w->d.incValsAlt,
                            w->d.scalars + S_NUM_INC, 2LL * cap, w->bodyBits, w->d.incSortScratch,
                            w->d.incSortScratchBytes, w->d.scalars + S_ERR, st, &alt, w->ctx->numSMs, 6LL * N, true));
    k_body_ranges<<<g, 256, 0, st>>>(alt ? w->d.incKeysAlt : w->d.incKeys, alt ? w->d.incValsAlt : w->d.incVals,
                                    w->d.scalars + S_NUM_INC, w->d.bodyIncStart, w->d.bodyIncEnd, w->d.incPos, N,
                                    (unsigned long long*)w->d.incSortScratch);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

int launch_solver(b3World_t* w, cudaStream_t st) { return launch_solver_taped(w, st, nullptr); }

int launch_solver_taped(b3World_t* w, cudaStream_t st, const JacobiTape* tape) {
    if (w->cfg.maxPairs == 0 || w->bodies.empty()) return B3_OK;
    if (w->gs) {
        if (tape) {
            b3_set_error("the adjoint form runs the Jacobi solver only");
            return B3_ERR_UNSUPPORTED;
        }
        return launch_gs_solver(w, st);
    }
    SolverView V = solver_view(w);
    SetupParams SP;
    SP.dt = w->sim.dt;
    SP.erp = w->sim.erp;
    SP.contactProcessing = w->sim.contactProcessing;
    SP.slopOffset = w->sim.slopOffset;
    const int g = w->ctx->numSMs * 8;
    const bool worlds = w->solverMode == 1 && w->cfg.numWorlds > 1, pass = w->solverGather == 1;
    k_setup_rows<<<g, 128, 0, st>>>(w->bodiesDev(), V, w->d.manifoldPair, w->d.contacts, SP,
                                    (unsigned long long*)(w->d.scalars + S_BAR_COUNT));
    B3_CHECK_LAUNCH();
    if (w->timing && w->setupEv) B3_CUDA(cudaEventRecord(w->setupEv, st));
    if (worlds) {
        // one block per world at a time, block barriers between phases
        const int nw = w->cfg.numWorlds;
        B3_CUDA(cudaMemsetAsync(w->d.worldMStart, 0x7f, sizeof(int) * nw, st));  // 0x7f7f7f7f: above any index
        B3_CUDA(cudaMemsetAsync(w->d.worldMEnd, 0, sizeof(int) * nw, st));
        k_world_ranges<<<w->ctx->numSMs * 4, 256, 0, st>>>(V, w->d.worldId, w->d.worldMStart, w->d.worldMEnd);
        B3_CHECK_LAUNCH();
        const int threads = w->solverThreads;
        const void* kw = tape ? (const void*)k_jacobi_worlds<true> : (const void*)k_jacobi_worlds<false>;
        int occ = 1;
        B3_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kw, threads, 0));
        occ = occ < 1 ? 1 : occ;
        const int grid = std::min(nw, w->ctx->numSMs * occ);
        int iters = w->sim.iterations;
        int nwv = nw;
        JacobiTape T = tape ? *tape : JacobiTape{};
        int* ws = w->d.worldMStart;
        int* we = w->d.worldMEnd;
        const int* wid = w->d.worldId;
        void* args[] = {&V, &iters, &ws, &we, &nwv, &wid, &T};
        B3_CUDA(cudaLaunchKernel(kw, dim3(grid), dim3(threads), args, 0, st));
        return B3_OK;
    }
    // persistent cooperative Jacobi: k_jacobi where the rows fit the shared
    // memories, the pass over the bodies beyond; where the body count leaves it
    // open both are launched and the one that the manifolds call for runs
    int iters = w->sim.iterations;
    uint32_t* bar = (uint32_t*)(w->d.scalars + S_BAR_COUNT);
    int32_t* err = w->d.scalars + S_ERR;
    b3Counters* ctr = w->d.counters;
    JacobiTape T = tape ? *tape : JacobiTape{};
    auto launch = [&](const void* kern, int threads, int occCap, int want, size_t smem, void** args) -> int {
        if (smem > 48 * 1024) B3_TRY(allow_dynamic_smem(w->ctx, kern));
        int occ = 1;
        B3_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem));
        occ = std::max(1, std::min(occ, occCap));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(std::min(w->ctx->numSMs * occ, want));
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        B3_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
        return B3_OK;
    };
    const long long est = std::min<long long>((long long)w->cfg.maxPairs, w->expectedManifolds());
    const bool open = pass && est <= 512 * 1024;
    int above = -1;
    if (!pass || open) {
        // shared memory for as many of a thread's manifolds as the scene is
        // expected to have, up to one block's share of an SM
        const int threads = open ? 128 : w->solverThreads, share = threads / 2;
        const int occCap = open ? 4 : w->solverOccCap;
        const int want = (int)std::max<long long>(1, (est + share - 1) / share);
        const size_t one = (size_t)(kLaneSlots * threads + kPairSlots * share) * sizeof(float4);
        const int blocks = std::min(w->ctx->numSMs * occCap, want);
        const int perSm = (blocks + w->ctx->numSMs - 1) / w->ctx->numSMs;
        const int need = open ? 1 : (int)((est + (long long)blocks * share - 1) / ((long long)blocks * share));
        int resident = std::min(need, (int)(((size_t)w->ctx->maxSmemOptin - 1024 * (perSm - 1)) / perSm / one));
        int most = 0x7fffffff;
        if (open) above = most = blocks * share * resident;
        void* args[] = {&V, &iters, &resident, &most, &bar, &err, &ctr, &T};
        B3_TRY(launch(tape ? (const void*)k_jacobi<true> : (const void*)k_jacobi<false>, threads, occCap, want,
                      one * resident, args));
    }
    if (pass) {
        const int threads = w->solverThreads;
        const int want = (int)std::max<long long>(1, (est + threads - 1) / threads);
        void* args[] = {&V, &iters, &above, &bar, &err, &ctr, &T};
        B3_TRY(launch(tape ? (const void*)k_jacobi_pass<true> : (const void*)k_jacobi_pass<false>, threads,
                      w->solverOccCap, want, 0, args));
    }
    return B3_OK;
}

int launch_integrate(b3World_t* w, cudaStream_t st) {
    const int N = (int)w->bodies.size();
    if (N == 0) return B3_OK;
    IntegrateParams P;
    P.dt = w->sim.dt;
    P.damping = w->sim.angularDamping;
    P.threshold = 0.25f * 3.14159254f;
    const int iters = w->sim.iterations;
    // the batched Gauss-Seidel solver leaves final velocities in the bodies
    k_integrate<<<(N + 255) / 256, 256, 0, st>>>(w->bodiesDev(), solver_view(w), (2 * iters - 1) & 1, P,
                                                iters > 0 && !w->gs ? 1 : 0);
    B3_CHECK_LAUNCH();
    return B3_OK;
}

}  // namespace b3
