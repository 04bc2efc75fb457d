// Shared by the Jacobi solver (solver.cu) and its adjoint (adjoint.cu):
// constraint-row storage, the solver view of the world's buffers, the row
// update, the per-body averaging and the bounded grid barrier.
#pragma once
#include "b3_math.cuh"
#include "b3_world.h"

namespace b3solver {

using namespace b3m;

// Row storage: kRowSlots float4 streams of length cap (slot major), one
// element per manifold.
//   kHead0  sA, eA, pA, sB as ints: [s, e) is the body's range of the copy
//           array, p this manifold's own copy in it (s = e for a static side)
//   kHead1  eB, pB, nRows | dyn << 16 as ints, mu
//   kNorm   n.xyz, invMassA
//   kInA    invInertiaA.xyz, invMassB
//   kInB    invInertiaB.xyz, -
//   kIds    bodies A and B as ints, copy counts A and B (set-up and the
//           adjoint only; no phase reads it)
//   point j (j < 4), kPoint0 + 4j: (r1, rhs) and (r2, 1/diag) of its normal
//           row, (d2, rhs) and (d1, rhs) of its two friction rows
//   kFJac   1/diag of the friction rows, two streams of four (row 2j: d2,
//           row 2j + 1: d1)
//   kLamN   impulses of the four normal rows; kLamF, + 1: of the friction rows
// A row's angular parts are r1 x axis and -(r2 x axis): recomputing them (12
// FMAs) costs less than the 32 bytes a row they would take, since the large
// scenes' solve is bound by these streams: 592 B per manifold and iteration
// at three points, 752 B with every row's angular parts stored.
constexpr int kHead0 = 0, kHead1 = 1, kNorm = 2, kInA = 3, kInB = 4;
constexpr int kPoint0 = 5;
constexpr int kFJac = 21;
constexpr int kLamN = 23;
constexpr int kLamF = 24;
constexpr int kIds = 26;
constexpr int kRowSlots = 27;
static_assert(kRowSlots == b3::kSolverRowSlots, "the allocation holds every stream");

struct SolverView {
    float4* rows;       // [kRowSlots][cap]
    int cap;            // manifold capacity (stride)
    // solver-body copies, (linear, angular) pairs sorted by body: the copies
    // of body b are [incStart[b], incEnd[b]), in manifold order
    float4* copies;     // [2 buffers][2 cap][2]
    const uint32_t* incPos;    // manifold side 2m + side -> its copy
    const uint32_t* incStart;  // per body
    const uint32_t* incEnd;
    const int32_t* numManifolds;
    int numBodies;
    // bounded waits of the persistent Jacobi kernel: polls of a grid
    // barrier before it gives up, and (testing the give-up path only) how
    // long block 0 holds back before its first barrier, in microseconds
    int spinLimit;
    int holdMicros;
};

__device__ __forceinline__ float4& R(const SolverView& v, int slot, int m) {
    return v.rows[(size_t)slot * v.cap + m];
}

// btPlaneSpace1 (LinearMath/btVector3.h), published construction of two
// unit tangents orthogonal to n.
__device__ __forceinline__ void plane_space(float3 n, float3& p, float3& q) {
    const float SQRT12 = 0.7071067811865475244008443621048490f;
    if (fabsf(n.z) > SQRT12) {
        const float a = n.y * n.y + n.z * n.z;
        const float k = rsqrtf(a);
        p = make_float3(0.f, -n.z * k, n.y * k);
        q = make_float3(a * k, -n.x * p.z, n.x * p.y);
    } else {
        const float a = n.x * n.x + n.y * n.y;
        const float k = rsqrtf(a);
        p = make_float3(-n.y * k, n.x * k, 0.f);
        q = make_float3(-n.z * p.y, n.z * p.x, a * k);
    }
}

// ---------------------------------------------------------------------------
// Persistent-kernel helpers
// ---------------------------------------------------------------------------
using b3dev::GridBarrier;

// Angular part of a row, r x axis, formed again in every phase: one multiply
// and one fused multiply-add per component, by name.
__device__ __forceinline__ float3 arm(float3 r, float3 axis) {
    return make_float3(__fmaf_rn(r.y, axis.z, -__fmul_rn(r.z, axis.y)), __fmaf_rn(r.z, axis.x, -__fmul_rn(r.x, axis.z)),
                       __fmaf_rn(r.x, axis.y, -__fmul_rn(r.y, axis.x)));
}

// The other body's part, -(r x axis): of a normal row the negated product above,
// of a friction row r x -axis, with the subtraction turned round.
__device__ __forceinline__ float3 arm_neg(float3 r, float3 axis) {
    return make_float3(__fmaf_rn(-r.y, axis.z, __fmul_rn(r.z, axis.y)), __fmaf_rn(-r.z, axis.x, __fmul_rn(r.x, axis.z)),
                       __fmaf_rn(-r.x, axis.y, __fmul_rn(r.y, axis.x)));
}
__device__ __forceinline__ float3 arm_rev(float3 r, float3 axis) {
    return make_float3(__fmaf_rn(r.z, axis.y, -__fmul_rn(r.y, axis.z)), __fmaf_rn(r.x, axis.z, -__fmul_rn(r.z, axis.x)),
                       __fmaf_rn(r.y, axis.x, -__fmul_rn(r.x, axis.y)));
}
__device__ __forceinline__ float dot_fma(float3 a, float3 b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ float3 fma3(float3 a, float s, float3 c) {
    return make_float3(__fmaf_rn(a.x, s, c.x), __fmaf_rn(a.y, s, c.y), __fmaf_rn(a.z, s, c.z));
}

// One row: axis n, angular parts t1 and t2, applied impulse lam in and out.
__device__ __forceinline__ void solve_row(float3 n, float3 t1, float3 t2, float rhs, float jac, float& lam, float lo,
                                          float hi, float imA, float imB, float3 iiA, float3 iiB, float3& dvA,
                                          float3& dwA, float3& dvB, float3& dwB) {
    float delta = rhs;  // - applied * cfm (cfm = 0)
    // every product and sum by name: the compiler contracts such expressions
    // by their surroundings (unrolled or not, velocities known to be zero or
    // not), and all forms of the solve have to give the same bits
    const float dv1 = __fadd_rn(dot_fma(n, dvA), dot_fma(t1, dwA));
    const float dv2 = __fsub_rn(dot_fma(t2, dwB), dot_fma(n, dvB));
    delta = __fmaf_rn(-dv1, jac, delta);
    delta = __fmaf_rn(-dv2, jac, delta);
    const float sum = lam + delta;
    float na;
    if (sum < lo) {
        delta = lo - lam;
        na = lo;
    } else if (sum > hi) {
        delta = hi - lam;
        na = hi;
    } else {
        na = sum;
    }
    lam = na;
    dvA = fma3(n, imA * delta, dvA);
    dwA = fma3(mulv(iiA, t1), delta, dwA);
    dvB = fma3(-n * imB, delta, dvB);
    dwB = fma3(mulv(iiB, t2), delta, dwB);
}

// a * s rounded by itself: fused into the row that adds to it, an average
// would round differently where it is formed next to the rows and where it is
// read back from memory.
__device__ __forceinline__ float3 scaled(float3 a, float s) {
    return make_float3(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s));
}

// Average over the copies [s, e) of one body (averageVelocities,
// P2/btPgsJacobiSolver.cpp:1683-1720): copies in manifold order, sum then
// multiply by 1/count. K records are in flight at a time; the order of the
// sum does not depend on K.
template <int K>
__device__ __forceinline__ void copy_average(const float4* __restrict__ copies, uint32_t s, uint32_t e, float3& lin,
                                             float3& ang) {
    float3 sl = make_float3(0.f, 0.f, 0.f), sa = sl;
    for (uint32_t i0 = s; i0 < e; i0 += K) {
        float4 l[K], a[K];
#pragma unroll
        for (int u = 0; u < K; ++u) {  // past the end: the last record again
            const float4* r = copies + 2 * (size_t)min(i0 + u, e - 1u);
            l[u] = __ldcg(r);
            a[u] = __ldcg(r + 1);
        }
#pragma unroll
        for (int u = 0; u < K; ++u) {
            if (i0 + u < e) {
                sl += f3(l[u]);
                sa += f3(a[u]);
            }
        }
    }
    lin = scaled(sl, 1.f / (float)(e - s));
    ang = scaled(sa, 1.f / (float)(e - s));
}

// Streams of one manifold: in global memory (slot major, stride cap), or in the
// adjoint in the block's shared memory (slot major, stride blockDim), where a
// thread keeps the manifolds that it takes in every phase.
struct GlobalRows {
    float4* at;
    size_t stride;
    __device__ __forceinline__ float4& operator()(int slot) const { return at[(size_t)slot * stride]; }
};
// streams a phase reads or writes (all but kIds)
constexpr int kPhaseSlots = kIds;
static_assert(kIds == kRowSlots - 1, "the ids are the last stream");

struct Heads {
    uint32_t sA, eA, pA, sB, eB, pB;
    int nRows, dyn;
    float mu;
};
template <class Rows>
__device__ __forceinline__ Heads load_heads(const Rows& S) {
    const float4 a = S(kHead0), b = S(kHead1);
    const int f = __float_as_int(b.z);
    return Heads{__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z), __float_as_uint(a.w),
                 __float_as_uint(b.x), __float_as_uint(b.y), f & 0xffff, f >> 16, b.w};
}

// Both bodies' averages, the first K copies of each side in flight at once
// (past a range's end the last record again, which the sum leaves out).
template <int K>
__device__ __forceinline__ void gather_averages(const float4* __restrict__ copies, const Heads& H, float3& vA,
                                                float3& wA, float3& vB, float3& wB) {
    float4 l[2][K], a[2][K];
    const uint32_t s[2] = {H.sA, H.sB}, e[2] = {H.eA, H.eB};
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < K; ++u) {
            const float4* r = copies + 2 * (size_t)min(s[h] + u, max(e[h], 1u) - 1u);
            l[h][u] = __ldcg(r);
            a[h][u] = __ldcg(r + 1);
        }
    float3 sl[2], sa[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        sl[h] = sa[h] = make_float3(0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (s[h] + u < e[h]) {
                sl[h] += f3(l[h][u]);
                sa[h] += f3(a[h][u]);
            }
        for (uint32_t i0 = s[h] + K; i0 < e[h]; i0 += K) {
#pragma unroll
            for (int u = 0; u < K; ++u) {
                const float4* r = copies + 2 * (size_t)min(i0 + u, e[h] - 1u);
                l[h][u] = __ldcg(r);
                a[h][u] = __ldcg(r + 1);
            }
#pragma unroll
            for (int u = 0; u < K; ++u)
                if (i0 + u < e[h]) {
                    sl[h] += f3(l[h][u]);
                    sa[h] += f3(a[h][u]);
                }
        }
    }
    if (H.dyn & 1) {
        const float f = 1.f / (float)(H.eA - H.sA);
        vA = scaled(sl[0], f);
        wA = scaled(sa[0], f);
    }
    if (H.dyn & 2) {
        const float f = 1.f / (float)(H.eB - H.sB);
        vB = scaled(sl[1], f);
        wB = scaled(sa[1], f);
    }
}

SolverView solver_view(b3World_t* w);

}  // namespace b3solver
