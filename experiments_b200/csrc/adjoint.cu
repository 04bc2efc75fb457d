// Adjoint (reverse-mode) form of the rigid-body step, for sm_100a.
//
// Gradients of a scalar loss of the final state with respect to the initial
// linear and angular velocities, the masses and the friction coefficients
// of the dynamic bodies, through every step of the plain pipeline:
//
//   integration   x' = x + v2 dt, q' = exp(phi(w2)) q (world-frame exp map
//                 with the 0.25 pi / dt clamp), v2 = v1 + dv, w2 = d (w + dw)
//   Jacobi solve  piecewise linear in the rows: the reverse sweep replays
//                 each phase from its recorded inputs (velocities and
//                 impulses) to recover the clamp masks, then runs the rows
//                 backwards; friction bounds carry mu and the normal impulse
//   constraint    rows (n, rhs, r x n, 1/diag) as functions of the contact
//   setup         points, normal, depths, positions, velocities, inverse
//                 masses / inertias: differentiated in forward mode, one
//                 dual-number pass per input, through the same arithmetic
//   contact       points, depths and normal as functions of both poses: each
//   geometry      reduced point is classified as an incident vertex, an
//                 incident edge cut by a side plane of the reference face, or
//                 a corner of two side planes on the incident face plane, and
//                 the normal as a face normal of A or B or an edge-edge cross
//                 product; then differentiated in forward mode over the 12
//                 pose directions (dx, dtheta of both bodies)
//   gravity       v1 = v + g dt (identity for the gradient)
//
// The discrete choices of the step (pair set, separating axis, clip
// topology, point selection, row activity, clamp masks) are held fixed, so
// the gradient is that of the smooth piece the trajectory lies on; finite
// differences agree with it on worlds whose active set does not change.
//
// Memory: body state is checkpointed every K steps; the reverse pass
// recomputes each segment but the last from its checkpoint, storing the K
// pre-step states (the forward run leaves the last segment's), then re-runs
// every step of the segment once more with the Jacobi tape (every phase's
// input velocities and impulses) before reversing it.
// The inverse inertia is the inverse mass times a fixed shape factor (the
// registration AABB rule), so its gradient folds into the mass gradient.
#include "solver_common.cuh"

#include <cfloat>
#include <vector>

using namespace b3m;
using namespace b3solver;

namespace {

// the float3 operators stay visible next to the dual-number ones below
using b3m::operator+;
using b3m::operator-;
using b3m::operator*;
using b3m::operator+=;
using b3m::operator-=;

// ---------------------------------------------------------------------------
// Dual numbers (value + one tangent) for the forward-mode derivatives
// ---------------------------------------------------------------------------
struct Du {
    float v, d;
};
__device__ __forceinline__ Du du(float v, float d = 0.f) { return Du{v, d}; }
__device__ __forceinline__ Du operator+(Du a, Du b) { return Du{a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Du operator-(Du a, Du b) { return Du{a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Du operator-(Du a) { return Du{-a.v, -a.d}; }
// Products and sums of products by name: the compiler contracts them by their
// surroundings, and where a contact hardly slides the direction of friction is a
// quotient of two rounded sums (by other contractions the gradients of 16 steps
// move by up to 3e-4 of their size).
__device__ __forceinline__ Du operator*(Du a, Du b) {
    return Du{a.v * b.v, __fmaf_rn(a.d, b.v, __fmul_rn(a.v, b.d))};
}
__device__ __forceinline__ Du operator*(Du a, float s) { return Du{a.v * s, a.d * s}; }
__device__ __forceinline__ Du operator/(Du a, Du b) {
    const float r = 1.f / b.v;
    const float q = a.v * r;
    return Du{q, (a.d - q * b.d) * r};
}
__device__ __forceinline__ Du dsqrt(Du a) {
    const float s = sqrtf(a.v);
    return Du{s, s > 0.f ? 0.5f * a.d / s : 0.f};
}
__device__ __forceinline__ Du drsqrt(Du a) {
    const float r = rsqrtf(a.v);
    return Du{r, -0.5f * a.d * r * r * r};
}

struct D3 {
    Du x, y, z;
};
__device__ __forceinline__ D3 d3(float3 v, float3 t) { return D3{du(v.x, t.x), du(v.y, t.y), du(v.z, t.z)}; }
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return D3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return D3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 operator-(D3 a) { return D3{-a.x, -a.y, -a.z}; }
__device__ __forceinline__ D3 operator*(D3 a, Du s) { return D3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ Du ddot(D3 a, D3 b) {
    return Du{dot_fma(make_float3(a.x.v, a.y.v, a.z.v), make_float3(b.x.v, b.y.v, b.z.v)),
              (a.x * b.x + a.y * b.y + a.z * b.z).d};
}
__device__ __forceinline__ Du dminor(Du a, Du b, Du c, Du d) {  // a b - c d
    return Du{__fmaf_rn(a.v, b.v, -__fmul_rn(c.v, d.v)), (a * b - c * d).d};
}
__device__ __forceinline__ D3 dcross(D3 a, D3 b) {
    return D3{dminor(a.y, b.z, a.z, b.y), dminor(a.z, b.x, a.x, b.z), dminor(a.x, b.y, a.y, b.x)};
}
__device__ __forceinline__ D3 dmulv(D3 a, D3 b) { return D3{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ D3 dnormalize(D3 a) {
    const Du l2 = ddot(a, a);
    return l2.v > 0.f ? a * drsqrt(l2) : a;
}
__device__ __forceinline__ float3 tan3(D3 a) { return make_float3(a.x.d, a.y.d, a.z.d); }

// btPlaneSpace1 in dual numbers (same branches as plane_space)
__device__ void dplane_space(D3 n, D3& p, D3& q) {
    const float SQRT12 = 0.7071067811865475244008443621048490f;
    if (fabsf(n.z.v) > SQRT12) {
        const Du a = n.y * n.y + n.z * n.z;
        const Du k = drsqrt(a);
        p = D3{du(0.f), -n.z * k, n.y * k};
        q = D3{a * k, -n.x * p.z, n.x * p.y};
    } else {
        const Du a = n.x * n.x + n.y * n.y;
        const Du k = drsqrt(a);
        p = D3{-n.y * k, n.x * k, du(0.f)};
        q = D3{-n.z * p.y, n.z * p.x, a * k};
    }
}

// ---------------------------------------------------------------------------
// Adjoint buffers
// ---------------------------------------------------------------------------
// Row adjoints, float4 streams: 1..3 the header's (invMassA, invMassB, mu),
// invInertiaA, invInertiaB; then three per row, of (axis, rhs), (angular part
// A, 1/diag) and (angular part B, -): normal row j at kNormal0 + 3j, friction
// row r at kFric0 + 3r.
constexpr int kAdjSlots = 40;
constexpr int kNormal0 = 4;
constexpr int kFric0 = 16;
constexpr int kContrib = 5;  // float4 per (manifold, side): (gx, gim), (gth, gmu), gv, gw, gii

struct AdjView {
    float4 *gX, *gTh, *gV, *gW;   // per body: adjoint of the state (x, rotation, v, w)
    float4 *gDv, *gDw;            // per body: adjoint of the solver's velocity change
    float* gInvMass;              // per body accumulators over all steps
    float* gMu;
    float4* rowAdj;               // [kAdjSlots][cap]: adjoint of the header and the rows
    float4* gIn;                  // [2 parity][2 cap][2]: adjoint of each phase's inputs, copies sorted by body
    float4* gLam;                 // [3][cap]: adjoint of the row impulses
    float4* contrib;              // [kContrib][2 cap], copies sorted by body
    int cap;
};

struct StepParams {
    float dt;
    float damping;
    float threshold;
    float3 gravity;
    float erp;
    float contactProcessing;
    float slopOffset;
    int frictionCombine;
    int iterations;
};

// Rodrigues rotation of v by the rotation vector phi
__device__ __forceinline__ float3 rotvec(float3 phi, float3 v) {
    const float a = length(phi);
    if (a < 1e-12f) return v + cross(phi, v);
    const float3 k = phi * (1.f / a);
    const float c = cosf(a), s = sinf(a);
    return v * c + cross(k, v) * s + k * (dot(k, v) * (1.f - c));
}

// ---------------------------------------------------------------------------
// Seeds: dL/dq -> world rotation adjoint 0.5 vec(gq (x) q*)
// ---------------------------------------------------------------------------
__global__ void k_adj_seed(int n, const float4* __restrict__ quat, const float4* __restrict__ gq,
                           float4* __restrict__ gTh) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 q = quat[i];
    const float4 g = gq[i];
    const float4 qc = make_float4(-q.x, -q.y, -q.z, q.w);
    const float4 r = quat_mult(g, qc);
    gTh[i] = make_float4(0.5f * r.x, 0.5f * r.y, 0.5f * r.z, 0.f);
}

// ---------------------------------------------------------------------------
// Integration adjoint (one thread per body)
// ---------------------------------------------------------------------------
__global__ void k_adj_integrate(int n, const float* __restrict__ invMass, const float4* __restrict__ angVelPost,
                                const uint32_t* __restrict__ incStart, const uint32_t* __restrict__ incEnd,
                                AdjView A, StepParams P) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || invMass[i] == 0.f) return;
    const float3 gx = f3(A.gX[i]), gth = f3(A.gTh[i]);
    const float3 gvPost = f3(A.gV[i]), gwPost = f3(A.gW[i]);
    const float3 w2 = f3(angVelPost[i]);
    // v2 feeds x' and the next state
    const float3 gv2 = gvPost + gx * P.dt;
    // q' = exp(phi) q: dtheta' = R(phi) dtheta + J_l(phi) dphi
    const float wl = length(w2);
    const bool clamped = wl * P.dt > P.threshold;
    const float ang = clamped ? P.threshold : wl * P.dt;
    const float3 axis = wl > 0.f ? w2 * (1.f / wl) : make_float3(0.f, 0.f, 0.f);
    const float3 phi = axis * ang;
    const float3 gthPre = rotvec(-phi, gth);
    // J_l^T g = g - c1 phi x g + c2 phi x (phi x g)
    float c1, c2;
    if (ang < 1e-3f) {
        c1 = 0.5f - ang * ang / 24.f;
        c2 = 1.f / 6.f - ang * ang / 120.f;
    } else {
        c1 = (1.f - cosf(ang)) / (ang * ang);
        c2 = (ang - sinf(ang)) / (ang * ang * ang);
    }
    const float3 pg = cross(phi, gth);
    const float3 gphi = gth - pg * c1 + cross(phi, pg) * c2;
    float3 gw2 = gwPost;
    if (clamped) {
        // phi = threshold * w2 / |w2|
        gw2 += (gphi - axis * dot(axis, gphi)) * (P.threshold / wl);
    } else {
        gw2 += gphi * P.dt;
    }
    // w2 = damping (w + dw), v2 = v1 + dv (dv, dw only with solver copies)
    const float3 gw = gw2 * P.damping;
    A.gX[i] = f4(gx);
    A.gTh[i] = f4(gthPre);
    A.gV[i] = f4(gv2);
    A.gW[i] = f4(gw);
    const bool solved = incEnd[i] > incStart[i];
    A.gDv[i] = f4(solved ? gv2 : make_float3(0.f, 0.f, 0.f));
    A.gDw[i] = f4(solved ? gw : make_float3(0.f, 0.f, 0.f));
}

// ---------------------------------------------------------------------------
// Jacobi adjoint: persistent cooperative kernel, phases in reverse
// ---------------------------------------------------------------------------
__device__ __forceinline__ void add4(float4& a, float3 v, float w = 0.f) {
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += w;
}

__device__ __forceinline__ float pick(const float4& v, int j) { return j < 2 ? (j ? v.y : v.x) : (j == 2 ? v.z : v.w); }
__device__ __forceinline__ void put(float4& v, int j, float x) {
    if (j == 0) v.x = x;
    else if (j == 1) v.y = x;
    else if (j == 2) v.z = x;
    else v.w = x;
}
// Row adjoints are summed where they lie: the sum of one manifold's row is this
// thread's alone, so the order is fixed, and nothing waits for the old value.
__device__ __forceinline__ void red4(float4* p, float3 v, float w = 0.f) { atomicAdd(p, f4(v, w)); }

// What the tape holds of one phase of one manifold.
struct Taped {
    float4 in[4];    // linear and angular velocity of A and B the phase started from
    float4 lam[2];   // impulses of its rows before it
    float4 normal;   // friction phase: impulses of the normal rows
};
__device__ __forceinline__ Taped load_tape(const b3::JacobiTape& T, int m, int p, size_t cap) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    Taped t;
#pragma unroll
    for (int k = 0; k < 4; ++k) t.in[k] = T.in[((size_t)p * 4 + k) * cap + m];
    const int it = p >> 1;
    if (p & 1) {
        const float4* f = T.lamF + ((size_t)2 * it * cap + m);
        t.lam[0] = it > 0 ? f[-2 * (ptrdiff_t)cap] : zero;
        t.lam[1] = it > 0 ? f[-(ptrdiff_t)cap] : zero;
        t.normal = T.lamN[(size_t)it * cap + m];
    } else {
        t.lam[0] = it > 0 ? T.lamN[(size_t)(it - 1) * cap + m] : zero;
        t.lam[1] = t.normal = zero;
    }
    return t;
}

// Row r of a phase: axis, angular parts, rhs and 1/diag (as normal_rows and
// friction_rows form them).
struct Row {
    float3 n, t1, t2;
    float rhs, jac;
};
template <bool kFriction>
__device__ __forceinline__ Row form_row(const GlobalRows& S, const float4& norm, const float4& a, const float4& b, int j,
                                        int q) {
    Row w;
    const float4 dir = kFriction ? S(kPoint0 + 4 * j + 2 + q) : norm;
    w.n = f3(dir);
    w.rhs = kFriction ? dir.w : a.w;
    w.t1 = arm(f3(a), w.n);
    w.t2 = kFriction ? arm_rev(f3(b), w.n) : arm_neg(f3(b), w.n);
    w.jac = kFriction ? pick(S(kFJac + (j >> 1)), 2 * (j & 1) + q) : b.w;
    return w;
}

// One phase of one manifold in reverse: the rows are solved again from the
// tape, then run backwards. J dv of each row is kept in the impulses' streams,
// which nothing reads after the solve.
template <bool kFriction>
__device__ __forceinline__ void reverse_rows(const GlobalRows& S, const AdjView& A, int m, int nRows, float mu,
                                             const Taped& t, float4& g0, float4& g1, float4& g2, float3& gvA, float3& gwA,
                                             float3& gvB, float3& gwB) {
    constexpr int kPer = kFriction ? 2 : 1;
    const size_t cap = (size_t)A.cap;
    const float4 norm = S(kNorm), ia = S(kInA), ib = S(kInB);
    const float imA = norm.w, imB = ia.w;
    const float3 iiA = f3(ia), iiB = f3(ib);
    float3 dvA = f3(t.in[0]), dwA = f3(t.in[1]), dvB = f3(t.in[2]), dwB = f3(t.in[3]);
    float4 applied[2];
    int clamped = 0;  // two bits a row: 1 at its lower limit, 2 at its upper one
#pragma unroll 1
    for (int j = 0; j < nRows; ++j) {
        float lo = 0.f, hi = 1e10f;
        if (kFriction) {
            if (!(pick(t.normal, j) > 0.f)) continue;
            hi = mu * pick(t.normal, j);
            lo = -hi;
        }
        const float4 a = S(kPoint0 + 4 * j), b = S(kPoint0 + 4 * j + 1);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const Row w = form_row<kFriction>(S, norm, a, b, j, q);
            const int r = kPer * j + q;
            // by name, as the solve forms them: the limits are decided by these
            const float dv1 = __fadd_rn(dot_fma(w.n, dvA), dot_fma(w.t1, dwA));
            const float dv2 = __fsub_rn(dot_fma(w.t2, dwB), dot_fma(w.n, dvB));
            put(S(kLamF + (r >> 2)), r & 3, dv1 + dv2);
            const float delta = __fmaf_rn(-dv2, w.jac, __fmaf_rn(-dv1, w.jac, w.rhs));
            const float lam = pick(r < 4 ? t.lam[0] : t.lam[1], r & 3);
            const float sum = lam + delta;
            float na;
            if (sum < lo) { na = lo; clamped |= 1 << 2 * r; }
            else if (sum > hi) { na = hi; clamped |= 2 << 2 * r; }
            else { na = sum; }
            const float d = na - lam;
            put(r < 4 ? applied[0] : applied[1], r & 3, d);
            dvA = fma3(w.n, imA * d, dvA);
            dwA = fma3(mulv(iiA, w.t1), d, dwA);
            dvB = fma3(-w.n * imB, d, dvB);
            dwB = fma3(mulv(iiB, w.t2), d, dwB);
        }
    }
    float gimA = 0.f, gimB = 0.f, gmu = 0.f;
    float3 giiA = make_float3(0.f, 0.f, 0.f), giiB = giiA;
#pragma unroll 1
    for (int j = nRows - 1; j >= 0; --j) {
        const float ln = pick(t.normal, j);
        if (kFriction && !(ln > 0.f)) continue;
        const float4 a = S(kPoint0 + 4 * j), b = S(kPoint0 + 4 * j + 1);
#pragma unroll
        for (int q = kPer - 1; q >= 0; --q) {
            const Row w = form_row<kFriction>(S, norm, a, b, j, q);
            const int r = kPer * j + q;
            const float3 n = w.n, t1 = w.t1, t2 = w.t2;
            const float jac = w.jac, d = pick(r < 4 ? applied[0] : applied[1], r & 3);
            const int st = clamped >> (2 * r) & 3;
            const float3 ktA = mulv(iiA, t1), ktB = mulv(iiB, t2);
            // inputs of this row (step back through its update)
            const float3 dvAi = dvA - n * (imA * d), dwAi = dwA - ktA * d;
            const float3 dvBi = dvB + n * (imB * d), dwBi = dwB - ktB * d;
            const float S0 = imA * dot(n, gvA) + dot(ktA, gwA) - imB * dot(n, gvB) + dot(ktB, gwB);
            float3 gn = (gvA * imA - gvB * imB) * d;
            float3 gt1 = mulv(iiA, gwA) * d;
            float3 gt2 = mulv(iiB, gwB) * d;
            gimA += d * dot(n, gvA);
            gimB -= d * dot(n, gvB);
            giiA += mulv(t1, gwA) * d;
            giiB += mulv(t2, gwB) * d;
            float4& gl = kFriction ? (j < 2 ? g1 : g2) : g0;
            const int c = kFriction ? 2 * (j & 1) + q : j;
            const float gna = pick(gl, c) + S0;
            float glIn = -S0;
            float grhs = 0.f, gjac = 0.f;
            if (st == 0) {
                glIn += gna;
                const float gdelta = gna;
                grhs = gdelta;
                gjac = -gdelta * pick(S(kLamF + (r >> 2)), r & 3);
                gn += (dvAi - dvBi) * (-gdelta * jac);
                gt1 += dwAi * (-gdelta * jac);
                gt2 += dwBi * (-gdelta * jac);
                gvA += n * (-gdelta * jac);
                gwA += t1 * (-gdelta * jac);
                gvB += n * (gdelta * jac);
                gwB += t2 * (-gdelta * jac);
            } else if (kFriction) {
                // bound +-mu * lambda_n
                const float sg = st == 2 ? 1.f : -1.f;
                gmu += sg * ln * gna;
                put(g0, j, pick(g0, j) + sg * mu * gna);
            }
            put(gl, c, glIn);
            float4* at = A.rowAdj + (size_t)((kFriction ? kFric0 : kNormal0) + 3 * r) * cap + m;
            red4(at, gn, grhs);
            red4(at + cap, gt1, gjac);
            red4(at + 2 * cap, gt2);
            dvA = dvAi; dwA = dwAi; dvB = dvBi; dwB = dwBi;
        }
    }
    red4(A.rowAdj + cap + m, make_float3(gimA, gimB, gmu));
    red4(A.rowAdj + 2 * cap + m, giiA);
    red4(A.rowAdj + 3 * cap + m, giiB);
}

// The phases of the solve in reverse, one thread per manifold, a grid barrier
// between phases. As in the solve the chain of a phase counts: a thread's first
// `resident` manifolds keep their rows in shared memory, the tape's streams (read
// in order, the phase's input velocities by manifold instead of every body's
// copies again) are fetched before the barrier, and behind it one round of
// L2 reads is left, the copies' adjoints. 32,308 manifolds, 20 phases: 521 -> 185
// us; before, every phase read its rows and the row adjoints it adds to one after
// another, with the rows' states in local memory.
__global__ void __launch_bounds__(128, 2)
k_jacobi_adjoint(SolverView V, b3::JacobiTape T, AdjView A, int iterations, int resident, uint32_t* bar, int32_t* err,
                 b3Counters* counters) {
    extern __shared__ float4 kept[];  // [resident][kPhaseSlots][blockDim]
    GridBarrier barrier(bar, err, counters, b3dev::kSpinLimit, true);
    const int M = *V.numManifolds;
    const size_t cap = (size_t)V.cap;
    const int phases = 2 * iterations;
    const int m0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    const int tb = (int)blockDim.x;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < resident; ++k) {
        const int m = m0 + k * stride;
        if (m < M) {
            float4* at = kept + (size_t)k * kPhaseSlots * tb + threadIdx.x;
#pragma unroll
            for (int s = 0; s < kPhaseSlots; ++s) at[s * tb] = R(V, s, m);
        }
    }
    for (int m = m0; m < M; m += stride)
        for (int s = 1; s < kAdjSlots; ++s) A.rowAdj[(size_t)s * cap + m] = zero;
    for (int p = phases - 1; p >= 0; --p) {
        const bool last = p == phases - 1;
        const float4* in = A.gIn + (size_t)((p + 1) & 1) * 4 * cap;
        float4* out = A.gIn + (size_t)(p & 1) * 4 * cap;
        int m = m0;
        for (int k = 0; k == 0 || m < M; ++k, m += stride) {
            const GlobalRows S = k < resident ? GlobalRows{kept + (size_t)k * kPhaseSlots * tb + threadIdx.x, (size_t)tb}
                                              : GlobalRows{V.rows + m, cap};
            Taped t;
            float4 g0 = zero, g1 = zero, g2 = zero;
            if (m < M) {
                t = load_tape(T, m, p, cap);
                if (!last) {
                    g0 = A.gLam[m];
                    g1 = A.gLam[cap + m];
                    g2 = A.gLam[2 * cap + m];
                }
            }
            if (k == 0 && !last && !barrier.wait()) return;
            if (m >= M) continue;
            const Heads H = load_heads(S);
            // adjoint of this phase's copy outputs
            float3 gvA = make_float3(0.f, 0.f, 0.f), gwA = gvA, gvB = gvA, gwB = gvA;
            if (last) {
                const float4 ids = R(V, kIds, m);
                const int bA = __float_as_int(ids.x), bB = __float_as_int(ids.y);
                if (H.dyn & 1) { gvA = f3(A.gDv[bA]); gwA = f3(A.gDw[bA]); }
                if (H.dyn & 2) { gvB = f3(A.gDv[bB]); gwB = f3(A.gDw[bB]); }
            } else {
                gather_averages<4>(in, H, gvA, gwA, gvB, gwB);
            }
            if (H.nRows > 0) {
                if (p & 1) reverse_rows<true>(S, A, m, H.nRows, H.mu, t, g0, g1, g2, gvA, gwA, gvB, gwB);
                else reverse_rows<false>(S, A, m, H.nRows, H.mu, t, g0, g1, g2, gvA, gwA, gvB, gwB);
            }
            if (p > 0) {
                A.gLam[m] = g0;
                A.gLam[cap + m] = g1;
                A.gLam[2 * cap + m] = g2;
                // adjoint of the phase inputs (the averages read at its start)
                if (H.dyn & 1) {
                    __stcg(&out[2 * (size_t)H.pA], f4(gvA));
                    __stcg(&out[2 * (size_t)H.pA + 1], f4(gwA));
                }
                if (H.dyn & 2) {
                    __stcg(&out[2 * (size_t)H.pB], f4(gvB));
                    __stcg(&out[2 * (size_t)H.pB + 1], f4(gwB));
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Constraint-setup and contact-geometry adjoint (kLanes lanes per manifold)
// ---------------------------------------------------------------------------
struct SetupIn {
    D3 xA, xB, vA, wA, vB, wB;
    Du imA, imB;
    D3 iiA, iiB;
    D3 n;
    const float4* p;       // points and depths
    int k;                 // the input whose tangent is one
};
// inputs: xA 0-2, xB 3-5, vA 6-8, wA 9-11, vB 12-14, wB 15-17, imA 18, imB 19,
// iiA 20-22, iiB 23-25, n 26-28, p 29-40, depth 41-44
constexpr int kInputs = 45, kInNormal = 26, kInPoint = 29, kInDepth = 41;
__device__ __forceinline__ float3 unit_at(int k, int base) {
    return make_float3(k == base ? 1.f : 0.f, k == base + 1 ? 1.f : 0.f, k == base + 2 ? 1.f : 0.f);
}

// k_setup_rows restated in dual numbers; returns the tangent of the rows
// contracted with their adjoint.
__device__ float setup_tangent(const SetupIn& I, const SolverView& V, const AdjView& A, int m, int npts, float kA,
                               float kB, float restitution, const StepParams& P) {
    const size_t cap = (size_t)V.cap;
    float acc = 0.f;
    int nRows = 0;
    for (int j = 0; j < npts; ++j) {
        const float4 at = I.p[j];
        const float3 tp = unit_at(I.k, kInPoint + 3 * j);
        const float td = I.k == kInDepth + j ? 1.f : 0.f;
        const Du dist = du(at.w, td) + du(P.slopOffset);
        if (!(dist.v <= P.contactProcessing)) continue;
        const D3 n = I.n;
        const D3 posB = d3(f3(at), tp);
        const D3 posA = posB + n * dist;
        const D3 r1 = posA - I.xA;
        const D3 r2 = posB - I.xB;
        const D3 t0 = dcross(r1, n);
        const D3 t1 = dcross(r2, n);
        const D3 angA = dmulv(I.iiA, t0);
        const D3 angB = dmulv(I.iiB, -t1);
        const Du d0 = I.imA + ddot(n, dcross(angA, r1));
        const Du d1 = I.imB + ddot(n, dcross(-angB, r2));
        const Du denom = du(1.f) / (d0 + d1);
        const Du scaled = du(1.f) / (d0 * kA + d1 * kB);
        const D3 vel1 = I.vA + dcross(I.wA, r1);
        const D3 vel2 = I.vB + dcross(I.wB, r2);
        const D3 vel = vel1 - vel2;
        const Du relv0 = ddot(n, vel);
        Du rest = relv0 * (-restitution);
        if (rest.v <= 0.f) rest = du(0.f);
        const Du v1n = ddot(n, I.vA) + ddot(t0, I.wA);
        const Du v2n = -ddot(n, I.vB) + ddot(-t1, I.wB);
        const Du relv = v1n + v2n;
        Du posErr = du(0.f);
        Du velErr = rest - relv;
        if (dist.v > 0.f) velErr = velErr - dist * (1.f / P.dt);
        else posErr = -dist * (P.erp / P.dt);
        const Du rhs = posErr * scaled + velErr * scaled;
        {
            const int s = kNormal0 + 3 * nRows;
            const float4 g0 = A.rowAdj[(size_t)s * cap + m];
            const float4 g1 = A.rowAdj[(size_t)(s + 1) * cap + m];
            const float4 g2 = A.rowAdj[(size_t)(s + 2) * cap + m];
            acc += dot(f3(g0), tan3(n)) + g0.w * rhs.d + dot(f3(g1), tan3(t0)) + g1.w * denom.d -
                   dot(f3(g2), tan3(t1));
        }
        D3 d1v = vel - n * relv0;
        const Du lat = ddot(d1v, d1v);
        D3 d2v;
        if (lat.v > FLT_EPSILON) {
            d1v = d1v * (du(1.f) / dsqrt(lat));
            d2v = dnormalize(dcross(d1v, n));
        } else {
            dplane_space(n, d1v, d2v);
        }
        for (int q = 0; q < 2; ++q) {
            const D3 dir = q == 0 ? d2v : d1v;
            const D3 ft1 = dcross(r1, dir);
            const D3 ft2 = dcross(r2, -dir);
            const D3 fA = dmulv(I.iiA, ft1);
            const D3 fB = dmulv(I.iiB, ft2);
            const Du e0 = I.imA + ddot(dir, dcross(fA, r1));
            const Du e1 = I.imB + ddot(dir, dcross(-fB, r2));
            const Du fden = du(1.f) / (e0 + e1);
            const Du fsc = du(1.f) / (e0 * kA + e1 * kB);
            const Du frel = (ddot(dir, I.vA) + ddot(ft1, I.wA)) + (-ddot(dir, I.vB) + ddot(ft2, I.wB));
            const Du frhs = -frel * fsc;
            const int s = kFric0 + 3 * (2 * nRows + q);
            const float4 g0 = A.rowAdj[(size_t)s * cap + m];
            const float4 g1 = A.rowAdj[(size_t)(s + 1) * cap + m];
            const float4 g2 = A.rowAdj[(size_t)(s + 2) * cap + m];
            acc += dot(f3(g0), tan3(dir)) + g0.w * frhs.d + dot(f3(g1), tan3(ft1)) + g1.w * fden.d +
                   dot(f3(g2), tan3(ft2));
        }
        ++nRows;
    }
    return acc;
}

// Contact geometry of one manifold as a function of the two poses.
enum PointKind { PK_VERTEX = 0, PK_EDGE = 1, PK_CORNER = 2, PK_ATTACHED = 3 };
enum AxisKind { AX_FACE_A = 0, AX_FACE_B = 1, AX_EDGES = 2, AX_ATTACHED = 3 };

struct GeoPoint {
    int kind;
    int i0, i1;   // vertex / edge endpoints (incident face slots) or planes k, l
    int k;        // side plane for an edge point
    float3 local; // attached fallback: the point in B's frame
};

struct Geo {
    int faceA, faceB;       // reference face (A), incident face (B)
    int axisKind, ax0, ax1; // face index or edge pair
    float axisSign;
    float3 nLocalA;         // fallback: the axis in A's frame
    GeoPoint pt[4];
};

__device__ __forceinline__ float3 vtx(const b3::ShapesDev& S, const b3ConvexPolyhedron& h, int local) {
    return f3(S.verts[h.vertexOffset + local]);
}
__device__ __forceinline__ int face_vertex(const b3::ShapesDev& S, const b3Face& f, int k) {
    return S.indices[f.indexOffset + k];
}

// Pose with a first-order perturbation: world-relative-to-origin vector of a
// body-attached local vector u (rotation part only) and a point.
struct PoseD {
    Mat3 R;
    D3 x;      // position relative to the origin, with tangent
    float3 th; // rotation tangent (dtheta)
};
__device__ __forceinline__ D3 pose_dir(const PoseD& P, float3 u) {
    const float3 r = mul(P.R, u);
    return d3(r, cross(P.th, r));
}
__device__ __forceinline__ D3 pose_point(const PoseD& P, float3 u) { return P.x + pose_dir(P, u); }

// 3 x 3 solve M p = h by Cramer's rule, rows a, b, c
__device__ D3 solve3(D3 a, D3 b, D3 c, Du ha, Du hb, Du hc) {
    const D3 bc = dcross(b, c), ca = dcross(c, a), ab = dcross(a, b);
    const Du det = ddot(a, bc);
    const Du inv = du(1.f) / det;
    return (bc * ha + ca * hb + ab * hc) * inv;
}

// Tangent of the contact geometry along the two poses' perturbation, contracted
// with its adjoint gin (the axis at kInNormal, points, depths).
__device__ float geo_tangent(const Geo& G, const b3::ShapesDev& S, const b3ConvexPolyhedron& hA,
                             const b3ConvexPolyhedron& hB, const PoseD& PA, const PoseD& PB, int npts,
                             const float* gin) {
    D3 nOut;
    const b3Face fa = S.faces[hA.faceOffset + G.faceA];
    const b3Face fb = S.faces[hB.faceOffset + G.faceB];
    // separating axis
    if (G.axisKind == AX_FACE_A) {
        const b3Face f = S.faces[hA.faceOffset + G.ax0];
        nOut = pose_dir(PA, make_float3(f.plane[0], f.plane[1], f.plane[2])) * du(G.axisSign);
    } else if (G.axisKind == AX_FACE_B) {
        const b3Face f = S.faces[hB.faceOffset + G.ax0];
        nOut = pose_dir(PB, make_float3(f.plane[0], f.plane[1], f.plane[2])) * du(G.axisSign);
    } else if (G.axisKind == AX_EDGES) {
        const D3 ea = pose_dir(PA, f3(S.edges[hA.uniqueEdgesOffset + G.ax0]));
        const D3 eb = pose_dir(PB, f3(S.edges[hB.uniqueEdgesOffset + G.ax1]));
        nOut = dnormalize(dcross(ea, eb)) * du(G.axisSign);
    } else {
        // not matched to a feature: rotates with A
        nOut = pose_dir(PA, G.nLocalA);
    }
    const float3 nAl = make_float3(fa.plane[0], fa.plane[1], fa.plane[2]);
    const D3 nAw = pose_dir(PA, nAl);
    const int nvA = fa.numIndices;
    const float* gn = gin + kInNormal;
    float acc = gn[0] * nOut.x.d + gn[1] * nOut.y.d + gn[2] * nOut.z.d;
    for (int j = 0; j < npts; ++j) {
        const GeoPoint& g = G.pt[j];
        D3 p;
        if (g.kind == PK_VERTEX) {
            p = pose_point(PB, vtx(S, hB, face_vertex(S, fb, g.i0)));
        } else if (g.kind == PK_EDGE) {
            const D3 a = pose_point(PB, vtx(S, hB, face_vertex(S, fb, g.i0)));
            const D3 b = pose_point(PB, vtx(S, hB, face_vertex(S, fb, g.i1)));
            const float3 va = vtx(S, hA, face_vertex(S, fa, g.k));
            const float3 vb = vtx(S, hA, face_vertex(S, fa, (g.k + 1) % nvA));
            const D3 pn = -dcross(pose_dir(PA, va - vb), nAw);
            const D3 P0 = pose_point(PA, va);
            const D3 u = b - a;
            const Du t = ddot(pn, P0 - a) / ddot(pn, u);
            p = a + u * t;
        } else if (g.kind == PK_CORNER) {
            const float3 ka = vtx(S, hA, face_vertex(S, fa, g.i0));
            const float3 kb = vtx(S, hA, face_vertex(S, fa, (g.i0 + 1) % nvA));
            const float3 la = vtx(S, hA, face_vertex(S, fa, g.i1));
            const float3 lb = vtx(S, hA, face_vertex(S, fa, (g.i1 + 1) % nvA));
            const D3 pk = -dcross(pose_dir(PA, ka - kb), nAw);
            const D3 pl = -dcross(pose_dir(PA, la - lb), nAw);
            const D3 nBw = pose_dir(PB, make_float3(fb.plane[0], fb.plane[1], fb.plane[2]));
            const D3 Pk = pose_point(PA, ka), Pl = pose_point(PA, la);
            const D3 Pb = pose_point(PB, vtx(S, hB, face_vertex(S, fb, 0)));
            p = solve3(pk, pl, nBw, ddot(pk, Pk), ddot(pl, Pl), ddot(nBw, Pb));
        } else {
            p = pose_point(PB, g.local);
        }
        const Du depth = ddot(nAw, p - PA.x) + du(fa.plane[3]);
        const float* gp = gin + kInPoint + 3 * j;
        acc += gp[0] * p.x.d + gp[1] * p.y.d + gp[2] * p.z.d + gin[kInDepth + j] * depth.d;
    }
    return acc;
}

// The corner of side planes k, l on the incident face plane is well defined
// (the three normals are not close to coplanar).
__device__ bool corner_ok(const b3::ShapesDev& S, const b3ConvexPolyhedron& hA, const b3ConvexPolyhedron& hB,
                          const b3Face& fa, const b3Face& fb, const Mat3& RA, const Mat3& RB, float3 nAw, int k,
                          int l) {
    const int nvA = fa.numIndices;
    const float3 ka = vtx(S, hA, face_vertex(S, fa, k)), kb = vtx(S, hA, face_vertex(S, fa, (k + 1) % nvA));
    const float3 la = vtx(S, hA, face_vertex(S, fa, l)), lb = vtx(S, hA, face_vertex(S, fa, (l + 1) % nvA));
    const float3 pk = normalize(-cross(mul(RA, ka - kb), nAw));
    const float3 pl = normalize(-cross(mul(RA, la - lb), nAw));
    const float3 nb = mul(RB, make_float3(fb.plane[0], fb.plane[1], fb.plane[2]));
    return fabsf(dot(pk, cross(pl, nb))) > 1e-3f;
}

// Classify a point of the manifold against reference face faceA and incident
// face faceB (values only); true if it fits neither an incident vertex, an
// incident edge cut by a side plane, nor a corner of two side planes.
__device__ bool geo_point(GeoPoint& g, int faceA, int faceB, const b3::ShapesDev& S, const b3ConvexPolyhedron& hA,
                          const b3ConvexPolyhedron& hB, const Mat3& RA, const Mat3& RB, float3 xB, float3 p) {
    // origin at body A's position (p and xB are given relative to it)
    const b3Face fa = S.faces[hA.faceOffset + faceA];
    const b3Face fb = S.faces[hB.faceOffset + faceB];
    const int nvA = fa.numIndices, nvB = fb.numIndices;
    const float3 nAw = mul(RA, make_float3(fa.plane[0], fa.plane[1], fa.plane[2]));
    const float tol = 5e-5f;
    g.kind = PK_ATTACHED;
    g.local = mul_t(RB, p - xB);
    float bestV = tol;
    for (int i = 0; i < nvB; ++i) {
        const float3 w = mul(RB, vtx(S, hB, face_vertex(S, fb, i))) + xB;
        const float e = length(w - p);
        if (e < bestV) { bestV = e; g.kind = PK_VERTEX; g.i0 = i; }
    }
    if (g.kind == PK_VERTEX) return false;
    // side planes containing the point
    int on[2] = {-1, -1};
    float onErr[2] = {tol, tol};
    for (int k = 0; k < nvA; ++k) {
        const float3 va = vtx(S, hA, face_vertex(S, fa, k));
        const float3 vb = vtx(S, hA, face_vertex(S, fa, (k + 1) % nvA));
        float3 pn = -cross(mul(RA, va - vb), nAw);
        const float l = length(pn);
        if (l <= 0.f) continue;
        pn = pn * (1.f / l);
        const float e = fabsf(dot(pn, p - mul(RA, va)));
        if (e < onErr[0]) { onErr[1] = onErr[0]; on[1] = on[0]; onErr[0] = e; on[0] = k; }
        else if (e < onErr[1]) { onErr[1] = e; on[1] = k; }
    }
    if (on[0] < 0) return true;
    // an incident edge through the point, crossing the side plane
    // (not lying in it: the intersection must be well defined)
    const float3 vk = vtx(S, hA, face_vertex(S, fa, on[0]));
    const float3 vk1 = vtx(S, hA, face_vertex(S, fa, (on[0] + 1) % nvA));
    const float3 pnk = normalize(-cross(mul(RA, vk - vk1), nAw));
    int edge = -1;
    float bestE = tol;
    for (int i = 0; i < nvB; ++i) {
        const float3 a = mul(RB, vtx(S, hB, face_vertex(S, fb, i))) + xB;
        const float3 b = mul(RB, vtx(S, hB, face_vertex(S, fb, (i + 1) % nvB))) + xB;
        const float3 u = b - a;
        const float uu = dot(u, u);
        if (uu <= 0.f) continue;
        if (fabsf(dot(pnk, u)) < 1e-3f * sqrtf(uu)) continue;
        const float t = dot(p - a, u) / uu;
        if (t < -1e-4f || t > 1.f + 1e-4f) continue;
        const float e = length(a + u * t - p);
        if (e < bestE) { bestE = e; edge = i; }
    }
    if (edge >= 0) {
        g.kind = PK_EDGE;
        g.i0 = edge;
        g.i1 = (edge + 1) % nvB;
        g.k = on[0];
    } else if (on[1] >= 0 && corner_ok(S, hA, hB, fa, fb, RA, RB, nAw, on[0], on[1])) {
        g.kind = PK_CORNER;
        g.i0 = on[0];
        g.i1 = on[1];
    } else {
        return true;
    }
    return false;
}

// The lanes of a manifold's group are half a warp; both halves go through the
// same votes and shuffles, each with its own values.
constexpr int kLanes = 16;
__device__ __forceinline__ unsigned group_ballot(bool x) {
    return __ballot_sync(0xffffffffu, x) >> (threadIdx.x & 16) & 0xffffu;
}
// Smallest value of the group and its index, the lowest index of equal ones.
__device__ __forceinline__ void group_least(float& v, int& i) {
#pragma unroll
    for (int d = kLanes / 2; d > 0; d >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, d);
        const int oi = __shfl_xor_sync(0xffffffffu, i, d);
        if (ov < v || (ov == v && oi < i)) {
            v = ov;
            i = oi;
        }
    }
}

// Faces of h whose sign * (n . sep) is within the forward's FP32 window
// (4e-6) of the extreme, extreme first: clipHullAgainstHull's choice, or
// its candidates where faces tie within FP32 (the forward decides those in
// float-float, exact ties to the lowest index). By a group's lanes, to out.
__device__ int face_candidates(const b3::ShapesDev& S, const b3ConvexPolyhedron& h, const Mat3& R, float3 sep,
                               float sign, int* out, int maxOut) {
    const int lane = threadIdx.x & (kLanes - 1);
    auto extent = [&](int f) {
        const b3Face fc = S.faces[h.faceOffset + f];
        return sign * dot(mul(R, make_float3(fc.plane[0], fc.plane[1], fc.plane[2])), sep);
    };
    float best = FLT_MAX;
    int bi = 0;
    for (int f = lane; f < h.numFaces; f += kLanes) {
        const float d = extent(f);
        if (d < best) { best = d; bi = f; }
    }
    group_least(best, bi);
    if (lane == 0) out[0] = bi;
    int n = 1;
    const int faces = __reduce_max_sync(0xffffffffu, h.numFaces);
    for (int f0 = 0; f0 < faces; f0 += kLanes) {
        const int f = f0 + lane;
        const bool near = f < h.numFaces && f != bi && extent(f) <= best + 4e-6f;
        const unsigned all = group_ballot(near);
        const int at = n + __popc(all & ((1u << lane) - 1u));
        if (near && at < maxOut) out[at] = f;
        n += __popc(all);
    }
    return min(n, maxOut);
}

// Classify the stored manifold against the forward poses (values only), by a
// group's lanes; G and cand lie in shared memory.
__device__ void geo_classify(Geo& G, int (*cand)[4], const b3::ShapesDev& S, const b3ConvexPolyhedron& hA,
                             const b3ConvexPolyhedron& hB, const Mat3& RA, const Mat3& RB, float3 xB, float3 sep,
                             float3 p, int npts, bool on, int* unclassified) {
    const int lane = threadIdx.x & (kLanes - 1);
    // separating axis: the feature whose direction matches sep best, in the
    // order faces of A, faces of B, pairs of edges, each with both signs
    const int nfA = hA.numFaces, nf = nfA + hB.numFaces;
    const int total = nf + hA.numUniqueEdges * hB.numUniqueEdges;
    float best = 1e-4f;
    int bi = 0x7fffffff;
    for (int c = lane; c < total; c += kLanes) {
        float3 dir;
        if (c < nf) {
            const b3Face fc = S.faces[c < nfA ? hA.faceOffset + c : hB.faceOffset + c - nfA];
            dir = mul(c < nfA ? RA : RB, make_float3(fc.plane[0], fc.plane[1], fc.plane[2]));
        } else {
            const int ea = (c - nf) / hB.numUniqueEdges, eb = (c - nf) % hB.numUniqueEdges;
            const float3 a = mul(RA, f3(S.edges[hA.uniqueEdgesOffset + ea]));
            const float3 b = mul(RB, f3(S.edges[hB.uniqueEdgesOffset + eb]));
            dir = cross(a, b);
            const float l = length(dir);
            if (l < 1e-6f) continue;
            dir = dir * (1.f / l);
        }
        for (int sg = 0; sg < 2; ++sg) {
            const float3 dlt = dir * (sg ? -1.f : 1.f) - sep;
            const float e = fmaxf(fabsf(dlt.x), fmaxf(fabsf(dlt.y), fabsf(dlt.z)));
            if (e < best) { best = e; bi = 2 * c + sg; }
        }
    }
    group_least(best, bi);
    const bool attached = bi == 0x7fffffff;
    if (lane == 0) {
        const int c = bi >> 1;
        G.axisKind = attached ? AX_ATTACHED : c < nfA ? AX_FACE_A : c < nf ? AX_FACE_B : AX_EDGES;
        G.ax0 = G.ax1 = 0;
        if (!attached) {
            G.ax0 = c < nfA ? c : c < nf ? c - nfA : (c - nf) / hB.numUniqueEdges;
            if (c >= nf) G.ax1 = (c - nf) % hB.numUniqueEdges;
        }
        G.axisSign = !attached && (bi & 1) ? -1.f : 1.f;
        G.nLocalA = mul_t(RA, sep);
    }
    // reference / incident faces: clipHullAgainstHull's choice, trying the
    // faces tied within FP32 until the points fit one pair of them
    const int nA = face_candidates(S, hA, RA, sep, 1.f, cand[0], 4);
    const int nB = face_candidates(S, hB, RB, sep, -1.f, cand[1], 4);
    __syncwarp();
    int least = 1 << 30, bestA = 0, bestB = 0;
    GeoPoint g = {}, found = {};
    for (int k = 0;; ++k) {
        const bool run = k < nA * nB && least > 0;
        if (!__any_sync(0xffffffffu, run)) break;
        const int fA = run ? cand[0][k / nB] : 0, fB = run ? cand[1][k % nB] : 0;
        bool miss = false;
        if (run && lane < npts) miss = geo_point(g, fA, fB, S, hA, hB, RA, RB, xB, p);
        const int misses = __popc(group_ballot(miss));
        if (run && misses < least) {
            least = misses;
            bestA = fA;
            bestB = fB;
            found = g;
        }
    }
    if (lane < npts) G.pt[lane] = found;
    if (lane == 0) {
        G.faceA = bestA;
        G.faceB = bestB;
        if (on && attached) atomicAdd(unclassified, 1);
        if (on && least) atomicAdd(unclassified, least);
    }
    __syncwarp();
}

struct ManifoldArgs {
    b3::BodiesDev Bd;       // invMass, invInertia, friction, restitution
    const float4* pos;      // pre-step state
    const float4* quat;
    const float4* linVel;   // before gravity
    const float4* angVel;
    b3::ShapesDev S;
    const int* manifoldPair;
    const b3Contact4* contacts;
    int* unclassified;
};

// A manifold's 45 set-up directions and 12 pose directions are passes of their
// own over the same values, and the searches of the classification are minima:
// a group of 16 lanes shares them. Bound by the instructions of the 45 passes;
// 32,308 manifolds: 473 -> 268 us against a thread per manifold, whose arrays
// went through local memory. One pass in reverse in place of the 45 takes 101
// us, but rounds otherwise where a contact slides at 4e-4 m/s: the direction
// of friction is a quotient of two such values there, and the gradients of 16
// steps move by 1.5e-4 of their size.
__global__ void __launch_bounds__(128)
k_adj_manifold(SolverView V, AdjView A, ManifoldArgs MA, StepParams P) {
    constexpr int kGroups = 128 / kLanes;
    __shared__ struct {
        Geo G;
        int cand[2][4];
        float4 p[4];     // points relative to body A, depths
        float gin[kInputs];
        float pose[12];
    } shared[kGroups];
    const int M = *V.numManifolds;
    const size_t cap = (size_t)V.cap;
    const int lane = threadIdx.x & (kLanes - 1), group = threadIdx.x / kLanes;
    auto& sh = shared[group];
    const float3 z3 = make_float3(0.f, 0.f, 0.f);
    for (int m0 = blockIdx.x * kGroups; m0 < M; m0 += gridDim.x * kGroups) {
        const bool on = m0 + group < M;
        const int m = min(m0 + group, M - 1);
        const float4 ids = R(V, kIds, m), nn = R(V, kNorm, m), ia = R(V, kInA, m), ib = R(V, kInB, m);
        const int bA = __float_as_int(ids.x), bB = __float_as_int(ids.y);
        const int dyn = __float_as_int(R(V, kHead1, m).z) >> 16;
        const float kA = ids.z, kB = ids.w;
        const b3Contact4* const c = MA.contacts + MA.manifoldPair[m];
        const int npts = (int)c->worldNormal[3];
        const bool dynA = dyn & 1, dynB = dyn & 2;
        // forward values; positions relative to body A's position
        const float3 oA = f3(MA.pos[bA]);
        const float3 xB = f3(MA.pos[bB]) - oA;
        const float3 g = P.gravity * P.dt;
        const float3 vA = dynA ? f3(MA.linVel[bA]) + g : z3;
        const float3 wA = dynA ? f3(MA.angVel[bA]) : z3;
        const float3 vB = dynB ? f3(MA.linVel[bB]) + g : z3;
        const float3 wB = dynB ? f3(MA.angVel[bB]) : z3;
        const float3 iiA = f3(ia), iiB = f3(ib);
        const float imA = nn.w, imB = ia.w;
        const float3 n0 = normalize(make_float3(-c->worldNormal[0], -c->worldNormal[1], -c->worldNormal[2]));
        const float restitution = MA.Bd.restitution[bA] * MA.Bd.restitution[bB];
        const float* at = c->worldPos[lane & 3];
        const float3 p = make_float3(at[0], at[1], at[2]) - oA;
        if (lane < 4) sh.p[lane] = f4(p, at[3]);
        __syncwarp();
        // --- setup: one forward-mode pass per input ---------------------
        for (int k = lane; k < kInputs; k += kLanes) {
            const bool aSide = (k < 3) || (k >= 6 && k < 12) || k == 18 || (k >= 20 && k < 23);
            const bool bSide = (k >= 3 && k < 6) || (k >= 12 && k < 18) || k == 19 || (k >= 23 && k < 26);
            const bool unused = (aSide && !dynA) || (bSide && !dynB) ||
                                (k >= kInPoint && k < kInDepth && (k - kInPoint) / 3 >= npts) ||
                                (k >= kInDepth && k - kInDepth >= npts);
            float acc = 0.f;
            if (!unused) {
                SetupIn I;
                I.xA = d3(z3, unit_at(k, 0));
                I.xB = d3(xB, unit_at(k, 3));
                I.vA = d3(vA, unit_at(k, 6));
                I.wA = d3(wA, unit_at(k, 9));
                I.vB = d3(vB, unit_at(k, 12));
                I.wB = d3(wB, unit_at(k, 15));
                I.imA = du(imA, k == 18 ? 1.f : 0.f);
                I.imB = du(imB, k == 19 ? 1.f : 0.f);
                I.iiA = d3(iiA, unit_at(k, 20));
                I.iiB = d3(iiB, unit_at(k, 23));
                I.n = d3(n0, unit_at(k, kInNormal));
                I.p = sh.p;
                I.k = k;
                acc = setup_tangent(I, V, A, m, npts, kA, kB, restitution, P);
            }
            sh.gin[k] = acc;
        }
        // --- geometry: 12 pose directions -------------------------------
        const int colA = MA.Bd.collidable[bA], colB = MA.Bd.collidable[bB];
        const b3ConvexPolyhedron hA = MA.S.polys[MA.S.cols[colA].shapeIndex];
        const b3ConvexPolyhedron hB = MA.S.polys[MA.S.cols[colB].shapeIndex];
        const Mat3 RA = quat_to_mat(MA.quat[bA]), RB = quat_to_mat(MA.quat[bB]);
        geo_classify(sh.G, sh.cand, MA.S, hA, hB, RA, RB, xB, n0, p, npts, on, MA.unclassified);
        if (lane < 12) {
            const int body = lane < 6 ? 0 : 1, kk = lane - 6 * body;
            float acc = 0.f;
            if (body == 0 ? dynA : dynB) {
                const float3 ex = unit_at(kk, 0), et = unit_at(kk, 3);
                PoseD PA, PB;
                PA.R = RA;
                PB.R = RB;
                PA.x = d3(z3, body == 0 ? ex : z3);
                PA.th = body == 0 ? et : z3;
                PB.x = d3(xB, body == 1 ? ex : z3);
                PB.th = body == 1 ? et : z3;
                acc = geo_tangent(sh.G, MA.S, hA, hB, PA, PB, npts, sh.gin);
                if (!isfinite(acc)) {
                    // a degenerate feature slipped through the classification
                    if (on) atomicAdd(MA.unclassified, 1);
                    acc = 0.f;
                }
            }
            sh.pose[lane] = acc;
        }
        __syncwarp();
        // --- one lane per dynamic side: the body's contribution ----------
        if (on && lane < 2 && (dyn & (1 << lane))) {
            // friction of the pair -> the bodies' coefficients
            const float4 head = A.rowAdj[cap + m];
            const float gmu = head.z;
            const float muA = MA.Bd.friction[bA], muB = MA.Bd.friction[bB];
            float gmuSide;
            if (P.frictionCombine == 1) {
                gmuSide = gmu * (lane ? muA : muB);
            } else {
                const float mc = sqrtf(muA * muB);
                gmuSide = mc > 0.f ? gmu * 0.5f * mc / (lane ? muB : muA) : 0.f;
            }
            // header adjoints from the solve (inverse masses, inertias)
            const float gim = (lane ? head.y : head.x) + sh.gin[18 + lane];
            auto three = [&](int k) { return make_float3(sh.gin[k], sh.gin[k + 1], sh.gin[k + 2]); };
            const float* ps = sh.pose + 6 * lane;
            const size_t slot = V.incPos[2 * m + lane];
            const size_t stride = 2 * cap;
            float4* C = A.contrib;
            C[0 * stride + slot] = f4(three(3 * lane) + make_float3(ps[0], ps[1], ps[2]), gim);
            C[1 * stride + slot] = f4(make_float3(ps[3], ps[4], ps[5]), gmuSide);
            C[2 * stride + slot] = f4(three(6 + 6 * lane));
            C[3 * stride + slot] = f4(three(9 + 6 * lane));
            C[4 * stride + slot] = f4(f3(A.rowAdj[(size_t)(2 + lane) * cap + m]) + three(20 + 3 * lane));
        }
        __syncwarp();  // before the next manifold's values
    }
}

// Sum each dynamic body's per-copy contributions (deterministic order).
__global__ void k_adj_gather(int n, const float* __restrict__ invMass, const float4* __restrict__ invInertia,
                             SolverView V, AdjView A) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || invMass[i] == 0.f) return;
    const uint32_t s = V.incStart[i], e = V.incEnd[i];
    if (e <= s) return;
    float4 sx = make_float4(0.f, 0.f, 0.f, 0.f), sth = sx, sv = sx, sw = sx, sii = sx;
    const size_t stride = 2 * (size_t)V.cap;
    for (uint32_t k = s; k < e; ++k) {
        const size_t slot = k;
        const float4 a = A.contrib[slot], b = A.contrib[stride + slot], c = A.contrib[2 * stride + slot];
        const float4 d = A.contrib[3 * stride + slot], f = A.contrib[4 * stride + slot];
        sx.x += a.x; sx.y += a.y; sx.z += a.z; sx.w += a.w;
        sth.x += b.x; sth.y += b.y; sth.z += b.z; sth.w += b.w;
        sv.x += c.x; sv.y += c.y; sv.z += c.z;
        sw.x += d.x; sw.y += d.y; sw.z += d.z;
        sii.x += f.x; sii.y += f.y; sii.z += f.z;
    }
    add4(A.gX[i], make_float3(sx.x, sx.y, sx.z));
    add4(A.gTh[i], make_float3(sth.x, sth.y, sth.z));
    add4(A.gV[i], make_float3(sv.x, sv.y, sv.z));
    add4(A.gW[i], make_float3(sw.x, sw.y, sw.z));
    // inverse inertia = inverse mass x shape factor
    const float im = invMass[i];
    const float3 ii = f3(invInertia[i]);
    A.gInvMass[i] += sx.w + (sii.x * ii.x + sii.y * ii.y + sii.z * ii.z) / im;
    A.gMu[i] += sth.w;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct b3Adjoint_t {
    b3World w = nullptr;
    int numSteps = 0, K = 1, N = 0, cap = 0, iterations = 0;
    int numCkpt = 0;
    float4* ckpt = nullptr;   // [numCkpt][4][N]
    float4* seg = nullptr;    // [K][4][N]: pre-step states of one segment
    float4* lastPre = nullptr;  // [4][N]: state before the last step
    int segHeld = -1;         // segment whose states seg holds
    b3::JacobiTape tape{};
    float4 *gX = nullptr, *gTh = nullptr, *gV = nullptr, *gW = nullptr, *gDv = nullptr, *gDw = nullptr;
    float *gInvMass = nullptr, *gMu = nullptr;
    float4 *rowAdj = nullptr, *gIn = nullptr, *gLam = nullptr, *contrib = nullptr;
    float4* seedQ = nullptr;
    int* unclassified = nullptr;
    bool forwardDone = false, backwardDone = false;
    std::vector<void*> owned;
};

namespace {

template <typename T>
int aalloc(b3Adjoint_t* a, T*& p, size_t count) {
    if (count == 0) count = 1;
    B3_CUDA(cudaMalloc((void**)&p, sizeof(T) * count));
    a->owned.push_back((void*)p);
    return B3_OK;
}

int copy_state(b3World_t* w, float4* dst, cudaStream_t st, bool toWorld) {
    const size_t N = w->bodies.size();
    float4* bufs[4] = {w->d.pos, w->d.quat, w->d.linVel, w->d.angVel};
    for (int k = 0; k < 4; ++k) {
        if (toWorld)
            B3_CUDA(cudaMemcpyAsync(bufs[k], dst + k * N, N * sizeof(float4), cudaMemcpyDeviceToDevice, st));
        else
            B3_CUDA(cudaMemcpyAsync(dst + k * N, bufs[k], N * sizeof(float4), cudaMemcpyDeviceToDevice, st));
    }
    return B3_OK;
}

AdjView adj_view(b3Adjoint_t* a) {
    AdjView A;
    A.gX = a->gX; A.gTh = a->gTh; A.gV = a->gV; A.gW = a->gW;
    A.gDv = a->gDv; A.gDw = a->gDw;
    A.gInvMass = a->gInvMass; A.gMu = a->gMu;
    A.rowAdj = a->rowAdj; A.gIn = a->gIn; A.gLam = a->gLam;
    A.contrib = a->contrib;
    A.cap = a->cap;
    return A;
}

StepParams step_params(b3World_t* w) {
    StepParams P;
    P.dt = w->sim.dt;
    P.damping = w->sim.angularDamping;
    P.threshold = 0.25f * 3.14159254f;
    P.gravity = w->sim.gravity;
    P.erp = w->sim.erp;
    P.contactProcessing = w->sim.contactProcessing;
    P.slopOffset = w->sim.slopOffset;
    P.frictionCombine = w->sim.frictionCombine;
    P.iterations = w->sim.iterations;
    return P;
}

// Reverse one step whose pre-step state is in `pre` ([4][N]); the world's
// buffers hold that step re-run with the tape.
int reverse_step(b3Adjoint_t* a, const float4* pre, cudaStream_t st) {
    b3World_t* w = a->w;
    const int N = a->N;
    const StepParams P = step_params(w);
    SolverView V = solver_view(w);
    AdjView A = adj_view(a);
    k_adj_integrate<<<(N + 255) / 256, 256, 0, st>>>(N, w->d.invMass, w->d.angVel, w->d.bodyIncStart,
                                                    w->d.bodyIncEnd, A, P);
    B3_CHECK_LAUNCH();
    if (a->iterations > 0) {
        B3_CUDA(cudaMemsetAsync(w->d.scalars + b3::S_BAR_COUNT, 0, sizeof(int32_t) * 2, st));
        // as in the solve: the grid from the expected manifolds (about 3 per
        // body), up to two blocks an SM, shared memory for a thread's share
        const int threads = 128, perSm = 2;
        const long long est = std::min<long long>((long long)w->cfg.maxPairs, 3LL * (long long)N);
        const int want = (int)std::max<long long>(1, (est + threads - 1) / threads);
        const int blocks = std::min(w->ctx->numSMs * perSm, want);
        const size_t one = (size_t)kPhaseSlots * threads * sizeof(float4);
        const int need = (int)((est + (long long)blocks * threads - 1) / ((long long)blocks * threads));
        int resident = std::min(need, (int)((size_t)w->ctx->maxSmemOptin / perSm / one));
        const size_t smem = one * resident;
        if (smem > 48 * 1024) B3_TRY(allow_dynamic_smem(w->ctx, (const void*)k_jacobi_adjoint));
        int occ = 1;
        B3_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_jacobi_adjoint, threads, smem));
        const int grid = std::min(w->ctx->numSMs * std::max(1, std::min(occ, perSm)), want);
        int iters = a->iterations;
        uint32_t* bar = (uint32_t*)(w->d.scalars + b3::S_BAR_COUNT);
        int32_t* err = w->d.scalars + b3::S_ERR;
        b3Counters* ctr = w->d.counters;
        b3::JacobiTape T = a->tape;
        void* args[] = {&V, &T, &A, &iters, &resident, &bar, &err, &ctr};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        B3_CUDA(cudaLaunchKernelExC(&cfg, (const void*)k_jacobi_adjoint, args));
    }
    ManifoldArgs MA;
    MA.Bd = w->bodiesDev();
    MA.pos = pre;
    MA.quat = pre + N;
    MA.linVel = pre + 2 * (size_t)N;
    MA.angVel = pre + 3 * (size_t)N;
    MA.S = w->shapesDev();
    MA.manifoldPair = w->d.manifoldPair;
    MA.contacts = w->d.contacts;
    MA.unclassified = a->unclassified;
    if (a->iterations > 0) {
        const int g = w->ctx->numSMs * 16;
        k_adj_manifold<<<g, 128, 0, st>>>(V, A, MA, P);
        B3_CHECK_LAUNCH();
        k_adj_gather<<<(N + 255) / 256, 256, 0, st>>>(N, w->d.invMass, w->d.invInertia, V, A);
        B3_CHECK_LAUNCH();
    }
    return B3_OK;
}

}  // namespace

extern "C" int b3_adjoint_create(b3World w, int numSteps, int checkpointEvery, b3Adjoint* out) {
    if (!w || !out || numSteps <= 0 || checkpointEvery <= 0) return B3_ERR_INVALID_ARG;
    *out = nullptr;
    if (!w->written) return B3_ERR_STATE;
    if (w->gs) {
        b3_set_error("the adjoint form differentiates the Jacobi solver; this world runs batched Gauss-Seidel");
        return B3_ERR_UNSUPPORTED;
    }
    if (w->numSpheres || w->numPlanes || w->numCompounds || w->numMeshes) {
        b3_set_error("the adjoint form differentiates hull-hull contact geometry; this world has spheres, planes, "
                     "compounds or meshes");
        return B3_ERR_UNSUPPORTED;
    }
    B3_CUDA(cudaSetDevice(w->ctx->device));
    b3Adjoint_t* a = new b3Adjoint_t();
    a->w = w;
    a->numSteps = numSteps;
    a->K = std::min(checkpointEvery, numSteps);
    a->N = (int)w->bodies.size();
    a->cap = w->cfg.maxPairs;
    a->iterations = w->sim.iterations;
    a->numCkpt = (numSteps + a->K - 1) / a->K;
    const size_t N = (size_t)a->N, cap = (size_t)a->cap;
    const size_t phases = 2 * (size_t)a->iterations;
    int rc = B3_OK;
    // HBM sizing: checkpoints, one segment of pre-step states, the tape of
    // one step and the adjoint buffers, checked against free device memory
    {
        const size_t f4 = sizeof(float4);
        const size_t need = f4 * ((size_t)a->numCkpt * 4 * N + (size_t)a->K * 4 * N + 4 * N + phases * 4 * cap +
                                  (size_t)a->iterations * 3 * cap + 7 * N + (size_t)kAdjSlots * cap + 8 * cap +
                                  3 * cap + (size_t)kContrib * 2 * cap) +
                            2 * sizeof(float) * N;
        size_t freeB = 0, totalB = 0;
        if (cudaMemGetInfo(&freeB, &totalB) == cudaSuccess && need > freeB / 100 * 95) {
            delete a;
            b3_set_error("adjoint needs %.2f GB, %.2f GB free", need / 1e9, freeB / 1e9);
            return B3_ERR_CAPACITY;
        }
    }
    auto fail = [&](int r) {
        for (void* p : a->owned) cudaFree(p);
        delete a;
        return r;
    };
    if ((rc = aalloc(a, a->ckpt, (size_t)a->numCkpt * 4 * N)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->seg, (size_t)a->K * 4 * N)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->lastPre, 4 * N)) != B3_OK) return fail(rc);
    if (phases > 0) {
        if ((rc = aalloc(a, a->tape.in, phases * 4 * cap)) != B3_OK) return fail(rc);
        if ((rc = aalloc(a, a->tape.lamN, (size_t)a->iterations * cap)) != B3_OK) return fail(rc);
        if ((rc = aalloc(a, a->tape.lamF, (size_t)a->iterations * 2 * cap)) != B3_OK) return fail(rc);
    }
    float4** pb[] = {&a->gX, &a->gTh, &a->gV, &a->gW, &a->gDv, &a->gDw, &a->seedQ};
    for (auto p : pb)
        if ((rc = aalloc(a, *p, N)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->gInvMass, N)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->gMu, N)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->rowAdj, (size_t)kAdjSlots * cap)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->gIn, 8 * cap)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->gLam, 3 * cap)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->contrib, (size_t)kContrib * 2 * cap)) != B3_OK) return fail(rc);
    if ((rc = aalloc(a, a->unclassified, 1)) != B3_OK) return fail(rc);
    *out = a;
    return B3_OK;
}

extern "C" int b3_adjoint_destroy(b3Adjoint a) {
    if (!a) return B3_OK;
    for (void* p : a->owned) cudaFree(p);
    delete a;
    return B3_OK;
}

extern "C" int b3_adjoint_forward(b3Adjoint a, void* stream) {
    if (!a) return B3_ERR_INVALID_ARG;
    b3World_t* w = a->w;
    B3_CUDA(cudaSetDevice(w->ctx->device));
    cudaStream_t st = as_stream(stream);
    const size_t N = (size_t)a->N;
    // the last segment's pre-step states are kept as they come by, so that the
    // reverse sweep starts without running that segment again
    const int lastStart = (a->numCkpt - 1) * a->K;
    a->segHeld = -1;
    for (int t = 0; t < a->numSteps; ++t) {
        if (t % a->K == 0) B3_TRY(copy_state(w, a->ckpt + (size_t)(t / a->K) * 4 * N, st, false));
        if (t >= lastStart) B3_TRY(copy_state(w, a->seg + (size_t)(t - lastStart) * 4 * N, st, false));
        if (t == a->numSteps - 1) B3_TRY(copy_state(w, a->lastPre, st, false));
        B3_TRY(b3_step(w, 1, stream));
    }
    a->segHeld = a->numCkpt - 1;
    a->forwardDone = true;
    a->backwardDone = false;
    return B3_OK;
}

extern "C" int b3_adjoint_backward(b3Adjoint a, const float* dPos4, const float* dQuat4, const float* dLinVel4,
                                   const float* dAngVel4, void* stream) {
    if (!a) return B3_ERR_INVALID_ARG;
    if (!a->forwardDone) return B3_ERR_STATE;
    b3World_t* w = a->w;
    B3_CUDA(cudaSetDevice(w->ctx->device));
    cudaStream_t st = as_stream(stream);
    const size_t N = (size_t)a->N;
    const size_t bytes = N * sizeof(float4);
    // seeds (dL/dq is turned into a world-rotation adjoint at the final pose)
    float4* dst[4] = {a->gX, a->seedQ, a->gV, a->gW};
    const float* src[4] = {dPos4, dQuat4, dLinVel4, dAngVel4};
    for (int k = 0; k < 4; ++k) {
        if (src[k]) B3_CUDA(cudaMemcpyAsync(dst[k], src[k], bytes, cudaMemcpyHostToDevice, st));
        else B3_CUDA(cudaMemsetAsync(dst[k], 0, bytes, st));
    }
    k_adj_seed<<<(int)((N + 255) / 256), 256, 0, st>>>((int)N, w->d.quat, a->seedQ, a->gTh);
    B3_CHECK_LAUNCH();
    B3_CUDA(cudaMemsetAsync(a->gInvMass, 0, N * sizeof(float), st));
    B3_CUDA(cudaMemsetAsync(a->gMu, 0, N * sizeof(float), st));
    B3_CUDA(cudaMemsetAsync(a->unclassified, 0, sizeof(int), st));
    for (int sgi = a->numCkpt - 1; sgi >= 0; --sgi) {
        const int t0 = sgi * a->K;
        const int t1 = std::min(t0 + a->K, a->numSteps);
        // recompute the segment's pre-step states from its checkpoint
        if (a->segHeld != sgi) {
            a->segHeld = -1;
            B3_TRY(copy_state(w, a->ckpt + (size_t)sgi * 4 * N, st, true));
            for (int t = t0; t < t1; ++t) {
                B3_TRY(copy_state(w, a->seg + (size_t)(t - t0) * 4 * N, st, false));
                if (t + 1 < t1) B3_TRY(b3::run_step(w, st, nullptr));
            }
            a->segHeld = sgi;
        }
        for (int t = t1 - 1; t >= t0; --t) {
            const float4* pre = a->seg + (size_t)(t - t0) * 4 * N;
            B3_TRY(copy_state(w, const_cast<float4*>(pre), st, true));
            B3_TRY(b3::run_step(w, st, &a->tape));
            B3_TRY(reverse_step(a, pre, st));
        }
    }
    // leave the world at the final state of the forward run
    B3_TRY(copy_state(w, a->lastPre, st, true));
    B3_TRY(b3::run_step(w, st, nullptr));
    a->backwardDone = true;
    return B3_OK;
}

extern "C" int b3_adjoint_gradients(b3Adjoint a, float* dLinVel4, float* dAngVel4, float* dMass, float* dFriction) {
    if (!a) return B3_ERR_INVALID_ARG;
    if (!a->backwardDone) return B3_ERR_STATE;
    b3World_t* w = a->w;
    B3_CUDA(cudaSetDevice(w->ctx->device));
    const size_t N = (size_t)a->N;
    B3_CUDA(cudaDeviceSynchronize());
    if (dLinVel4) B3_CUDA(cudaMemcpy(dLinVel4, a->gV, N * sizeof(float4), cudaMemcpyDeviceToHost));
    if (dAngVel4) B3_CUDA(cudaMemcpy(dAngVel4, a->gW, N * sizeof(float4), cudaMemcpyDeviceToHost));
    if (dMass || dFriction) {
        std::vector<float> gim(N), gmu(N);
        B3_CUDA(cudaMemcpy(gim.data(), a->gInvMass, N * sizeof(float), cudaMemcpyDeviceToHost));
        B3_CUDA(cudaMemcpy(gmu.data(), a->gMu, N * sizeof(float), cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < N; ++i) {
            const float im = w->bodies[i].invMass;
            // invMass = 1 / mass  ->  dL/dmass = -dL/dinvMass * invMass^2
            if (dMass) dMass[i] = im != 0.f ? -gim[i] * im * im : 0.f;
            if (dFriction) dFriction[i] = im != 0.f ? gmu[i] : 0.f;
        }
    }
    return B3_OK;
}

extern "C" int b3_adjoint_info(b3Adjoint a, int* unclassified) {
    if (!a || !unclassified) return B3_ERR_INVALID_ARG;
    B3_CUDA(cudaMemcpy(unclassified, a->unclassified, sizeof(int), cudaMemcpyDeviceToHost));
    return B3_OK;
}
