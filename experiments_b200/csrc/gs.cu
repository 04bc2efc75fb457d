// Batched Gauss-Seidel contact solver: the reference's GPU solver
// (btGpuNarrowphaseAndSolver::solveContacts, P1/btGpuNarrowPhaseAndSolver.cpp:
// 1073-1353, driving ST/Solver.cpp) for worlds created with
// B3_WORLD_BATCHED_GS_SOLVER.
//
// Per step, after the manifolds:
//   k_gs_keys      cell of each manifold on the 16 x 16 xz grid from its
//                  dynamic body (SetSortDataKernel, ST/solverSetup2.cl:457-478)
//                  and its parity class (BatchSolveKernelContact's cell
//                  mapping, ST/solveContact.cl:418-426); radix sort by
//                  (class, cell), stable, so each class lists its manifolds
//                  in (cell, manifold) order
//   k_gs_sides     one entry per manifold and dynamic body; radix sort by
//   k_gs_links     body: each body's manifolds in slot order, and for every
//                  entry the one before it on the same body and class
//   k_gs_colour    greedy colouring of every class at once: a manifold takes
//                  the lowest batch that no earlier manifold on its bodies
//                  has, which is what the sequential greedy pass of
//                  sortConstraintByBatch (P1/btGpuNarrowPhaseAndSolver.cpp:
//                  752-852) arrives at batch after batch, run over the class
//                  in order, with exact body identities
//   k_gs_rank      each entry's place in its body's solve order
//   k_gs_inertia   world inverse inertia R diag(I^-1) R^T per body
//                  (setupBodiesKernel, broadphaseKernel.cl:189-201)
//   k_gs_setup     Constraint4 per manifold (setConstraint4,
//                  ST/solverSetup.cl:520-609), stored grouped by
//                  (class, batch) (counting sort)
//   k_gs_solve     4 contact then 4 friction iterations; in each, the
//                  classes in order and their batches in order
//                  (ST/Solver.cpp:561-700; solveContact.cl:272-365,
//                  solveFriction.cl:297-391)
//
// B200 mapping: both passes are sequential per body and independent elsewhere,
// so a manifold waits for its own two bodies and not for the whole grid. In the
// colouring it waits for the previous entry on each body, in the solve until
// each body's velocity carries the version that its place in the body's order
// calls for. A wait is about one L2 round trip after what it waits for, against
// a grid barrier per batch (8 x some 50 batches) and three per colouring round
// (some 290 rounds): 65,537 mixed bodies (196 K manifolds), colouring 2,619 and
// solve 2,499 us with barriers. All waits are bounded.
// Velocities are written to the bodies directly; integration then applies
// no Jacobi averages.
#include <algorithm>

#include "b3_internal.h"
#include "b3_math.cuh"
#include "b3_world.h"
#include "solver_common.cuh"

using namespace b3m;

namespace {

constexpr int kSplit = 16;        // SolverBase::N_SPLIT
constexpr int kIterations = 4;    // m_nIterations (P1/btGpuNarrowPhaseAndSolver.cpp:1330)
constexpr float kScale = 0.5f;    // 1 / (N_OBJ_PER_SPLIT * m_averageExtent) = 1 / (10 * 0.2)
constexpr float kFriction = 0.7f; // m_linear.w (ST/solverSetup.cl:541), ST/solveFriction.cl:319
constexpr float kDrift = 0.005f;  // ConstraintCfg::m_positionDrift
constexpr float kPosCoeff = 0.2f; // ConstraintCfg::m_positionConstraintCoeff

__device__ __forceinline__ int class_of(int cell) { return (cell & 1) + 2 * ((cell / kSplit) & 1); }

// cell and class of every manifold; keys (class, cell), values manifold
__global__ void k_gs_keys(const b3Contact4* __restrict__ contacts, const int* __restrict__ manifoldPair,
                          const int32_t* __restrict__ numManifolds, const float4* __restrict__ pos,
                          const float* __restrict__ invMass, uint32_t* __restrict__ keys,
                          uint32_t* __restrict__ vals, int* __restrict__ cellOf) {
    const int M = *numManifolds;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const b3Contact4& c = contacts[manifoldPair[m]];
        const int A = abs(c.bodyAPtrAndSignBit), B = abs(c.bodyBPtrAndSignBit);
        // the dynamic body's position (A unless A is static)
        const int body = invMass[A] != 0.f ? A : B;
        const float4 p = pos[body];
        const int xi = (int)((p.x - (p.x < 0.f ? 1.f : 0.f)) * kScale) & (kSplit - 1);
        const int zi = (int)((p.z - (p.z < 0.f ? 1.f : 0.f)) * kScale) & (kSplit - 1);
        const int cell = xi + zi * kSplit;
        keys[m] = (uint32_t)((class_of(cell) << 8) | cell);
        vals[m] = (uint32_t)m;
        cellOf[m] = cell;
    }
}

// Polls of a wait on another manifold before it gives up (about a microsecond
// each).
constexpr int kGsSpins = 1 << 20;

// A wait gave up: the step's error flag, as a grid barrier sets it.
__device__ __forceinline__ void gave_up(int32_t* err, b3Counters* counters) {
    if (atomicExch(err, 1) == 0) atomicAdd(&counters->timeouts, 1);
}

// One entry per manifold side: key = its dynamic body (numBodies for a static
// one, past every body), value = 2 slot + side. (A sort that gave up may leave
// other values than manifolds.)
__global__ void k_gs_sides(const uint32_t* __restrict__ vals, const b3Contact4* __restrict__ contacts,
                           const int* __restrict__ manifoldPair, const float* __restrict__ invMass,
                           const int32_t* __restrict__ numManifolds, int numBodies, uint32_t* __restrict__ bodyKeys,
                           uint32_t* __restrict__ bodyVals, int* __restrict__ slotBatch,
                           unsigned long long* __restrict__ used, int32_t* __restrict__ numSides) {
    const int M = *numManifolds;
    if (blockIdx.x == 0 && threadIdx.x == 0) *numSides = 2 * M;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < M; s += gridDim.x * blockDim.x) {
        const b3Contact4& c = contacts[manifoldPair[min(vals[s], (uint32_t)(M - 1))]];
        const int A = abs(c.bodyAPtrAndSignBit), B = abs(c.bodyBPtrAndSignBit);
        bodyKeys[2 * s] = invMass[A] != 0.f ? (uint32_t)A : (uint32_t)numBodies;
        bodyKeys[2 * s + 1] = invMass[B] != 0.f ? (uint32_t)B : (uint32_t)numBodies;
        bodyVals[2 * s] = 2u * s;
        bodyVals[2 * s + 1] = 2u * s + 1u;
        slotBatch[s] = -1;
        used[2 * s] = used[2 * s + 1] = 0ull;
    }
}

// What the colouring needs of an entry: the previous one on the same body in the
// same class (-1: none, -2: a static side), and where more than 63 entries of a
// body are of one class (a run) that run's set of late batches, -1 otherwise. Runs
// of 64 and more start 64 places apart at least, so that the place of a run's 64th
// entry, by 64, numbers its set.
constexpr int kLateWords = b3::kGsMaxBatch / 64;
static_assert(b3::kGsMaxBatch % 64 == 0, "a set is whole words");

// Per body its range of the sorted entries; per entry its links. With an error of
// this step's sorts or an earlier step the solve is void: no links, no colouring
// and no places then (the sorts may not have ended, and the entries are indexes).
__global__ void k_gs_links(const uint32_t* __restrict__ bodyKeys, const uint32_t* __restrict__ bodyVals,
                           const uint32_t* __restrict__ keys, const int32_t* __restrict__ numSides, int numBodies,
                           uint32_t* __restrict__ start, uint32_t* __restrict__ end, int2* __restrict__ link,
                           unsigned long long* __restrict__ late, const int32_t* __restrict__ err,
                           int32_t* __restrict__ stop) {
    const int n = *numSides, e = *err;
    if (blockIdx.x == 0 && threadIdx.x == 0) *stop = e;
    if (e) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = bodyKeys[i], v = bodyVals[i];
        if (k >= (uint32_t)numBodies) {
            link[v] = make_int2(-2, -1);
            continue;
        }
        const bool first = i == 0 || bodyKeys[i - 1] != k;
        if (first) start[k] = (uint32_t)i;
        if (i == n - 1 || bodyKeys[i + 1] != k) end[k] = (uint32_t)(i + 1);
        const uint32_t before = first ? 0u : bodyVals[i - 1];
        const uint32_t cls = keys[v >> 1] >> 8;
        int set = -1;
        // a run of 64 reaches 32 places before or after each of its entries
        if ((i >= 32 && bodyKeys[i - 32] == k) || (i + 32 < n && bodyKeys[i + 32] == k)) {
            auto same = [&](int j) { return bodyKeys[j] == k && keys[bodyVals[j] >> 1] >> 8 == cls; };
            int lo = i, step = 1;  // the run's first entry: in steps of growing size, then by halves
            while (lo - step >= 0 && same(lo - step)) {
                lo -= step;
                step *= 2;
            }
            for (; step > 0; step /= 2)
                if (lo - step >= 0 && same(lo - step)) lo -= step;
            if (lo + 63 < n && same(lo + 63)) {
                set = (lo + 63) / 64;
                if (i == lo)
                    for (int w = 0; w < kLateWords; ++w) late[(size_t)set * kLateWords + w] = 0ull;
            }
        }
        link[v] = make_int2(!first && keys[before >> 1] >> 8 == cls ? (int)before : -1, set);
    }
}

struct ColourView {
    const int2* link;          // per entry
    unsigned long long* late;  // sets of batches, kLateWords words each
    const int32_t* numManifolds;
    unsigned long long* used;  // per entry: batches taken on its body up to it, kDone when final
    int* slotBatch;            // per slot
    const int32_t* stop;
    int32_t* err;
    b3Counters* counters;
    int maxBatch;
};
constexpr unsigned long long kDone = 1ull << 63;  // the 63 bits below: batches 0 to 62

// The lowest batch that no earlier entry of either side has, once 0 to 62 are
// taken; maxBatch if there is none. A run's batches from 63 on are in its set,
// which is the slot's own by then: the run's entries are coloured one after
// another. A side without a set has 62 entries before this one at most, and they
// are looked at one by one, for the words that the sets leave open. A step of 500
// cubes on a dynamic plate: 4.1 ms, of 1,500 11.9; walking a run of k entries for
// every candidate batch, k^3 / 6 reads, took 18.5 ms and more than the waits last.
// Word by word and in line: the colouring counts on its eight blocks an SM (out of
// line with the words in an array it took 48 registers, five blocks, and 65,537
// mixed bodies 0.13 ms more).
__device__ __forceinline__ int late_batch(const int2* link, unsigned long long* late, const int* slotBatch, int4 sides) {
    __threadfence();
    for (int w = 0; w < kLateWords; ++w) {
        unsigned long long taken = w ? 0ull : kDone - 1;
        if (sides.y >= 0) taken |= __ldcg(&late[(size_t)sides.y * kLateWords + w]);
        if (sides.w >= 0) taken |= __ldcg(&late[(size_t)sides.w * kLateWords + w]);
        for (int h = 0; h < 2 && ~taken; ++h)
            if ((h ? sides.w : sides.y) < 0)
                for (int p = h ? sides.z : sides.x; p >= 0; p = link[p].x) {
                    const int t = __ldcg(&slotBatch[p >> 1]);
                    if (t >> 6 == w) taken |= 1ull << (t & 63);
                }
        if (!~taken) continue;
        const unsigned long long bit = ~taken & (taken + 1);
        if (sides.y >= 0) __stcg(&late[(size_t)sides.y * kLateWords + w], __ldcg(&late[(size_t)sides.y * kLateWords + w]) | bit);
        if (sides.w >= 0) __stcg(&late[(size_t)sides.w * kLateWords + w], __ldcg(&late[(size_t)sides.w * kLateWords + w]) | bit);
        return 64 * w + __ffsll((long long)bit) - 1;
    }
    return b3::kGsMaxBatch;
}

// One thread per slot, slots in order. A block hands batches on within its 256
// slots through shared memory (most chains run through neighbouring slots: a
// body's manifolds follow each other), other blocks read them from L2. The grid
// is resident and its blocks go through the slots in order, so the first slot
// without a batch always has all it waits for.
constexpr int kColourThreads = 256;
__global__ void __launch_bounds__(kColourThreads, 8) k_gs_colour(ColourView V) {
    __shared__ volatile unsigned long long local[2 * kColourThreads];
    const int M = *V.numManifolds;
    const int t = threadIdx.x;
    if (*V.stop) return;
    for (int s0 = blockIdx.x * kColourThreads; s0 < M; s0 += gridDim.x * kColourThreads) {
        const int s = s0 + t;
        local[2 * t] = local[2 * t + 1] = 0ull;
        __syncthreads();
        bool done = s >= M;
        const int4 link = done ? make_int4(-1, -1, -1, -1) : reinterpret_cast<const int4*>(V.link)[s];
        const int pa = link.x, pb = link.z;
        unsigned long long ua = 0, ub = 0;
        bool hasA = pa < 0, hasB = pb < 0;
        auto look = [&](int p, unsigned long long& u) {
            const int at = p - 2 * s0;
            u = at >= 0 ? local[at] : b3dev::ld_acquire_u64(V.used + p);
            return u != 0ull;
        };
        int spins = 0;
        while (!__all_sync(0xffffffffu, done)) {
            if (!done) {
                if (!hasA) hasA = look(pa, ua);
                if (!hasB) hasB = look(pb, ub);
                if (hasA && hasB) {
                    const unsigned long long free = ~(ua | ub) & (kDone - 1);
                    int batch = free ? __ffsll((long long)free) - 1
                                     : late_batch(V.link, V.late, V.slotBatch, link);
                    if (batch >= V.maxBatch) {
                        atomicExch(V.err, 2);
                        batch = -1;
                    }
                    __stcg(&V.slotBatch[s], batch);
                    if (batch >= 63) __threadfence();
                    const unsigned long long mine = kDone | (batch >= 0 && batch < 63 ? 1ull << batch : 0ull);
                    local[2 * t] = ua | mine;
                    local[2 * t + 1] = ub | mine;
                    b3dev::st_release_u64(V.used + 2 * s, ua | mine);
                    b3dev::st_release_u64(V.used + 2 * s + 1, ub | mine);
                    done = true;
                } else if (++spins > kGsSpins || ((spins & 1023) == 0 && *(volatile int32_t*)V.err == 1)) {
                    gave_up(V.err, V.counters);
                    done = true;
                }
            }
        }
        __syncthreads();
    }
}

// Place of each entry in its body's solve order: how many of the body's
// entries have an earlier (class, batch), and how many there are. (No batch has
// a body twice.)
__global__ void k_gs_rank(const uint32_t* __restrict__ bodyKeys, const uint32_t* __restrict__ bodyVals,
                          const uint32_t* __restrict__ keys, const int* __restrict__ slotBatch,
                          const int32_t* __restrict__ numSides, int numBodies, const uint32_t* __restrict__ start,
                          const uint32_t* __restrict__ end, int maxBatch, int2* __restrict__ place,
                          const int32_t* __restrict__ stop) {
    const int n = *numSides;
    if (*stop) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = bodyKeys[i], v = bodyVals[i];
        int2 r = make_int2(0, 0);
        if (k < (uint32_t)numBodies) {
            const uint32_t s = start[k], e = end[k];
            auto order = [&](uint32_t at) { return (int)(keys[at >> 1] >> 8) * maxBatch + slotBatch[at >> 1]; };
            const int mine = order(v);
            for (uint32_t j = s; j < e; ++j) r.x += order(bodyVals[j]) < mine ? 1 : 0;
            r.y = (int)(e - s);
        }
        place[v] = r;
    }
}

// world inverse inertia rows per body (zero for static bodies), and the
// velocities as the solve passes them on, (linear, angular) with version 0
__global__ void k_gs_inertia(b3::BodiesDev Bd, float4* __restrict__ Iw, float4* __restrict__ vel) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Bd.n) return;
    float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
    if (Bd.invMass[i] != 0.f) {
        const Mat3 R = quat_to_mat(Bd.quat[i]);
        const float3 d = f3(Bd.invInertia[i]);
        // (R diag(d) R^T)_ab = sum_k R_ak d_k R_bk
        const float3 a0 = make_float3(R.r0.x * d.x, R.r0.y * d.y, R.r0.z * d.z);
        const float3 a1 = make_float3(R.r1.x * d.x, R.r1.y * d.y, R.r1.z * d.z);
        const float3 a2 = make_float3(R.r2.x * d.x, R.r2.y * d.y, R.r2.z * d.z);
        r0 = make_float4(dot(a0, R.r0), dot(a0, R.r1), dot(a0, R.r2), 0.f);
        r1 = make_float4(dot(a1, R.r0), dot(a1, R.r1), dot(a1, R.r2), 0.f);
        r2 = make_float4(dot(a2, R.r0), dot(a2, R.r1), dot(a2, R.r2), 0.f);
    }
    Iw[3 * i + 0] = r0;
    Iw[3 * i + 1] = r1;
    Iw[3 * i + 2] = r2;
    vel[2 * i] = f4(f3(Bd.linVel[i]));
    vel[2 * i + 1] = f4(f3(Bd.angVel[i]));
}

struct M3 {
    float3 r0, r1, r2;
};
__device__ __forceinline__ M3 load_iw(const float4* Iw, int i) {
    return M3{f3(__ldg(&Iw[3 * i])), f3(__ldg(&Iw[3 * i + 1])), f3(__ldg(&Iw[3 * i + 2]))};
}
__device__ __forceinline__ float3 mul(const M3& m, float3 v) {
    return make_float3(dot(m.r0, v), dot(m.r1, v), dot(m.r2, v));
}

// calcJacCoeff (ST/solverSetup.cl:445-454); symmetric inverse inertias
__device__ __forceinline__ float jac_coeff(float3 ang0, float3 ang1, float imA, const M3& IA, float imB,
                                           const M3& IB) {
    return -1.f / (imA + dot(mul(IA, ang0), ang0) + imB + dot(mul(IB, ang1), ang1));
}

// btPlaneSpace1 as the solver kernels write it (ST/solverSetup.cl:477-501)
__device__ __forceinline__ void plane_space1(float3 n, float3& p, float3& q) {
    if (fabsf(n.z) > 0.70710678f) {
        const float a = n.y * n.y + n.z * n.z;
        const float k = 1.f / sqrtf(a);
        p = make_float3(0.f, -n.z * k, n.y * k);
        q = make_float3(a * k, -n.x * p.z, n.x * p.y);
    } else {
        const float a = n.x * n.x + n.y * n.y;
        const float k = 1.f / sqrtf(a);
        p = make_float3(-n.y * k, n.x * k, 0.f);
        q = make_float3(-n.z * p.y, n.z * p.x, a * k);
    }
}

// per (class, batch) key: counts, then offsets (exclusive scan), then the
// constraints scattered to their group with setConstraint4
__global__ void k_gs_count(const uint32_t* __restrict__ keys, const int* __restrict__ slotBatch,
                           const int32_t* __restrict__ numManifolds, int maxBatch, uint32_t* __restrict__ groupCount) {
    const int M = *numManifolds;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < M; s += gridDim.x * blockDim.x) {
        const int cls = (int)(keys[s] >> 8);
        const int b = slotBatch[s];
        if (b >= 0 && b < maxBatch) atomicAdd(&groupCount[cls * maxBatch + b], 1u);
    }
}

// exclusive scan of the group counts, one block (groups <= 4 * 1024)
__global__ void __launch_bounds__(1024) k_gs_offsets(const uint32_t* __restrict__ count, uint32_t* __restrict__ offset,
                                                     int groups) {
    __shared__ uint32_t warpSum[32];
    const int per = (groups + blockDim.x - 1) / blockDim.x;
    const int i0 = threadIdx.x * per;
    uint32_t local = 0;
    for (int i = i0; i < min(i0 + per, groups); ++i) local += count[i];
    // inclusive scan of the per-thread sums
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warpSum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) / 32;
        uint32_t v = lane < nw ? warpSum[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane < nw) warpSum[lane] = v;
    }
    __syncthreads();
    uint32_t run = x - local + (wid > 0 ? warpSum[wid - 1] : 0u);
    for (int i = i0; i < min(i0 + per, groups); ++i) {
        offset[i] = run;
        run += count[i];
    }
    if (threadIdx.x == blockDim.x - 1) offset[groups] = run;
}

struct SetupParams {
    float dtInv;
    int maxBatch;
};

__global__ void k_gs_setup(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                           const int* __restrict__ slotBatch, const int32_t* __restrict__ numManifolds,
                           const uint32_t* __restrict__ groupOffset, uint32_t* __restrict__ groupFill,
                           const b3Contact4* __restrict__ contacts, const int* __restrict__ manifoldPair,
                           b3::BodiesDev Bd, const float4* __restrict__ Iw, const int2* __restrict__ place,
                           b3Constraint4* __restrict__ cs, int4* __restrict__ turn, int* __restrict__ slotOfManifold,
                           SetupParams P) {
    const int M = *numManifolds;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < M; s += gridDim.x * blockDim.x) {
        const int cls = (int)(keys[s] >> 8);
        const int batch = slotBatch[s];
        const int m = (int)min(vals[s], (uint32_t)(M - 1));
        if (batch < 0 || batch >= P.maxBatch) {  // colouring stopped (error flag set)
            slotOfManifold[m] = -1;
            continue;
        }
        const int g = cls * P.maxBatch + batch;
        const int q = (int)(groupOffset[g] + atomicAdd(&groupFill[g], 1u));
        slotOfManifold[m] = q;
        const int2 ta = place[2 * s], tb = place[2 * s + 1];
        turn[q] = make_int4(ta.x, ta.y, tb.x, tb.y);
        const b3Contact4 c = contacts[manifoldPair[m]];
        const int A = abs(c.bodyAPtrAndSignBit), B = abs(c.bodyBPtrAndSignBit);
        const float imA = Bd.invMass[A], imB = Bd.invMass[B];
        const M3 IA = load_iw(Iw, A), IB = load_iw(Iw, B);
        const float3 posA = f3(Bd.pos[A]), posB = f3(Bd.pos[B]);
        const float3 n = make_float3(c.worldNormal[0], c.worldNormal[1], c.worldNormal[2]);
        const int np = (int)c.worldNormal[3];
        b3Constraint4 d;
        d.bodyA = (uint32_t)A;
        d.bodyB = (uint32_t)B;
        d.batchIdx = batch;
        d.padding = 0u;
        d.linear[0] = -n.x;
        d.linear[1] = -n.y;
        d.linear[2] = -n.z;
        d.linear[3] = kFriction;
#pragma unroll
        for (int ic = 0; ic < 4; ++ic) {
            d.appliedRambdaDt[ic] = 0.f;
            d.jacCoeffInv[ic] = 0.f;
            d.b[ic] = 0.f;
            d.worldPos[ic][0] = d.worldPos[ic][1] = d.worldPos[ic][2] = d.worldPos[ic][3] = 0.f;
            if (ic < np) {
                const float3 p = make_float3(c.worldPos[ic][0], c.worldPos[ic][1], c.worldPos[ic][2]);
                const float3 ang0 = -cross(p - posA, n), ang1 = cross(p - posB, n);
                d.jacCoeffInv[ic] = jac_coeff(ang0, ang1, imA, IA, imB, IB);
                // restitution 0: the position term alone
                d.b[ic] = (c.worldPos[ic][3] + kDrift) * kPosCoeff * P.dtInv;
                d.worldPos[ic][0] = p.x;
                d.worldPos[ic][1] = p.y;
                d.worldPos[ic][2] = p.z;
                d.worldPos[ic][3] = c.worldPos[ic][3];
            }
        }
        float3 center = make_float3(0.f, 0.f, 0.f);
        for (int i = 0; i < np; ++i) center += make_float3(c.worldPos[i][0], c.worldPos[i][1], c.worldPos[i][2]);
        center = center * (1.f / (float)np);
        float3 t[2];
        plane_space1(n, t[0], t[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float3 ang0 = -cross(center - posA, t[i]), ang1 = cross(center - posB, t[i]);
            d.fJacCoeffInv[i] = jac_coeff(ang0, ang1, imA, IA, imB, IB);
            d.fAppliedRambdaDt[i] = 0.f;
        }
        d.center[0] = center.x;
        d.center[1] = center.y;
        d.center[2] = center.z;
        d.center[3] = 0.f;
        cs[q] = d;
    }
}

struct SolveView {
    b3Constraint4* cs;             // grouped by (class, batch)
    const int4* turn;              // per constraint: place and count on A, on B
    const int32_t* numManifolds;
    float4* vel;                   // [bodies][2]: linear and angular velocity, w = version
    float4* pos;
    float4* linVel;
    float4* angVel;
    const float* invMass;
    const float4* Iw;
    int32_t* err;
    b3Counters* counters;
};

// One constraint with the data that does not change during the solve: its
// Constraint4 record, its turn, and its bodies' inverse masses and world
// inverse inertias (positions are read with the rest). All of it is fetched
// before the wait, so that after it only the velocities are still to come.
struct Pending {
    union {
        b3Constraint4 c;
        float4 raw[11];
    };
    int4 turn;
    int A, B;
    float imA, imB;
    float3 posA, posB;
    M3 IA, IB;
};
static_assert(sizeof(b3Constraint4) == 11 * sizeof(float4), "Constraint4 is 176 bytes");

__device__ __forceinline__ void fetch(const SolveView& V, int q, Pending& P) {
    const float4* src = reinterpret_cast<const float4*>(V.cs + q);
#pragma unroll
    for (int k = 0; k < 11; ++k) P.raw[k] = src[k];
    P.turn = __ldg(&V.turn[q]);
    P.A = (int)P.c.bodyA;
    P.B = (int)P.c.bodyB;
    P.imA = V.invMass[P.A];
    P.imB = V.invMass[P.B];
    P.posA = f3(V.pos[P.A]);
    P.posB = f3(V.pos[P.B]);
    P.IA = load_iw(V.Iw, P.A);
    P.IB = load_iw(V.Iw, P.B);
}

// the constraint, contact (phase 0) or friction (phase 1), on its bodies'
// velocities
__device__ void solve_one(const SolveView& V, Pending& P, int q, int phase, float3& vA, float3& wA, float3& vB,
                          float3& wB) {
    b3Constraint4& c = P.c;
    const float imA = P.imA, imB = P.imB;
    const bool dA = imA != 0.f, dB = imB != 0.f;
    const float3 posA = P.posA, posB = P.posB;
    const M3& IA = P.IA;
    const M3& IB = P.IB;
    const float3 lin = make_float3(c.linear[0], c.linear[1], c.linear[2]);
    const float3 n = -lin;
    float4* dst = reinterpret_cast<float4*>(V.cs + q);
    if (phase == 0) {
        // solveContact (ST/solveContact.cl:272-309): impulses clamped to [0, inf)
#pragma unroll
        for (int ic = 0; ic < 4; ++ic) {
            if (c.jacCoeffInv[ic] == 0.f) continue;
            const float3 p = make_float3(c.worldPos[ic][0], c.worldPos[ic][1], c.worldPos[ic][2]);
            const float3 ang0 = -cross(p - posA, n), ang1 = cross(p - posB, n);
            float l = dot(lin, vA) + dot(ang0, wA) + dot(-lin, vB) + dot(ang1, wB) + c.b[ic];
            l *= c.jacCoeffInv[ic];
            const float prev = c.appliedRambdaDt[ic];
            const float upd = fmaxf(prev + l, 0.f);
            l = upd - prev;
            c.appliedRambdaDt[ic] = upd;
            vA += lin * (imA * l);
            vB += -lin * (imB * l);
            wA += mul(IA, ang0) * l;
            wB += mul(IB, ang1) * l;
        }
        dst[8] = P.raw[8];  // appliedRambdaDt
    } else {
        // solveFrictionConstraint (ST/solveFriction.cl:297-391)
        if (c.fJacCoeffInv[0] == 0.f && c.fJacCoeffInv[1] == 0.f) return;
        const float sum = ((c.appliedRambdaDt[0] + c.appliedRambdaDt[1]) + c.appliedRambdaDt[2]) + c.appliedRambdaDt[3];
        const float maxR = kFriction * sum, minR = -maxR;
        float3 t[2];
        plane_space1(n, t[0], t[1]);
        const float3 center = make_float3(c.center[0], c.center[1], c.center[2]);
        const float3 r0 = center - posA, r1 = center - posB;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float3 fl = -t[i], ang0 = -cross(r0, t[i]), ang1 = cross(r1, t[i]);
            float l = dot(fl, vA) + dot(ang0, wA) + dot(-fl, vB) + dot(ang1, wB);
            l *= c.fJacCoeffInv[i];
            const float prev = c.fAppliedRambdaDt[i];
            const float upd = fminf(fmaxf(prev + l, minR), maxR);
            l = upd - prev;
            c.fAppliedRambdaDt[i] = upd;
            vA += fl * (imA * l);
            vB += -fl * (imB * l);
            wA += mul(IA, ang0) * l;
            wB += mul(IB, ang1) * l;
        }
        // angular damping about the normal (:368-379)
        const float3 ab = normalize(posB - posA), ac = normalize(center - posA);
        if (dot(ab, ac) > 0.95f || !dA || !dB) {
            const float angNA = dot(n, wA), angNB = dot(n, wB);
            wA -= n * (angNA * 0.1f);
            wB -= n * (angNB * 0.1f);
        }
        dst[9] = P.raw[9];  // fJacCoeffInv, fAppliedRambdaDt
    }
}

// Iterations in order, constraints in order; a thread has the same constraints
// in every iteration, so their impulses are its own. Constraint q's turn on a
// body comes when the body's velocity has version it * count + place; static
// bodies take no turns: their velocity is read and written as zero. The warp's
// lanes look in turn and solve as they can. The grid is resident and each
// thread goes through its constraints in order, so the first one unsolved
// always has its turn.
__global__ void __launch_bounds__(128) k_gs_solve(SolveView V) {
    const int M = *V.numManifolds;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    if (*(volatile int32_t*)V.err) return;  // the colouring stopped: the records are not complete
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int it = 0; it < 2 * kIterations; ++it) {
        const int phase = it / kIterations;
        for (int q0 = tid & ~31; q0 < M; q0 += stride) {
            const int q = q0 + (tid & 31);
            bool done = q >= M;
            Pending P;
            if (!done) fetch(V, q, P);
            const bool dA = !done && P.imA != 0.f, dB = !done && P.imB != 0.f;
            const int turnA = done ? 0 : it * P.turn.y + P.turn.x, turnB = done ? 0 : it * P.turn.w + P.turn.z;
            int spins = 0;
            while (!__all_sync(0xffffffffu, done)) {
                if (!done) {
                    float4 lA = zero, aA = zero, lB = zero, aB = zero;
                    if (dA) {
                        lA = b3dev::ld_whole(&V.vel[2 * P.A]);
                        aA = b3dev::ld_whole(&V.vel[2 * P.A + 1]);
                    }
                    if (dB) {
                        lB = b3dev::ld_whole(&V.vel[2 * P.B]);
                        aB = b3dev::ld_whole(&V.vel[2 * P.B + 1]);
                    }
                    const bool ready = (!dA || (__float_as_int(lA.w) == turnA && __float_as_int(aA.w) == turnA)) &&
                                       (!dB || (__float_as_int(lB.w) == turnB && __float_as_int(aB.w) == turnB));
                    if (ready) {
                        float3 vA = f3(lA), wA = f3(aA), vB = f3(lB), wB = f3(aB);
                        solve_one(V, P, q, phase, vA, wA, vB, wB);
                        if (dA) {
                            b3dev::st_whole(&V.vel[2 * P.A], f4(vA, __int_as_float(turnA + 1)));
                            b3dev::st_whole(&V.vel[2 * P.A + 1], f4(wA, __int_as_float(turnA + 1)));
                        }
                        if (dB) {
                            b3dev::st_whole(&V.vel[2 * P.B], f4(vB, __int_as_float(turnB + 1)));
                            b3dev::st_whole(&V.vel[2 * P.B + 1], f4(wB, __int_as_float(turnB + 1)));
                        }
                        // the last turn of a body leaves its velocity
                        if (!dA || turnA + 1 == 2 * kIterations * P.turn.y) {
                            V.linVel[P.A] = dA ? f4(vA) : zero;
                            V.angVel[P.A] = dA ? f4(wA) : zero;
                        }
                        if (!dB || turnB + 1 == 2 * kIterations * P.turn.w) {
                            V.linVel[P.B] = dB ? f4(vB) : zero;
                            V.angVel[P.B] = dB ? f4(wB) : zero;
                        }
                        done = true;
                    } else if (++spins > kGsSpins || ((spins & 1023) == 0 && *(volatile int32_t*)V.err)) {
                        gave_up(V.err, V.counters);
                        done = true;
                    } else if (spins > 4) {
                        __nanosleep(50);
                    }
                }
            }
        }
    }
}

// Blocks of a resident grid: at most perSm on each SM, and no more than the work.
int cooperative_grid(const void* kern, int threads, int numSMs, int perSm, long long work) {
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, 0) != cudaSuccess || occ < 1) occ = 1;
    occ = std::min(occ, perSm);
    const long long want = std::max<long long>(1, (work + threads - 1) / threads);
    return (int)std::min<long long>((long long)numSMs * occ, want);
}

int launch_cooperative(const void* kern, int grid, int threads, void** args, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B3_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
    return B3_OK;
}

}  // namespace

namespace b3 {

int launch_gs_solver(b3World_t* w, cudaStream_t st) {
    if (w->cfg.maxPairs == 0 || w->bodies.empty()) return B3_OK;
    auto& d = w->d;
    const int N = (int)w->bodies.size();
    const int cap = w->cfg.maxPairs;
    const int maxBatch = kGsMaxBatch;
    const int32_t* M = d.scalars + S_NUM_MANIFOLDS;
    const int g = w->ctx->numSMs * 8;
    // 1. cells and classes, sorted by (class, cell)
    k_gs_keys<<<g, 256, 0, st>>>(d.contacts, d.manifoldPair, M, d.pos, d.invMass, d.incKeys, d.incVals, d.gsCell);
    B3_CHECK_LAUNCH();
    bool alt = false;
    B3_TRY(radix_sort_pairs(d.incKeys, d.incVals, d.incKeysAlt, d.incValsAlt, M, cap, 10, d.incSortScratch,
                            d.incSortScratchBytes, d.scalars + S_ERR, st, &alt, w->ctx->numSMs, 3LL * N));
    const uint32_t* keys = alt ? d.incKeysAlt : d.incKeys;
    const uint32_t* vals = alt ? d.incValsAlt : d.incVals;
    // 2. colouring. The Constraint4 records take 11 of a manifold's row streams;
    // the entries' buffers lie in the others.
    static_assert(11 * sizeof(float4) + 2 * (4 * sizeof(uint32_t) + sizeof(unsigned long long) + 2 * sizeof(int2)) +
                          sizeof(int4) + (1 + 32) * sizeof(unsigned long long) * kLateWords / 32 <=
                      kSolverRowSlots * sizeof(float4),
                  "the solver's buffers fit a manifold's rows (a set for 32 manifolds, and one more)");
    const size_t c = (size_t)cap;
    int4* turn = reinterpret_cast<int4*>(d.rows + 11 * c);
    unsigned long long* used = reinterpret_cast<unsigned long long*>(turn + c);
    int2* place = reinterpret_cast<int2*>(used + 2 * c);
    uint32_t* bodyKeys = reinterpret_cast<uint32_t*>(place + 2 * c);
    uint32_t* bodyVals = bodyKeys + 2 * c;
    uint32_t* bodyKeysAlt = bodyVals + 2 * c;
    uint32_t* bodyValsAlt = bodyKeysAlt + 2 * c;
    int2* link = reinterpret_cast<int2*>(bodyValsAlt + 2 * c);
    unsigned long long* late = reinterpret_cast<unsigned long long*>(link + 2 * c);  // one set for 64 entries
    int32_t* numSides = d.scalars + S_NUM_INC;
    k_gs_sides<<<g, 256, 0, st>>>(vals, d.contacts, d.manifoldPair, d.invMass, M, N, bodyKeys, bodyVals, d.gsSlotBatch,
                                  used, numSides);
    B3_CHECK_LAUNCH();
    bool altB = false;
    B3_TRY(radix_sort_pairs(bodyKeys, bodyVals, bodyKeysAlt, bodyValsAlt, numSides, 2LL * cap, w->bodyBits,
                            d.incSortScratch, d.incSortScratchBytes, d.scalars + S_ERR, st, &altB, w->ctx->numSMs,
                            6LL * N));
    if (altB) {
        std::swap(bodyKeys, bodyKeysAlt);
        std::swap(bodyVals, bodyValsAlt);
    }
    k_gs_links<<<g, 256, 0, st>>>(bodyKeys, bodyVals, keys, numSides, N, d.bodyIncStart, d.bodyIncEnd, link,
                                  late, d.scalars + S_ERR, d.scalars + S_GS_STOP);
    B3_CHECK_LAUNCH();
    ColourView CV;
    CV.link = link;
    CV.late = late;
    CV.numManifolds = M;
    CV.used = used;
    CV.slotBatch = d.gsSlotBatch;
    CV.stop = d.scalars + S_GS_STOP;
    CV.err = d.scalars + S_ERR;
    CV.counters = d.counters;
    CV.maxBatch = maxBatch;
    // Resident threads are the slots (constraints) looked ahead of the first one
    // undone. Colouring, 196 K and 900 K manifolds: 1 block an SM 747 / 3,779
    // us, 2 blocks 434 / 2,290, 4 blocks 334 / 1,411, 8 blocks 207 / 840. Solve:
    // 1 block (of 128) 587 / 1,269 us, 2 blocks 505 / 1,052, 3 blocks 522 /
    // 1,044. solverMode 1 (the narrow width) halves both.
    const int narrow = w->solverMode == 1 ? 2 : 1;
    const long long estM = std::min<long long>((long long)cap, 3LL * N);
    {
        const int grid = cooperative_grid((const void*)k_gs_colour, kColourThreads, w->ctx->numSMs, 8 / narrow, estM);
        void* args[] = {&CV};
        B3_TRY(launch_cooperative((const void*)k_gs_colour, grid, kColourThreads, args, st));
    }
    // 3. groups (class, batch): counts, offsets, turns, constraints
    const int groups = 4 * maxBatch;
    B3_CUDA(cudaMemsetAsync(d.gsGroupCount, 0, sizeof(uint32_t) * groups, st));
    B3_CUDA(cudaMemsetAsync(d.gsGroupFill, 0, sizeof(uint32_t) * groups, st));
    k_gs_count<<<g, 256, 0, st>>>(keys, d.gsSlotBatch, M, maxBatch, d.gsGroupCount);
    B3_CHECK_LAUNCH();
    k_gs_offsets<<<1, 1024, 0, st>>>(d.gsGroupCount, d.gsGroupOffset, groups);
    B3_CHECK_LAUNCH();
    k_gs_rank<<<g, 256, 0, st>>>(bodyKeys, bodyVals, keys, d.gsSlotBatch, numSides, N, d.bodyIncStart, d.bodyIncEnd,
                                 maxBatch, place, d.scalars + S_GS_STOP);
    B3_CHECK_LAUNCH();
    k_gs_inertia<<<(N + 255) / 256, 256, 0, st>>>(w->bodiesDev(), d.gsInertia, d.gsVel);
    B3_CHECK_LAUNCH();
    SetupParams SP;
    SP.dtInv = 1.f / w->sim.dt;
    SP.maxBatch = maxBatch;
    k_gs_setup<<<g, 128, 0, st>>>(keys, vals, d.gsSlotBatch, M, d.gsGroupOffset, d.gsGroupFill, d.contacts,
                                  d.manifoldPair, w->bodiesDev(), d.gsInertia, place, d.gsConstraints, turn,
                                  d.gsSlotOfManifold, SP);
    B3_CHECK_LAUNCH();
    // 4. Gauss-Seidel iterations
    SolveView SV;
    SV.cs = d.gsConstraints;
    SV.turn = turn;
    SV.numManifolds = M;
    SV.vel = d.gsVel;
    SV.pos = d.pos;
    SV.linVel = d.linVel;
    SV.angVel = d.angVel;
    SV.invMass = d.invMass;
    SV.Iw = d.gsInertia;
    SV.err = d.scalars + S_ERR;
    SV.counters = d.counters;
    {
        const void* kg = (const void*)k_gs_solve;
        const int grid = cooperative_grid(kg, 128, w->ctx->numSMs, 2 / narrow, estM);
        void* args[] = {&SV};
        B3_TRY(launch_cooperative(kg, grid, 128, args, st));
    }
    return B3_OK;
}

}  // namespace b3

extern "C" int b3_solver_solve_batched_gs(b3World w, void* stream) {
    if (!w) return B3_ERR_INVALID_ARG;
    if (!w->gs) {
        b3_set_error("the world was not created with B3_WORLD_BATCHED_GS_SOLVER");
        return B3_ERR_STATE;
    }
    return b3_stage_solve(w, stream);
}

extern "C" int b3_get_gs_batches(b3World w, int32_t* cellBatch2, int max, int* count, void* stream) {
    if (!w || !count) return B3_ERR_INVALID_ARG;
    if (!w->gs) return B3_ERR_STATE;
    if (!w->written) return B3_ERR_STATE;
    cudaStream_t st = (cudaStream_t)stream;
    int32_t nm = 0;
    B3_CUDA(cudaMemcpyAsync(&nm, w->d.scalars + b3::S_NUM_MANIFOLDS, 4, cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaStreamSynchronize(st));
    *count = nm;
    if (!cellBatch2 || nm <= 0 || max <= 0) return B3_OK;
    const int n = std::min(nm, max);
    std::vector<int> cell(nm), slot(nm);
    std::vector<b3Constraint4> cs(nm);
    B3_CUDA(cudaMemcpyAsync(cell.data(), w->d.gsCell, 4 * (size_t)nm, cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaMemcpyAsync(slot.data(), w->d.gsSlotOfManifold, 4 * (size_t)nm, cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaMemcpyAsync(cs.data(), w->d.gsConstraints, sizeof(b3Constraint4) * (size_t)nm,
                            cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaStreamSynchronize(st));
    for (int m = 0; m < n; ++m) {
        cellBatch2[2 * m] = cell[m];
        cellBatch2[2 * m + 1] = slot[m] >= 0 && slot[m] < nm ? cs[slot[m]].batchIdx : -1;
    }
    return B3_OK;
}

extern "C" int b3_get_gs_constraints(b3World w, b3Constraint4* out, int max, int* count, void* stream) {
    if (!w || !count) return B3_ERR_INVALID_ARG;
    if (!w->gs) return B3_ERR_STATE;
    if (!w->written) return B3_ERR_STATE;
    cudaStream_t st = (cudaStream_t)stream;
    int32_t nm = 0;
    B3_CUDA(cudaMemcpyAsync(&nm, w->d.scalars + b3::S_NUM_MANIFOLDS, 4, cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaStreamSynchronize(st));
    *count = nm;
    if (!out || nm <= 0 || max <= 0) return B3_OK;
    std::vector<int> slot(nm);
    std::vector<b3Constraint4> cs(nm);
    B3_CUDA(cudaMemcpyAsync(slot.data(), w->d.gsSlotOfManifold, 4 * (size_t)nm, cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaMemcpyAsync(cs.data(), w->d.gsConstraints, sizeof(b3Constraint4) * (size_t)nm,
                            cudaMemcpyDeviceToHost, st));
    B3_CUDA(cudaStreamSynchronize(st));
    for (int m = 0; m < std::min(nm, max); ++m) out[m] = slot[m] >= 0 && slot[m] < nm ? cs[slot[m]] : b3Constraint4{};
    return B3_OK;
}
