// The separating-axis sweep by lane groups, for pairs of few axes (included by
// narrowphase.cu).
//
// Two boxes have 6 distinct face axes and 9 edge pairs. A warp per such pair
// gave 15 lanes work once and paid the pair's set-up, reductions and clip
// decision in full; most of that is straight code, which is bound by the
// instruction fetch. Here eight lanes take a pair, four pairs go through each
// instruction, and every lane has one axis in each of two rounds:
//   * round 1, the face axes, and the edge pairs past the eighth in the lanes
//     that are left over; round 2, the first eight edge pairs;
//   * a face whose normal is another's negative is one axis: its depth, error
//     and orientation are the other's bit for bit (ShapesDev.axisFaces).
// 406,661 pairs of cubes: 1.30 -> 0.46 ns a pair; the sweep of 1,048,576 cubes
// (7.32 M pairs) 7.44 -> 2.21 ms, of 131,072 mixed bodies (a quarter of the
// 1.60 M pairs boxes) 2.74 -> 2.14 ms, before pairs that are apart were
// left out.
// All 32 lanes go through one control flow, with whole-warp masks throughout:
// a vote or reduction with a group's own mask splits the warp, and the four
// groups then run one after another.
//
// Pairs with more axes stay with the warp sweep, whose lanes they fill (eight
// lanes measured: hull-hull 3.9 ns a pair against 1.7, icosphere-icosphere 14
// against 7). k_np_bin sorts the pairs into the two queues and leaves out
// most of those that are apart.
// Each axis is computed with the warp sweep's arithmetic, the candidates are
// the same set, and the winner and its tests are the same. What a group cannot
// hold (more than kGroupCand near-minimum axes) goes to the warp sweep, which
// does it from the start.

// Products and sums by name: the same axis is evaluated in several places,
// which have to agree to the bit.
__device__ __forceinline__ float xdot(float3 a, float3 b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ float3 xmul(const Mat3& m, float3 v) {
    return make_float3(xdot(m.r0, v), xdot(m.r1, v), xdot(m.r2, v));
}
__device__ __forceinline__ float3 xmul_t(const Mat3& m, float3 v) {
    return make_float3(xdot(make_float3(m.r0.x, m.r1.x, m.r2.x), v), xdot(make_float3(m.r0.y, m.r1.y, m.r2.y), v),
                       xdot(make_float3(m.r0.z, m.r1.z, m.r2.z), v));
}
__device__ __forceinline__ float3 xcross(float3 a, float3 b) {
    return make_float3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
                       __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}

constexpr int kGroupCand = 8;   // near-minimum axes a group ranks, one per lane
constexpr int kSweepChunk = 32; // pairs per work grab at most, one prefetched by each lane

struct __align__(16) SweepScratch {
    PairPre pre[kSweepChunk];
    int cand[32 / kClipGroup][kGroupCand];
};

// One pair as its group's lanes see it.
struct SweepPair {
    Mat3 RA, RB;
    float3 rel, D;   // posB - posA; A's local centre minus B's
    float delta;     // FP32 depth error of a well-conditioned axis
    float rinSum;    // both inradii, less a margin
    int pa, pb;
};

__device__ __forceinline__ void sweep_pair(SweepPair& q, const PairPre& pre, const b3::ShapesDev& S) {
    q.pa = pre.shapeA;
    q.pb = pre.shapeB;
    q.RA = quat_to_mat(pre.qA);
    q.RB = quat_to_mat(pre.qB);
    const float4 cA = __ldg(&S.info[3 * q.pa]), cB = __ldg(&S.info[3 * q.pb]);
    q.rel = f3(pre.pB) - f3(pre.pA);
    q.D = xmul(q.RA, f3(cA)) - (xmul(q.RB, f3(cB)) + q.rel);
    q.delta = 1e-6f * (1.f + cA.w + cB.w + len_ub(q.rel));
    q.rinSum = fmaxf(0.f, S.inradius[q.pa] + S.inradius[q.pb] - 1e-4f);
}
// (face offset, face axes, edge offset, edges) and (vertex pairs, their number
// (< 0: symmetric), faces, -) of a polyhedron
__device__ __forceinline__ int4 poly_axes(const b3::ShapesDev& S, int p) {
    return __ldg(reinterpret_cast<const int4*>(&S.info[3 * p + 1]));
}
__device__ __forceinline__ int4 poly_pack(const b3::ShapesDev& S, int p) {
    return __ldg(reinterpret_cast<const int4*>(&S.info[3 * p + 2]));
}

// Extent of a hull along the local direction ld over its vertex pairs
// first, first + step, ..: x * ld.x, then + y * ld.y, then + z * ld.z.
__device__ __forceinline__ void extent(const b3::ShapesDev& S, int4 pk, float3 ld, int first, int step, float& lo,
                                       float& hi) {
    const unsigned long long lx = pack2(ld.x, ld.x), ly = pack2(ld.y, ld.y), lz = pack2(ld.z, ld.z);
    const int np = abs(pk.y);
    lo = FLT_MAX;
    hi = -FLT_MAX;
#pragma unroll 2
    for (int j = first; j < np; j += step) {
        const float4 xy = __ldg(&S.vpXY[pk.x + j]);
        const float2 z = __ldg(&S.vpZ[pk.x + j]);
        unsigned long long d = mul2(pack2(xy.x, xy.y), lx);
        d = fma2(pack2(xy.z, xy.w), ly, d);
        d = fma2(pack2(z.x, z.y), lz, d);
        float d0, d1;
        unpack2(d, d0, d1);
        lo = fminf(lo, fminf(d0, d1));
        hi = fmaxf(hi, fmaxf(d0, d1));
    }
}
// A symmetric hull keeps one vertex of each v, -v: rounding is symmetric too,
// so its extent is +-max |v . d|, the same bits.
__device__ __forceinline__ void mirror(int4 pk, float& lo, float& hi) {
    const float e = fmaxf(hi, -lo);
    if (pk.y < 0) {
        lo = -e;
        hi = e;
    }
}
__device__ __forceinline__ float pair_depth(const SweepPair& q, const b3::ShapesDev& S, float3 n) {
    float lo0, hi0, lo1, hi1;
    const int4 ka = poly_pack(S, q.pa), kb = poly_pack(S, q.pb);
    extent(S, ka, xmul_t(q.RA, n), 0, 1, lo0, hi0);
    mirror(ka, lo0, hi0);
    extent(S, kb, xmul_t(q.RB, n), 0, 1, lo1, hi1);
    mirror(kb, lo1, hi1);
    const float off = xdot(q.rel, n);
    lo1 += off;
    hi1 += off;
    return fminf(hi0 - lo1, hi1 - lo0);
}

// axis_dir of an edge pair: the oriented direction, its depth error and the
// lower bound of its depth; false when the edges are parallel.
__device__ __forceinline__ bool edge_axis(const SweepPair& q, float4 ea, float4 eb, float3& n, float& err, float& lb) {
    const float3 wa = xmul(q.RA, f3(ea)), wb = xmul(q.RB, f3(eb));
    const float3 cr = xcross(wa, wb);
    if (!(fabsf(cr.x) > 1e-6f || fabsf(cr.y) > 1e-6f || fabsf(cr.z) > 1e-6f)) return false;
    const float cl = sqrtf(xdot(cr, cr));
    n = cr * (1.f / cl);
    const float isin = ea.w * eb.w / cl, lD = len_ub(q.D), dn = xdot(q.D, n);
    err = q.delta + 0.3f * q.delta * isin;
    lb = q.rinSum - fabsf(dn) - 1e-5f * (1.f + lD) - 1e-6f * lD * isin - 2.f * err;
    if (dn < 0.f) n = -n;
    return true;
}

// Reductions and votes within the eight lanes of each group, by the whole warp.
constexpr unsigned kAll = 0xffffffffu;
__device__ __forceinline__ float group_min(float v) {
#pragma unroll
    for (int o = kClipGroup / 2; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kAll, v, o));
    return v;
}
__device__ __forceinline__ float group_max(float v) { return -group_min(-v); }
__device__ __forceinline__ int group_min(int v) {
#pragma unroll
    for (int o = kClipGroup / 2; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(kAll, v, o));
    return v;
}
// (value, index) minimum
__device__ __forceinline__ void group_argmin(float& v, int& idx) {
    const float m = group_min(v);
    idx = group_min(v == m ? idx : kNone);
    v = m;
}
// the group's bits of a vote, its own eight lowest
__device__ __forceinline__ unsigned group_ballot(bool p) {
    return __ballot_sync(kAll, p) >> (threadIdx.x & 31 & ~(kClipGroup - 1)) & ((1u << kClipGroup) - 1u);
}
__device__ __forceinline__ bool group_any(bool p) { return group_ballot(p) != 0u; }
// v of the group's lane src
__device__ __forceinline__ float3 group_from(float3 v, int src) {
    return make_float3(__shfl_sync(kAll, v.x, src, kClipGroup), __shfl_sync(kAll, v.y, src, kClipGroup),
                       __shfl_sync(kAll, v.z, src, kClipGroup));
}

// sweep_axes for the four pairs of a warp, one per group (on: the group has
// one): 0 = separated (or no axis), 1 = decided in FP32 (sepf), 2 =
// near-minimum axes left in cand[0..count) for the float-float ranking, 3 = to
// the warp sweep. Votes are taken by all lanes before anything that depends on
// a lane's own condition.
__device__ __forceinline__ int group_sweep(const PairPre& pre, bool on, const b3::ShapesDev& S, int* cand,
                                           float3& sepf, int& count) {
    const int gl = grp_lane();
    SweepPair q;
    sweep_pair(q, pre, S);
    const int4 aA = poly_axes(S, q.pa), aB = poly_axes(S, q.pb);
    const int FA = poly_pack(S, q.pa).z, nFace = FA + poly_pack(S, q.pb).z;
    const int nAx = aA.y + aB.y, EB = aB.w, nE = aA.w * EB;
    auto edge = [&](int e, float3& n, float& err, float& lb) {
        const int e0 = e * ((1 << 12) / EB + 1) >> 12;  // e / EB for e < 16
        return edge_axis(q, __ldg(&S.edges[aA.z + e0]), __ldg(&S.edges[aB.z + e - e0 * EB]), n, err, lb);
    };
    // round 1
    float3 n1 = make_float3(0.f, 0.f, 0.f), n2 = n1;
    float d1 = FLT_MAX, err1 = 0.f, lb1 = -FLT_MAX;
    int idx1 = kNone;
    const bool face = on && gl < nAx;
    if (face) {
        const bool onA = gl < aA.y;
        const int at = onA ? aA.x : aB.x;
        const int f = __ldg(&S.axisFaces[at + (onA ? gl : gl - aA.y)]);
        n1 = xmul(onA ? q.RA : q.RB, f3(__ldg((const float4*)&S.faces[at + f].plane[0])));
        if (xdot(q.D, n1) < 0.f) n1 = -n1;
        err1 = q.delta;
        idx1 = onA ? f : FA + f;
    } else if (on && 8 + gl - nAx < nE) {
        const int e = 8 + gl - nAx;
        if (edge(e, n1, err1, lb1)) idx1 = nFace + e;
    }
    __syncwarp();
    if (idx1 != kNone) d1 = pair_depth(q, S, n1);
    __syncwarp();
    // clearly separated by a face axis (the reference returns early too,
    // P2/sat.cl:527-530)
    const bool apart = group_any(face && d1 < -q.delta);
    on = on && !apart;
    if (!__any_sync(kAll, on)) return 0;
    const bool amb = face && fabsf(d1) <= q.delta;  // its separation test is ambiguous in FP32
    const float lbHi = group_min(face ? fminf(d1 + err1, FLT_MAX) : FLT_MAX);
    if (lb1 > lbHi) idx1 = kNone;  // an edge out of reach of the best face, as below
    // round 2
    float d2 = FLT_MAX, err2 = 0.f;
    int idx2 = kNone;
    if (on && gl < nE) {
        float lb;
        if (edge(gl, n2, err2, lb) && !(lb > lbHi)) {
            d2 = pair_depth(q, S, n2);
            idx2 = nFace + gl;
        }
    }
    __syncwarp();
    const float up1 = idx1 != kNone ? fminf(d1 + err1, FLT_MAX) : FLT_MAX;
    const float up2 = idx2 != kNone ? fminf(d2 + err2, FLT_MAX) : FLT_MAX;
    const float lim = group_min(fminf(up1, up2));
    on = on && lim < FLT_MAX;
    const bool take1 = on && idx1 != kNone && d1 - err1 <= lim, take2 = on && idx2 != kNone && d2 - err2 <= lim;
    const unsigned b1 = group_ballot(take1), b2 = group_ballot(take2), bA = group_ballot(on && amb);
    count = __popc(b1) + __popc(b2) + __popc(bA);
    int what = !on ? 0 : count > kGroupCand ? 3 : 2;
    const float tol = 1e-5f * (len_ub(q.D) + 1e-3f);  // orientation test not near zero
    // A single well-conditioned winner needs no refinement: a face axis, or an
    // edge axis with |e0 x e1| >= 0.01 (FP32 normal error < 1e-5).
    const int src = b1 ? __ffs(b1) - 1 : b2 ? __ffs(b2) - 1 : 0;
    const bool mine1 = b1 != 0u;
    const float3 w1 = group_from(mine1 ? n1 : n2, src);
    const float werr = __shfl_sync(kAll, mine1 ? err1 : err2, src, kClipGroup);
    if (what == 2 && count == 1 && werr <= 31.f * q.delta && fabsf(xdot(q.D, w1)) > tol) {
        sepf = w1;
        what = 1;
    }
    if (!__any_sync(kAll, what == 2)) return what;
    // the list: faces and late edges, edges, ambiguous faces
    const unsigned below = (1u << gl) - 1u;
    if (what == 2) {
        if (take1) cand[__popc(b1 & below)] = idx1;
        if (take2) cand[__popc(b1) + __popc(b2 & below)] = idx2;
        if (amb) cand[__popc(b1) + __popc(b2) + __popc(bA & below)] = idx1;
    }
    __syncwarp();
    // Several candidates that are the same direction within 1e-5 (parallel
    // faces, or edge pairs spanning a face's normal): whichever the exact
    // arithmetic picks, the normal agrees within tolerance and the clip faces
    // follow from it, so the FP32 first minimum is kept. An ambiguous face
    // decides separation and goes to float-float. The direction they are
    // compared with is the warp sweep's first candidate, of its lowest lane
    // (face k and edge k in lane k, the lower of two first).
    const bool several = what == 2 && count > 1 && bA == 0u;
    if (!__any_sync(kAll, several)) return what;
    auto lane32 = [&](int idx) { return (idx < nFace ? idx : idx - nFace) & 31; };
    const int l1 = take1 ? lane32(idx1) : kNone, l2 = take2 ? lane32(idx2) : kNone;
    const int low = group_min(min(l1, l2));
    float lo = FLT_MAX;
    int first = kNone;
    if (take1 && l1 == low) {
        lo = d1 - err1;
        first = idx1;
    }
    if (take2 && l2 == low && (d2 - err2 < lo || (d2 - err2 == lo && idx2 < first))) {
        lo = d2 - err2;
        first = idx2;
    }
    group_argmin(lo, first);
    const unsigned f1 = group_ballot(take1 && idx1 == first), f2 = group_ballot(take2 && idx2 == first);
    const float3 ref = group_from(f1 ? n1 : n2, f1 ? __ffs(f1) - 1 : f2 ? __ffs(f2) - 1 : 0);
    auto agrees = [&](float3 n, float err) {
        const float3 dd = n - ref;
        return err <= 31.f * q.delta && fabsf(xdot(q.D, n)) > tol &&
               !(fmaxf(fabsf(dd.x), fmaxf(fabsf(dd.y), fabsf(dd.z))) > 1e-5f);
    };
    const bool odd = group_any((take1 && !agrees(n1, err1)) || (take2 && !agrees(n2, err2)));
    float d = FLT_MAX;
    int win = kNone;
    if (take1) {
        d = d1;
        win = idx1;
    }
    if (take2 && (d2 < d || (d2 == d && idx2 < win))) {
        d = d2;
        win = idx2;
    }
    group_argmin(d, win);
    const unsigned g1 = group_ballot(take1 && idx1 == win), g2 = group_ballot(take2 && idx2 == win);
    const float3 w = group_from(g1 ? n1 : n2, g1 ? __ffs(g1) - 1 : g2 ? __ffs(g2) - 1 : 0);
    if (several && !odd && (g1 | g2)) {
        sepf = w;
        what = 1;
    }
    return what;
}

// Whether a pair of polyhedra is one for the groups: its axes fill two rounds
// of eight lanes at most.
__device__ __forceinline__ bool sweep_small(const b3::ShapesDev& S, int pa, int pb) {
    const int4 a = poly_axes(S, pa), b = poly_axes(S, pb);
    const int nAx = a.y + b.y;
    return nAx <= kClipGroup && a.w * b.w <= 2 * kClipGroup - nAx && a.w > 0 && b.w > 0;
}

// A pair is apart if the face of A that B's centre is farthest outside of, or the
// face of B for A's centre, separates them by four times the bound on the FP32
// depth's error: the sweep would then find that axis' depth below its own limit
// (one such bound) and end there, so nothing but the work is different.
__device__ __noinline__ bool pair_apart(const PairPre& pre, const b3::ShapesDev& S) {
    SweepPair q;
    sweep_pair(q, pre, S);
    for (int side = 0; side < 2; ++side) {
        const int pi = side ? q.pb : q.pa;
        const Mat3& R = side ? q.RB : q.RA;
        const float3 lc = f3(__ldg(&S.info[3 * pi])), ld = xmul_t(R, q.D);
        const float3 x = side ? lc + ld : lc - ld;  // the other's centre in this one's frame
        const b3ConvexPolyhedron& h = S.polys[pi];
        const int f0 = h.faceOffset, nf = h.numFaces;
        float best = -FLT_MAX;
        float3 pn = make_float3(0.f, 0.f, 0.f);
        for (int f = 0; f < nf; ++f) {
            const float4 pl = __ldg((const float4*)&S.faces[f0 + f].plane[0]);
            const float out = pl.x * x.x + pl.y * x.y + pl.z * x.z + pl.w;
            if (out > best) {
                best = out;
                pn = f3(pl);
            }
        }
        const float3 n = xmul(R, pn);
        float mn0, mx0, mn1, mx1;
        project_packed(S, q.pa, q.RA, n, mn0, mx0);
        project_packed(S, q.pb, q.RB, n, mn1, mx1);
        const float off = xdot(q.rel, n);
        if (fminf(mx0 - (mn1 + off), (mx1 + off) - mn0) < -4.f * q.delta) return true;
    }
    return false;
}

// The queue of an item: 0 the groups', 1 the warps', -1 none (the narrowphase
// skips it, or it is apart).
template <bool kSub>
__device__ __forceinline__ int bin_of(int slot, const int2* __restrict__ pairs, const int4* __restrict__ subs, int base,
                                      const b3::BodiesDev& Bd, const b3::ShapesDev& S) {
    PairPre q;
    item_prefetch<kSub>(q, slot, pairs, subs, base, Bd, S);
    if (q.shapeA < 0) return -1;
    const int bin = sweep_small(S, q.shapeA, q.shapeB) ? 0 : 1;
    return pair_apart(q, S) ? -1 : bin;
}

// Sorts the items into the groups' queue and the warps', up to 2,048 to a round so
// that the counters see one addition each per round; items the narrowphase
// skips, and pairs that are apart, get their flag cleared here. Three quarters of
// the pairs in a settled heap are apart, and a thread finds most of them with two
// faces in place of a warp's or a group's search. Bin and sweeps, the bin without
// -> with the test: 4,096 piles (3.95 M pairs) 4.03 -> 2.07 ms, 131,072 mixed
// bodies (1.60 M) 2.16 -> 1.67, 1,048,576 cubes (7.32 M, no bin before) 2.21 -> 1.54.
constexpr int kBinThreads = 128, kBinItems = 16;
template <bool kSub>
__global__ void __launch_bounds__(kBinThreads, 6)
k_np_bin(const int2* __restrict__ pairs, const int4* __restrict__ subs, const int32_t* __restrict__ numPairsDev,
         b3::BodiesDev Bd, b3::ShapesDev S, int32_t* __restrict__ scalars, uint32_t* __restrict__ manifoldFlag,
         int* __restrict__ smallQ, int* __restrict__ warpQ, int unsortedUpTo) {
    __shared__ int cnt[2], at[2];
    __shared__ int list[kBinThreads * kBinItems];  // the groups' from the front, the warps' from the back
    constexpr int kLast = kBinThreads * kBinItems - 1;
    const int tid = (int)threadIdx.x;
    const int numItems = kSub ? scalars[b3::S_NUM_SUB] : *numPairsDev;
    const int base = kSub ? *numPairsDev : 0;
    if (numItems <= unsortedUpTo) return;
    const int all = (int)gridDim.x * kBinThreads;
    const int items = min(kBinItems, (numItems + all - 1) / all);  // per thread and round
    for (int start = blockIdx.x * kBinThreads * items; start < numItems; start += all * items) {
        if (tid < 2) cnt[tid] = 0;
        __syncthreads();
        for (int u = 0; u < items; ++u) {
            const int i = start + u * kBinThreads + tid;
            const int bin = i < numItems ? bin_of<kSub>(base + i, pairs, subs, base, Bd, S) : -1;
            if (bin < 0 && i < numItems) manifoldFlag[base + i] = 0u;
            const unsigned m0 = __ballot_sync(kAll, bin == 0), m1 = __ballot_sync(kAll, bin == 1);
            int r = 0;
            if ((tid & 31) == 0 && m0) r = atomicAdd(&cnt[0], __popc(m0));
            if ((tid & 31) == 1 && m1) r = atomicAdd(&cnt[1], __popc(m1));
            const int r0 = __shfl_sync(kAll, r, 0), r1 = __shfl_sync(kAll, r, 1);
            if (bin == 0) list[r0 + __popc(m0 & b3dev::lanemask_lt())] = base + i;
            if (bin == 1) list[kLast - (r1 + __popc(m1 & b3dev::lanemask_lt()))] = base + i;
        }
        __syncthreads();
        if (tid < 2 && cnt[tid]) at[tid] = atomicAdd(scalars + (tid ? b3::S_NP_BIG : b3::S_NP_SMALL), cnt[tid]);
        __syncthreads();
        for (int k = tid; k < cnt[0]; k += kBinThreads) smallQ[at[0] + k] = list[k];
        for (int k = tid; k < cnt[1]; k += kBinThreads) warpQ[at[1] + k] = list[kLast - k];
        __syncthreads();
    }
}

// Stage 1, pairs of few axes: see above. Separated pairs are finished here, pairs
// whose axis the sweep decides go to the FP32 clip queue with that axis, pairs
// with near-minimum candidates to the float-float queue. kSub: the items are
// the sub-pairs of compound and mesh pairs, in the slots after the pairs'.
// queue: their slots, or null when every item is one (as they are up to
// unsortedUpTo items).
template <bool kSub>
__global__ void __launch_bounds__(128, 5)
k_np_sweep_groups(const int2* __restrict__ pairs, const int4* __restrict__ subs,
                  const int32_t* __restrict__ numPairsDev, b3::BodiesDev Bd, b3::ShapesDev S,
                  const int* __restrict__ queue, int unsortedUpTo, uint32_t* __restrict__ manifoldFlag,
                  float4* __restrict__ pairSep, int* __restrict__ fastQ, int* __restrict__ slowQ,
                  int* __restrict__ warpQ, int* __restrict__ cand, int candSlots, int32_t* __restrict__ scalars) {
    extern __shared__ __align__(16) unsigned char np_smem[];
    const int lane = threadIdx.x & 31, grp = lane / kClipGroup, gl = grp_lane();
    SweepScratch& W = reinterpret_cast<SweepScratch*>(np_smem)[threadIdx.x >> 5];
    const int base = kSub ? *numPairsDev : 0;
    const int items = kSub ? scalars[b3::S_NUM_SUB] : *numPairsDev;
    if (items <= unsortedUpTo) queue = nullptr;
    const int total = queue ? scalars[b3::S_NP_SMALL] : items;
    // pairs per grab: one round of the groups while the pairs are few, so that
    // all warps have some; 32 once there are enough
    const int warps = gridDim.x * (blockDim.x >> 5);
    int per = 32 / kClipGroup;
    while (per < kSweepChunk && total > 2 * per * warps) per *= 2;
    int i0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per;
    while (i0 < total) {
        const int m = min(per, total - i0);
        int p = -1;
        if (lane < m) {
            p = queue ? queue[i0 + lane] : base + i0 + lane;
            item_prefetch<kSub>(W.pre[lane], p, pairs, subs, base, Bd, S);
            W.pre[lane].aux.w = 0.f;
        }
        __syncwarp();
        for (int r0 = 0; r0 < m; r0 += 32 / kClipGroup) {
            const int r = r0 + grp;
            const PairPre& pre = W.pre[min(r, m - 1)];
            const bool has = r < m && pre.shapeA >= 0;
            // a group without a pair goes along with another's
            const unsigned who = __ballot_sync(kAll, has);
            if (!who) continue;
            const int stand = __shfl_sync(kAll, r, __ffs(who) - 1);
            int count = 0;
            float3 sepf = make_float3(0.f, 0.f, 0.f);
            const int what = group_sweep(has ? pre : W.pre[stand], has, S, W.cand[grp], sepf, count);
            const unsigned near = __ballot_sync(kAll, gl == 0 && what == 2);
            const unsigned big = __ballot_sync(kAll, gl == 0 && what == 3);
            int slot = 0;
            if (lane == 0 && near) slot = atomicAdd(scalars + b3::S_NP_SLOW, __popc(near));
            if (lane == 0 && big) {
                int at = atomicAdd(scalars + b3::S_NP_BIG, __popc(big));
                for (unsigned l = big; l; l &= l - 1) warpQ[at++] = W.pre[r0 + (__ffs(l) - 1) / kClipGroup].p;
            }
            slot = __shfl_sync(kAll, slot, 0) + __popc(near & ((1u << (lane & ~(kClipGroup - 1))) - 1u));
            if (what == 2) {
                const bool kept = slot < candSlots;
                if (kept && gl < count) cand[(size_t)slot * kMaxCand + gl] = W.cand[grp][gl];
                if (gl == 0) {
                    slowQ[slot] = pre.p;
                    pairSep[pre.p] = make_float4(__int_as_float(kept ? count : -1), 0.f, 0.f, (float)kSepRefine);
                }
            }
            if (gl == 0 && what != 0)
                W.pre[r].aux = make_float4(sepf.x, sepf.y, sepf.z, what == 1 ? 1.f : 2.f);
            __syncwarp();
        }
        __syncwarp();
        // the chunk's decided pairs enter the clip queue with one addition
        const float4 s = lane < m ? W.pre[lane].aux : make_float4(0.f, 0.f, 0.f, 2.f);
        const unsigned fast = __ballot_sync(0xffffffffu, s.w == 1.f);
        int at = 0;
        if (lane == 0 && fast) at = atomicAdd(scalars + b3::S_NP_FAST, __popc(fast));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (s.w == 1.f) {
            pairSep[p] = make_float4(s.x, s.y, s.z, (float)kSepDecided);
            fastQ[at + __popc(fast & b3dev::lanemask_lt())] = p;
        } else if (s.w == 0.f) {
            manifoldFlag[p] = 0u;
        }
        if (lane == 0) i0 = (warps + atomicAdd(scalars + b3::S_NP_WORK, 1)) * per;
        i0 = __shfl_sync(0xffffffffu, i0, 0);
    }
}
