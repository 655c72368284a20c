// Fixed-radius search and flat-COO edge construction.
//
// Replaces _count_edges_kernel! / _fill_edges_kernel_{3d,2d}! /
// _build_edges_cuda! (ext/OctopusCUDAExt.jl:262-415) and reproduces the CPU
// path's output exactly (src/cpu/edges_cpu.jl:36-247):
//
//   * The build lays the points out in the order in which the reference's
//     depth-first search visits them (build.cu sections 6 and 7), so each
//     query's neighbors, in the reference's order, are the in-radius points
//     in ascending position of that layout, whatever structure finds them.
//   * One warp serves one chunk of the query set's layout (at most 32 points,
//     a run of sibling leaves).  It walks the box hierarchy over the target's
//     layout, one lane per child box (fan-out 32), in ascending position,
//     down to the target chunks.  The box tests are conservative
//     (QueryBox), and the exact per-pair test
//     d2 = ((dx*dx + dy*dy) + dz*dz) <= r*r decides membership.
//   * Target points are staged in shared memory and broadcast to the 32 lanes.
//   * counts -> int64 exclusive scan -> fill at the per-query cursor.

#include <algorithm>

#include "internal.h"
#include "scan.cuh"

namespace oct {

constexpr int kEdgeWarps = 4;
// Blocks of k_edges per SM: the most that leave it without spills (Float32 count
// of 1M lattice points with 7 / 8 / 10: 269 / 260 / 290 us).
template <class T> constexpr int kEdgeBlocks = sizeof(T) == 4 ? 8 : 5;
constexpr int kEdgeThreads = kEdgeWarps * 32;
constexpr int kStage = 32;  // staged hits per lane, and points per chunk

// The three passes of k_edges.
enum EdgePass {
    EP_COUNT = 0,   // per-query neighbor counts only
    EP_RECORD = 1,  // counts, plus each query's hit records (up to rec_cap of them)
    EP_FILL = 2,    // the COO at the scanned offsets by a second walk (groups whose records overflowed)
    EP_STATS = 3,   // the count pass with traversal statistics (a diagnostic, oct_edges_traversal_stats)
};

// Traversal statistics of EP_STATS, summed over the launch.
enum TraversalStat {
    TS_GROUPS = 0,     // query groups (warps)
    TS_QUERIES,        // query points
    TS_EXPANSIONS,     // rounds of box tests (up to 32 boxes each)
    TS_CHILDREN,       // boxes tested
    TS_CHUNKS,         // target chunks staged
    TS_TARGETS,        // target points staged
    TS_STEPS,          // pair-loop steps executed (four targets each)
    TS_PAIR_TESTS,     // query-target distance tests issued (steps x 4 x queries of the group)
    TS_HITS,           // pairs within the radius (self pair excluded when asked)
    TS_CYCLES_TOTAL,   // SM cycles of the warps, summed
    TS_CYCLES_LEAF,    // ... of which in target chunks (staging and pair tests)
    TS_CYCLES_PAIRS,   // ... of which in the pair loop
    TS_NUM
};

// A hit record: the visiting position of a target chunk's first point and the
// bit mask of the chunk's points within the radius of one query.  A query's
// records, in order, list its neighbors in the reference's order.
constexpr int kMaxRecords = 65000;  // per query: the record count is stored in 16 bits
constexpr uint16_t kOverflowMark = 0xffff;  // record count of the queries of an overflowed group

// Edge k of the COO: sender = target point t, receiver = query qi at px
// (src/cpu/edges_cpu.jl:200-215: rel_displacement = (x_q - x_t) * inv(r),
// rel_dist_norm = sqrt(d2) * inv(r), 1-based indices).
template <class T, int D>
__device__ __forceinline__ void write_edge(int64_t k, const SPt<T, D>& t, const T* px, int32_t qi, int32_t base,
                                           T inv_r, int32_t* __restrict__ senders, int32_t* __restrict__ receivers,
                                           T* __restrict__ rdisp, T* __restrict__ rdist) {
    senders[k] = t.idx - base + 1;
    if (rdisp == nullptr) return;  // neighbor lists (CSR values) only
    T diff[D];
    const T d2 = dist2<T, D>(t.x, px, diff);
    receivers[k] = qi - base + 1;
#pragma unroll
    for (int d = 0; d < D; ++d) rdisp[(int64_t)D * k + d] = mul_rn(-diff[d], inv_r);
    rdist[k] = mul_rn(sqrt_rn(d2), inv_r);
}

// Radius and index base of the point set (cloud) holding position p (sorted
// and visiting positions of a cloud share one range).
template <class T>
__device__ __forceinline__ void cloud_params(const Batch& bt, int64_t p, T& r2, T& inv_r, int32_t& base) {
    if (bt.n_clouds) {
        const int c = cloud_of_position(bt, p);
        const double* cp = bt.cparam + (size_t)c * kCloudParams;
        r2 = (T)cp[4];
        inv_r = (T)cp[5];
        base = (int32_t)bt.coff[c];
    }
}

// sqrt to within 2^-22 of its value (the slack of the bounds it goes into is 2^-20)
__device__ __forceinline__ float sqrt_near(float a) {
    float s;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(a));
    return s;
}
__device__ __forceinline__ double sqrt_near(double a) { return sqrt_rn(a); }

// The pair test of one staged chunk of targets against the warp's queries.
//
// EXACT: d2 in the reference's operation order, packed differences and
// squares for two float targets at a time and scalar sums (packed
// add.rn.f32x2 sums after the packed squares changed results, as a fused
// multiply-add would).  About ten issue slots per target.
//
// FAST decides the same test from another expression.  With c the middle of
// the query chunk's box, t' = t - c and q' = q - c rounded to the element
// type, and |t'|^2 stored beside the target,
//     d = (|t'|^2 + (|q'|^2 - r2)) - 2 q' . t'
// by fused multiply-adds: half an addition, 3/2 multiply-adds, one funnel
// shift collecting the sign and half a three-way minimum per target.  Every
// coordinate and intermediate is bounded through the boxes: a target that
// passed the box test has |t - c| <= half extent + r per axis.  With
// S = 2 (sum h^2 + sum (h + r)^2) + r2, which bounds every intermediate,
// u the unit roundoff: the coordinates' rounding contributes 2 u S, the two
// squared norms 3 u S, the sums and multiply-adds 4 u S, and the reference's
// own rounding of d2 near r2 5 u S, so the sign of d decides as the reference
// does whenever |d| > 14 u S.  eps = 32 u S leaves more than a factor of two;
// a chunk with a smaller |d| in any lane (about 0.4% of them at 28 neighbors
// per point) is tested again by EXACT.  Groups whose box is large against r
// (eps above 2^-11 r2: the uncertain shell would be met too often) and
// radii near the ends of the type's range use EXACT alone.
template <class T> struct PairConst;
template <> struct PairConst<float> {
    static constexpr float eps = 1.0f / (1 << 19);  // 32 u
    static constexpr float shell = 1.0f / (1 << 11);
    static constexpr float slack = 1.0f / (1 << 20);
    static constexpr float place = 1.0f / (1 << 20);  // rounding of a box's middle against its coordinates
    static constexpr float tiny = 1e-30f, huge = 1e36f, far = 1e38f;
};
template <> struct PairConst<double> {
    static constexpr double eps = 1.0 / (1ULL << 48);  // 32 u
    static constexpr double shell = 1.0 / (1 << 11);
    static constexpr double slack = 1.0 / (1 << 15);  // also the slack of QueryBox
    static constexpr double place = 1.0 / (1ULL << 48);
    static constexpr double tiny = 1e-290, huge = 1e290, far = 1e300;
};

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
// max(a, b, 0)
__device__ __forceinline__ float gap(float a, float b) {
    float d;
    asm("max.f32 %0, %1, %2, 0f00000000;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// The box of a warp's queries against the search's boxes and target points.
// No pair within r is lost; how near the rest may be decides only the work.
template <class T, int D> struct QueryBox;

// Float32: per-axis gaps of the coordinates, squared and summed by fused
// multiply-adds, against lim = r2 (1 + 2^-20) + 7 subnormals.  A pair of points
// inside with d2 <= r2 has per-axis gaps of at most its own differences, and
// the roundings of the two sums (4 u each, and less than a subnormal per
// square) are far inside the bound's slack.
template <int D> struct QueryBox<float, D> {
    float lo[D], hi[D], lim;
    __device__ __forceinline__ bool near(const float* blo, const float* bhi) const {
        float acc = 0.f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const float g = gap(__fsub_rn(blo[d], hi[d]), __fsub_rn(lo[d], bhi[d]));
            acc = d == 0 ? __fmul_rn(g, g) : __fmaf_rn(g, g, acc);
        }
        return acc <= lim;
    }
    __device__ __forceinline__ bool near(const BoxNode<float, D>& nd) const { return near(nd.lo, nd.hi); }
    __device__ __forceinline__ bool near_point(const float* x, const float*) const { return near(x, x); }
};

// Float64: gaps of the fixed-point boxes (BoxUnits) in integers.  For a pair
// within r, with u = (x - o) s rounded to 2^-21 at most, two floors differ by
// less than |u_t - u_q| + 1 <= r s + 1 on an axis; lo and hi hold the queries'
// extremes less and plus that 1, so the squared gaps sum to less than
// (r s)^2 + 1 = lim (lim's extra 1 covers the 2^-21).  A gap is cut at 2^15,
// above any r s, which keeps the sum below 2^32.
//
// A target point is tested by its offset from the box's middle, which the pair
// test needs anyway, in radii and Float32 (`half` has room for its rounding).
template <int D> struct QueryBox<double, D> {
    int32_t lo[D], hi[D];
    unsigned lim;
    float half[D];
    double per_r;  // 1 / r
    __device__ __forceinline__ bool near(const BoxNode<double, D>& nd) const {
        unsigned acc = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const unsigned g = min(__vimax3_s32(nd.lo[d] - hi[d], lo[d] - nd.hi[d], 0), 1 << 15);
            acc += g * g;
        }
        return acc <= lim;
    }
    __device__ __forceinline__ bool near_point(const double*, const double* x) const {
        float acc = 0.f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const float g = fmaxf(__fsub_rn(fabsf((float)__dmul_rn(x[d], per_r)), half[d]), 0.f);
            acc = d == 0 ? __fmul_rn(g, g) : __fmaf_rn(g, g, acc);
        }
        return acc <= 1.f + 0x1p-16f;
    }
};

// Bits of the targets (those of `keep`) within the radius of query q; sx[d] =
// the targets' coordinates.
template <int D>
__device__ __forceinline__ unsigned pairs_exact(const float (*sx)[32], unsigned keep, const float* q, float r2) {
    unsigned hm = 0;
    unsigned long long P[D];
#pragma unroll
    for (int d = 0; d < D; ++d) P[d] = pack2(q[d], q[d]);
    // one bit per step of four targets with a target kept
    for (unsigned km = (keep | keep >> 1 | keep >> 2 | keep >> 3) & 0x11111111u; km; km &= km - 1) {
        const int j = __ffs(km) - 1;
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const ulonglong2 px = *reinterpret_cast<const ulonglong2*>(&sx[d][j]);
            const unsigned long long da = sub2_rn(px.x, P[d]);
            const unsigned long long db = sub2_rn(px.y, P[d]);
            const unsigned long long qa = mul2_rn(da, da);
            const unsigned long long qb = mul2_rn(db, db);
            s0 = (d == 0) ? lo2(qa) : __fadd_rn(s0, lo2(qa));
            s1 = (d == 0) ? hi2(qa) : __fadd_rn(s1, hi2(qa));
            s2 = (d == 0) ? lo2(qb) : __fadd_rn(s2, lo2(qb));
            s3 = (d == 0) ? hi2(qb) : __fadd_rn(s3, hi2(qb));
        }
        hm |= ((s0 <= r2 ? 1u : 0u) | (s1 <= r2 ? 2u : 0u) | (s2 <= r2 ? 4u : 0u) | (s3 <= r2 ? 8u : 0u)) << j;
    }
    return hm & keep;
}
template <int D>
__device__ __forceinline__ unsigned pairs_exact(const double (*sx)[32], unsigned keep, const double* q, double r2) {
    unsigned hm = 0;
    for (unsigned km = keep; km; km &= km - 1) {
        const int j = __ffs(km) - 1;
        double t[D], diff[D];
#pragma unroll
        for (int d = 0; d < D; ++d) t[d] = sx[d][j];
        hm |= (dist2<double, D>(t, q, diff) <= r2 ? 1u : 0u) << j;
    }
    return hm;
}

// The same by FAST: sx[d] = t', sx[D] = |t'|^2 (PairConst::far for a target
// outside `keep`); m2q = -2 q', off = |q'|^2 - r2.  *close: some |d| <= eps.
template <int D>
__device__ __forceinline__ unsigned pairs_fast(const float (*sx)[32], unsigned keep, const float* m2q, float off,
                                               float eps, bool* close) {
    unsigned hm = 0;
    float u = PairConst<float>::far;
    unsigned long long M[D];
#pragma unroll
    for (int d = 0; d < D; ++d) M[d] = pack2(m2q[d], m2q[d]);
    const unsigned long long O = pack2(off, off);
    const unsigned steps = keep | keep >> 1 | keep >> 2 | keep >> 3;
#pragma unroll
    for (int j = 28; j >= 0; j -= 4) {
        if (steps >> j & 1u) {
            const ulonglong2 tt = *reinterpret_cast<const ulonglong2*>(&sx[D][j]);
            unsigned long long a = add2_rn(tt.x, O), b = add2_rn(tt.y, O);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const ulonglong2 px = *reinterpret_cast<const ulonglong2*>(&sx[d][j]);
                a = fma2_rn(px.x, M[d], a);
                b = fma2_rn(px.y, M[d], b);
            }
            u = min3_abs(lo2(a), hi2(a), u);
            u = min3_abs(lo2(b), hi2(b), u);
            hm = __funnelshift_l((unsigned)(b >> 32), hm, 1);
            hm = __funnelshift_l((unsigned)b, hm, 1);
            hm = __funnelshift_l((unsigned)(a >> 32), hm, 1);
            hm = __funnelshift_l((unsigned)a, hm, 1);
        } else {
            hm <<= 4;
        }
    }
    *close = u <= eps;
    return hm;
}
template <int D>
__device__ __forceinline__ unsigned pairs_fast(const double (*sx)[32], unsigned keep, const double* m2q, double off,
                                               double eps, bool* close) {
    unsigned hm = 0, u = 0x7fffffffu;  // u: smallest high word of |d|
    for (unsigned km = (keep | keep >> 1) & 0x55555555u; km; km &= km - 1) {
        const int j = __ffs(km) - 1;
        const double2 tt = *reinterpret_cast<const double2*>(&sx[D][j]);
        double a = __dadd_rn(tt.x, off), b = __dadd_rn(tt.y, off);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double2 px = *reinterpret_cast<const double2*>(&sx[d][j]);
            a = __fma_rn(px.x, m2q[d], a);
            b = __fma_rn(px.y, m2q[d], b);
        }
        const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
        u = min(u, min(ha & 0x7fffffffu, hb & 0x7fffffffu));
        hm |= ((ha >> 31) | (hb >> 31) << 1) << j;
    }
    *close = u <= (unsigned)__double2hiint(eps);
    return hm;
}

// Bound by instruction issue and the latency of a warp's dependent steps (63%
// of issue slots at 38% of the warp slots on a 343,000-point lattice, where
// k_edges over the tree with an exact test per pair executed 100 M warp
// instructions, this one 64 M).  Count, before and after: 1M lattice points
// 313 -> 258 us, 2M uniform points at 14 neighbors 792 -> 663, 1M clustered 2D
// points at 151 neighbors 373 -> 298, 200,003 Float64 points 152 -> 147, 250,007
// queries against 1M points 329 -> 255.  Not faster: loading the next chunk's
// points while this one is tested (72 registers), spans of 256 or 1024
// positions, two or eight warps per block, two chunks of queries per warp.
//
// ocount: in the record pass, ocount[0] counts the groups whose records
// overflowed (those groups are walked again by the fill pass) and ocount[1]
// is the largest record count of a query; in the fill pass, ocount[0] is
// the bounds-guard word.  recs[qpos * rec_cap + r] = record r of the query at
// visiting position qpos, rcount[qpos] = its record count, gflag[g] = 1 when a
// query of group g had more than rec_cap records.  qpos_of[i] = the visiting
// position of query point i (when given), which the fill reads.
template <class T, int D, int PASS>
__global__ void __launch_bounds__(kEdgeThreads, kEdgeBlocks<T>) k_edges(
    const SPt<T, D>* __restrict__ qpts, const BoxNode<T, D>* __restrict__ qchunks, int64_t n_groups,
    const __grid_constant__ Bvh<T, D> bv, const __grid_constant__ BoxUnits bu, const SPt<T, D>* __restrict__ tpts,
    int64_t n_targets, T r2, T inv_r, int exclude_self,
    int32_t* __restrict__ counts, int32_t* __restrict__ qpos_of, const int64_t* __restrict__ offsets,
    int32_t* __restrict__ senders, int32_t* __restrict__ receivers, T* __restrict__ rdisp, T* __restrict__ rdist,
    int* __restrict__ ocount, int2* __restrict__ recs, int64_t rec_cap, uint16_t* __restrict__ rcount,
    uint8_t* __restrict__ gflag, Batch bt, unsigned long long* __restrict__ stats) {
    pdl_wait();
    pdl_trigger();
    constexpr bool STAGE = PASS == EP_FILL;
    constexpr bool STATS = PASS == EP_STATS;
    constexpr unsigned FULL = 0xffffffffu;
    long long st_t0 = 0, st_leaf = 0, st_pairs = 0;
    unsigned long long st_exp = 0, st_children = 0, st_chunks = 0, st_targets = 0, st_steps = 0;
    if constexpr (STATS) st_t0 = clock64();
    // The current target chunk, structure of arrays so that four targets load
    // as 16 bytes per axis (row D: |t'|^2).
    __shared__ __align__(16) T sx[kEdgeWarps][D + 1][32];
    // Upper levels of the walk: the child boxes still to visit, their first index.
    __shared__ uint2 swalk[kEdgeWarps][kBvhLevels];
    // Fill pass: each lane stages the positions of its next hits; a flush
    // writes them as runs of consecutive edges of one query.
    __shared__ int32_t obuf[STAGE ? kEdgeWarps : 1][32][STAGE ? kStage + 1 : 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t g = (int64_t)blockIdx.x * kEdgeWarps + w;
    if (g >= n_groups) return;  // warp-uniform
    if (PASS == EP_FILL && recs != nullptr && gflag[g] == 0) return;  // expanded from its records
    const BoxNode<T, D> gc = qchunks[g];
    const bool valid = lane < gc.b;
    const int64_t qpos = gc.a + (valid ? lane : 0);  // position of this lane's query
    const SPt<T, D> q = qpts[qpos];
    // A batch searches each cloud in its own positions with its own radius and
    // reports cloud-local indices.
    int32_t base = 0, cloud = 0;
    int32_t plo = 0, phi = (int32_t)n_targets;
    if (bt.n_clouds) {
        cloud = cloud_of_position(bt, gc.a);
        const double* cp = bt.cparam + (size_t)cloud * kCloudParams;
        r2 = (T)cp[4];
        inv_r = (T)cp[5];
        base = plo = (int32_t)bt.coff[cloud];
        phi = (int32_t)bt.coff[cloud + 1];
    }
    // The queries' box and the fast pair test's constants (see pairs_fast).
    using PC = PairConst<T>;
    QueryBox<T, D> qb;
    T ctr[D], m2q[D], off, eps;  // ctr: the middle of the queries' box
    bool fast = r2 >= PC::tiny;
    {
        const T r = sqrt_near(r2) * (T(1) + PC::slack);
        T h[D];  // |x - ctr| of a query is no more
        if constexpr (sizeof(T) == 4) {
            qb.lim = r2 * (T(1) + PC::slack) + 1e-44f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                qb.lo[d] = gc.lo[d];
                qb.hi[d] = gc.hi[d];
                const T half = T(0.5) * (gc.hi[d] - gc.lo[d]);
                ctr[d] = gc.lo[d] + half;
                h[d] = half * (T(1) + PC::slack) + fabs(ctr[d]) * PC::place;
            }
        } else {
            BoxUnits un = bu;
            if (bt.n_clouds) {
                un = cloud_units(bt, cloud);
                un.width = div_rn(1.0, un.s);
            }
            const T half_unit = T(0.5) * un.width, half_more = half_unit * (T(1) + PC::slack);
            qb.lim = (un.mul > 1.0 ? (unsigned)(un.mul * un.mul) : 1u) + 1u;
            qb.per_r = un.s / un.mul;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                // The box in the target's units: another query set's from its
                // points, cut at +-kFar (beyond that no target is near, and the
                // fast test's bounds do not hold).
                constexpr int32_t kFar = (1 << 30) - 1;
                int32_t lo = gc.lo[d], hi = gc.hi[d];
                if (qchunks != bv.chunk) {
                    const int32_t u = min(max(box_coord(q.x[d], d, un), -kFar), kFar);
                    lo = box_min(u);
                    hi = box_max(u);
                    fast = fast && lo > -kFar && hi < kFar;
                }
                qb.lo[d] = lo - 1;
                qb.hi[d] = hi + 1;
                ctr[d] = fma_rn((T)(lo + hi + 1), half_unit, un.o[d]);
                h[d] = fma_rn((T)(hi - lo + 1), half_more, (fabs(ctr[d]) + fabs(un.o[d])) * PC::place);
                qb.half[d] = __fmaf_rn(__double2float_ru(h[d] * qb.per_r), 1.f + 0x1p-20f, 0x1p-20f);
            }
        }
        T qq = T(0), tt = T(0), qn = T(0);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            qq += h[d] * h[d];
            tt += (h[d] + r) * (h[d] + r);
            const T x = q.x[d] - ctr[d];
            m2q[d] = T(-2) * x;
            qn += x * x;
        }
        const T S = T(2) * (qq + tt) + r2;
        eps = PC::eps * S;
        off = valid ? qn - r2 : PC::far;  // a lane without a query hits nothing
        fast = fast && eps <= PC::shell * r2 && S <= PC::huge;  // false for a NaN
    }
    int32_t cnt = 0;
    int64_t cur = 0, cur_end = 0;
    if (PASS == EP_FILL && valid) {
        cur = offsets[q.idx];
        cur_end = offsets[q.idx + 1];
    }
    int ocnt = 0;
    int nrec = 0;
    const int cap = (int)rec_cap;
    int2* myrec = PASS == EP_RECORD ? recs + qpos * rec_cap : nullptr;  // this query's records

    // One query per round: lane e writes the query's e-th staged edge, so a
    // round stores a run of consecutive edges of one segment.  Only the lanes
    // passing `need` are flushed, so each query leaves in long runs.
    auto flush = [&](bool need) {
        __syncwarp();
        unsigned busy = __ballot_sync(FULL, need && ocnt > 0);
        while (busy) {
            const int ql = __ffs(busy) - 1;
            busy &= busy - 1;
            const int nql = __shfl_sync(FULL, ocnt, ql);
            const long long cq = __shfl_sync(FULL, (long long)cur, ql);
            const long long ce = __shfl_sync(FULL, (long long)cur_end, ql);
            const int32_t qi = __shfl_sync(FULL, q.idx, ql);
            T px[D];
#pragma unroll
            for (int d = 0; d < D; ++d) px[d] = __shfl_sync(FULL, q.x[d], ql);
            if (lane < nql) {
                const int64_t k = cq + lane;
                if (k < ce)
                    write_edge<T, D>(k, tpts[obuf[w][ql][lane]], px, qi, base, inv_r, senders, receivers, rdisp,
                                     rdist);
                else
                    atomicOr(ocount, 1);  // never taken when count and fill agree
            }
        }
        if (need) {
            cur += ocnt;
            ocnt = 0;
        }
        __syncwarp();
    };

    // One target chunk: positions [first, first + num); t = this lane's point
    // of it (lane < num).
    auto visit = [&](int32_t first, int num, const SPt<T, D>& t) {
        long long st_c0 = 0;
        if constexpr (STATS) st_c0 = clock64();
        // A target farther than r from the group's box can be no query's
        // neighbor: the pair loop skips the steps whose targets all are.
        T x[D];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = t.x[d] - ctr[d];
        const bool near = lane < num && qb.near_point(t.x, x);
        const unsigned keep = __ballot_sync(FULL, near);
        if (keep == 0) return;
        long long st_p0 = 0;
        if constexpr (STATS) {
            st_p0 = clock64();
            ++st_chunks;
            st_targets += num;
            st_steps += __popc((keep | keep >> 1 | keep >> 2 | keep >> 3) & 0x11111111u);
        }
        unsigned hm = 0;
        bool exact = !fast;
        if (fast) {
            T tt = T(0);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                if (!near) x[d] = T(0);
                tt = d == 0 ? x[d] * x[d] : fma_rn(x[d], x[d], tt);
            }
            if (!near) tt = PC::far;
            __syncwarp();  // every lane is done with the previous chunk
#pragma unroll
            for (int d = 0; d < D; ++d) sx[w][d][lane] = x[d];
            sx[w][D][lane] = tt;
            __syncwarp();
            bool close;
            hm = pairs_fast<D>(sx[w], keep, m2q, off, eps, &close);
            exact = __any_sync(FULL, close);
        }
        if (exact) {
            __syncwarp();
#pragma unroll
            for (int d = 0; d < D; ++d) sx[w][d][lane] = near ? t.x[d] : T(INFINITY);
            __syncwarp();
            hm = valid ? pairs_exact<D>(sx[w], keep, q.x, r2) : 0u;
        }
        if constexpr (STATS) st_pairs += clock64() - st_p0;
        if (exclude_self && first == gc.a) hm &= ~(1u << lane);  // the group's own chunk (same tree)
        const int nh = __popc(hm);
        cnt += nh;
        if (PASS == EP_RECORD) {
            if (hm != 0) {
                if (nrec < cap) myrec[nrec] = make_int2(first, (int32_t)hm);
                ++nrec;
            }
        } else if (STAGE) {
            if (__any_sync(FULL, ocnt + nh > kStage)) flush(ocnt + nh > kStage);
            while (hm) {
                const int j = __ffs(hm) - 1;
                hm &= hm - 1;
                obuf[w][lane][ocnt++] = first + j;
            }
        }
        if constexpr (STATS) st_leaf += clock64() - st_c0;
    };

    // The walk: level `l` nodes from `b0` on, `m` those of the current round
    // still to descend into; the levels above wait in swalk.  It starts at the
    // lowest level with at most 64 nodes over the positions searched.
    int top = 0;
    while (top < bv.top && ((phi - 1) >> (kSpanShift + 5 * top)) - (plo >> (kSpanShift + 5 * top)) >= 64) ++top;
    const int32_t i1 = ((phi - 1) >> (kSpanShift + 5 * top)) + 1;
    int32_t na = 0, nb = 0;  // the last level-0 round's nodes, one per lane: first chunk, chunks
    auto test = [&](int l, int32_t b0, int32_t end) {
        const int32_t i = b0 + lane;
        bool pass = false;
        if (i < end) {
            const BoxNode<T, D> nd = bv.lev[l][i];
            pass = qb.near(nd);
            if (l == 0) {
                na = nd.a;
                nb = nd.b;
            }
        }
        if constexpr (STATS) {
            ++st_exp;
            st_children += min(32, end - b0);
        }
        return __ballot_sync(FULL, pass);
    };
    int l = top;
    int32_t b0 = plo >> (kSpanShift + 5 * top);
    unsigned m = test(l, b0, i1);
    while (true) {
        if (m == 0) {
            if (l == top) {
                b0 += 32;
                if (b0 >= i1) break;
                m = test(l, b0, i1);
            } else {
                ++l;
                __syncwarp();
                const uint2 up = swalk[w][l];
                m = up.x;
                b0 = (int32_t)up.y;
            }
            continue;
        }
        const int i = __ffs(m) - 1;
        m &= m - 1;
        if (l > 0) {
            __syncwarp();
            if (lane == 0) swalk[w][l] = make_uint2(m, (unsigned)b0);
            b0 = (b0 + i) * 32;
            --l;
            m = test(l, b0, min(b0 + 32, bv.cnt[l]));
            continue;
        }
        const int32_t c0 = __shfl_sync(FULL, na, i);
        const int nc = __shfl_sync(FULL, nb, i);
        for (int cb = 0; cb < nc; cb += 32) {
            int32_t first = 0, num = 0;
            bool pass = false;
            if (cb + lane < nc) {
                const BoxNode<T, D> nd = bv.chunk[c0 + cb + lane];
                pass = qb.near(nd) && nd.a >= plo && nd.a < phi;
                first = nd.a;
                num = nd.b;
            }
            if constexpr (STATS) {
                ++st_exp;
                st_children += min(32, nc - cb);
            }
            unsigned cm = __ballot_sync(FULL, pass);
            while (cm) {
                const int j = __ffs(cm) - 1;
                cm &= cm - 1;
                const int32_t f = __shfl_sync(FULL, first, j);
                const int k = __shfl_sync(FULL, num, j);
                SPt<T, D> t;
                if (lane < k) t = tpts[f + lane];
                visit(f, k, t);
            }
        }
    }
    if (STAGE) flush(true);
    if (PASS != EP_FILL && valid) {
        counts[q.idx] = cnt;
        if (PASS == EP_RECORD || PASS == EP_COUNT) {
            if (qpos_of) qpos_of[q.idx] = (int32_t)qpos;
        }
    }
    if constexpr (STATS) {
        const unsigned long long hits = warp_sum((unsigned long long)cnt);
        const int nv = __popc(__ballot_sync(FULL, valid));
        if (lane == 0) {
            const unsigned long long v[TS_NUM] = {1ull, (unsigned long long)nv, st_exp, st_children, st_chunks,
                                                  st_targets, st_steps, 4ull * st_steps * (unsigned long long)nv, hits,
                                                  (unsigned long long)(clock64() - st_t0), (unsigned long long)st_leaf,
                                                  (unsigned long long)st_pairs};
#pragma unroll
            for (int k = 0; k < TS_NUM; ++k) atomicAdd(stats + k, v[k]);
        }
    }
    if (PASS == EP_RECORD) {
        const bool over = __any_sync(FULL, nrec > cap);
        if (valid) rcount[qpos] = over ? kOverflowMark : (uint16_t)nrec;
        const int mx = __reduce_max_sync(FULL, nrec);
        if (lane == 0) {
            gflag[g] = over ? 1 : 0;
            if (over) atomicAdd(ocount, 1);
            // The maximum settles after a few groups: most groups only read it.
            if (mx > __ldcg(ocount + 1)) atomicMax(ocount + 1, mx);
        }
    }
}

// The D values of rel_displacement column k (T-aligned D-tuples).  PAIRS: the
// array is aligned to two values, so two of them leave as one word: in 3D the
// first two of an even column and the last two of an odd one, which halves the
// columns' strided stores in the same two instructions for every lane.
template <class T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };
template <class T, int D>
__device__ __forceinline__ void store_column(T* __restrict__ rdisp, int64_t k, const T* v, bool pairs) {
    using P = typename Pair<T>::type;
    T* p = rdisp + (int64_t)D * k;
    if (!pairs) {
#pragma unroll
        for (int d = 0; d < D; ++d) p[d] = v[d];
    } else if constexpr (D == 2) {
        P w;
        w.x = v[0];
        w.y = v[1];
        *reinterpret_cast<P*>(p) = w;
    } else {
        const bool odd = k & 1;
        P w;
        w.x = odd ? v[1] : v[0];
        w.y = odd ? v[2] : v[1];
        *reinterpret_cast<P*>(p + (odd ? 1 : 0)) = w;
        p[odd ? 0 : 2] = odd ? v[0] : v[2];
    }
}

// Position (0..31) of the k-th set bit (k from 0) of m; k < popc(m).
__device__ __forceinline__ int kth_set_bit(unsigned m, int k) {
    int pos = 0;
    int c = __popc(m & 0xffffu);
    if (k >= c) { k -= c; m >>= 16; pos += 16; }
    c = __popc(m & 0xffu);
    if (k >= c) { k -= c; m >>= 8; pos += 8; }
    c = __popc(m & 0xfu);
    if (k >= c) { k -= c; m >>= 4; pos += 4; }
    c = __popc(m & 0x3u);
    if (k >= c) { k -= c; m >>= 2; pos += 2; }
    c = (int)(m & 1u);
    if (k >= c) pos += 1;
    return pos;
}

// Fill pass from the records with direct stores, in original index order
// (the default fill; k_expand below writes through bulk copies instead: a
// tuned alternative, and the fill of more than 2^27 targets).  Warp v owns
// queries 32v .. 32v+31, one per lane; their records, query after query, form
// one flat list, and so do their edges, in the same order (a record's hits are
// consecutive edges of its query).  The warp loads the records 32 at a time
// (one per lane), scans their hit counts and appends each hit (query lane <<
// 27 | target position) to a list in shared memory; whenever the list holds a
// round of 64 edges it writes them, one per lane and window of 32:
//   * a record's query: the queries whose records reach into the 32-record
//     window set one bit each at their first record in the window (the one
//     running into the window at bit 0), so the query of record l is the
//     (popc of the bits up to l)-th of them (ballot, reduce-or, popc; no search);
//   * windows start at multiples of 32 COO slots, so a window's index and
//     distance stores are one 128-byte line each (4-byte elements), and are
//     full except at the two ends of the warp's range;
//   * consecutive lanes take consecutive edges: their targets share chunks
//     and their queries' data (one 16-byte load of shared memory) is mostly
//     the same.
// Edge f of the flat list goes to COO slot kb[q] + f of its query q.  Queries
// of an overflowed group (record count kOverflowMark) are left to the walking
// fill.
//
// Bound by L1 (76% on a 343,000-point lattice: the gathered targets and the
// strided columns) and instruction issue (68%), at 3.5 to 3.8 TB/s of COO.
// Against windows that start and end with each batch of 32 records, with the
// query's data by shuffles and one store per value: 1M lattice points 225 ->
// 193 us, 1M clustered 2D points (151 M edges) 985 -> 800, 2M uniform points
// 299 -> 288, 100,000 points 35 -> 32.  Rounds of one or three windows, lists
// of 256 or 960 further hits, 7 to 12 blocks per SM were equal or slower; four
// consecutive edges per lane with 16-byte stores was 5 to 25% slower (its
// gathers touch four times as many lines per instruction).
constexpr int kDirectWarps = 4;
// Above this many hits per record on average the warp lists a record at a time,
// lane l the hit of bit l: full masks put the lanes' own lists 32 words apart,
// on one bank.  8,000 points that are all neighbors: 2.36 ms, 2.78 with the
// lanes' lists alone; 1M clustered 2D points 793 us with 12 or 16, 818 with 8.
constexpr int kDenseHits = 16;
constexpr int64_t kDirectTargets = 1LL << 27;

template <class T, int D>
struct ExpandSmem {
    static constexpr int kRound = 64;
    static constexpr int kList = kRound + 512;  // an incomplete round, and the hits of the records taken next
    uint32_t edge[kList];
    SPt<T, D> q[32];  // the queries (idx: 1-based, cloud-local)
    long long kb[32];
    T ir[32];
    int32_t base[32];
};

template <class T, int D>
__global__ void __launch_bounds__(kDirectWarps * 32, sizeof(T) == 4 ? 10 : 4) k_expand_direct(
    int64_t nq, const int32_t* __restrict__ qpos_of, const SPt<T, D>* __restrict__ qpts,
    const SPt<T, D>* __restrict__ tpts, const int64_t* __restrict__ offsets, const int2* __restrict__ recs,
    int64_t rec_cap, const uint16_t* __restrict__ rcount, T inv_r, int32_t* __restrict__ senders,
    int32_t* __restrict__ receivers, T* __restrict__ rdisp, T* __restrict__ rdist, Batch bt) {
    pdl_wait();
    pdl_trigger();
    constexpr unsigned full = 0xffffffffu;
    using Smem = ExpandSmem<T, D>;
    constexpr int ROUND = Smem::kRound, U = ROUND / 32;
    __shared__ __align__(16) Smem smem[kDirectWarps];
    Smem& sm = smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t i0 = ((int64_t)blockIdx.x * kDirectWarps + (threadIdx.x >> 5)) * 32;
    if (i0 >= nq) return;  // warp-uniform
    const int64_t i = i0 + lane;
    const bool valid = i < nq;
    const int64_t K0 = offsets[i0];  // the warp's first COO slot
    const int32_t qp = valid ? qpos_of[i] : 0;
    int nr = valid ? rcount[qp] : 0;
    int ne = 0;
    long long k0 = 0;
    const bool over = nr == kOverflowMark;
    if (valid && !over) {
        k0 = offsets[i];
        ne = (int)(offsets[i + 1] - k0);
    } else {
        nr = 0;
    }
    const bool feat = rdisp != nullptr;  // false: neighbor lists (CSR values) only
    const bool pairs = ((uintptr_t)rdisp & (2 * sizeof(T) - 1)) == 0;
    const bool gaps = __any_sync(full, over);  // some query's slots are left out
    const unsigned le = full >> (31 - lane);  // lanes up to this one
    // flat record and edge ranges of the queries
    int rinc = nr, einc = ne;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(full, rinc, o);
        const int b = __shfl_up_sync(full, einc, o);
        if (lane >= o) {
            rinc += a;
            einc += b;
        }
    }
    const int rexc = rinc - nr;
    {
        SPt<T, D> q = qpts[qp];
        T r2 = T(0), ir = inv_r;
        int32_t base = 0;
        cloud_params<T>(bt, qp, r2, ir, base);
        q.idx = q.idx - base + 1;
        sm.q[lane] = q;
        sm.ir[lane] = ir;
        sm.base[lane] = base;
        sm.kb[lane] = k0 - (einc - ne);  // slot of flat edge f of this query: kb + f
    }
    const int R = __shfl_sync(full, rinc, 31), E = __shfl_sync(full, einc, 31);
    // List entry b holds flat edge f0 + b.
    const int head = (int)(K0 & 31);
    int f0 = -head, cnt = head;
    // The round at list index `at`: U windows, all target loads before any store.
    auto write = [&](int at) {
        SPt<T, D> t[U];
        int ql[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int b = at + 32 * u + lane, f = f0 + b;
            ok[u] = b < cnt && f >= 0 && f < E;  // the last always holds when records and counts agree
            const uint32_t e = ok[u] ? sm.edge[b] : 0u;
            ql[u] = (int)(e >> 27);
            if (ok[u]) t[u] = tpts[e & 0x07ffffffu];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!ok[u]) continue;
            const int f = f0 + at + 32 * u + lane;
            const int64_t k = (gaps ? sm.kb[ql[u]] : K0) + f;
            int32_t base = 0;
            T ir = inv_r;
            if (bt.n_clouds) {
                base = sm.base[ql[u]];
                ir = sm.ir[ql[u]];
            }
            senders[k] = t[u].idx - base + 1;
            if (feat) {
                const SPt<T, D> q = sm.q[ql[u]];
                T diff[D], disp[D];
                const T d2 = dist2<T, D>(t[u].x, q.x, diff);
                receivers[k] = q.idx;
                rdist[k] = mul_rn(sqrt_rn(d2), ir);
#pragma unroll
                for (int d = 0; d < D; ++d) disp[d] = mul_rn(-diff[d], ir);
                store_column<T, D>(rdisp, k, disp, pairs);
            }
        }
    };
    for (int rb = 0, take; rb < R; rb += take) {
        // record rho = rb + lane and its query
        // (queries without records set no bit, so the k-th bit belongs to the
        // k-th query lane that reaches into the window)
        const bool qin = nr > 0 && rexc < rb + 32 && rinc > rb;
        const unsigned qm = __ballot_sync(full, qin);
        const unsigned qs = __reduce_or_sync(full, qin ? 1u << max(rexc - rb, 0) : 0u);
        const int rq = kth_set_bit(qm, __popc(qs & le) - 1);  // query lane of this lane's record
        const int32_t rqp = __shfl_sync(full, qp, rq);
        const int rqx = __shfl_sync(full, rexc, rq);
        const int rho = rb + lane;
        int2 rec = make_int2(0, 0);
        if (rho < R) rec = recs[(int64_t)rqp * rec_cap + (rho - rqx)];
        const int c = __popc((unsigned)rec.y);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += a;
        }
        // the records whose hits fit the list (one always does)
        const bool fits = cnt + incl <= Smem::kList;
        take = __popc(__ballot_sync(full, fits));
        // each record's hits listed at their edges' places
        int k = cnt + incl - c;
        const uint32_t first = (uint32_t)rq << 27 | (uint32_t)rec.x;
        const int hits = __shfl_sync(full, incl, take - 1);
        if (hits > kDenseHits * take) {  // by the warp, a record at a time
            for (int j = 0; j < take; ++j) {
                const unsigned m = __shfl_sync(full, (unsigned)rec.y, j);
                const uint32_t f = __shfl_sync(full, first, j);
                const int b = __shfl_sync(full, k, j);
                if (m >> lane & 1u) sm.edge[b + __popc(m & lanemask_lt())] = f + (uint32_t)lane;
            }
        } else {  // by each record's lane
            for (unsigned mb = fits ? (unsigned)rec.y : 0u; mb; mb &= mb - 1, ++k)
                sm.edge[k] = first + (uint32_t)(__ffs(mb) - 1);
        }
        cnt += hits;
        __syncwarp();
        int at = 0;
        for (; cnt - at >= ROUND; at += ROUND) write(at);
        if (at) {
            // the incomplete round moves to the front
            uint32_t e[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int b = at + 32 * u + lane;
                e[u] = b < cnt ? sm.edge[b] : 0u;
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < U; ++u) sm.edge[32 * u + lane] = e[u];
            cnt -= at;
            f0 += at;
            __syncwarp();
        }
    }
    if (cnt) write(0);
}

// Fill pass from the records, in original index order.  Warp v writes the
// edges of queries 32v .. 32v+31, which own one contiguous range [K0, K1) of
// the COO, query after query, each query's edges in record order.  The warp
// takes the records of all its queries as one flat list, 32 per round (one per
// lane, the record's query found by a binary search of the queries' record
// counts), scans their hit counts, and then writes the round's hits with the
// lanes on consecutive hits, two per lane in flight: each lane finds its hit's
// record by a binary search of the scanned counts (shuffles), its point as the
// k-th set bit of the record's mask, and its query's coordinates, index and
// radius by shuffles from the query's lane.
//
// Output goes through a per-warp ring of NCH chunks of CHUNK edges in shared
// memory, one array per COO array, in the COO's own layout; a completed chunk
// is written to global memory by 1-D bulk copies (cp.async.bulk, issued by
// lane 0), so the stores leave the load/store pipe.  Ring slot s holds COO
// edge k with s = (k - base) mod RING, base = K0 rounded down to a multiple of
// 4: a bulk copy starts at an edge index that is a multiple of 4, which makes
// every source and destination address a multiple of 16 bytes (4-byte and
// 8-byte elements, D values per edge for rel_displacement) given 16-byte
// aligned output arrays, and every size a multiple of 16.  The at most three
// edges at each end of the warp's range that do not fill an aligned group of
// four are stored by lanes.  A warp with a query whose records overflowed
// (left to the walking fill), or with unaligned outputs, stores every edge
// from registers instead.
constexpr int kFillWarps = 4;

__device__ __forceinline__ void bulk_store(void* gdst, const void* ssrc, uint32_t bytes) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(ssrc);
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(s), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Orders this thread's shared-memory writes before later bulk-copy reads.
__device__ __forceinline__ void fence_smem_to_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }


// Shared-memory bytes of one warp's ring of `ring` edges.
template <class T, int D, bool FEAT>
__host__ __device__ constexpr size_t fill_ring_bytes(int ring) {
    return FEAT ? (size_t)ring * (8 + (D + 1) * sizeof(T)) : (size_t)ring * 4;
}

template <class T, int D, bool FEAT, int CHUNK, int NCH>
__global__ void __launch_bounds__(kFillWarps * 32) k_expand(
    int64_t nq, const int32_t* __restrict__ qpos_of, const SPt<T, D>* __restrict__ qpts,
    const SPt<T, D>* __restrict__ tpts, const int64_t* __restrict__ offsets, const int2* __restrict__ recs,
    int64_t rec_cap, const uint16_t* __restrict__ rcount, T inv_r, int32_t* __restrict__ senders,
    int32_t* __restrict__ receivers, T* __restrict__ rdisp, T* __restrict__ rdist, Batch bt, int bulk_ok) {
    constexpr int RING = CHUNK * NCH;
    constexpr int U = 2;                                  // hits per lane in flight
    constexpr int SUB = 32 * U;                           // hits written per sub-round
    constexpr int SPAN = (SUB - 1 + CHUNK - 1) / CHUNK;   // chunk boundaries a sub-round may cross
    static_assert(CHUNK % 32 == 0 && (RING & (RING - 1)) == 0 && NCH - 1 - SPAN >= 0, "ring shape");
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(128) unsigned char fill_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i0 = ((int64_t)blockIdx.x * kFillWarps + w) * 32;
    if (i0 >= nq) return;  // warp-uniform
    unsigned char* wsm = fill_smem + (size_t)w * fill_ring_bytes<T, D, FEAT>(RING);
    int32_t* r_snd = reinterpret_cast<int32_t*>(wsm);
    int32_t* r_rcv = r_snd + RING;
    T* r_dist = reinterpret_cast<T*>(r_rcv + RING);
    T* r_disp = r_dist + RING;

    // Lane j: query i0 + j.
    const int64_t i = i0 + lane;
    const bool valid = i < nq;
    const int nval = nq - i0 < 32 ? (int)(nq - i0) : 32;
    const int32_t qp = valid ? qpos_of[i] : 0;
    int nr = valid ? rcount[qp] : 0;
    const bool over = valid && nr == kOverflowMark;
    const long long k0 = valid ? offsets[i] : 0;
    const long long kn = valid ? offsets[i + 1] : 0;
    int ne = (int)(kn - k0);
    if (over) {  // written by the walking fill
        nr = 0;
        ne = 0;
    }
    const SPt<T, D> q = qpts[qp];
    T r2 = T(0), ir = inv_r;
    int32_t base = 0;
    cloud_params<T>(bt, qp, r2, ir, base);
    const int32_t qi = q.idx - base + 1;
    // record and hit prefixes over the queries
    int rincl = nr, eincl = ne;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(FULL, rincl, o);
        const int b = __shfl_up_sync(FULL, eincl, o);
        if (lane >= o) {
            rincl += a;
            eincl += b;
        }
    }
    const int rexcl = rincl - nr;
    const int total_r = __shfl_sync(FULL, rincl, 31);
    // COO index of this query's flat hit 0 (flat hits count only the queries
    // written here): hit F of query j is COO edge kq_j + F
    const long long kq = k0 - (eincl - ne);
    const long long K0 = __shfl_sync(FULL, k0, 0);
    const long long K1 = __shfl_sync(FULL, kn, nval - 1);
    const bool bulk = bulk_ok && !__any_sync(FULL, over) && K1 - K0 >= 32;
    const long long kbase = K0 & ~3LL;  // ring slot 0 <-> COO edge kbase (mod RING)
    long long next_flush = 0;           // next ring chunk to write out (chunk c: [kbase + c*CHUNK, +CHUNK))
    long long cur_chunk = -1;           // highest chunk written so far

    // Writes out the chunks that end at or before `upto` (all that remain of
    // the range when `last`): the aligned part by bulk copies (one group per
    // chunk), the unaligned ends by lanes.
    auto flush = [&](long long upto, bool last) {
        while (true) {
            const long long cs = kbase + next_flush * CHUNK, ce = cs + CHUNK;
            if (cs >= K1 || (ce > upto && !last)) break;
            const long long lo = cs > K0 ? cs : K0, hi = ce < K1 ? ce : K1;
            long long a = (lo + 3) & ~3LL;
            if (a > hi) a = hi;
            const long long b = a + ((hi - a) & ~3LL);
            if (lane == 0) {
                if (b > a) {
                    const int sl = (int)((a - kbase) & (RING - 1));
                    const uint32_t m = (uint32_t)(b - a);
                    bulk_store(senders + a, r_snd + sl, 4u * m);
                    if (FEAT) {
                        bulk_store(receivers + a, r_rcv + sl, 4u * m);
                        bulk_store(rdist + a, r_dist + sl, (uint32_t)sizeof(T) * m);
                        bulk_store(rdisp + (long long)D * a, r_disp + D * sl, (uint32_t)(D * sizeof(T)) * m);
                    }
                }
                bulk_commit();  // one group per chunk, empty or not
            }
            // [lo, a) and [b, hi): at most three edges each
            const long long k = lane < 4 ? lo + lane : b + (lane - 4);
            if ((lane < 4 && k < a) || (lane >= 4 && lane < 8 && k < hi)) {
                const int sl = (int)((k - kbase) & (RING - 1));
                senders[k] = r_snd[sl];
                if (FEAT) {
                    receivers[k] = r_rcv[sl];
                    rdist[k] = r_dist[sl];
#pragma unroll
                    for (int d = 0; d < D; ++d) rdisp[(long long)D * k + d] = r_disp[D * sl + d];
                }
            }
            ++next_flush;
        }
    };

    int fbase = 0;  // flat hits of the earlier record rounds
    for (int r0 = 0; r0 < total_r; r0 += 32) {
        // record r0 + lane and its query: the last query whose first record is <= it
        const int rho = r0 + lane;
        int jr = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
            const int v = __shfl_sync(FULL, rexcl, jr + st);
            if (v <= rho) jr += st;
        }
        const int32_t qpr = __shfl_sync(FULL, qp, jr);
        const int rx0 = __shfl_sync(FULL, rexcl, jr);
        int2 rec = make_int2(0, 0);
        if (rho < total_r) rec = recs[(int64_t)qpr * rec_cap + (rho - rx0)];
        const int p = __popc((unsigned)rec.y);
        int hincl = p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(FULL, hincl, o);
            if (lane >= o) hincl += a;
        }
        const int hexcl = hincl - p;
        const int tot = __shfl_sync(FULL, hincl, 31);
        for (int e0 = 0; e0 < tot; e0 += SUB) {
            const int cnt = min(SUB, tot - e0);
            if (bulk) {
                // the sub-round writes COO edges [K0 + fbase + e0, + cnt): its
                // last chunk reuses the slots of that chunk minus NCH
                const long long c = (K0 + fbase + e0 + cnt - 1 - kbase) / CHUNK;
                if (c > cur_chunk) {
                    if (c >= NCH) {
                        if (lane == 0) bulk_wait_read<NCH - 1 - SPAN>();
                        __syncwarp();
                    }
                    cur_chunk = c;
                }
            }
            SPt<T, D> tp[U];
            int jq[U], tpos[U];
            long long kk[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + 32 * u + lane;
                int r = 0;
#pragma unroll
                for (int st = 16; st > 0; st >>= 1) {
                    const int v = __shfl_sync(FULL, hexcl, r + st);
                    if (v <= e) r += st;
                }
                const unsigned m = (unsigned)__shfl_sync(FULL, rec.y, r);
                const int rx = __shfl_sync(FULL, rec.x, r);
                const int er = __shfl_sync(FULL, hexcl, r);
                jq[u] = __shfl_sync(FULL, jr, r);
                kk[u] = __shfl_sync(FULL, kq, jq[u]) + fbase + e;
                tpos[u] = 0;
                if (e < tot) {
                    tpos[u] = rx + kth_set_bit(m, e - er);
                    tp[u] = tpts[tpos[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + 32 * u + lane;
                T px[D];
#pragma unroll
                for (int d = 0; d < D; ++d) px[d] = __shfl_sync(FULL, q.x[d], jq[u]);
                const T irq = __shfl_sync(FULL, ir, jq[u]);
                const int32_t bq = __shfl_sync(FULL, base, jq[u]);
                const int32_t qiq = __shfl_sync(FULL, qi, jq[u]);
                if (e >= tot) continue;
                const long long k = kk[u];
                const int32_t snd = tp[u].idx - bq + 1;
                T dv[D], dist = T(0);
                if (FEAT) {
                    T diff[D];
                    const T d2 = dist2<T, D>(tp[u].x, px, diff);
                    dist = mul_rn(sqrt_rn(d2), irq);
#pragma unroll
                    for (int d = 0; d < D; ++d) dv[d] = mul_rn(-diff[d], irq);
                }
                if (bulk) {
                    const int sl = (int)((k - kbase) & (RING - 1));
                    r_snd[sl] = snd;
                    if (FEAT) {
                        r_rcv[sl] = qiq;
                        r_dist[sl] = dist;
#pragma unroll
                        for (int d = 0; d < D; ++d) r_disp[D * sl + d] = dv[d];
                    }
                } else {
                    senders[k] = snd;
                    if (FEAT) {
                        receivers[k] = qiq;
                        rdist[k] = dist;
#pragma unroll
                        for (int d = 0; d < D; ++d) rdisp[(long long)D * k + d] = dv[d];
                    }
                }
            }
            if (bulk) {
                fence_smem_to_bulk();
                __syncwarp();
                flush(K0 + fbase + e0 + cnt, false);
            }
        }
        fbase += tot;
    }
    if (bulk) {
        __syncwarp();
        flush(K1, true);
        if (lane == 0) bulk_wait_all();
    }
}

// Per-thread reference-order DFS for a handful of query points (the
// get_neighborlist / for_each_neighbor accessors, src/api.jl:282-292 and
// src/cpu/iterator_cpu.jl:245-263).  No self filter.
template <class T, int D>
__global__ void k_neighbors_of(const T* __restrict__ qcoords, int64_t nsel, const TNode<T, D>* __restrict__ tnode,
                               const SPt<T, D>* __restrict__ tpts, int64_t n_tnodes, T r2,
                               int32_t* __restrict__ out_counts, int32_t* __restrict__ out_idx, int64_t cap) {
    constexpr int SD = stack_depth<D>();
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsel) return;
    T p[D];
#pragma unroll
    for (int d = 0; d < D; ++d) p[d] = qcoords[(int64_t)D * s + d];
    int32_t stack[SD];
    int sp = 0;
    int64_t c = 0;
    if (n_tnodes > 0) stack[sp++] = 0;
    while (sp > 0) {
        const int32_t ent = stack[--sp];
        const int32_t nid = ent & 0x7fffffff;
        const bool asc = ent < 0;
        const TNode<T, D> nd = tnode[nid];
        if (box_gap2<T, D>(p, p, nd.lo, nd.hi) > r2) continue;
        if (nd.b > 0) {
            for (int32_t k = nd.a; k < nd.a + nd.b; ++k) {
                const SPt<T, D> t = tpts[k];
                T diff[D];
                if (dist2<T, D>(t.x, p, diff) <= r2) {
                    if (c < cap) out_idx[s * cap + c] = t.idx + 1;
                    ++c;
                }
            }
        } else {
            const unsigned slots = (unsigned)(-nd.b);
            const bool casc = asc || !(slots & 1u);
            const int nc = __popc(slots);
            int pushed[Dims<D>::nch];
            int np = 0;
            for (int j = 0; j < nc; ++j) {
                const TNode<T, D> ch = tnode[nd.a + j];
                if (box_gap2<T, D>(p, p, ch.lo, ch.hi) <= r2) pushed[np++] = nd.a + j;
            }
            for (int j = 0; j < np; ++j)
                stack[sp++] = casc ? (pushed[np - 1 - j] | (int32_t)0x80000000) : pushed[j];
        }
    }
    out_counts[s] = (int32_t)c;
}

namespace {

// Hit records per query for the next count: 32 to start, then 1.25x the
// largest record count of the last count (at most kMaxRecords), within a
// budget of 4 GiB or 8 bytes per edge of the last count (a third of the
// COO's own size), whichever is larger, and at most 32 GiB.
constexpr int64_t kRecordBudget = 4LL << 30;
constexpr int64_t kRecordBudgetMax = 32LL << 30;

// A caller-set record count (OCT_OPT_RECORD_CAP) replaces the hint, within
// the same budget; records are used when there is room for 8 per query point
// (for a caller-set count, for 1).
int64_t record_cap(const Ctx& ctx, int64_t nq) {
    const int64_t budget = std::min(std::max(kRecordBudget, 8 * ctx.rec_edges_hint), kRecordBudgetMax);
    const int64_t fit = budget / (8 * std::max<int64_t>(nq, 1));
    const int64_t want = ctx.rec_cap_override > 0 ? std::min<int64_t>(ctx.rec_cap_override, kMaxRecords)
                                                  : ctx.rec_cap_hint;
    const int64_t cap = std::min<int64_t>(want, fit);
    return cap >= (ctx.rec_cap_override > 0 ? 1 : 8) ? cap : 0;
}

template <class T, int D>
int count_typed(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, int64_t* n_edges) {
    cudaError_t err;
    cudaStream_t s = ctx.stream;
    const int64_t nq = q.n;
    if ((err = ensure(ctx.counts, (size_t)std::max<int64_t>(nq, 1) * 4)) ||
        (err = ensure(ctx.qpos, (size_t)std::max<int64_t>(nq, 1) * 4)) || (err = ensure(ctx.offsets, (size_t)(nq + 1) * 8)) ||
        (err = ensure(ctx.scan_tmp, (size_t)scan_tmp_elems(nq) * 8)) || (err = ensure(ctx.total, 16)) ||
        (err = ensure(ctx.dstatus, 8)))
        return cuda_status(ctx, err, "allocating edge scratch");
    if ((err = cudaMemsetAsync(ctx.dstatus.p, 0, 4, s)) || (err = cudaMemsetAsync(ctx.total.p, 0, 16, s)))
        return cuda_status(ctx, err, "status reset");
    if (!ctx.total_host) {
        if ((err = cudaMallocHost((void**)&ctx.total_host, 16))) return cuda_status(ctx, err, "pinned total");
    }
    const T r = (T)t.radius;
    const T r2 = r * r;  // src/cpu/edges_cpu.jl:184
    const Tuning tn = ctx.tuning_for(t.ndims, t.dtype, nq, q.nbrs_hint);
    ctx.plan_tuning = tn;
    ctx.rec_cap = 0;
    if (t.n_nodes == 0) {
        if ((err = cudaMemsetAsync(ctx.counts.p, 0, (size_t)nq * 4, s))) return cuda_status(ctx, err, "zero counts");
    } else {
        // Record each query's hits while counting, so that the fill pass
        // need not walk the tree again.
        const int64_t cap = record_cap(ctx, nq);
        if (cap > 0) {
            if ((err = ensure(ctx.recs, (size_t)nq * cap * 8)) || (err = ensure(ctx.rcount, (size_t)nq * 2)) ||
                (err = ensure(ctx.gflag, (size_t)std::max<int64_t>(q.n_groups, 1))))
                return cuda_status(ctx, err, "allocating hit records");
            ctx.rec_cap = cap;
        }
        PhaseTimer pt_(ctx, PH_COUNT);
        const int64_t ng = q.n_groups;
        const auto kern = ctx.rec_cap ? k_edges<T, D, EP_RECORD> : k_edges<T, D, EP_COUNT>;
        launch_pdl(kern, div_up(ng, kEdgeWarps), kEdgeThreads, 0, s, q.dpts.as<SPt<T, D>>(),
            q.chunk.as<BoxNode<T, D>>(), ng, t.search_layout<T, D>(), t.box_units(), t.dpts.as<SPt<T, D>>(), t.n, r2, T(0),
            exclude_self ? 1 : 0, ctx.counts.as<int32_t>(), ctx.qpos.as<int32_t>(), nullptr, nullptr, nullptr, nullptr,
            nullptr, (int*)(ctx.total.as<int64_t>() + 1), ctx.rec_cap ? ctx.recs.as<int2>() : nullptr, ctx.rec_cap,
            ctx.rcount.as<uint16_t>(), ctx.gflag.as<uint8_t>(), t.batch(), nullptr);
        ctx.kernel_launches += 1;
    }
    {
        PhaseTimer pt_(ctx, PH_SCAN);
        ctx.kernel_launches += exclusive_scan_i32_i64(ctx.counts.as<int32_t>(), ctx.offsets.as<int64_t>(), nq,
                                                      ctx.total.as<int64_t>(), ctx.scan_tmp.as<int64_t>(), s);
    }
    if ((err = cudaMemcpyAsync(ctx.total_host, ctx.total.p, 16, cudaMemcpyDeviceToHost, s)) ||
        (err = wait_stream(s)))
        return cuda_status(ctx, err, "edge count");
    *n_edges = ctx.total_host[0];
    q.nbrs_hint = (double)*n_edges / (double)std::max<int64_t>(nq, 1);
    ctx.rec_overflow = 0;
    if (ctx.rec_cap) {
        // Size the next count's records for this one's largest query.
        const int32_t* w = reinterpret_cast<const int32_t*>(ctx.total_host + 1);
        ctx.rec_overflow = w[0];
        const int64_t need = ((int64_t)w[1] * 5 / 4 + 7) / 8 * 8;
        ctx.rec_cap_hint = std::min<int64_t>(std::max<int64_t>(need, 16), kMaxRecords);
        ctx.rec_edges_hint = *n_edges;
    }
    return OK;
}

// Ring of the fill: kFillRing chunks of CHUNK edges (32, 64 or 128: a tuned shape).
constexpr int kFillRing = 4;

template <class T, int D, bool FEAT, int CHUNK>
cudaError_t launch_expand_shape(Ctx& ctx, const Tree& q, const Tree& t, T inv_r, int32_t* senders, int32_t* receivers,
                                void* rel_disp, void* rel_dist, int bulk_ok) {
    constexpr size_t smem = kFillWarps * fill_ring_bytes<T, D, FEAT>(CHUNK * kFillRing);
    auto kern = k_expand<T, D, FEAT, CHUNK, kFillRing>;
    if (smem > 48 * 1024) {
        static bool attr_set = false;  // per instantiation
        if (!attr_set) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            attr_set = true;
        }
    }
    kern<<<div_up(q.n, 32 * kFillWarps), kFillWarps * 32, smem, ctx.stream>>>(
        q.n, ctx.qpos.as<int32_t>(), q.dpts.as<SPt<T, D>>(), t.dpts.as<SPt<T, D>>(), ctx.offsets.as<int64_t>(),
        ctx.recs.as<int2>(), ctx.rec_cap, ctx.rcount.as<uint16_t>(), inv_r, senders, receivers, (T*)rel_disp,
        (T*)rel_dist, t.batch(), bulk_ok);
    return cudaGetLastError();
}

// The fill of the last count's records with the tuned stores: direct
// (k_expand_direct) or bulk copies of 32-, 64- or 128-edge chunks (k_expand).
template <class T, int D, bool FEAT>
cudaError_t launch_expand(Ctx& ctx, const Tree& q, const Tree& t, T inv_r, int32_t* senders, int32_t* receivers,
                          void* rel_disp, void* rel_dist, int bulk_ok) {
    int chunk = ctx.plan_tuning.fill_chunk;
    if (chunk == 0 && t.n > kDirectTargets) chunk = 64;  // positions too wide for the direct fill's list entries
    switch (chunk) {
        case 32:
            return launch_expand_shape<T, D, FEAT, 32>(ctx, q, t, inv_r, senders, receivers, rel_disp, rel_dist,
                                                       bulk_ok);
        case 64:
            return launch_expand_shape<T, D, FEAT, 64>(ctx, q, t, inv_r, senders, receivers, rel_disp, rel_dist,
                                                       bulk_ok);
        case 128:
            return launch_expand_shape<T, D, FEAT, 128>(ctx, q, t, inv_r, senders, receivers, rel_disp, rel_dist,
                                                        bulk_ok);
        default:  // direct stores
            launch_pdl(k_expand_direct<T, D>, div_up(q.n, 32 * kDirectWarps), kDirectWarps * 32, 0, ctx.stream, q.n,
                ctx.qpos.as<int32_t>(), q.dpts.as<SPt<T, D>>(), t.dpts.as<SPt<T, D>>(), ctx.offsets.as<int64_t>(),
                ctx.recs.as<int2>(), ctx.rec_cap, ctx.rcount.as<uint16_t>(), inv_r, senders, receivers, (T*)rel_disp,
                (T*)rel_dist, t.batch());
            return cudaGetLastError();
    }
}

template <class T, int D>
int fill_typed(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, int32_t* senders, int32_t* receivers,
               void* rel_disp, void* rel_dist) {
    const T r = (T)t.radius;
    const T r2 = r * r;
    const T inv_r = T(1) / r;  // inv(r), src/cpu/edges_cpu.jl:185
    cudaStream_t s = ctx.stream;
    PhaseTimer pt_(ctx, PH_FILL);
    const int64_t ng = q.n_groups;
    if (ctx.rec_cap) {
        const bool feat = rel_disp != nullptr;
        auto aligned = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
        const int bulk_ok = aligned(senders) && (!feat || (aligned(receivers) && aligned(rel_disp) && aligned(rel_dist)));
        cudaError_t err = feat ? launch_expand<T, D, true>(ctx, q, t, inv_r, senders, receivers, rel_disp, rel_dist,
                                                           bulk_ok)
                               : launch_expand<T, D, false>(ctx, q, t, inv_r, senders, receivers, rel_disp, rel_dist,
                                                            bulk_ok);
        if (err != cudaSuccess) return cuda_status(ctx, err, "edge fill launch");
        ctx.kernel_launches += 1;
    }
    if (!ctx.rec_cap || ctx.rec_overflow) {
        // Groups without complete records walk the tree again.
        k_edges<T, D, EP_FILL><<<div_up(ng, kEdgeWarps), kEdgeThreads, 0, s>>>(
            q.dpts.as<SPt<T, D>>(), q.chunk.as<BoxNode<T, D>>(), ng, t.search_layout<T, D>(), t.box_units(), t.dpts.as<SPt<T, D>>(),
            t.n, r2, inv_r, exclude_self ? 1 : 0, nullptr, nullptr, ctx.offsets.as<int64_t>(), senders, receivers,
            (T*)rel_disp, (T*)rel_dist, ctx.dstatus.as<int>(), ctx.rec_cap ? ctx.recs.as<int2>() : nullptr,
            ctx.rec_cap, nullptr, ctx.gflag.as<uint8_t>(), t.batch(), nullptr);
        ctx.kernel_launches += 1;
    }
    return cuda_status(ctx, cudaGetLastError(), "edge fill launch");
}

template <class T, int D>
int neighbors_typed(Ctx& ctx, const Tree& t, const void* qcoords, int64_t nsel, int32_t* out_counts,
                    int32_t* out_idx, int64_t cap) {
    const T r = (T)t.radius;
    const T r2 = r * r;
    k_neighbors_of<T, D><<<div_up(nsel, 128), 128, 0, ctx.stream>>>(
        (const T*)qcoords, nsel, t.tnode.as<TNode<T, D>>(), t.spts.as<SPt<T, D>>(), t.n_nodes, r2, out_counts,
        out_idx, cap);
    ctx.kernel_launches += 1;
    return cuda_status(ctx, cudaGetLastError(), "neighbor query launch");
}

template <class T, int D>
cudaError_t count_into_typed(const Tree& q, const Tree& t, bool exclude_self, int32_t* counts, cudaStream_t s) {
    const T r = (T)t.radius;
    const T r2 = r * r;
    k_edges<T, D, EP_COUNT><<<div_up(q.n_groups, kEdgeWarps), kEdgeThreads, 0, s>>>(
        q.dpts.as<SPt<T, D>>(), q.chunk.as<BoxNode<T, D>>(), q.n_groups, t.search_layout<T, D>(), t.box_units(),
        t.dpts.as<SPt<T, D>>(), t.n, r2, T(0), exclude_self ? 1 : 0, counts, nullptr, nullptr, nullptr, nullptr,
        nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr, t.batch(), nullptr);
    return cudaGetLastError();
}

template <class T, int D>
int stats_typed(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, unsigned long long* stats_dev) {
    const T r = (T)t.radius;
    const T r2 = r * r;
    k_edges<T, D, EP_STATS><<<div_up(q.n_groups, kEdgeWarps), kEdgeThreads, 0, ctx.stream>>>(
        q.dpts.as<SPt<T, D>>(), q.chunk.as<BoxNode<T, D>>(), q.n_groups, t.search_layout<T, D>(), t.box_units(),
        t.dpts.as<SPt<T, D>>(), t.n, r2, T(0), exclude_self ? 1 : 0, ctx.counts.as<int32_t>(), nullptr, nullptr,
        nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr, t.batch(), stats_dev);
    ctx.kernel_launches += 1;
    return cuda_status(ctx, cudaGetLastError(), "traversal statistics launch");
}

}  // namespace

// Launches only the per-query count kernel into caller memory; allocates
// nothing (used by the allocation-free count entry point).
cudaError_t count_into(const Tree& q, const Tree& t, bool exclude_self, int32_t* counts, cudaStream_t s) {
    if (q.n == 0) return cudaSuccess;
    if (t.n_nodes == 0) return cudaMemsetAsync(counts, 0, (size_t)q.n * 4, s);
    if (t.dtype == 0)
        return t.ndims == 3 ? count_into_typed<float, 3>(q, t, exclude_self, counts, s)
                            : count_into_typed<float, 2>(q, t, exclude_self, counts, s);
    return t.ndims == 3 ? count_into_typed<double, 3>(q, t, exclude_self, counts, s)
                        : count_into_typed<double, 2>(q, t, exclude_self, counts, s);
}

int traversal_stats(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, uint64_t* out, int n_out) {
    cudaError_t err;
    if ((err = ensure(ctx.counts, (size_t)std::max<int64_t>(q.n, 1) * 4)) || (err = ensure(ctx.tstats, TS_NUM * 8)))
        return cuda_status(ctx, err, "allocating statistics");
    if ((err = cudaMemsetAsync(ctx.tstats.p, 0, TS_NUM * 8, ctx.stream))) return cuda_status(ctx, err, "statistics");
    ctx.plan_query = nullptr;  // the counts buffer is reused: no fill may follow
    if (q.n > 0 && t.n_nodes > 0) {
        unsigned long long* sd = ctx.tstats.as<unsigned long long>();
        const int st = t.dtype == 0 ? (t.ndims == 3 ? stats_typed<float, 3>(ctx, q, t, exclude_self, sd)
                                                    : stats_typed<float, 2>(ctx, q, t, exclude_self, sd))
                                    : (t.ndims == 3 ? stats_typed<double, 3>(ctx, q, t, exclude_self, sd)
                                                    : stats_typed<double, 2>(ctx, q, t, exclude_self, sd));
        if (st != OK) return st;
    }
    uint64_t host[TS_NUM];
    if ((err = cudaMemcpyAsync(host, ctx.tstats.p, TS_NUM * 8, cudaMemcpyDeviceToHost, ctx.stream)) ||
        (err = cudaStreamSynchronize(ctx.stream)))
        return cuda_status(ctx, err, "statistics read");
    for (int k = 0; k < n_out && k < TS_NUM; ++k) out[k] = host[k];
    for (int k = TS_NUM; k < n_out; ++k) out[k] = 0;
    return OK;
}

int edges_count(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, int64_t* n_edges) {
    ctx.plan_query = nullptr;
    int st = OK;
    if (q.n == 0) {
        *n_edges = 0;
    } else if (t.dtype == 0) {
        st = t.ndims == 3 ? count_typed<float, 3>(ctx, q, t, exclude_self, n_edges)
                          : count_typed<float, 2>(ctx, q, t, exclude_self, n_edges);
    } else {
        st = t.ndims == 3 ? count_typed<double, 3>(ctx, q, t, exclude_self, n_edges)
                          : count_typed<double, 2>(ctx, q, t, exclude_self, n_edges);
    }
    if (st != OK) return st;
    ctx.plan_query = &q;
    ctx.plan_target = &t;
    ctx.plan_qgen = q.generation;
    ctx.plan_tgen = t.generation;
    ctx.plan_exclude = exclude_self ? 1 : 0;
    ctx.plan_edges = *n_edges;
    return OK;
}

int edges_fill(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, int32_t* senders, int32_t* receivers,
               void* rel_disp, void* rel_dist, int64_t n_edges) {
    if (ctx.plan_query != &q || ctx.plan_target != &t || ctx.plan_qgen != q.generation ||
        ctx.plan_tgen != t.generation || ctx.plan_exclude != (exclude_self ? 1 : 0))
        return set_error(ctx, ERR_STATE, "oct_edges_fill: no matching oct_edges_count for this pair and build");
    if (n_edges < ctx.plan_edges)
        return set_error(ctx, ERR_CAPACITY, "oct_edges_fill: output capacity is smaller than the edge count");
    if (ctx.plan_edges == 0 || q.n == 0 || t.n_nodes == 0) return OK;
    if (t.dtype == 0)
        return t.ndims == 3 ? fill_typed<float, 3>(ctx, q, t, exclude_self, senders, receivers, rel_disp, rel_dist)
                            : fill_typed<float, 2>(ctx, q, t, exclude_self, senders, receivers, rel_disp, rel_dist);
    return t.ndims == 3 ? fill_typed<double, 3>(ctx, q, t, exclude_self, senders, receivers, rel_disp, rel_dist)
                        : fill_typed<double, 2>(ctx, q, t, exclude_self, senders, receivers, rel_disp, rel_dist);
}

int edges_fill_diff(Ctx& ctx, const Tree& t, int32_t* senders, int32_t* receivers, void* rel_disp, void* rel_dist,
                    int32_t* mirror, int64_t n_edges) {
    if (ctx.plan_query != &t || ctx.plan_target != &t || ctx.plan_qgen != t.generation ||
        ctx.plan_tgen != t.generation || ctx.plan_exclude != 1)
        return set_error(ctx, ERR_STATE, "oct_edges_fill_diff: no matching self-pair oct_edges_count for this build");
    if (t.n_clouds) return set_error(ctx, ERR_ARGUMENT, "oct_edges_fill_diff: not defined for a batched tree");
    if (n_edges < ctx.plan_edges)
        return set_error(ctx, ERR_CAPACITY, "oct_edges_fill_diff: output capacity is smaller than the edge count");
    if (ctx.plan_edges > INT32_MAX)
        return set_error(ctx, ERR_OVERFLOW, "oct_edges_fill_diff: more than 2^31 - 1 edges overflow the Int32 mirrors");
    if (ctx.plan_edges == 0 || t.n == 0 || t.n_nodes == 0) return OK;
    // The COO first, then each edge's mirror by a scan of its sender's
    // segment.
    int st;
    if (t.dtype == 0)
        st = t.ndims == 3 ? fill_typed<float, 3>(ctx, t, t, true, senders, receivers, rel_disp, rel_dist)
                          : fill_typed<float, 2>(ctx, t, t, true, senders, receivers, rel_disp, rel_dist);
    else
        st = t.ndims == 3 ? fill_typed<double, 3>(ctx, t, t, true, senders, receivers, rel_disp, rel_dist)
                          : fill_typed<double, 2>(ctx, t, t, true, senders, receivers, rel_disp, rel_dist);
    if (st != OK) return st;
    return edges_mirror_scan(ctx, senders, receivers, ctx.plan_edges, t.n, ctx.offsets.as<int64_t>(), mirror);
}

namespace {
__global__ void k_offsets_i32(const int64_t* __restrict__ in, int64_t n, int32_t* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (int32_t)in[i];
}
}  // namespace

int csr_fill(Ctx& ctx, const Tree& q, const Tree& t, bool exclude_self, int32_t* offsets, int32_t* flat,
             int64_t capacity) {
    if (ctx.plan_query != &q || ctx.plan_target != &t || ctx.plan_qgen != q.generation ||
        ctx.plan_tgen != t.generation || ctx.plan_exclude != (exclude_self ? 1 : 0))
        return set_error(ctx, ERR_STATE, "oct_csr_fill: no matching oct_edges_count for this pair and build");
    if (ctx.plan_edges > INT32_MAX)
        return set_error(ctx, ERR_OVERFLOW, "oct_csr_fill: more than 2^31 - 1 neighbors overflow the Int32 offsets");
    if (capacity < ctx.plan_edges)
        return set_error(ctx, ERR_CAPACITY, "oct_csr_fill: flat capacity is smaller than the neighbor count");
    if (q.n == 0) return cuda_status(ctx, cudaMemsetAsync(offsets, 0, 4, ctx.stream), "csr offsets");
    k_offsets_i32<<<div_up(q.n + 1, 256), 256, 0, ctx.stream>>>(ctx.offsets.as<int64_t>(), q.n + 1, offsets);
    ctx.kernel_launches += 1;
    if (ctx.plan_edges == 0 || t.n_nodes == 0) return cuda_status(ctx, cudaGetLastError(), "csr offsets");
    if (t.dtype == 0)
        return t.ndims == 3 ? fill_typed<float, 3>(ctx, q, t, exclude_self, flat, nullptr, nullptr, nullptr)
                            : fill_typed<float, 2>(ctx, q, t, exclude_self, flat, nullptr, nullptr, nullptr);
    return t.ndims == 3 ? fill_typed<double, 3>(ctx, q, t, exclude_self, flat, nullptr, nullptr, nullptr)
                        : fill_typed<double, 2>(ctx, q, t, exclude_self, flat, nullptr, nullptr, nullptr);
}

int neighbors_of(Ctx& ctx, const Tree& t, const void* qcoords, int64_t nsel, int32_t* out_counts, int32_t* out_idx,
                 int64_t cap) {
    if (nsel == 0) return OK;
    if (t.n_nodes == 0) {
        return cuda_status(ctx, cudaMemsetAsync(out_counts, 0, (size_t)nsel * 4, ctx.stream), "neighbor query");
    }
    if (t.dtype == 0)
        return t.ndims == 3 ? neighbors_typed<float, 3>(ctx, t, qcoords, nsel, out_counts, out_idx, cap)
                            : neighbors_typed<float, 2>(ctx, t, qcoords, nsel, out_counts, out_idx, cap);
    return t.ndims == 3 ? neighbors_typed<double, 3>(ctx, t, qcoords, nsel, out_counts, out_idx, cap)
                        : neighbors_typed<double, 2>(ctx, t, qcoords, nsel, out_counts, out_idx, cap);
}

}  // namespace oct
