// Shared device/host helpers for the B200 octree neighbor-search library.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace oct {

// ---------------------------------------------------------------- status --
// Mirrors the exception classes the reference raises on this path
// (src/api.jl, src/morton.jl:84, ext/cuda_build.jl:156-163).
enum Status : int {
    OK = 0,
    ERR_ARGUMENT = 1,    // ArgumentError
    ERR_DIMENSION = 2,   // DimensionMismatch
    ERR_INEXACT = 3,     // InexactError from floor(Int32, (p - o) * inv_cs)
    ERR_CUDA = 4,        // a CUDA runtime call failed
    ERR_OVERFLOW = 5,    // internal capacity exceeded (the library retries)
    ERR_CAPACITY = 6,    // caller-supplied buffer too small
    ERR_TIMEOUT = 7,     // a bounded device wait ran out
    ERR_STATE = 8,       // ErrorException: wrong call order / missing build
};

// Device-side status word bits (OctHeader::status).
enum DevFlag : int {
    DF_NONFINITE = 1,    // a coordinate is NaN or +-Inf
    DF_NODE_OVERFLOW = 2,
    DF_RANGE = 4,        // binning out of Int32 range
    DF_TIMEOUT = 8,
    DF_KEY_WIDTH = 16,   // a re-encoded key does not fit the previous build's key width
};

constexpr int kWarp = 32;
constexpr int kLeafSize = 32;  // src/types.jl:177 (target_leaf_size)

template <int D> struct Dims;
template <> struct Dims<3> { static constexpr int bits = 21; static constexpr int nch = 8; };
template <> struct Dims<2> { static constexpr int bits = 31; static constexpr int nch = 4; };

// Worst-case DFS frontier: src/cpu/build_cpu.jl:39-43 (148 in 3D, 94 in 2D).
template <int D> __host__ __device__ constexpr int stack_depth() { return 1 + (Dims<D>::nch - 1) * Dims<D>::bits; }

// Sorted point record: coordinates in Morton order plus the point's original
// 0-based index, packed to a 16-byte multiple for vector loads.
template <class T, int D> struct alignas(16) SPt {
    T x[D];
    int32_t idx;
};

// Packed traversal node.  Internal: a = first child id (0-based, children are
// consecutive in BFS order), b = -(occupied-slot mask).  Leaf: a = first
// sorted position (0-based), b = point count (> 0).
template <class T, int D> struct alignas(16) TNode {
    T lo[D];
    T hi[D];
    int32_t a;
    int32_t b;
};

// Search layout of a built tree: the points in the order in which the
// reference's depth-first search visits them, cut into chunks of at most 32
// (runs of sibling leaves) with their boxes (TNode: a = first position, b =
// count), under a hierarchy of boxes with fan-out 32 over fixed spans of
// positions.  lev[0] holds one node per kSpan positions (a = first chunk
// starting in the span, b = number of such chunks); lev[l] one node per 32 of
// lev[l - 1].
//
// A Float32 box is in coordinates.  A Float64 box is in 32-bit fixed point:
// floor((x - o) s) of its corners, o the set's (or cloud's) origin and s =
// mul / radius with mul = 2^14, or less when the set is wider than 2^15 radii
// (BoxUnits), so that every value stays below 2^29.  The units follow the radius
// and the set's own place, so the boxes reject as much at any offset and scale
// (float boxes of coordinates reject nothing once a float step is a radius
// wide: count and fill of 200,003 points shifted by 3e6, r = 0.03, took 57 ms
// and take 0.25).  A node is half of one in doubles, whose loads and Float64
// latency cost more (8M uniform points in the unit cube: 4.42 ms, 4.9 with
// doubles, 4.26 with floats).
template <class T> struct BoxCoord { using type = T; };
template <> struct BoxCoord<double> { using type = int32_t; };
template <class T, int D> using BoxNode = TNode<typename BoxCoord<T>::type, D>;

struct BoxUnits {
    double o[3];
    double s;
    double width;  // 1 / s (for the search)
    double mul;    // units per radius, a power of two
};
// `mul` for a set `cells` radii wide, 2^-2 to 2^14: cells * mul < 2^29 for
// cells below 2^31 (the host refuses more).
__host__ __device__ inline double box_mul(double cells) {
    union { double d; unsigned long long u; } v;
    v.d = cells;
    const int bits = (int)(v.u >> 52 & 0x7ff) - 1022;  // cells < 2^bits
    const int k = 29 - bits > 14 ? 14 : 29 - bits < -2 ? -2 : 29 - bits;
    v.u = (unsigned long long)(k + 1023) << 52;
    return v.d;
}
constexpr int kSpanShift = 9;
constexpr int kSpan = 1 << kSpanShift;
constexpr int kBvhLevels = 4;
template <class T, int D> struct Bvh {
    BoxNode<T, D>* chunk = nullptr;
    BoxNode<T, D>* lev[kBvhLevels] = {};
    int32_t cnt[kBvhLevels] = {};
    int32_t top = 0;  // highest level built: the first with at most 64 nodes, or the last
};

// Per-tree device header, copied to pinned host memory at the end of a build.
struct OctHeader {
    int32_t status;
    int32_t nan_flag;
    int64_t n_nodes;
    int64_t capacity;
    double gmin[3];
    double gmax[3];
    int32_t n_blocks_done;
    int32_t pad;
    int64_t n_groups;   // chunks of the search layout
    int32_t guard_bad;  // canary bytes found overwritten (guard-check mode)
    int32_t asc_key;    // 2^31 - 1 - the first node whose first child slot is empty (0: none)
    int64_t n_moved;    // refit mode: keys that changed since the previous build
};

// Packed pairs of floats with per-element IEEE round-to-nearest (sm_100+).
// Each operation alone is rounded exactly as the scalar __f*_rn operation.
// Chaining a packed add onto packed products is NOT: measured on B200 with
// CUDA 12.9, add.rn.f32x2(mul.rn.f32x2(..), mul.rn.f32x2(..)) disagreed with
// the separately rounded scalar sum in ~39% of random pairs (also with
// volatile asm and -Xptxas --fmad=false), while packed products summed with
// scalar __fadd_rn agreed in all 2M pairs tested.  Sums therefore stay scalar.
__device__ __forceinline__ unsigned long long sub2_rn(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long mul2_rn(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long add2_rn(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2_rn(unsigned long long a, unsigned long long b,
                                                      unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// min(|a|, |b|, |c|) in one instruction.
__device__ __forceinline__ float min3_abs(float a, float b, float c) {
    float d;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    return ((unsigned long long)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
__device__ __forceinline__ float lo2(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }

// A batch of independent point sets ("clouds") built as one forest.  Cloud c
// occupies positions [coff[c], coff[c+1]) both in input order and in sorted
// order, because the sort key is (c << kbits) | morton.  n_clouds == 0 means
// a single point set (every field unused).
constexpr int kCloudParams = 12;  // origin[3], inv_cs, r2, inv_r, bmin[3], bmax[3]
struct Batch {
    int32_t n_clouds = 0;
    int32_t kbits = 0;
    const int64_t* coff = nullptr;   // [n_clouds + 1]
    const double* cparam = nullptr;  // [n_clouds * kCloudParams], values exact in the element type
    double mul = 1.0;                // BoxUnits::mul of every cloud
};

// Box units of one cloud.
__device__ __forceinline__ BoxUnits cloud_units(const Batch& b, int cloud) {
    const double* cp = b.cparam + (size_t)cloud * kCloudParams;
    BoxUnits u;
    u.o[0] = cp[0];
    u.o[1] = cp[1];
    u.o[2] = cp[2];
    u.s = cp[3] * b.mul;
    u.mul = b.mul;
    return u;
}

// Cloud containing input (== sorted) position i: binary search of coff.
__device__ __forceinline__ int cloud_of_position(const Batch& b, int64_t i) {
    int lo = 0, hi = b.n_clouds - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (b.coff[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// --------------------------------------------------- Julia float semantics --
// Correctly rounded arithmetic without contraction (Julia never fuses).
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float sqrt_rn(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double sqrt_rn(double a) { return __dsqrt_rn(a); }
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }

// Squared distance (x_t - x_q), summed left to right: ((dx*dx + dy*dy) + dz*dz),
// src/cpu/iterator_cpu.jl:96-97.
template <class T, int D>
__device__ __forceinline__ T dist2(const T* t, const T* q, T* diff) {
    T acc;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        diff[d] = sub_rn(t[d], q[d]);
        const T s = mul_rn(diff[d], diff[d]);
        acc = (d == 0) ? s : add_rn(acc, s);
    }
    return acc;
}

// Box-to-box squared gap, conservative for the point test above: for a query
// point inside [qlo,qhi] and a target inside [lo,hi], each per-axis gap is <=
// |x_t - x_q| under monotone rounding, so the sum never exceeds dist2.
template <class T, int D>
__device__ __forceinline__ T box_gap2(const T* qlo, const T* qhi, const T* lo, const T* hi) {
    T acc;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        T g = sub_rn(lo[d], qhi[d]);
        const T g2 = sub_rn(qlo[d], hi[d]);
        g = g > g2 ? g : g2;
        g = g > T(0) ? g : T(0);
        const T s = mul_rn(g, g);
        acc = (d == 0) ? s : add_rn(acc, s);
    }
    return acc;
}

// Minimum / maximum of a warp's values, in every lane (which zero a tie
// keeps is unspecified: for boxes, not for the reference's bounds).
__device__ __forceinline__ float box_min(float v) {
    float m;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}
__device__ __forceinline__ float box_max(float v) {
    float m;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}
__device__ __forceinline__ int32_t box_min(int32_t v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ int32_t box_max(int32_t v) { return __reduce_max_sync(0xffffffffu, v); }
// A coordinate as a box holds it (monotone, so boxes of coordinates map to boxes).
__device__ __forceinline__ float box_coord(float x, int, const BoxUnits&) { return x; }
__device__ __forceinline__ int32_t box_coord(double x, int d, const BoxUnits& u) {
    return __double2int_rd(__dmul_rn(__dsub_rn(x, u.o[d]), u.s));
}

// Morton interleave, src/morton.jl:13-23 and :50-58.
__host__ __device__ __forceinline__ uint64_t split_by_3(uint64_t x) {
    x &= 0x00000000001fffffULL;
    x = (x | (x << 32)) & 0x001f00000000ffffULL;
    x = (x | (x << 16)) & 0x001f0000ff0000ffULL;
    x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
    x = (x | (x << 2)) & 0x1249249249249249ULL;
    return x;
}
__host__ __device__ __forceinline__ uint64_t split_by_2(uint64_t x) {
    x &= 0x000000007fffffffULL;
    x = (x | (x << 16)) & 0x0000ffff0000ffffULL;
    x = (x | (x << 8)) & 0x00ff00ff00ff00ffULL;
    x = (x | (x << 4)) & 0x0f0f0f0f0f0f0f0fULL;
    x = (x | (x << 2)) & 0x3333333333333333ULL;
    x = (x | (x << 1)) & 0x5555555555555555ULL;
    return x;
}

// ------------------------------------------- programmatic dependent launch --
// A kernel launched with launch_pdl may be scheduled while the kernel before
// it in the stream is still running.  Its first statement is pdl_wait(),
// which returns once every earlier grid of the stream has completed and its
// memory is visible, so nothing it reads or writes overlaps the earlier
// kernel; pdl_trigger() then lets the next kernel be scheduled early in turn.
// What overlaps is the launch and block scheduling between the kernels.  In
// a launch without the attribute both are no-ops.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
__host__ inline cudaError_t launch_pdl(void (*kern)(P...), int64_t grid, int block, size_t smem, cudaStream_t s,
                                       A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<A&&>(args)...);
}

// ---------------------------------------------------------- warp helpers --
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <class T> __device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

inline int div_up(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

}  // namespace oct
