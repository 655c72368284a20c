// Device-resident tree build: bounds reduce -> Morton encode -> stable LSD
// radix sort -> sorted point gather -> BFS topology -> bottom-up bounds.
//
// Replaces _build_gpu_tree! (ext/cuda_build.jl:227-288) and reproduces the
// CPU build exactly (src/cpu/bin_cpu.jl, src/sort.jl, src/cpu/build_cpu.jl,
// src/cpu/refit_cpu.jl): the same keys, the same stable order, the same
// leaves and BFS node numbering, and bit-identical bounds.
//
// Topology without per-level launches: a node at level L starts at sorted
// position k iff the level-L key prefix changes at k and the level-(L-1)
// group containing k holds more than 32 points (or k is the root).  A group
// holds more than 32 points iff some window of 33 consecutive positions
// around k shares its prefix, which one pass over the sorted keys detects.
// Each position therefore owns a contiguous range of levels [lo, hi], with
// hi the level of the leaf that contains it.  BFS ids are level-major,
// position-minor, so they come from one exclusive scan of per-block,
// per-level node counts; children of a node are consecutive ids.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include <cuda/atomic>

#include "internal.h"
#include "pointsort.cuh"
#include "scan.cuh"
#include "sort.cuh"

namespace oct {

constexpr int kThreads = 256;

// ------------------------------------------------------------ 1. bounds --
// Order key of an IEEE value: its bits with the magnitude bits flipped when
// the sign is set, so that signed integer order is the value order of every
// non-NaN value, -0.0 below +0.0 (Julia's min/max); the map is its own inverse.
template <class T> struct OrdKey;
template <> struct OrdKey<float> {
    using I = int32_t;
    static constexpr I kMag = 0x7fffffff, kExp = 0x7f800000;
    static constexpr I kMaxKey = 0x7fffffff, kMinKey = (I)0x80000000;
    __device__ static I bits(float x) { return __float_as_int(x); }
    __device__ static I key(I b) { return b ^ ((b >> 31) & kMag); }
    __device__ static float value(I k) { return __int_as_float(key(k)); }
};
template <> struct OrdKey<double> {
    using I = long long;
    static constexpr I kMag = 0x7fffffffffffffffLL, kExp = 0x7ff0000000000000LL;
    static constexpr I kMaxKey = 0x7fffffffffffffffLL, kMinKey = (I)0x8000000000000000ULL;
    __device__ static I bits(double x) { return __double_as_longlong(x); }
    __device__ static I key(I b) { return b ^ ((b >> 63) & kMag); }
    __device__ static double value(I k) { return __longlong_as_double(key(k)); }
};
__device__ __forceinline__ int32_t ord_warp_min(int32_t v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ int32_t ord_warp_max(int32_t v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ long long ord_warp_min(long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ long long ord_warp_max(long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Minima, maxima (Julia order, as order keys) and largest magnitude of a
// block's values, in every lane of its first warp; `sm` holds a warp's per row.
template <class T, int D>
__device__ __forceinline__ void block_bounds(typename OrdKey<T>::I* lo, typename OrdKey<T>::I* hi,
                                             typename OrdKey<T>::I& mag,
                                             typename OrdKey<T>::I (*sm)[2 * D + 1]) {
    using K = OrdKey<T>;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        lo[d] = ord_warp_min(lo[d]);
        hi[d] = ord_warp_max(hi[d]);
    }
    mag = ord_warp_max(mag);
    if (lane == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            sm[w][2 * d] = lo[d];
            sm[w][2 * d + 1] = hi[d];
        }
        sm[w][2 * D] = mag;
    }
    __syncthreads();
    if (w == 0) {
        const bool in = lane < kThreads / 32;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            lo[d] = ord_warp_min(in ? sm[lane][2 * d] : K::kMaxKey);
            hi[d] = ord_warp_max(in ? sm[lane][2 * d + 1] : K::kMinKey);
        }
        mag = ord_warp_max(in ? sm[lane][2 * D] : 0);
    }
}

// Per-axis min/max (Julia min/max order) and a non-finite flag.  The last
// block to finish folds the per-block partials (rows of eight order keys: D
// minima, D maxima, the largest magnitude) into the header.  The fold runs on
// order keys (OrdKey): integer min/max give Julia's min/max of finite values,
// and a magnitude at or above the exponent mask marks a NaN or Inf (whose
// bounds then do not matter: the build fails).  Bound by latency up to a
// million points: the loads, then the two folds, in parallel through redux
// (1000 points 7.5 us, 11.4 with one thread folding the warps' floats; 1M
// lattice points 13, 17; 1M 2D points and 200,003 Float64 points, which read
// one value per load before, 11.4 and 13.3, 17.5 and 19.3).
template <class T, int D>
__global__ void __launch_bounds__(kThreads) k_bounds(const T* __restrict__ coords, int64_t n,
                                                     typename OrdKey<T>::I* __restrict__ partials, OctHeader* hdr) {
    pdl_wait();
    pdl_trigger();
    using K = OrdKey<T>;
    using I = typename K::I;
    __shared__ I sm[kThreads / 32][2 * D + 1];
    __shared__ bool is_last;
    I lo[D], hi[D], mag = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) { lo[d] = K::kMaxKey; hi[d] = K::kMinKey; }
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nthr = (int64_t)gridDim.x * blockDim.x;
    auto take = [&](int d, T x) {
        const I b = K::bits(x);
        const I k = K::key(b);
        lo[d] = min(lo[d], k);
        hi[d] = max(hi[d], k);
        mag = max(mag, b & K::kMag);
    };
    int64_t done = 0;  // points folded by the vector loop
    if (((uintptr_t)coords & 15) == 0) {
        // D words of 16 bytes = E points (their values in order, so an axis
        // each), kGroups of them in flight per thread.
        constexpr int E = 16 / (int)sizeof(T), kGroups = D == 3 ? 2 : 3;
        const uint4* v = reinterpret_cast<const uint4*>(coords);
        const int64_t groups = n / E;
        for (int64_t g = tid; g < groups; g += kGroups * nthr) {
            uint4 q[kGroups][D];
#pragma unroll
            for (int u = 0; u < kGroups; ++u) {
                const int64_t gu = g + u * nthr < groups ? g + u * nthr : g;
#pragma unroll
                for (int c = 0; c < D; ++c) q[u][c] = v[D * gu + c];
            }
#pragma unroll
            for (int u = 0; u < kGroups; ++u) {
                T x[D * E];
                memcpy(x, q[u], sizeof(x));
#pragma unroll
                for (int c = 0; c < D * E; ++c) take(c % D, x[c]);
            }
        }
        done = groups * E;
    }
    for (int64_t i = done + tid; i < n; i += nthr) {
#pragma unroll
        for (int d = 0; d < D; ++d) take(d, coords[D * i + d]);
    }
    block_bounds<T, D>(lo, hi, mag, sm);
    if (threadIdx.x == 0) {
        I* p = partials + (size_t)blockIdx.x * 8;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            p[d] = lo[d];
            p[3 + d] = hi[d];
        }
        p[6] = mag;
        is_last = cuda::atomic_ref<int32_t, cuda::thread_scope_device>(hdr->n_blocks_done)
                      .fetch_add(1, cuda::memory_order_acq_rel) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
#pragma unroll
    for (int d = 0; d < D; ++d) { lo[d] = K::kMaxKey; hi[d] = K::kMinKey; }
    mag = 0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads) {
        const I* p = partials + (size_t)b * 8;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            lo[d] = min(lo[d], __ldcg(p + d));
            hi[d] = max(hi[d], __ldcg(p + 3 + d));
        }
        mag = max(mag, __ldcg(p + 6));
    }
    block_bounds<T, D>(lo, hi, mag, sm);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            hdr->gmin[d] = (double)K::value(lo[d]);
            hdr->gmax[d] = (double)K::value(hi[d]);
        }
        hdr->nan_flag = mag >= K::kExp ? 1 : 0;
        hdr->n_blocks_done = 0;
    }
}

// ------------------------------------------------------------ 2. encode --
// Morton key of one point's cell (src/cpu/bin_cpu.jl:12-31 with
// src/morton.jl:13-60): floor((x - origin) * inv_cs) per axis, clamped to the
// key's bits per axis, bit-interleaved with x in the lowest bit.
template <class T, int D>
__device__ __forceinline__ uint64_t cell_key(const T* __restrict__ x, const T* o, T inv_cs) {
    constexpr int64_t cmax = (1LL << Dims<D>::bits) - 1;
    uint64_t c[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const T v = mul_rn(sub_rn(x[d], o[d]), inv_cs);
        int64_t ci = (int64_t)floor(v);
        ci = ci < 0 ? 0 : (ci > cmax ? cmax : ci);
        c[d] = (uint64_t)ci;
    }
    return (D == 3) ? ((split_by_3(c[2]) << 2) | (split_by_3(c[1]) << 1) | split_by_3(c[0]))
                    : ((split_by_2(c[1]) << 1) | split_by_2(c[0]));
}

// bin_point + clamp + morton_encode (src/cpu/bin_cpu.jl:52-95).  The host has
// already proven every cell index fits Int32 (the max coordinate bins last).
template <class T, int D, class K>
__global__ void __launch_bounds__(kThreads) k_encode(const T* __restrict__ coords, int64_t n, T o0, T o1, T o2,
                                                     T inv_cs, K* __restrict__ keys,
                                                     Batch bt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    T o[3] = {o0, o1, o2};
    int cloud = 0;
    if (bt.n_clouds) {
        // Each cloud has its own origin and cell size (one TNS per cloud).
        cloud = cloud_of_position(bt, i);
        const double* cp = bt.cparam + (size_t)cloud * kCloudParams;
        o[0] = (T)cp[0];
        o[1] = (T)cp[1];
        o[2] = (T)cp[2];
        inv_cs = (T)cp[3];
    }
    const uint64_t key = cell_key<T, D>(coords + D * i, o, inv_cs);
    keys[i] = bt.n_clouds ? (K)(((uint64_t)cloud << bt.kbits) | key) : (K)key;
}

// ------------------------------------------------------------ 4. gather --
// A permutation entry outside [0, n) can only come from a sort whose
// look-back wait ran out (DF_TIMEOUT is then set already): it is skipped, so
// that the coordinate read stays inside its array.
template <class T, int D>
__global__ void __launch_bounds__(kThreads) k_gather(const T* __restrict__ coords, const int32_t* __restrict__ perm,
                                                     int64_t n, SPt<T, D>* __restrict__ spts,
                                                     int* __restrict__ status) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int32_t j = perm ? perm[k] : (int32_t)k;
    if ((uint64_t)(uint32_t)j >= (uint64_t)n) {
        atomicOr(status, (int)DF_TIMEOUT);
        return;
    }
    SPt<T, D> p;
#pragma unroll
    for (int d = 0; d < D; ++d) p.x[d] = coords[(int64_t)D * j + d];
    p.idx = j;
    spts[k] = p;
}

// ---------------------------------------------------------- 5. topology --
// Number of leading D-bit digits (of Dims<D>::bits) two keys share.
template <int D, class K> __device__ __forceinline__ int common_levels(K a, K b) {
    // the highest differing bit, -1 for equal keys
    const int hb = sizeof(K) == 4 ? 31 - __clz((int)(a ^ b)) : 63 - __clzll((long long)(a ^ b));
    return Dims<D>::bits - (int)((unsigned)(hb + D) / (unsigned)D);
}

// Same, where keys of different clouds share no level (-1).
template <int D, class K> __device__ __forceinline__ int common_levels_b(K a, K b, const Batch& bt) {
    if (!bt.n_clouds) return common_levels<D, K>(a, b);
    if ((uint64_t)a >> bt.kbits != (uint64_t)b >> bt.kbits) return -1;
    const uint64_t m = (1ULL << bt.kbits) - 1;
    return common_levels<D, uint64_t>((uint64_t)a & m, (uint64_t)b & m);
}

// Digit (child slot) of a key at level L, from its Morton part.
template <int D, class K> __device__ __forceinline__ int slot_digit(K key, int shd, const Batch& bt) {
    uint64_t v = (uint64_t)key;
    if (bt.n_clouds) v &= (1ULL << bt.kbits) - 1;
    return (int)((v >> shd) & (uint64_t)(Dims<D>::nch - 1));
}

// Each warp of mark / emit takes kStrips consecutive strips of 32 positions
// (both passes and their scan, 16M uniform / 1M lattice points: 342 / 41 us
// with one position per thread and the keys and counters in shared memory,
// 243 / 35 us with 1 strip, 198 / 32 with 2, 191 / 36 with 4).
constexpr int kStrips = 2;
constexpr int kMarkTile = kThreads * kStrips;  // positions per block

// lohi[k] = lo | hi << 8: the levels whose node starts at position k are
// lo..hi (empty when lo > hi); hi is the level of the leaf containing k
// (src/cpu/build_cpu.jl:146: leaf iff count <= 32 or level >= max_levels).
// Also counts the block's nodes per level.
//
// A lane holds the same lane of kStrips + 2 consecutive strips, so the levels
// that positions j and j + 32 share are one comparison of two of its
// registers.  Bound by instructions.
template <int D, class K>
__global__ void __launch_bounds__(kThreads) k_mark(const K* __restrict__ skeys, int64_t n,
                                                   uint16_t* __restrict__ lohi, int32_t* __restrict__ blockcnt,
                                                   int nblocks, uint8_t* __restrict__ dstart,
                                                   int32_t* __restrict__ bvh_arrive, int n_arrive, OctHeader* hdr,
                                                   Batch bt) {
    pdl_wait();
    pdl_trigger();
    constexpr int MAXLEV = Dims<D>::bits;
    constexpr int NLEV = MAXLEV + 1;
    static_assert(NLEV <= 32, "one counter per lane");
    __shared__ int32_t cnt[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < 32) cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kMarkTile + w * (32 * kStrips) + lane;
    // key[i]: position base + 32 (i - 1)
    K key[kStrips + 2];
#pragma unroll
    for (int i = 0; i < kStrips + 2; ++i) {
        const int64_t p = base + 32 * (i - 1);
        key[i] = p >= 0 && p < n ? skeys[p] : K(0);
    }
    // share[i]: levels shared by the positions of key[i] and key[i + 1]
    int share[kStrips + 1];
#pragma unroll
    for (int i = 0; i < kStrips + 1; ++i) {
        const int64_t p = base + 32 * (i - 1);
        share[i] = p >= 0 && p + 32 < n ? common_levels_b<D, K>(key[i], key[i + 1], bt) : -1;
    }
#pragma unroll
    for (int r = 0; r < kStrips; ++r) {
        const int64_t k = base + 32 * r;
        // the maximum over the 33 positions k - 32 .. k: the suffix of the
        // strip before, with the prefix of this one (a shuffle past the end
        // returns the lane's own value)
        int sa = share[r], pb = share[r + 1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            sa = max(sa, __shfl_down_sync(0xffffffffu, sa, o));
            pb = max(pb, __shfl_up_sync(0xffffffffu, pb, o));
        }
        const K up = __shfl_up_sync(0xffffffffu, key[r + 1], 1), last = __shfl_sync(0xffffffffu, key[r], 31);
        if (k < n) {
            const int lo = k == 0 ? 0 : common_levels_b<D, K>(lane ? up : last, key[r + 1], bt) + 1;
            const int hi = min(max(sa, pb) + 1, MAXLEV);
            lohi[k] = (uint16_t)(lo | (hi << 8));
            // the search layout's flags and counters start at zero (sections 6, 7)
            dstart[k] = 0;
            if (k < n_arrive) bvh_arrive[k] = 0;
            if (k == 0) {
                hdr->n_groups = 0;
                hdr->asc_key = 0;
            }
            for (int L = lo; L <= hi; ++L) atomicAdd(&cnt[L], 1);
        }
    }
    __syncthreads();
    if (threadIdx.x < NLEV) blockcnt[(int64_t)threadIdx.x * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

// Node (L, k) -> BFS id.  Writes nrange[id] = {k, L}, first_child[id] = the
// id of the first child (the node (L+1, k)) or -1 for a leaf, and
// node_end[id] = one past the node's last position; k_emit_nodes completes
// each node from these.
template <int D>
__global__ void __launch_bounds__(kThreads) k_emit_ids(int64_t n, const uint16_t* __restrict__ lohi,
                                                       const int64_t* __restrict__ blockoff, int nblocks,
                                                       int64_t capacity, int32_t* __restrict__ first_child,
                                                       int2* __restrict__ nrange, int32_t* __restrict__ node_end,
                                                       OctHeader* hdr, Batch bt) {
    pdl_wait();
    pdl_trigger();
    constexpr int NLEV = Dims<D>::bits + 1;
    constexpr int NW = kThreads / 32;
    // per warp and level: its nodes, then the next id
    __shared__ int32_t next[NW][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kMarkTile + w * (32 * kStrips) + lane;
    next[w][lane] = 0;
    int v[kStrips + 1];  // lo | hi << 8 of this lane's positions, and of the position after the last strip
#pragma unroll
    for (int r = 0; r < kStrips; ++r) v[r] = base + 32 * r < n ? lohi[base + 32 * r] : 1;
    v[kStrips] = lane == 0 && base + 32 * kStrips < n ? lohi[base + 32 * kStrips] : 1;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kStrips; ++r)
        for (int L = v[r] & 0xff; L <= v[r] >> 8; ++L) atomicAdd(&next[w][L], 1);
    __syncthreads();
    if (hdr->n_nodes > capacity) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&hdr->status, (int)DF_NODE_OVERFLOW);
        return;
    }
    if (threadIdx.x < NLEV) {
        int32_t run = (int32_t)blockoff[(int64_t)threadIdx.x * nblocks + blockIdx.x];
#pragma unroll
        for (int j = 0; j < NW; ++j) {
            const int32_t c = next[j][threadIdx.x];
            next[j][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
    // Node ends.  A level-L node ends where the level-L key prefix changes, so
    // the nodes holding position k that end at k + 1 are those of levels
    // lo(k + 1) .. hi(k) (every level at the end of the array).  The level-L
    // node holding k is the last one starting at or before k.
    int nlo[kStrips], from = NLEV, to = -1;
#pragma unroll
    for (int r = 0; r < kStrips; ++r) {
        const int64_t k = base + 32 * r;
        const int nv = __shfl_down_sync(0xffffffffu, v[r], 1), nv0 = __shfl_sync(0xffffffffu, v[r + 1], 0);
        nlo[r] = k >= n ? NLEV : k + 1 == n ? 0 : (lane == 31 ? nv0 : nv) & 0xff;
        const int lo = min(v[r] & 0xff, nlo[r]), hi = v[r] >> 8;
        if (lo <= hi) {
            from = min(from, lo);
            to = max(to, hi);
        }
    }
    from = __reduce_min_sync(0xffffffffu, from);
    to = __reduce_max_sync(0xffffffffu, to);
    // All strips of a level together, levels downward (a node's first child is
    // the next level's node at the same position).
    int32_t prev[kStrips];
#pragma unroll
    for (int r = 0; r < kStrips; ++r) prev[r] = -1;
    for (int L = to; L >= from; --L) {
        unsigned b[kStrips];
#pragma unroll
        for (int r = 0; r < kStrips; ++r)
            b[r] = __ballot_sync(0xffffffffu, (v[r] & 0xff) <= L && L <= v[r] >> 8);
        int32_t first = next[w][L];
#pragma unroll
        for (int r = 0; r < kStrips; ++r) {
            const int64_t k = base + 32 * r;
            const int hi = v[r] >> 8;
            const bool in = b[r] >> lane & 1u;
            const int32_t id = first + __popc(b[r] & lanemask_lt());  // of a node starting here
            if (in) {
                nrange[id] = make_int2((int)k, L);
                first_child[id] = L < hi ? prev[r] : -1;
                prev[r] = id;
            }
            if (nlo[r] <= L && L <= hi) node_end[in ? id : id - 1] = (int32_t)(k + 1);
            first += __popc(b[r]);
        }
    }
}

// What climbing the tree needs of a node, in one 16-byte load: its parent (-1
// for a root; written by the parent's thread), its first child, and its
// numbers of children (bits 0-7) and internal children (8-15), kLinkFull when
// it covers its whole point set.
struct alignas(16) NodeLink {
    int32_t parent, pad, first, meta;
};
constexpr int kLinkFull = 1 << 16;

// Completes node `id`: its last position (from the end k_emit_ids left in
// `arrive`, which is then reset for the refit), its occupied child slots and
// the children's parent links.
template <class T, int D, class K>
__global__ void __launch_bounds__(kThreads) k_emit_nodes(const K* __restrict__ skeys, int64_t n, int64_t capacity,
                                                         const int32_t* __restrict__ first_child_in,
                                                         TNode<T, D>* __restrict__ tnode, int2* __restrict__ nrange,
                                                         NodeLink* __restrict__ link, int32_t* __restrict__ arrive,
                                                         const int64_t* __restrict__ blockoff, int nblocks,
                                                         OctHeader* hdr, Batch bt) {
    pdl_wait();
    pdl_trigger();
    constexpr int BITS = Dims<D>::bits;
    constexpr int NCH = Dims<D>::nch;
    const int64_t nn = hdr->n_nodes;
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (nn > capacity || id >= nn) return;
    const int2 kl = nrange[id];
    const int64_t k = kl.x;
    const int L = kl.y;
    const int32_t first_child = first_child_in[id];
    // The point set holding k: [s0, s1) (a cloud, or everything).
    int cloud = 0;
    int64_t s0 = 0, s1 = n;
    if (bt.n_clouds) {
        cloud = cloud_of_position(bt, k);
        s0 = bt.coff[cloud];
        s1 = bt.coff[cloud + 1];
    }
    const int64_t e = arrive[id];  // the end written by k_emit_ids
    TNode<T, D> nd;
    int inner = 0;  // internal children
    if (first_child < 0) {
        nd.a = (int32_t)k;
        nd.b = (int32_t)(e - k);
    } else {
        // The children are the consecutive level-(L+1) ids from first_child
        // whose ranges start inside [k, e) (nrange[c].x, written by the id
        // pass, is their first position); each one's slot is its key's digit.
        const int shd = D * BITS - D * (L + 1);
        const int64_t lend = L + 2 <= BITS ? blockoff[(int64_t)(L + 2) * nblocks] : nn;  // first id past level L+1
        // (all of them read at once: a loop that stopped at the first child
        // past the range would wait for each in turn)
        int32_t cs[NCH];
#pragma unroll
        for (int j = 0; j < NCH; ++j) cs[j] = first_child + j < lend ? nrange[first_child + j].x : INT32_MAX;
        K ck[NCH];
        int32_t cf[NCH];
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
            ck[j] = cs[j] < e ? skeys[cs[j]] : K(0);
            cf[j] = cs[j] < e ? first_child_in[first_child + j] : -1;
        }
        unsigned slots = 0u;
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
            if (cs[j] < e) {
                slots |= 1u << slot_digit<D, K>(ck[j], shd, bt);
                inner += cf[j] >= 0;
                link[first_child + j].parent = (int32_t)id;
            }
        }
        nd.a = first_child;
        nd.b = -(int32_t)slots;
    }
    if (k == s0 && e == s1) {
        // A node covering its whole point set has that set's bounds.
        if (bt.n_clouds) {
            const double* cp = bt.cparam + (size_t)cloud * kCloudParams;
#pragma unroll
            for (int d = 0; d < D; ++d) { nd.lo[d] = (T)cp[6 + d]; nd.hi[d] = (T)cp[9 + d]; }
        } else {
#pragma unroll
            for (int d = 0; d < D; ++d) { nd.lo[d] = (T)hdr->gmin[d]; nd.hi[d] = (T)hdr->gmax[d]; }
        }
    } else {
#pragma unroll
        for (int d = 0; d < D; ++d) { nd.lo[d] = T(0); nd.hi[d] = T(0); }
    }
    tnode[id] = nd;
    nrange[id] = make_int2((int)k, (int)(e - 1));
    arrive[id] = 0;
    // the first node (in level-major order) whose first slot is empty: no
    // ascending unit lies above it (section 6)
    if (nd.b < 0 && !((unsigned)(-nd.b) & 1u) && 0x7fffffff - (int32_t)id > *(volatile int32_t*)&hdr->asc_key)
        atomicMax(&hdr->asc_key, 0x7fffffff - (int32_t)id);
    link[id].first = first_child;
    link[id].meta = (nd.b < 0 ? __popc((unsigned)(-nd.b)) : 0) | inner << 8 | (k == s0 && e == s1 ? kLinkFull : 0);
    if (L == 0) link[id].parent = -1;  // a root (one per cloud in a batch)
}

// ------------------------------------- 6. leaf bounds and visiting order --
// Visiting order: the reference's search pushes a node's children in slot
// order onto a stack, so it visits them last slot first, except below an
// internal node whose first slot is empty, which it scans as one leaf in
// ascending position order (src/cpu/iterator_cpu.jl:74-116).  The order does
// not depend on the query.  For a point at sorted position k let [s, e) be the
// range of its unit: the highest such node above it, or else its leaf.  The
// units of a point set holding positions [c0, c1) are visited in descending,
// the points inside a unit in ascending position order, so the point's
// visiting position is c0 + (c1 - e) + (k - s).  Each leaf copies its points
// there (dpts), which makes everything a search meets one after another
// contiguous in memory and ascending, and folds their bounds
// (src/cpu/refit_cpu.jl:39-48).
//
// The same pass makes the chunks: a chunk is a run of sibling leaves of at
// most gmax (<= 32, a tuned shape) points in total, or a piece of gmax points
// of a larger leaf.  Siblings share a parent box, so a chunk's points are
// spatially compact; 32 consecutive positions can instead straddle a jump of
// the curve and span the whole domain.  dstart[p] = point count of the chunk
// starting at visiting position p (kPiece set for a piece), else 0; a run's
// box and dstart index go to rbox at the run's first leaf's node, dnode[p].
//
// A warp collects the internal nodes among the ids it scans in a queue and
// reads what it needs of up to 32 of them at once, one per lane: their unit,
// set and children.  Four teams of eight lanes then take a node each: its leaf
// children's points, eight per round and child, four children's loads in
// flight, folded so that each lane ends with the box of one child, from which
// the runs and the node's own box follow by shuffles.  Bounded below by 32n
// bytes read and written; bound by the latency of a node's dependent loads at
// 16 warps per SM (long scoreboard 60% of the stalls, issue 28%; the loads of
// the points to L2 ahead of time gained nothing).  16M uniform points: 222 us,
// where teams that picked their own nodes and took one child after another
// took 279; 1M lattice points 17 (32), 5.2M points in 512 clouds 65 (87), 2M
// uniform points 44 (50), 8000 points 10 (14).  Eight children at once spill
// (Float32: 241 us at 16M); three blocks per SM, which spill too, 259.
constexpr int kTeam = 8;
constexpr int kTeamChildren = 4;  // children folded at once
constexpr int kTeamRounds = 4;    // rounds of eight points; more of a larger leaf follow alone
// points per lane in flight in a larger leaf's rest
template <class T> constexpr int kTeamPtsOf = sizeof(T) == 4 ? 4 : 2;
constexpr int kLayoutBlocks = 2;  // blocks per SM
// A warp takes up to kPickRounds x 32 ids at a time, in clusters of eight ids
// (a 128-byte line of links) when it has several rounds to come: level-major
// ids hold their internal nodes in runs, which smaller clusters spread.
constexpr int kPickRounds = 4;
constexpr int kClusterShift = 3;
// One wave of warps, or more when each still gets kWarpNodes ids: with fewer
// the teams stay half empty (2D points of 1M in a mixture: 44 us, 52 with two
// waves), with more the device waits for the slowest warp (the 512 clouds: 65
// us, 84 in one wave).
constexpr int kLayoutWave = 148 * kLayoutBlocks;
constexpr int kWarpNodes = 64;
constexpr int kPiece = 0x80;
constexpr int kAscending = 1 << 17;  // beside kLinkFull: the node's points are visited in ascending order

// Box of a team's lanes on order keys (integer min/max follow Julia's
// min/max of finite values, -0.0 below +0.0), in every lane.
template <class T, int D, int W = kTeam>
__device__ __forceinline__ void team_fold(typename OrdKey<T>::I* lo, typename OrdKey<T>::I* hi) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) {
            lo[d] = min(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = max(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    }
}

// Boxes of four children, every lane of a team holding its part of each: lane
// `sub` ends with the box of child sub % 4.  After one butterfly step the lanes
// exchange halves of what they still hold, so the four boxes take 7 shuffles
// per value where a butterfly for each would take 12.
template <class T>
__device__ __forceinline__ void fold_children(typename OrdKey<T>::I (&lo)[kTeamChildren],
                                              typename OrdKey<T>::I (&hi)[kTeamChildren]) {
    constexpr unsigned FULL = 0xffffffffu;
    using I = typename OrdKey<T>::I;
    const int sub = threadIdx.x & (kTeam - 1);
#pragma unroll
    for (int c = 0; c < kTeamChildren; ++c) {
        lo[c] = min(lo[c], __shfl_xor_sync(FULL, lo[c], kTeamChildren));
        hi[c] = max(hi[c], __shfl_xor_sync(FULL, hi[c], kTeamChildren));
    }
#pragma unroll
    for (int o = kTeamChildren / 2; o > 0; o >>= 1) {
        const bool up = sub & o;
#pragma unroll
        for (int c = 0; c < o; ++c) {
            const I gl = up ? lo[c] : lo[c + o], gh = up ? hi[c] : hi[c + o];
            const I kl = up ? lo[c + o] : lo[c], kh = up ? hi[c + o] : hi[c];
            lo[c] = min(kl, __shfl_xor_sync(FULL, gl, o));
            hi[c] = max(kh, __shfl_xor_sync(FULL, gh, o));
        }
    }
}

template <class T, int D>
__device__ __forceinline__ void store_bounds(TNode<T, D>* nd, const typename OrdKey<T>::I* lo,
                                             const typename OrdKey<T>::I* hi) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
        nd->lo[d] = OrdKey<T>::value(lo[d]);
        nd->hi[d] = OrdKey<T>::value(hi[d]);
    }
}

// Box units of a single set from this build's bounds, with the host's
// arithmetic (the origin as in k_resort_mark; Tree::box_units).
template <class T, int D>
__device__ __forceinline__ BoxUnits set_units(const OctHeader* hdr, T inv_r) {
    BoxUnits u;
    double cells = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const T o = sub_rn((T)hdr->gmin[d], T(1e-6));
        u.o[d] = (double)o;
        cells = fmax(cells, (double)mul_rn(sub_rn((T)hdr->gmax[d], o), inv_r));
    }
    u.mul = box_mul(cells);
    u.s = (double)inv_r * u.mul;
    return u;
}

template <class T, int D>
__global__ void __launch_bounds__(kThreads, kLayoutBlocks) k_layout(int64_t capacity, int64_t n, TNode<T, D>* __restrict__ tnode,
                                                     const int2* __restrict__ nrange,
                                                     const NodeLink* __restrict__ link,
                                                     const SPt<T, D>* __restrict__ spts, SPt<T, D>* __restrict__ dpts,
                                                     uint8_t* __restrict__ dstart, int32_t* __restrict__ dnode,
                                                     BoxNode<T, D>* __restrict__ rbox, int gmax, T inv_r,
                                                     const OctHeader* hdr,
                                                     Batch bt) {
    pdl_wait();
    pdl_trigger();
    using K = OrdKey<T>;
    using I = typename K::I;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int kTeamPts = kTeamPtsOf<T>;
    constexpr int NCH = Dims<D>::nch;
    constexpr int G = kTeamChildren;
    const int64_t nn = hdr->n_nodes;
    // After a sort whose wait ran out the ranges mean nothing (the build fails).
    if (nn > capacity || (hdr->status & DF_TIMEOUT)) return;
    const int32_t asc_min = 0x7fffffff - hdr->asc_key;  // no node above (before) this id is scanned ascending
    const int lane = threadIdx.x & 31, sub = lane & (kTeam - 1), w = threadIdx.x >> 5;
    const unsigned team = 0xffu << (lane & ~(kTeam - 1));
    const int64_t warps = min((int64_t)gridDim.x * (kThreads / 32), max((int64_t)kLayoutWave * (kThreads / 32), nn / kWarpNodes));
    // Nodes are taken in clusters of 2^csh ids, a warp's clusters `warps` apart.
    const int csh = nn >= warps * (32 * kPickRounds) ? kClusterShift : 0;
    int64_t next = (int64_t)blockIdx.x * (kThreads / 32) + w;
    __shared__ BoxUnits units;
    if constexpr (sizeof(T) == 8) {
        if (threadIdx.x == 0 && !bt.n_clouds) units = set_units<T, D>(hdr, inv_r);
        __syncthreads();
    }
    if (next >= warps) return;  // warp-uniform
    __shared__ int32_t queue[kThreads / 32][32 * (kPickRounds + 1)];
    int head = 0, queued = 0;
    while (true) {
        if (queued < 32 && (next << csh) < nn) {
            __syncwarp();
            const int32_t rest = queue[w][min(head + lane, 32 * kPickRounds + 31)];
            __syncwarp();
            if (lane < queued) queue[w][lane] = rest;
            head = 0;
            do {
                bool work[kPickRounds];  // internal nodes, and roots that are leaves
                int32_t ids[kPickRounds];
#pragma unroll
                for (int r = 0; r < kPickRounds; ++r) {
                    const int64_t id = ((next + ((lane >> csh) + r * (int64_t)(32 >> csh)) * warps) << csh) +
                                       (lane & ((1 << csh) - 1));
                    work[r] = false;
                    ids[r] = (int32_t)id;
                    if (id < nn) {
                        const NodeLink lk = link[id];
                        work[r] = (lk.meta & 0xff) != 0 || lk.parent < 0;
                    }
                }
#pragma unroll
                for (int r = 0; r < kPickRounds; ++r) {
                    const unsigned m = __ballot_sync(FULL, work[r]);
                    if (work[r]) queue[w][queued + __popc(m & ((1u << lane) - 1))] = ids[r];
                    queued += __popc(m);
                }
                next += (int64_t)(kPickRounds * 32 >> csh) * warps;
            } while (queued < 32 && (next << csh) < nn);
            __syncwarp();
        }
        if (queued == 0) break;
        const int take = min(queued, 32);
        // One node per lane: its first child (a leaf root is its own), its
        // children (0: a leaf root), whether its bounds are the set's, its
        // unit's direction and the shift to visiting positions.
        int32_t node = -1, first = 0, meta = 0, to = 0, cloud = 0;
        if (lane < take) {
            node = queue[w][head + lane];
            const NodeLink lk = link[node];
            const int2 range = nrange[node];
            meta = lk.meta & (kLinkFull | 0xff);
            first = meta & 0xff ? lk.first : node;
            // the children on their way to L2
            asm volatile("prefetch.global.L2 [%0];" ::"l"(tnode + first));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(tnode + first + max((meta & 0xff) - 1, 0)));
            int32_t c0 = 0, c1 = (int32_t)n;
            if (bt.n_clouds) {
                cloud = cloud_of_position(bt, range.x);
                c0 = (int32_t)bt.coff[cloud];
                c1 = (int32_t)bt.coff[cloud + 1];
            }
            to = (int32_t)((uint32_t)c0 + (uint32_t)c1);
            if ((lk.meta & 0xff) > (lk.meta >> 8 & 0xff)) {  // (some child is a leaf)
                NodeLink ul = lk;
                for (int32_t u = node; u >= asc_min; u = ul.parent, ul = link[max(u, 0)]) {
                    if (!((unsigned)(-tnode[u].b) & 1u)) {
                        const int2 ur = nrange[u];
                        to = c0 + (c1 - (ur.y + 1)) - ur.x;
                        meta |= kAscending;
                    }
                }
            }
        }
        head += take;
        queued -= take;
        for (int k = 0; k < take; k += 32 / kTeam) {
            // The warp's four teams run in step (every shuffle is warp-wide, a
            // team without a node idles): a team of its own mask would execute
            // alone.
            const int src = k + lane / kTeam;
            const int ms = __shfl_sync(FULL, meta, src & 31);
            const int32_t q = __shfl_sync(FULL, node, src & 31), ch0 = __shfl_sync(FULL, first, src & 31);
            const int32_t shift = __shfl_sync(FULL, to, src & 31);
            const int32_t cl = sizeof(T) == 8 ? __shfl_sync(FULL, cloud, src & 31) : 0;
            const bool internal = src < take && (ms & 0xff) != 0, asc = ms & kAscending;
            const int nc = src >= take ? 0 : internal ? ms & 0xff : 1;
            // the visiting position of the child's point at sorted position a is place(a, b) + its rank
            auto place = [&](int32_t a, int32_t b) {
                return asc ? a + shift : (int32_t)((uint32_t)shift - (uint32_t)a - (uint32_t)b);
            };
            int32_t ca = 0, cb = 0;
            if (sub < nc) {
                ca = tnode[ch0 + sub].a;
                cb = tnode[ch0 + sub].b;
            }
            const unsigned leaf_m = __ballot_sync(FULL, cb > 0), inner_m = __ballot_sync(FULL, sub < nc && cb <= 0);
            if (leaf_m == 0) continue;
            // The children's points, copied and folded: the first kTeamRounds
            // rounds take eight points of each of G children, all loads in
            // flight; lane `sub` gets the box of child `sub`.
            cb = max(cb, 0);  // 0: no leaf here
            const int bw = __reduce_max_sync(FULL, cb);
            I lo[D], hi[D];
#pragma unroll
            for (int h = 0; h < NCH; h += G) {
                int32_t a[G], b[G];
                I gl[D][G], gh[D][G];
#pragma unroll
                for (int c = 0; c < G; ++c) {
                    a[c] = __shfl_sync(FULL, ca, h + c, kTeam);
                    b[c] = __shfl_sync(FULL, cb, h + c, kTeam);
#pragma unroll
                    for (int d = 0; d < D; ++d) { gl[d][c] = K::kMaxKey; gh[d][c] = K::kMinKey; }
                }
                for (int32_t m = sub; m - sub < min(bw, kTeam * kTeamRounds); m += kTeam) {
                    SPt<T, D> p[G];
#pragma unroll
                    for (int c = 0; c < G; ++c)
                        if (m < b[c]) p[c] = spts[a[c] + m];
#pragma unroll
                    for (int c = 0; c < G; ++c) {
                        if (m < b[c]) {
                            dpts[place(a[c], b[c]) + m] = p[c];
#pragma unroll
                            for (int d = 0; d < D; ++d) {
                                const I k = K::key(K::bits(p[c].x[d]));
                                gl[d][c] = min(gl[d][c], k);
                                gh[d][c] = max(gh[d][c], k);
                            }
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    fold_children<T>(gl[d], gh[d]);
                    if (h == 0 || sub >= h) { lo[d] = gl[d][0]; hi[d] = gh[d][0]; }
                }
            }
            if (bw > kTeam * kTeamRounds) {  // the rest of larger leaves, one child after another
                for (int j = 0; j < NCH; ++j) {
                    const int32_t a = __shfl_sync(FULL, ca, j, kTeam), b = __shfl_sync(FULL, cb, j, kTeam);
                    const int32_t at = place(a, b);
                    I rl[D], rh[D];
#pragma unroll
                    for (int d = 0; d < D; ++d) { rl[d] = K::kMaxKey; rh[d] = K::kMinKey; }
                    const int32_t bj = __reduce_max_sync(FULL, b);
                    if (bj <= kTeam * kTeamRounds) continue;
                    for (int32_t m = kTeam * kTeamRounds + sub; m - sub < bj; m += kTeamPts * kTeam) {
                        SPt<T, D> p[kTeamPts];
#pragma unroll
                        for (int t = 0; t < kTeamPts; ++t)
                            if (m + t * kTeam < b) p[t] = spts[a + m + t * kTeam];
#pragma unroll
                        for (int t = 0; t < kTeamPts; ++t) {
                            if (m + t * kTeam < b) {
                                dpts[at + m + t * kTeam] = p[t];
#pragma unroll
                                for (int d = 0; d < D; ++d) {
                                    const I k = K::key(K::bits(p[t].x[d]));
                                    rl[d] = min(rl[d], k);
                                    rh[d] = max(rh[d], k);
                                }
                            }
                        }
                    }
                    __syncwarp();
                    team_fold<T, D>(rl, rh);
                    if (sub == j) {
#pragma unroll
                        for (int d = 0; d < D; ++d) { lo[d] = min(lo[d], rl[d]); hi[d] = max(hi[d], rh[d]); }
                    }
                }
            }
            if (cb > 0) store_bounds<T, D>(tnode + ch0 + sub, lo, hi);
            if (sub >= nc || cb == 0) {
#pragma unroll
                for (int d = 0; d < D; ++d) { lo[d] = K::kMaxKey; hi[d] = K::kMinKey; }
            }
            // Runs: bit j of `start`: child j opens one, of `cut`: child j opens one or is in none.
            unsigned start = 0, cut = 0;
            {
                int count = 0;
#pragma unroll
                for (int j = 0; j < NCH; ++j) {
                    const int32_t b = __shfl_sync(FULL, cb, j, kTeam);
                    const bool in = b > 0 && b <= gmax;
                    const bool opens = in && (count == 0 || count + b > gmax);
                    count = !in ? 0 : opens ? b : count + b;
                    start |= opens ? 1u << j : 0u;
                    cut |= opens || !in ? 1u << j : 0u;
                }
                cut |= ~0u << NCH;
            }
            {
                // the run's last child after `sub`, the run's box at its first child
                const int len = __ffs(cut >> (sub + 1));  // children from here to the run's end
                I rlo[D], rhi[D];
#pragma unroll
                for (int d = 0; d < D; ++d) { rlo[d] = lo[d]; rhi[d] = hi[d]; }
#pragma unroll
                for (int o = 1; o < NCH; o <<= 1) {
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        const I vl = __shfl_down_sync(FULL, rlo[d], o, kTeam), vh = __shfl_down_sync(FULL, rhi[d], o, kTeam);
                        if (o < len) { rlo[d] = min(rlo[d], vl); rhi[d] = max(rhi[d], vh); }
                    }
                }
                const int32_t run_end = __shfl_sync(FULL, ca + cb, (sub + len - 1) & (kTeam - 1), kTeam);
                if (start >> sub & 1u) {
                    // outside an ascending unit the run's last leaf is visited first
                    const int32_t pos = place(ca, run_end - ca);
                    dstart[pos] = (uint8_t)(run_end - ca);
                    dnode[pos] = ch0 + sub;
                    BoxNode<T, D> nd;
                    BoxUnits u;
                    if constexpr (sizeof(T) == 8) u = bt.n_clouds ? cloud_units(bt, cl) : units;
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        nd.lo[d] = box_coord(K::value(rlo[d]), d, u);
                        nd.hi[d] = box_coord(K::value(rhi[d]), d, u);
                    }
                    nd.a = pos;
                    nd.b = run_end - ca;
                    rbox[ch0 + sub] = nd;
                }
            }
            if (cb > gmax) {  // pieces of a larger leaf
                const int32_t at = place(ca, cb);
                for (int32_t c = 0; c < cb; c += gmax) dstart[at + c] = (uint8_t)(kPiece | min(gmax, cb - c));
            }
            __syncwarp();
            team_fold<T, D>(lo, hi);
            // (a node covering its whole set already has that set's bounds)
            if (internal && (inner_m & team) == 0 && sub == 0 && !(ms & kLinkFull))
                store_bounds<T, D>(tnode + q, lo, hi);
            __syncwarp();
        }
    }
}

// --------------------------------------------- 7. node bounds and chunks --
// One launch, two kinds of blocks that do not depend on each other (both need
// only section 6).
//
// Node bounds: a lane climbs from each internal node whose children are all
// leaves; at a parent, the boxes of all its children are folded for the last
// internal child to arrive (src/cpu/refit_cpu.jl:50-60).  No thread waits: a
// lane that is not last stops.  Only internal children count as arrivals, so the acquire-release
// counters (whose acquire drops the SM's L1) are an eighth of the nodes.
//
// Chunks: one warp per span of kSpan visiting positions lists the chunks that
// start in it (contiguous in the chunk array, at a place reserved with one
// atomic; the spans' order there affects no result), one lane per chunk, with
// their boxes from section 6 (a piece's from its points), and folds the
// span's.  The last warp to finish among 32 spans folds their boxes into the
// next level, and so on up.
constexpr int kSpansPerBlock = kThreads / 32;

// A level costs three dependent round trips: the release of the box with the
// counter, the children's boxes, and in their shade the next link.  A warp
// climbs from 32 nodes at once; those that arrive last at their parents are
// folded by teams of one lane per child, as many at a time as the warp holds,
// and every step is taken by the whole warp (teams with masks of their own
// execute one after another).  The whole launch, with such teams of eight and
// now: 16M uniform points 110 and 76 us, 500,009 2D points 25 and 17, 5.2M points
// in 512 clouds 28 and 21, 100,000 points 12 and 12; one lane folding all the
// children took 88, 17, 23 and 13, and 19 us instead of 15 for 200,003 Float64
// points.
template <class T, int D>
__device__ __forceinline__ void fold_nodes(int64_t first, int64_t stride, int64_t nn, TNode<T, D>* tnode,
                                           const NodeLink* __restrict__ link, int32_t* arrive) {
    using K = OrdKey<T>;
    using I = typename K::I;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NCH = Dims<D>::nch;
    const int lane = threadIdx.x & 31, sub = lane & (NCH - 1), team = lane / NCH;
    for (int64_t base = first; base < nn; base += stride) {
        // nodes whose children are all leaves: their boxes are done (section 6)
        int32_t q = -1;
        NodeLink lk;
        if (base + lane < nn) {
            lk = link[base + lane];
            if ((lk.meta & 0xff) != 0 && (lk.meta & (0xff00 | kLinkFull)) == 0) q = lk.parent;
            if (q >= 0) lk = link[q];
        }
        while (true) {
            if (q >= 0 && (lk.meta & kLinkFull)) q = -1;  // (a full node's bounds come from the set's reduce)
            if (!__any_sync(FULL, q >= 0)) break;
            NodeLink next;
            if (q >= 0) {
                if (lk.parent >= 0) next = link[lk.parent];
                if (cuda::atomic_ref<int32_t, cuda::thread_scope_device>(arrive[q]).fetch_add(
                        1, cuda::memory_order_acq_rel) != (lk.meta >> 8 & 0xff) - 1)
                    q = -1;
            }
            __syncwarp();  // a lane's acquire covers its team's reads
            for (unsigned won = __ballot_sync(FULL, q >= 0); won;) {
                int src = -1;
#pragma unroll
                for (int t = 0; t < 32 / NCH; ++t) {
                    if (won && t == team) src = __ffs(won) - 1;
                    won &= won - 1;
                }
                const int32_t node = __shfl_sync(FULL, q, src & 31);
                const int32_t ch0 = __shfl_sync(FULL, lk.first, src & 31);
                const int nc = __shfl_sync(FULL, lk.meta, src & 31) & 0xff;
                const bool in = src >= 0 && sub < nc;
                I lo[D], hi[D];
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    lo[d] = in ? K::key(K::bits(__ldcg(&tnode[ch0 + sub].lo[d]))) : K::kMaxKey;
                    hi[d] = in ? K::key(K::bits(__ldcg(&tnode[ch0 + sub].hi[d]))) : K::kMinKey;
                }
                team_fold<T, D, NCH>(lo, hi);
                if (src >= 0 && sub == 0) store_bounds<T, D>(tnode + node, lo, hi);
            }
            __syncwarp();  // the boxes' stores, before the lanes' next releases
            if (q >= 0) {
                q = lk.parent;
                lk = next;
            }
        }
    }
}

template <class T, int D>
__global__ void __launch_bounds__(kThreads) k_fold_chunks(int span_blocks, int64_t n, int64_t capacity,
                                                          TNode<T, D>* tnode, const NodeLink* __restrict__ link,
                                                          int32_t* arrive, const SPt<T, D>* __restrict__ dpts,
                                                          const uint8_t* __restrict__ dstart,
                                                          const int32_t* __restrict__ dnode,
                                                          const BoxNode<T, D>* __restrict__ rbox, int64_t chunk_cap,
                                                          const __grid_constant__ Bvh<T, D> bv,
                                                          int32_t* __restrict__ bvh_arrive, T inv_r, OctHeader* hdr,
                                                          Batch bt) {
    pdl_wait();
    pdl_trigger();
    __shared__ uint32_t list_sm[kSpansPerBlock][kSpan];  // (offset in the span << 8) | dstart
    const int64_t nn = hdr->n_nodes;
    if (nn > capacity || (hdr->status & DF_TIMEOUT)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((int)blockIdx.x >= span_blocks) {
        fold_nodes<T, D>(((int64_t)(blockIdx.x - span_blocks) * kSpansPerBlock + w) * 32,
                         (int64_t)(gridDim.x - span_blocks) * kThreads, nn, tnode, link, arrive);
        return;
    }
    int32_t node = blockIdx.x * kSpansPerBlock + w;
    if (node >= bv.cnt[0]) return;
    const int64_t s0 = (int64_t)node * kSpan;
    uint32_t* list = list_sm[w];
    // this lane's PL positions: which start chunks
    constexpr int PL = kSpan / 32;
    alignas(PL) uint8_t c[PL];
    const int64_t l0 = s0 + PL * lane;
    if (s0 + kSpan <= n) {
#pragma unroll
        for (int j = 0; j < PL; j += 8) *reinterpret_cast<uint2*>(c + j) = *reinterpret_cast<const uint2*>(dstart + l0 + j);
    } else {
#pragma unroll
        for (int j = 0; j < PL; ++j) c[j] = l0 + j < n ? dstart[l0 + j] : 0;
    }
    int mine = 0;
#pragma unroll
    for (int j = 0; j < PL; ++j) mine += c[j] != 0;
    const int incl = warp_inclusive_scan(mine);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int at = incl - mine;
#pragma unroll
    for (int j = 0; j < PL; ++j)
        if (c[j]) list[at++] = (uint32_t)(((PL * lane + j) << 8) | c[j]);
    int32_t cbase = 0;
    if (lane == 0) cbase = (int32_t)atomicAdd((unsigned long long*)&hdr->n_groups, (unsigned long long)total);
    cbase = __shfl_sync(0xffffffffu, cbase, 0);
    __syncwarp();
    using B = typename BoxCoord<T>::type;
    constexpr B kHigh = sizeof(T) == 8 ? B(1 << 30) : B(INFINITY), kLow = -kHigh;  // beyond every box
    B slo[D], shi[D];
#pragma unroll
    for (int d = 0; d < D; ++d) { slo[d] = kHigh; shi[d] = kLow; }
    for (int k = 0; k < total; k += 32) {
        const uint32_t v = k + lane < total ? list[k + lane] : 0;
        const int32_t first = (int32_t)(s0 + (v >> 8));
        const int cnt = (int)(v & (kPiece - 1));
        BoxNode<T, D> nd;
#pragma unroll
        for (int d = 0; d < D; ++d) { nd.lo[d] = kHigh; nd.hi[d] = kLow; }
        nd.a = first;
        nd.b = cnt;
        if (v && !(v & kPiece)) nd = rbox[dnode[first]];
        unsigned pm = __ballot_sync(0xffffffffu, (v & kPiece) != 0);
        BoxUnits u;
        if constexpr (sizeof(T) == 8) {
            if (pm && !bt.n_clouds) u = set_units<T, D>(hdr, inv_r);
        }
        for (; pm; pm &= pm - 1) {
            const int j = __ffs(pm) - 1;
            const int32_t f = __shfl_sync(0xffffffffu, first, j);
            const int m = __shfl_sync(0xffffffffu, cnt, j);
            SPt<T, D> p;
            if (lane < m) p = dpts[f + lane];
            if constexpr (sizeof(T) == 8) {
                if (bt.n_clouds) u = cloud_units(bt, cloud_of_position(bt, f));
            }
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const B x = lane < m ? box_coord(p.x[d], d, u) : kLow;
                const B lo = box_min(lane < m ? x : kHigh);
                const B hi = box_max(x);
                if (lane == j) { nd.lo[d] = lo; nd.hi[d] = hi; }
            }
        }
        if (v && (int64_t)cbase + k + lane < chunk_cap) bv.chunk[cbase + k + lane] = nd;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            slo[d] = min(slo[d], box_min(nd.lo[d]));
            shi[d] = max(shi[d], box_max(nd.hi[d]));
        }
    }
    auto store_box = [&](BoxNode<T, D>* out, int32_t a, int32_t b) {
        BoxNode<T, D> nd;
#pragma unroll
        for (int d = 0; d < D; ++d) { nd.lo[d] = slo[d]; nd.hi[d] = shi[d]; }
        nd.a = a;
        nd.b = b;
        *out = nd;
    };
    if (lane == 0) store_box(bv.lev[0] + node, cbase, total);
    for (int l = 1; l <= bv.top; ++l) {
        const int32_t up = node >> 5;
        const int need = min(32, bv.cnt[l - 1] - 32 * up);
        int old = 0;
        if (lane == 0)
            old = cuda::atomic_ref<int32_t, cuda::thread_scope_device>(bvh_arrive[up]).fetch_add(
                1, cuda::memory_order_acq_rel);
        old = __shfl_sync(0xffffffffu, old, 0);
        if (old != need - 1) return;
        __syncwarp();
        const BoxNode<T, D>* ch = bv.lev[l - 1] + 32 * up + lane;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            slo[d] = box_min(lane < need ? __ldcg(&ch->lo[d]) : kHigh);
            shi[d] = box_max(lane < need ? __ldcg(&ch->hi[d]) : kLow);
        }
        if (lane == 0) store_box(bv.lev[l] + up, 0, 0);
        bvh_arrive += bv.cnt[l];
        node = up;
    }
}

// --------------------------------------------------- 8. reference views --
template <class T, int D>
__global__ void k_view_nodes(const TNode<T, D>* __restrict__ tnode, const int2* __restrict__ nrange, int64_t nn,
                             int32_t* __restrict__ vf, int32_t* __restrict__ vl, int32_t* __restrict__ vc,
                             T* __restrict__ vmin, T* __restrict__ vmax) {
    constexpr int NCH = Dims<D>::nch;
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nn) return;
    const TNode<T, D> nd = tnode[id];
    const int2 rg = nrange[id];
    vf[id] = rg.x + 1;
    vl[id] = rg.y + 1;
    int j = 0;
    for (int c = 0; c < NCH; ++c) {
        int32_t v = -1;
        if (nd.b < 0 && (((unsigned)(-nd.b) >> c) & 1u)) v = nd.a + (j++) + 1;
        vc[id * NCH + c] = v;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) { vmin[id * D + d] = nd.lo[d]; vmax[id * D + d] = nd.hi[d]; }
}

template <class T, int D>
__global__ void k_view_perm(const SPt<T, D>* __restrict__ spts, int64_t n, int32_t* __restrict__ vp) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) vp[k] = spts[k].idx + 1;
}

// The retained per-point Morton codes of refit mode (src/api.jl:234-238),
// scattered from the sorted keys on demand: morton[perm[k]] = key[k].
template <class T, int D, class K>
__global__ void k_view_morton(const SPt<T, D>* __restrict__ spts, const K* __restrict__ skeys, int64_t n,
                              uint64_t* __restrict__ morton) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) morton[spts[k].idx] = (uint64_t)skeys[k];
}

// --------------------------------------------------------- 9. batches ----
// Per-cloud min/max (Julia order) and non-finite flag: out[c*8 + 0..2] = min,
// [3..5] = max, [6] = non-finite.  One block per cloud, kCloudLoads points per
// thread in flight, folded as order keys.  Bound by the latency of the largest
// cloud's loads (5.2M points in 512 clouds of up to 20,000: 21 us; one point
// per thread of 256 at a time, folded as floats, took 67).
constexpr int kCloudThreads = 512;
constexpr int kCloudLoads = 8;
template <class T, int D>
__global__ void __launch_bounds__(kCloudThreads) k_cloud_bounds(const T* __restrict__ coords,
                                                                const int64_t* __restrict__ coff,
                                                                double* __restrict__ out) {
    using K = OrdKey<T>;
    using I = typename K::I;
    __shared__ I smin[kCloudThreads / 32][D], smax[kCloudThreads / 32][D];
    __shared__ int snan;
    const int c = blockIdx.x;
    const int64_t s0 = coff[c], s1 = coff[c + 1];
    if (threadIdx.x == 0) snan = 0;
    __syncthreads();
    I lo[D], hi[D];
#pragma unroll
    for (int d = 0; d < D; ++d) { lo[d] = K::kMaxKey; hi[d] = K::kMinKey; }
    bool bad = false;
    for (int64_t i0 = s0 + threadIdx.x; i0 < s1; i0 += kCloudLoads * kCloudThreads) {
        T x[kCloudLoads][D];
#pragma unroll
        for (int u = 0; u < kCloudLoads; ++u) {
            const int64_t i = min(i0 + u * kCloudThreads, s1 - 1);  // (the last point again beyond the end)
#pragma unroll
            for (int d = 0; d < D; ++d) x[u][d] = coords[D * i + d];
        }
#pragma unroll
        for (int u = 0; u < kCloudLoads; ++u) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                bad |= !isfinite(x[u][d]);
                const I k = K::key(K::bits(x[u][d]));
                lo[d] = min(lo[d], k);
                hi[d] = max(hi[d], k);
            }
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        lo[d] = ord_warp_min(lo[d]);
        hi[d] = ord_warp_max(hi[d]);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&snan, 1);
    if (lane == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) { smin[w][d] = lo[d]; smax[w][d] = hi[d]; }
    }
    __syncthreads();
    if (threadIdx.x < D) {
        const int d = threadIdx.x;
        I l = smin[0][d], h = smax[0][d];
        for (int v = 1; v < kCloudThreads / 32; ++v) {
            l = min(l, smin[v][d]);
            h = max(h, smax[v][d]);
        }
        double* p = out + (size_t)c * 8;
        p[d] = (double)K::value(l);
        p[3 + d] = (double)K::value(h);
        if (d == 0) p[6] = snan ? 1.0 : 0.0;
    }
}

__global__ void k_gather_edge_offsets(const int64_t* __restrict__ offsets, const int64_t* __restrict__ coff,
                                      int n_clouds, int64_t* __restrict__ eoff) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c <= n_clouds) eoff[c] = offsets[coff[c]];
}

// ---------------------------------------------------- 10. time stepping --
// Refit mode keeps the previous build's sorted keys and permutation.  Points
// move little between steps, so most keys are unchanged: re-encoding every
// point at its previous sorted position leaves the unchanged keys U sorted by
// (key, index) in place.  The changed keys M are few; they are collected,
// sorted by (key, index) in shared-memory chunks and ranked across chunks,
// then merged with U: an unchanged key at position p lands at
// (p - changed keys before p) + (keys of M below it), and the keys of M that
// fall between two consecutive unchanged keys are placed by the first of
// the two.  The merged order is exactly the stable sort of the new keys
// (src/sort.jl:15-24), so the topology and everything after it equal a full
// rebuild.  When no key changed, order and topology are kept and only the
// bounds are recomputed.
constexpr int kChunk = 2048;
constexpr int64_t kMaxMerged = 65536;  // above this many changed keys a full sort is cheaper
inline int64_t merge_cap(int64_t n) { return std::min<int64_t>(kMaxMerged, std::max<int64_t>(kChunk, n / 8)); }
constexpr int64_t kSpeculate = -2;  // run_pipeline: merge with the count of changed keys still on the device
constexpr int kRetry = -1;          // run_pipeline: the speculative merge did not apply

template <class K>
__device__ __forceinline__ bool key_less(K ka, int32_t ia, K kb, int32_t ib) {
    return ka < kb || (ka == kb && ia < ib);
}

// Number of entries of the (key, index)-sorted array (k, v)[0, len) below (key, idx).
template <class K>
__device__ __forceinline__ int64_t count_below(const K* __restrict__ k, const int32_t* __restrict__ v, int64_t len,
                                               K key, int32_t idx) {
    int64_t a = 0, b = len;
    while (a < b) {
        const int64_t mid = (a + b) >> 1;
        if (key_less(k[mid], v[mid], key, idx)) a = mid + 1; else b = mid;
    }
    return a;
}

// Re-encodes point perm[p] at its previous sorted position p, flags a changed
// key, counts the changes per block and appends the changed (key, index)
// pairs to (mk, mv) in any order (slots past `cap` are counted, not
// written).  The origin comes from this build's bounds reduce, with the
// host's arithmetic (src/cpu/bin_cpu.jl:22).
template <class T, int D, class K>
__global__ void __launch_bounds__(kThreads) k_resort_mark(const T* __restrict__ coords, int64_t n,
                                                          const int32_t* __restrict__ perm,
                                                          const K* __restrict__ keys, T inv_cs, OctHeader* hdr,
                                                          uint8_t* __restrict__ changed, int32_t* __restrict__ blockcnt,
                                                          K* __restrict__ mk, int32_t* __restrict__ mv, int64_t cap) {
    pdl_wait();
    pdl_trigger();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool c = false;
    K nk = 0;
    int32_t i = 0;
    if (p < n) {
        T o[3] = {T(0), T(0), T(0)};
#pragma unroll
        for (int d = 0; d < D; ++d) o[d] = sub_rn((T)hdr->gmin[d], T(1e-6));
        i = perm[p];
        const uint64_t key = cell_key<T, D>(coords + (int64_t)D * i, o, inv_cs);
        nk = (K)key;
        if ((uint64_t)nk != key) atomicOr(&hdr->status, (int)DF_KEY_WIDTH);
        c = nk != keys[p];
        changed[p] = (uint8_t)c;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, c);
    if (bal) {
        const int lane = threadIdx.x & 31;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd((unsigned long long*)&hdr->n_moved, (unsigned long long)__popc(bal));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (c) {
            const int64_t slot = (int64_t)base + __popc(bal & lanemask_lt());
            if (slot < cap) {
                mk[slot] = nk;
                mv[slot] = i;
            }
        }
    }
    const int cnt = __syncthreads_count(c);
    if (threadIdx.x == 0) blockcnt[blockIdx.x] = cnt;
}

// Sorts each chunk of up to kChunk changed keys by (key, index) in shared
// memory: a bitonic network of `width` entries (a power of two, the chunk
// size rounded up), width / 2 compare-exchanges per stage shared by the
// block's threads.  The count m is read on the device (*m_ptr); nothing is sorted
// when m exceeds cap.
template <class K>
__global__ void __launch_bounds__(kChunk / 2) k_moved_sort(const int64_t* __restrict__ m_ptr, int64_t cap,
                                                           K* __restrict__ mk, int32_t* __restrict__ mv) {
    pdl_wait();
    pdl_trigger();
    __shared__ K sk[kChunk];
    __shared__ int32_t sv[kChunk];
    const int64_t m = *m_ptr;
    if (m > cap || (int64_t)blockIdx.x * kChunk >= m) return;  // block-uniform
    int width = 64;
    while (width < m && width < kChunk) width <<= 1;
    const int64_t base = (int64_t)blockIdx.x * kChunk;
    for (int t = threadIdx.x; t < width; t += blockDim.x) {
        const int64_t j = base + t;
        if (j < m) {
            sk[t] = mk[j];
            sv[t] = mv[j];
        } else {
            sk[t] = ~K(0);
            sv[t] = INT32_MAX;  // above every real index: padding sorts last
        }
    }
    __syncthreads();
    for (int size = 2; size <= width; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < width / 2; t += blockDim.x) {
                const int i = 2 * t - (t & (stride - 1));
                const int j = i + stride;
                const bool up = (i & size) == 0;
                const K ki = sk[i], kj = sk[j];
                const int32_t vi = sv[i], vj = sv[j];
                if (key_less(kj, vj, ki, vi) == up) {
                    sk[i] = kj;
                    sk[j] = ki;
                    sv[i] = vj;
                    sv[j] = vi;
                }
            }
            __syncthreads();
        }
    }
    for (int t2 = threadIdx.x; t2 < width; t2 += blockDim.x) {
        const int64_t j = base + t2;
        if (j < m) {
            mk[j] = sk[t2];
            mv[j] = sv[t2];
        }
    }
}

// Global rank of each changed key: its rank in its own chunk plus the number
// of smaller keys in every other chunk.
template <class K>
__global__ void __launch_bounds__(kThreads) k_moved_rank(const int64_t* __restrict__ m_ptr, int64_t cap,
                                                         const K* __restrict__ ck, const int32_t* __restrict__ cv,
                                                         K* __restrict__ sk, int32_t* __restrict__ sv) {
    pdl_wait();
    pdl_trigger();
    const int64_t m = *m_ptr;
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m > cap || m <= kChunk || j >= m) return;  // one chunk is already in order
    const K key = ck[j];
    const int32_t idx = cv[j];
    const int64_t own = j / kChunk;
    int64_t r = j - own * kChunk;
    const int64_t nchunks = (m + kChunk - 1) / kChunk;
    for (int64_t c = 0; c < nchunks; ++c) {
        if (c == own) continue;
        const int64_t b = c * kChunk;
        r += count_below(ck + b, cv + b, m - b < kChunk ? m - b : (int64_t)kChunk, key, idx);
    }
    sk[r] = key;
    sv[r] = idx;
}

template <class T, int D, class K>
__device__ __forceinline__ void put_sorted(int64_t pos, K key, int32_t idx, const T* __restrict__ coords,
                                           K* __restrict__ okeys, int32_t* __restrict__ operm,
                                           SPt<T, D>* __restrict__ spts) {
    okeys[pos] = key;
    operm[pos] = idx;
    SPt<T, D> sp;
#pragma unroll
    for (int d = 0; d < D; ++d) sp.x[d] = coords[(int64_t)D * idx + d];
    sp.idx = idx;
    spts[pos] = sp;
}

// Merges the unchanged keys (in place at their previous positions) with the
// sorted changed keys (mk, mv)[0, m) into (okeys, operm), and gathers the
// sorted points (the gather of section 4).  changed_before[b] counts the
// changed positions before block b.
template <class T, int D, class K>
__global__ void __launch_bounds__(kThreads) k_resort_merge(int64_t n, const int64_t* __restrict__ m_ptr, int64_t cap,
                                                           const K* __restrict__ keys,
                                                           const int32_t* __restrict__ perm,
                                                           const uint8_t* __restrict__ changed,
                                                           const int64_t* __restrict__ changed_before,
                                                           const K* __restrict__ mk1, const int32_t* __restrict__ mv1,
                                                           const K* __restrict__ mk2, const int32_t* __restrict__ mv2,
                                                           const T* __restrict__ coords, K* __restrict__ okeys,
                                                           int32_t* __restrict__ operm, SPt<T, D>* __restrict__ spts) {
    pdl_wait();
    pdl_trigger();
    __shared__ int wsum[kThreads / 32];
    __shared__ int64_t sbound[2];
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t m = *m_ptr;
    if (m > cap) {
        // Too many changed keys for a merge (the caller sorts afresh): keep
        // the previous order, so that what follows reads a valid permutation.
        if (p < n) put_sorted<T, D, K>(p, keys[p], perm[p], coords, okeys, operm, spts);
        return;
    }
    // Sorted changed keys: ranked across chunks when there are several.
    const K* __restrict__ mk = m > kChunk ? mk2 : mk1;
    const int32_t* __restrict__ mv = m > kChunk ? mv2 : mv1;
    if (m == n) {  // every key changed: the sorted changed keys are the result
        if (p < n) put_sorted<T, D, K>(p, mk[p], mv[p], coords, okeys, operm, spts);
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // The previous (key, index) order is sorted, so the changed keys below any
    // entry of this block lie between those below its first entry and those
    // below the next block's first: two full searches per block, then each
    // thread searches only that span (usually a few entries).
    const int64_t b0 = (int64_t)blockIdx.x * blockDim.x;
    if (threadIdx.x < 2) {
        const int64_t q = b0 + (threadIdx.x ? (int64_t)blockDim.x : 0);
        sbound[threadIdx.x] = q < n ? count_below(mk, mv, m, keys[q], perm[q]) : m;
    }
    const bool in = p < n;
    const bool c = in && changed[p];
    const bool u = in && !c;
    const unsigned cbal = __ballot_sync(0xffffffffu, c);
    const unsigned ubal = __ballot_sync(0xffffffffu, u);
    if (lane == 0) wsum[w] = __popc(cbal);
    __syncthreads();
    const int64_t blo = sbound[0], bhi = sbound[1];
    int before = __popc(cbal & lanemask_lt());
    for (int j = 0; j < w; ++j) before += wsum[j];
    K key = 0;
    int32_t idx = 0;
    int64_t s = 0;
    if (u) {
        key = keys[p];
        idx = perm[p];
        s = blo + count_below(mk + blo, mv + blo, bhi - blo, key, idx);
    }
    // Changed keys below the next unchanged key: from the next unchanged lane
    // of this warp, or found past the warp's end.
    const unsigned later = ubal & ~((2u << lane) - 1u);
    const int src = later ? __ffs(later) - 1 : lane;
    int64_t sn = __shfl_sync(0xffffffffu, s, src);
    if (!u) return;
    if (!later) {
        int64_t q = p - lane + 32;
        while (q < n && changed[q]) ++q;
        if (q >= n)
            sn = m;
        else if (q < b0 + (int64_t)blockDim.x)
            sn = blo + count_below(mk + blo, mv + blo, bhi - blo, keys[q], perm[q]);
        else if (q == b0 + (int64_t)blockDim.x)
            sn = bhi;
        else
            sn = count_below(mk, mv, m, keys[q], perm[q]);
    }
    const int64_t ui = p - (changed_before[blockIdx.x] + before);  // rank among unchanged keys
    put_sorted<T, D, K>(ui + s, key, idx, coords, okeys, operm, spts);
    for (int64_t j = s; j < sn; ++j) put_sorted<T, D, K>(j + ui + 1, mk[j], mv[j], coords, okeys, operm, spts);
    if (ui == 0)
        for (int64_t j = 0; j < s; ++j) put_sorted<T, D, K>(j, mk[j], mv[j], coords, okeys, operm, spts);
}

// Bounds-only step (no key changed): the topology is kept; reset the
// counters of sections 6 and 7 (chunk starts stay where they are) and preset
// the full-range nodes from this build's reduce.
template <class T, int D>
__global__ void __launch_bounds__(kThreads) k_refit_prepare(int64_t nn, int64_t n, TNode<T, D>* __restrict__ tnode,
                                                            const int2* __restrict__ nrange,
                                                            int32_t* __restrict__ arrive,
                                                            int32_t* __restrict__ bvh_arrive, int n_arrive,
                                                            int32_t asc_key, OctHeader* hdr) {
    pdl_wait();
    pdl_trigger();
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id == 0) {
        hdr->n_nodes = nn;
        hdr->n_groups = 0;
        hdr->asc_key = asc_key;
    }
    for (int64_t k = id; k < n_arrive; k += (int64_t)gridDim.x * blockDim.x) bvh_arrive[k] = 0;
    if (id >= nn) return;
    arrive[id] = 0;
    const int2 rg = nrange[id];
    if (rg.x == 0 && (int64_t)rg.y == n - 1) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            tnode[id].lo[d] = (T)hdr->gmin[d];
            tnode[id].hi[d] = (T)hdr->gmax[d];
        }
    }
}

// ----------------------------------------------------------- 11. guards --
// Guard-check mode (OCT_OPT_GUARD_CHECK): a canary region follows the part of
// each sort buffer and node array that the build may write; after each
// topology attempt every canary byte is compared and the mismatches are
// counted into hdr->guard_bad.
constexpr size_t kGuardBytes = 16384;
constexpr unsigned char kGuardByte = 0xA5;

__global__ void k_guard_check(const unsigned char* __restrict__ p, int64_t len, int* __restrict__ bad) {
    int c = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (int64_t)gridDim.x * blockDim.x)
        c += p[i] != kGuardByte;
    c = warp_sum(c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(bad, c);
}

// ------------------------------------------------------------- host side --
namespace {

// In guard-check mode, `b` holds `bytes` plus a canary region after them.
cudaError_t ensure_g(const Ctx& ctx, DevBuf& b, size_t bytes) {
    return ensure(b, bytes + (ctx.guard_check ? kGuardBytes : 0));
}
cudaError_t guard_fill(const Ctx& ctx, const DevBuf& b, size_t bytes) {
    if (!ctx.guard_check) return cudaSuccess;
    return cudaMemsetAsync(static_cast<unsigned char*>(b.p) + bytes, kGuardByte, kGuardBytes, ctx.stream);
}
void guard_check(Ctx& ctx, const DevBuf& b, size_t bytes, OctHeader* hdr) {
    if (!ctx.guard_check) return;
    k_guard_check<<<8, 256, 0, ctx.stream>>>(static_cast<const unsigned char*>(b.p) + bytes, (int64_t)kGuardBytes,
                                            &hdr->guard_bad);
    ctx.kernel_launches += 1;
}

// Bounds, visiting order, chunks and box hierarchy (sections 6 and 7) of the
// tree whose topology was just launched; `nodes` bounds its node count.
template <class T, int D>
void launch_layout(Ctx& ctx, Tree& t, const void* skeys, int64_t n, int64_t node_cap, int64_t chunk_cap, int64_t nodes,
                   int gmax, T inv_r) {
    OctHeader* hdr = t.hdr.as<OctHeader>();
    // Each run's first leaf, by visiting position, in the key buffer that does
    // not hold the sorted keys (4 or 8 bytes per point).
    int32_t* dnode = t.keys[skeys == t.keys[0].p ? 1 : 0].as<int32_t>();
    {
        PhaseTimer pt_(ctx, PH_REFIT);
        // a grid that fills the device; warps take further nodes in turn
        const int64_t blocks = std::min<int64_t>(div_up(nodes, kThreads), 2 * kLayoutWave);
        launch_pdl(k_layout<T, D>, blocks, kThreads, 0, ctx.stream, node_cap, n, t.tnode.as<TNode<T, D>>(),
            t.nrange.as<int2>(), t.link.as<NodeLink>(), t.spts.as<SPt<T, D>>(), t.dpts.as<SPt<T, D>>(),
            t.dstart.as<uint8_t>(), dnode, t.rbox.as<BoxNode<T, D>>(), gmax, inv_r, hdr, t.batch());
    }
    PhaseTimer pt_(ctx, PH_GROUPS);
    const int span_blocks = div_up(n, kSpan * kSpansPerBlock);
    const int64_t fold_blocks = std::min<int64_t>(div_up(nodes, kThreads), 148 * 16);
    launch_pdl(k_fold_chunks<T, D>, span_blocks + fold_blocks, kThreads, 0, ctx.stream, span_blocks, n, node_cap,
        t.tnode.as<TNode<T, D>>(), t.link.as<NodeLink>(), t.arrive.as<int32_t>(), t.dpts.as<SPt<T, D>>(),
        t.dstart.as<uint8_t>(), dnode, t.rbox.as<BoxNode<T, D>>(), chunk_cap,
        t.search_layout<T, D>(), t.bvh_arrive.as<int32_t>(), inv_r, hdr, t.batch());
    ctx.kernel_launches += 2;
}

template <class T, int D, class K>
int run_pipeline(Ctx& ctx, Tree& t, const T* coords, int64_t n, T radius, int64_t moved = -1, int prev = -1) {
    const Batch bt = t.batch();
    cudaStream_t s = ctx.stream;
    cudaError_t err;
    constexpr int BITS = Dims<D>::bits;
    constexpr int NLEV = BITS + 1;
    const T inv_cs = T(1) / radius;  // src/cpu/bin_cpu.jl:60
    T o[3] = {T(0), T(0), T(0)};
    for (int d = 0; d < D; ++d) o[d] = (T)t.origin[d];

    if ((err = ensure(t.spts, (size_t)n * sizeof(SPt<T, D>)))) return cuda_status(ctx, err, "allocating points");
    t.iperm_valid = false;
    int32_t lev[kBvhLevels];
    int64_t bvh_nodes = 0;
    t.bvh_levels(n, lev, &bvh_nodes);
    const int n_arrive = (int)(bvh_nodes - lev[0]);
    if ((err = ensure_g(ctx, t.dpts, (size_t)n * sizeof(SPt<T, D>))) || (err = ensure(t.dstart, (size_t)n)) ||
        (err = ensure(t.bvh, (size_t)bvh_nodes * sizeof(BoxNode<T, D>))) ||
        (err = ensure(t.bvh_arrive, (size_t)n_arrive * 4)))
        return cuda_status(ctx, err, "allocating the search layout");
    OctHeader* hdr = t.hdr.as<OctHeader>();
    const K* skeys;
    const int32_t* perm;
    int sorted = -1;  // buffer holding this build's sorted keys and permutation
    if (moved == -1) {  // a full sort
        // Keys and points sorted together (stable: ties keep ascending
        // original index, src/sort.jl:15-24), the encode fused into the sort.
        const int passes = t.sort_passes;
        if ((err = ensure_g(ctx, t.keys[0], (size_t)n * sizeof(K))) ||
            (err = ensure_g(ctx, t.keys[1], (size_t)n * sizeof(K))) || (err = ensure_g(ctx, t.vals[0], (size_t)n * 4)) ||
            (err = ensure_g(ctx, t.spts, (size_t)n * sizeof(SPt<T, D>))) ||
            (t.keep_morton && (err = ensure(t.vals[1], (size_t)n * 4))))  // the next step's merge writes here
            return cuda_status(ctx, err, "allocating sort buffers");
        for (int b = 0; b < 2; ++b)
            if ((err = guard_fill(ctx, t.keys[b], (size_t)n * sizeof(K)))) return cuda_status(ctx, err, "sort guards");
        if ((err = guard_fill(ctx, t.vals[0], (size_t)n * 4)) ||
            (err = guard_fill(ctx, t.spts, (size_t)n * sizeof(SPt<T, D>))) ||
            (err = guard_fill(ctx, t.dpts, (size_t)n * sizeof(SPt<T, D>))))
            return cuda_status(ctx, err, "sort guards");
        if (passes == 0) {
            // Every point in one cell: keys all equal, the input order stands.
            PhaseTimer pt_(ctx, PH_SORT);
            k_encode<T, D, K><<<div_up(n, kThreads), kThreads, 0, s>>>(coords, n, o[0], o[1], o[2], inv_cs,
                                                                        t.keys[0].as<K>(), bt);
            k_gather<T, D><<<div_up(n, kThreads), kThreads, 0, s>>>(coords, nullptr, n, t.spts.as<SPt<T, D>>(),
                                                                    &hdr->status);
            ctx.kernel_launches += 2;
            perm = nullptr;
        } else {
            if ((err = ensure(t.look, onesweep_words(n, passes) * 4)))
                return cuda_status(ctx, err, "allocating sort scratch");
            int sms = 0;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device);
            EncodeParams<T> ep;
            ep.o[0] = o[0];
            ep.o[1] = o[1];
            ep.o[2] = o[2];
            ep.inv_cs = inv_cs;
            ep.bt = bt;
            PhaseTimer pt_(ctx, PH_SORT);
            err = point_sort<T, D, K>(coords, ep, n, passes, t.keys[0].as<K>(), t.keys[1].as<K>(),
                                      t.spts.as<SPt<T, D>>(), t.dpts.as<SPt<T, D>>(), t.vals[0].as<int32_t>(),
                                      t.look.as<uint32_t>(), &hdr->status, sms, ctx.wait_limit,
                                      ctx.withhold_tile, s, &ctx.kernel_launches);
            if (err) return cuda_status(ctx, err, "key sort launch");
            perm = t.vals[0].as<int32_t>();
            if (!bt.n_clouds) sorted = 0;
        }
        skeys = t.keys[0].as<K>();
        t.last_path = 0;
    } else {
        // Refit mode, keys already re-encoded in the previous order (section 10).
        K* kp = t.keys[prev].as<K>();
        int32_t* vp = t.vals[prev].as<int32_t>();
        skeys = kp;
        perm = vp;
        sorted = prev;
        if (moved == 0) {
            // Same keys, same order, same topology: new bounds only.
            {
                PhaseTimer pt_(ctx, PH_GATHER);
                k_gather<T, D><<<div_up(n, kThreads), kThreads, 0, s>>>(coords, vp, n, t.spts.as<SPt<T, D>>(),
                                                                    &hdr->status);
                ctx.kernel_launches += 1;
            }
            {
                PhaseTimer pt_(ctx, PH_REFIT);
                launch_pdl(k_refit_prepare<T, D>, div_up(t.n_nodes, kThreads), kThreads, 0, s, t.n_nodes, n,
                    t.tnode.as<TNode<T, D>>(), t.nrange.as<int2>(), t.arrive.as<int32_t>(),
                    t.bvh_arrive.as<int32_t>(), n_arrive, t.asc_key, hdr);
                ctx.kernel_launches += 1;
            }
            launch_layout<T, D>(ctx, t, skeys, n, t.capacity, t.chunk_cap, t.n_nodes, t.group_cap, inv_cs);
            if ((err = cudaGetLastError())) return cuda_status(ctx, err, "bounds refit");
            t.last_path = 2;
            t.sorted_buf = sorted;
            t.perm_dev = vp;
            t.skeys_dev = skeys;
            t.key_bytes = (int)sizeof(K);
            return OK;
        }
        // The changed keys' count is read on the device; when it is not known
        // yet (a speculative build) the grids cover the merge capacity.
        const int nb = div_up(n, kThreads);
        const int64_t mcap = merge_cap(n);
        const int64_t mmax = moved == kSpeculate ? mcap : moved;
        const int64_t nchunks = div_up(mmax, kChunk);
        int width = 64;
        while (width < mmax && width < kChunk) width <<= 1;
        if ((err = ensure(t.mkeys2, (size_t)mmax * sizeof(K))) || (err = ensure(t.mvals2, (size_t)mmax * 4)) ||
            (err = ensure(t.vals[1 - prev], (size_t)n * 4)))
            return cuda_status(ctx, err, "allocating changed keys");
        K* mk = t.mkeys.as<K>();
        int32_t* mv = t.mvals.as<int32_t>();
        K* ok = t.keys[1 - prev].as<K>();
        int32_t* ov = t.vals[1 - prev].as<int32_t>();
        {
            PhaseTimer pt_(ctx, PH_SORT);
            // Threads per chunk: width / 2 when the count is known, else 256.
            const int tpb = moved == kSpeculate ? 256 : std::max(32, width / 2);
            launch_pdl(k_moved_sort<K>, (unsigned)nchunks, tpb, 0, s, &hdr->n_moved, mcap, mk, mv);
            ctx.kernel_launches += 1;
            if (nchunks > 1) {
                launch_pdl(k_moved_rank<K>, div_up(mmax, kThreads), kThreads, 0, s, &hdr->n_moved, mcap, mk, mv,
                    t.mkeys2.as<K>(), t.mvals2.as<int32_t>());
                ctx.kernel_launches += 1;
            }
            launch_pdl(k_resort_merge<T, D, K>, nb, kThreads, 0, s, n, &hdr->n_moved, mcap, kp, vp,
                t.rflag.as<uint8_t>(), t.roff.as<int64_t>(), mk, mv, t.mkeys2.as<K>(), t.mvals2.as<int32_t>(), coords,
                ok, ov, t.spts.as<SPt<T, D>>());
            ctx.kernel_launches += 1;
        }
        skeys = ok;
        perm = ov;
        sorted = 1 - prev;
        t.last_path = 1;
    }

    // --- topology + refit (retried with the exact node or chunk count on overflow)
    const int nblocks = div_up(n, kMarkTile);
    t.n_mark_blocks = nblocks;
    const int64_t nbc = (int64_t)NLEV * nblocks;
    if ((err = ensure(t.blockcnt, (size_t)nbc * 4)) ||
        (err = ensure(t.blockoff, (size_t)(nbc + 1) * 8)) ||
        (err = ensure(t.scan_tmp, (size_t)scan_tmp_elems(nbc) * 8)))
        return cuda_status(ctx, err, "allocating topology scratch");
    int64_t est = (int64_t)Dims<D>::nch * ((n + 31) / 32) + 2 * NLEV + 64;
    if (ctx.node_cap_override > 0)
        t.capacity = ctx.node_cap_override;  // the first attempt's capacity, as set by the caller
    else if (t.capacity < est)
        t.capacity = est;
    // Query points per traversal group (a tuned shape; 32 by default).
    const int gmax = ctx.tuning_for(t.ndims, t.dtype, n, t.nbrs_hint).group_cap;
    t.group_cap = gmax;
    // Two chunks per gmax points (32: n / 16; uniform, clustered, lattice, line
    // and sphere sets have n / 20 to n / 32) and one per cloud; a set that has
    // more is laid out again with its own count.
    t.chunk_cap = std::max(t.chunk_cap, 2 * n / gmax + t.n_clouds + 64);
    for (int attempt = 0; attempt < 4; ++attempt) {
        ctx.last_attempts = attempt + 1;
        const int64_t cap = t.capacity;
        const size_t gcap = (size_t)t.chunk_cap;
        const size_t lohi_at = ((size_t)cap * 4 + 15) / 16 * 16;  // behind the first child ids
        const size_t rbytes =
            std::max({(size_t)cap * sizeof(BoxNode<T, D>), (size_t)n * 4, lohi_at + (size_t)n * 2});
        if ((err = ensure_g(ctx, t.tnode, (size_t)cap * sizeof(TNode<T, D>))) ||
            (err = ensure_g(ctx, t.nrange, (size_t)cap * 8)) || (err = ensure_g(ctx, t.link, (size_t)cap * sizeof(NodeLink))) ||
            (err = ensure_g(ctx, t.arrive, (size_t)cap * 4)) ||
            (err = ensure(t.scan_tmp, (size_t)scan_tmp_elems(nbc) * 8)) ||
            (err = ensure_g(ctx, t.rbox, rbytes)) ||
            (err = ensure_g(ctx, t.chunk, gcap * sizeof(BoxNode<T, D>))))
            return cuda_status(ctx, err, "allocating node arrays");
        if ((err = guard_fill(ctx, t.tnode, (size_t)cap * sizeof(TNode<T, D>))) ||
            (err = guard_fill(ctx, t.nrange, (size_t)cap * 8)) || (err = guard_fill(ctx, t.link, (size_t)cap * sizeof(NodeLink))) ||
            (err = guard_fill(ctx, t.arrive, (size_t)cap * 4)) ||
            (err = guard_fill(ctx, t.rbox, rbytes)) ||
            (err = guard_fill(ctx, t.chunk, gcap * sizeof(BoxNode<T, D>))))
            return cuda_status(ctx, err, "node array guards");
        {
        PhaseTimer pt_(ctx, PH_TOPOLOGY);
        int32_t* fchild = t.rbox.as<int32_t>();
        uint16_t* lohi = reinterpret_cast<uint16_t*>(t.rbox.as<unsigned char>() + lohi_at);
        launch_pdl(k_mark<D, K>, nblocks, kThreads, 0, s, skeys, n, lohi, t.blockcnt.as<int32_t>(),
            nblocks, t.dstart.as<uint8_t>(), t.bvh_arrive.as<int32_t>(), n_arrive, hdr, bt);
        ctx.kernel_launches += exclusive_scan_i32_i64(t.blockcnt.as<int32_t>(), t.blockoff.as<int64_t>(), nbc,
                                                      &hdr->n_nodes, t.scan_tmp.as<int64_t>(), s);
        launch_pdl(k_emit_ids<D>, nblocks, kThreads, 0, s, n, lohi, t.blockoff.as<int64_t>(), nblocks,
            cap, fchild, t.nrange.as<int2>(), t.arrive.as<int32_t>(), hdr, bt);
        launch_pdl(k_emit_nodes<T, D, K>, div_up(cap, kThreads), kThreads, 0, s, skeys, n, cap, fchild,
            t.tnode.as<TNode<T, D>>(), t.nrange.as<int2>(), t.link.as<NodeLink>(), t.arrive.as<int32_t>(),
            t.blockoff.as<int64_t>(), nblocks, hdr, bt);
        ctx.kernel_launches += 3;
        }
        launch_layout<T, D>(ctx, t, skeys, n, cap, (int64_t)gcap, cap, gmax, inv_cs);
        if (ctx.guard_check) {
            guard_check(ctx, t.tnode, (size_t)cap * sizeof(TNode<T, D>), hdr);
            guard_check(ctx, t.nrange, (size_t)cap * 8, hdr);
            guard_check(ctx, t.link, (size_t)cap * sizeof(NodeLink), hdr);
            guard_check(ctx, t.arrive, (size_t)cap * 4, hdr);
            guard_check(ctx, t.rbox, rbytes, hdr);
            guard_check(ctx, t.chunk, gcap * sizeof(BoxNode<T, D>), hdr);
            if (moved == -1) {
                for (int b = 0; b < 2; ++b) guard_check(ctx, t.keys[b], (size_t)n * sizeof(K), hdr);
                guard_check(ctx, t.vals[0], (size_t)n * 4, hdr);
                guard_check(ctx, t.spts, (size_t)n * sizeof(SPt<T, D>), hdr);
                guard_check(ctx, t.dpts, (size_t)n * sizeof(SPt<T, D>), hdr);
            }
        }
        if ((err = cudaMemcpyAsync(t.hdr_host, hdr, sizeof(OctHeader), cudaMemcpyDeviceToHost, s)) ||
            (err = wait_stream(s)))
            return cuda_status(ctx, err, "tree build");
        if (t.hdr_host->guard_bad)
            return set_error(ctx, ERR_STATE, "tree build: a kernel wrote past the end of a sort buffer or node array");
        if (moved == kSpeculate &&
            (t.hdr_host->nan_flag || t.hdr_host->n_moved > merge_cap(n) || (t.hdr_host->status & DF_KEY_WIDTH)))
            return kRetry;  // the bounds say the merge did not apply: build again on the usual path
        if (t.hdr_host->status & DF_TIMEOUT)
            return set_error(ctx, ERR_TIMEOUT, "tree build: a radix-sort look-back wait ran out");
        if (t.hdr_host->status & DF_NODE_OVERFLOW) {
            t.capacity = t.hdr_host->n_nodes + t.hdr_host->n_nodes / 8 + 64;
            const int zero = 0;
            cudaMemcpyAsync(&hdr->status, &zero, sizeof(int), cudaMemcpyHostToDevice, s);
            continue;
        }
        if (t.hdr_host->n_groups > t.chunk_cap) {
            t.chunk_cap = t.hdr_host->n_groups + t.hdr_host->n_groups / 8;
            continue;
        }
        t.n_nodes = t.hdr_host->n_nodes;
        t.n_groups = t.hdr_host->n_groups;
        t.asc_key = t.hdr_host->asc_key;
        t.sorted_buf = sorted;
        t.perm_dev = perm;
        t.skeys_dev = skeys;
        t.key_bytes = (int)sizeof(K);
        return OK;
    }
    return set_error(ctx, ERR_OVERFLOW, "tree build: node or chunk capacity retry did not converge");
}

// Refit mode: re-encodes every point at its previous sorted position and
// counts the changed keys into hdr->n_moved (read with the bounds).
template <class T, int D, class K>
int resort_mark(Ctx& ctx, Tree& t, const T* coords, int64_t n, T radius, int prev, int64_t cap) {
    cudaStream_t s = ctx.stream;
    cudaError_t err;
    const int nb = div_up(n, kThreads);
    if ((err = ensure(t.rflag, (size_t)n)) || (err = ensure(t.rcnt, (size_t)nb * 4)) ||
        (err = ensure(t.roff, (size_t)(nb + 1) * 8)) || (err = ensure(t.scan_tmp, (size_t)scan_tmp_elems(nb) * 8)) ||
        (err = ensure(t.mkeys, (size_t)cap * sizeof(K))) || (err = ensure(t.mvals, (size_t)cap * 4)))
        return cuda_status(ctx, err, "allocating refit-mode scratch");
    OctHeader* hdr = t.hdr.as<OctHeader>();
    PhaseTimer pt_(ctx, PH_ENCODE);
    launch_pdl(k_resort_mark<T, D, K>, nb, kThreads, 0, s, coords, n, t.vals[prev].as<int32_t>(), t.keys[prev].as<K>(),
        T(1) / radius, hdr, t.rflag.as<uint8_t>(), t.rcnt.as<int32_t>(), t.mkeys.as<K>(), t.mvals.as<int32_t>(), cap);
    ctx.kernel_launches += 1 + exclusive_scan_i32_i64(t.rcnt.as<int32_t>(), t.roff.as<int64_t>(), nb, nullptr,
                                                      t.scan_tmp.as<int64_t>(), s);
    return OK;
}

// Origin and key width on the host from the bounds in t.hdr_host, in T
// (src/cpu/bin_cpu.jl:22,35,60); InexactError where the reference's
// floor(Int32, ...) throws.
template <class T, int D>
int host_key_width(Ctx& ctx, Tree& t, T radius) {
    if (t.hdr_host->nan_flag)
        return set_error(ctx, ERR_INEXACT, "InexactError: floor(Int32, NaN/Inf) in bin_point (non-finite coordinate)");
    const T inv_cs = T(1) / radius;
    int64_t cmax_all = 0;
    double cells = 0.0;
    for (int d = 0; d < D; ++d) {
        const T o = (T)t.hdr_host->gmin[d] - T(1e-6);
        t.origin[d] = (double)o;
        const T v = ((T)t.hdr_host->gmax[d] - o) * inv_cs;
        cells = std::max(cells, (double)v);
        const T f = std::floor(v);
        if (!(f >= T(-2147483648.0) && f < T(2147483648.0)))
            return set_error(ctx, ERR_INEXACT, "InexactError: floor(Int32, (p - origin) / radius) exceeds Int32");
        int64_t c = (int64_t)f;
        const int64_t cm = (1LL << Dims<D>::bits) - 1;
        c = c < 0 ? 0 : (c > cm ? cm : c);
        cmax_all = std::max(cmax_all, c);
    }
    t.mul = box_mul(cells);
    int nbits_axis = 0;
    while (nbits_axis < 63 && (cmax_all >> nbits_axis) != 0) ++nbits_axis;
    t.key_bits = D * nbits_axis;
    t.key_bytes = t.key_bits <= 32 ? 4 : 8;
    t.sort_passes = (t.key_bits + 7) / 8;
    return OK;
}

template <class T, int D>
int build_typed(Ctx& ctx, Tree& t, const T* coords, int64_t n, double radius_d) {
    cudaStream_t s = ctx.stream;
    cudaError_t err;
    const T radius = (T)radius_d;
    if ((err = ensure(t.hdr, sizeof(OctHeader)))) return cuda_status(ctx, err, "allocating header");
    if (!t.hdr_host) {
        if ((err = header_alloc(&t.hdr_host))) return cuda_status(ctx, err, "pinned header");
    }
    OctHeader* hdr = t.hdr.as<OctHeader>();
    if ((err = cudaMemsetAsync(hdr, 0, sizeof(OctHeader), s))) return cuda_status(ctx, err, "header reset");

    // --- 1. bounds (one host round trip, like ext/cuda_build.jl:235)
    const int nb = std::max(1, std::min(div_up(n, kThreads * 8), 4 * 148));
    if ((err = ensure(t.partials, (size_t)nb * 8 * 8))) return cuda_status(ctx, err, "allocating partials");
    {
        PhaseTimer pt_(ctx, PH_BOUNDS);
        launch_pdl(k_bounds<T, D>, nb, kThreads, 0, s, coords, n, t.partials.as<typename OrdKey<T>::I>(), hdr);
        ctx.kernel_launches += 1;
    }
    // Refit mode with a reusable previous order: re-encode in that order now,
    // so the count of changed keys arrives with the bounds.
    const int prev = t.sorted_buf;
    t.sorted_buf = -1;
    const bool try_resort = t.keep_morton && prev >= 0 && t.sorted_n == n && t.sorted_radius == radius_d;
    // Merge at most this many changed keys; more are cheaper to sort afresh.
    const int64_t cap = merge_cap(n);
    if (try_resort) {
        const int st = t.sorted_key_bytes == 4 ? resort_mark<T, D, uint32_t>(ctx, t, coords, n, radius, prev, cap)
                                               : resort_mark<T, D, uint64_t>(ctx, t, coords, n, radius, prev, cap);
        if (st != OK) return st;
    }
    // Steady time stepping: the previous build merged its changed keys, so
    // merge again without waiting for the bounds.  The round trip at the end
    // of the topology brings the bounds, the count of changed keys and the
    // key-width flag; if the merge did not apply, build again below.
    if (try_resort && t.last_path == 1) {
        const int st = t.sorted_key_bytes == 4
                           ? run_pipeline<T, D, uint32_t>(ctx, t, coords, n, radius, kSpeculate, prev)
                           : run_pipeline<T, D, uint64_t>(ctx, t, coords, n, radius, kSpeculate, prev);
        if (st != kRetry) {
            if (st != OK) return st;
            const int kw = host_key_width<T, D>(ctx, t, radius);
            if (kw != OK) return kw;
            t.key_bytes = t.sorted_key_bytes;  // the width the keys were built with
            t.last_moved = t.hdr_host->n_moved;
            t.last_path = 1;
            t.sorted_n = n;
            t.sorted_radius = radius_d;
            return OK;
        }
        t.sorted_buf = -1;
    } else if ((err = cudaMemcpyAsync(t.hdr_host, hdr, sizeof(OctHeader), cudaMemcpyDeviceToHost, s)) ||
               (err = wait_stream(s))) {
        return cuda_status(ctx, err, "bounds reduce");
    }
    const int kw = host_key_width<T, D>(ctx, t, radius);
    if (kw != OK) return kw;
    // Merge the changed keys into the previous order unless they are too many
    // (or the key width changed).
    int64_t moved = -1;
    t.last_moved = try_resort ? t.hdr_host->n_moved : -1;
    if (try_resort && t.key_bytes == t.sorted_key_bytes && t.hdr_host->n_moved <= cap) moved = t.hdr_host->n_moved;
    const int st = t.key_bytes == 4 ? run_pipeline<T, D, uint32_t>(ctx, t, coords, n, radius, moved, prev)
                                    : run_pipeline<T, D, uint64_t>(ctx, t, coords, n, radius, moved, prev);
    if (st == OK && t.sorted_buf >= 0) {
        t.sorted_n = n;
        t.sorted_radius = radius_d;
        t.sorted_key_bytes = t.key_bytes;
    }
    return st;
}

template <class T, int D>
int build_batch_typed(Ctx& ctx, Tree& t, const T* coords, int64_t n, const int64_t* coff_host,
                      const double* radii_host, int32_t nc) {
    cudaStream_t s = ctx.stream;
    cudaError_t err;
    if ((err = ensure(t.hdr, sizeof(OctHeader))) || (err = ensure(t.b_coff, (size_t)(nc + 1) * 8)) ||
        (err = ensure(t.b_cparam, (size_t)nc * kCloudParams * 8)) ||
        (err = ensure(t.b_cbounds, (size_t)nc * 8 * 8)) ||
        (err = ensure(t.b_eoff, (size_t)(nc + 1) * 8)))
        return cuda_status(ctx, err, "allocating batch arrays");
    if (!t.hdr_host) {
        if ((err = header_alloc(&t.hdr_host))) return cuda_status(ctx, err, "pinned header");
    }
    if ((err = cudaMemsetAsync(t.hdr.p, 0, sizeof(OctHeader), s)) ||
        (err = cudaMemcpyAsync(t.b_coff.p, coff_host, (size_t)(nc + 1) * 8, cudaMemcpyHostToDevice, s)))
        return cuda_status(ctx, err, "batch upload");
    {
        PhaseTimer pt_(ctx, PH_BOUNDS);
        k_cloud_bounds<T, D><<<nc, kCloudThreads, 0, s>>>(coords, t.b_coff.as<int64_t>(), t.b_cbounds.as<double>());
        ctx.kernel_launches += 1;
    }
    std::vector<double> cb((size_t)nc * 8);
    if ((err = cudaMemcpyAsync(cb.data(), t.b_cbounds.p, cb.size() * 8, cudaMemcpyDeviceToHost, s)) ||
        (err = wait_stream(s)))
        return cuda_status(ctx, err, "cloud bounds");
    // Per cloud, in T, exactly what a TNS of that cloud alone computes
    // (src/cpu/bin_cpu.jl:22,35,60; src/cpu/edges_cpu.jl:184-185).
    std::vector<double> cp((size_t)nc * kCloudParams, 0.0);
    int64_t cmax_all = 0;
    double cells = 0.0;
    for (int c = 0; c < nc; ++c) {
        if (coff_host[c + 1] == coff_host[c]) continue;
        const double* b = cb.data() + (size_t)c * 8;
        if (b[6] != 0.0)
            return set_error(ctx, ERR_INEXACT, "InexactError: floor(Int32, NaN/Inf) in bin_point (non-finite coordinate)");
        const T r = (T)radii_host[c];
        const T inv_cs = T(1) / r;
        double* p = cp.data() + (size_t)c * kCloudParams;
        for (int d = 0; d < D; ++d) {
            const T o = (T)b[d] - T(1e-6);
            p[d] = (double)o;
            const T v = ((T)b[3 + d] - o) * inv_cs;
            cells = std::max(cells, (double)v);
            const T f = std::floor(v);
            if (!(f >= T(-2147483648.0) && f < T(2147483648.0)))
                return set_error(ctx, ERR_INEXACT, "InexactError: floor(Int32, (p - origin) / radius) exceeds Int32");
            int64_t ci = (int64_t)f;
            const int64_t cm = (1LL << Dims<D>::bits) - 1;
            ci = ci < 0 ? 0 : (ci > cm ? cm : ci);
            cmax_all = std::max(cmax_all, ci);
            p[6 + d] = b[d];
            p[9 + d] = b[3 + d];
        }
        p[3] = (double)inv_cs;
        p[4] = (double)(r * r);
        p[5] = (double)(T(1) / r);
    }
    if ((err = cudaMemcpyAsync(t.b_cparam.p, cp.data(), cp.size() * 8, cudaMemcpyHostToDevice, s)))
        return cuda_status(ctx, err, "cloud parameters");
    t.mul = box_mul(cells);
    int nbits_axis = 0;
    while (nbits_axis < 63 && (cmax_all >> nbits_axis) != 0) ++nbits_axis;
    int cbits = 0;
    while (cbits < 31 && ((int64_t)(nc - 1) >> cbits) != 0) ++cbits;
    t.kbits = D * nbits_axis;
    t.key_bits = t.kbits + cbits;
    if (t.key_bits > 64) return set_error(ctx, ERR_ARGUMENT, "batch: cloud id and Morton code exceed 64 key bits");
    t.key_bytes = t.key_bits <= 32 ? 4 : 8;
    t.sort_passes = (t.key_bits + 7) / 8;
    if (t.key_bytes == 4) return run_pipeline<T, D, uint32_t>(ctx, t, coords, n, T(0));
    return run_pipeline<T, D, uint64_t>(ctx, t, coords, n, T(0));
}

}  // namespace

int build_tree_batch(Ctx& ctx, Tree& t, const void* coords, int64_t n, const int64_t* coff_host,
                     const double* radii_host, int32_t n_clouds) {
    t.sorted_buf = -1;
    t.built = false;
    t.view_valid = false;
    t.n = n;
    t.radius = 0.0;
    t.keep_morton = false;
    ++t.generation;
    t.n_clouds = n_clouds;
    if (n == 0) {
        t.n_nodes = 0;
        t.n_groups = 0;
        t.built = true;
        return OK;
    }
    int st;
    if (t.dtype == 0)
        st = t.ndims == 3 ? build_batch_typed<float, 3>(ctx, t, (const float*)coords, n, coff_host, radii_host, n_clouds)
                          : build_batch_typed<float, 2>(ctx, t, (const float*)coords, n, coff_host, radii_host, n_clouds);
    else
        st = t.ndims == 3 ? build_batch_typed<double, 3>(ctx, t, (const double*)coords, n, coff_host, radii_host, n_clouds)
                          : build_batch_typed<double, 2>(ctx, t, (const double*)coords, n, coff_host, radii_host, n_clouds);
    if (st == OK) t.built = true;
    return st;
}

int batch_edge_offsets(Ctx& ctx, Tree& t, int64_t* out_host) {
    const int nc = t.n_clouds;
    cudaError_t err;
    if (ctx.plan_query != &t || ctx.plan_target != &t || ctx.plan_qgen != t.generation)
        return set_error(ctx, ERR_STATE, "batch edge offsets: no matching oct_edges_count for this tree");
    if (t.n == 0 || ctx.plan_edges <= 0) {
        for (int c = 0; c <= nc; ++c) out_host[c] = 0;
        return OK;
    }
    k_gather_edge_offsets<<<div_up(nc + 1, 128), 128, 0, ctx.stream>>>(ctx.offsets.as<int64_t>(), t.b_coff.as<int64_t>(),
                                                                        nc, t.b_eoff.as<int64_t>());
    ctx.kernel_launches += 1;
    if ((err = cudaMemcpyAsync(out_host, t.b_eoff.p, (size_t)(nc + 1) * 8, cudaMemcpyDeviceToHost, ctx.stream)) ||
        (err = wait_stream(ctx.stream)))
        return cuda_status(ctx, err, "batch edge offsets");
    return OK;
}

int build_tree(Ctx& ctx, Tree& t, const void* coords, int64_t n, double radius) {
    t.built = false;
    t.view_valid = false;
    t.n = n;
    t.radius = radius;
    t.n_clouds = 0;
    ++t.generation;
    if (n == 0) {
        t.n_nodes = 0;
        t.sorted_buf = -1;
        t.built = true;
        return OK;
    }
    int st;
    if (t.dtype == 0)
        st = t.ndims == 3 ? build_typed<float, 3>(ctx, t, (const float*)coords, n, radius)
                          : build_typed<float, 2>(ctx, t, (const float*)coords, n, radius);
    else
        st = t.ndims == 3 ? build_typed<double, 3>(ctx, t, (const double*)coords, n, radius)
                          : build_typed<double, 2>(ctx, t, (const double*)coords, n, radius);
    if (st == OK) t.built = true;
    return st;
}

int ensure_iperm(Ctx& ctx, const Tree& t) {
    if (t.iperm_valid || t.n == 0 || !t.perm_dev) return OK;
    OctHeader* hdr = t.hdr.as<OctHeader>();
    k_inverse_perm<<<(unsigned)div_up(t.n, kSortThreads), kSortThreads, 0, ctx.stream>>>(
        t.perm_dev, t.n, t.rbox.as<int32_t>(), &hdr->status);
    ctx.kernel_launches += 1;
    const cudaError_t err = cudaGetLastError();
    if (err) return cuda_status(ctx, err, "inverse permutation launch");
    t.iperm_valid = true;
    return OK;
}

namespace {
template <class T, int D>
int view_typed(Ctx& ctx, Tree& t) {
    cudaError_t err;
    const int64_t nn = std::max<int64_t>(t.n_nodes, 1), n = std::max<int64_t>(t.n, 1);
    constexpr int NCH = Dims<D>::nch;
    if ((err = ensure(t.v_first, nn * 4)) || (err = ensure(t.v_last, nn * 4)) || (err = ensure(t.v_children, nn * 4 * NCH)) ||
        (err = ensure(t.v_bmin, nn * sizeof(T) * D)) || (err = ensure(t.v_bmax, nn * sizeof(T) * D)) ||
        (err = ensure(t.v_perm, n * 4)))
        return cuda_status(ctx, err, "allocating views");
    if (t.n_nodes > 0)
        k_view_nodes<T, D><<<div_up(t.n_nodes, kThreads), kThreads, 0, ctx.stream>>>(
            t.tnode.as<TNode<T, D>>(), t.nrange.as<int2>(), t.n_nodes, t.v_first.as<int32_t>(), t.v_last.as<int32_t>(),
            t.v_children.as<int32_t>(), t.v_bmin.as<T>(), t.v_bmax.as<T>());
    if (t.n > 0)
        k_view_perm<T, D><<<div_up(t.n, kThreads), kThreads, 0, ctx.stream>>>(t.spts.as<SPt<T, D>>(), t.n,
                                                                               t.v_perm.as<int32_t>());
    if (t.keep_morton && t.n > 0 && !t.n_clouds) {
        if ((err = ensure(t.morton, (size_t)t.n * 8))) return cuda_status(ctx, err, "allocating morton codes");
        if (t.key_bytes == 4)
            k_view_morton<T, D, uint32_t><<<div_up(t.n, kThreads), kThreads, 0, ctx.stream>>>(
                t.spts.as<SPt<T, D>>(), (const uint32_t*)t.skeys_dev, t.n, t.morton.as<uint64_t>());
        else
            k_view_morton<T, D, uint64_t><<<div_up(t.n, kThreads), kThreads, 0, ctx.stream>>>(
                t.spts.as<SPt<T, D>>(), (const uint64_t*)t.skeys_dev, t.n, t.morton.as<uint64_t>());
    }
    if ((err = cudaStreamSynchronize(ctx.stream))) return cuda_status(ctx, err, "materializing views");
    t.view_valid = true;
    return OK;
}
}  // namespace

int materialize_view(Ctx& ctx, Tree& t) {
    if (t.view_valid) return OK;
    if (t.dtype == 0) return t.ndims == 3 ? view_typed<float, 3>(ctx, t) : view_typed<float, 2>(ctx, t);
    return t.ndims == 3 ? view_typed<double, 3>(ctx, t) : view_typed<double, 2>(ctx, t);
}

}  // namespace oct
