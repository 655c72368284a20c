// Key sort of the build that carries the points along.
//
// The stable LSD radix sort of the Morton keys (ties keep ascending original
// index, src/sort.jl:15-24) with each point's record SPt {coordinates,
// original index} as the sorted value, so that the sorted points come out of
// the last pass instead of a gather at random original indices afterwards.
// The Morton encode (src/cpu/bin_cpu.jl:52-95) is fused in too:
//
//   k_point_counts  reads the coordinates once, encodes each key and counts
//                   every pass's 8-bit digits;
//   k_point_pass    one launch per digit: each block takes the next tile of
//                   2048 points (tile ids in the order blocks start), ranks
//                   its keys by digit (warp match, per-warp counters), adds the
//                   counts of the tiles before it by decoupled look-back
//                   (bounded waits) while the tile's points come into shared
//                   memory by asynchronous copies, and writes each digit's run
//                   contiguously.  The first pass encodes from the coordinates;
//                   the last writes the sorted keys, the sorted points and the
//                   permutation;
//   k_inverse_perm  the inverse permutation, launched by the first caller that
//                   needs it after a build.
//
// Every wait is bounded (spin_limit polling rounds); one that runs out sets
// DF_TIMEOUT, and every store still stays inside its array.
#pragma once

#include <algorithm>

#include <cuda/atomic>

#include "common.cuh"
#include "sort.cuh"

namespace oct {

// Per-point encode parameters: one origin and cell size, or per cloud.
template <class T>
struct EncodeParams {
    T o[3];
    T inv_cs;
    Batch bt;
};

// Bits of x spread to every third / second bit, for keys of at most 32 bits
// (10 bits per axis in 3D, 16 in 2D).
__device__ __forceinline__ uint32_t spread3_32(uint32_t x) {
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    return (x | (x << 2)) & 0x09249249u;
}
__device__ __forceinline__ uint32_t spread2_32(uint32_t x) {
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

// Cell index of one axis, floor(v) clamped below at 0; the caller has proven
// that it fits Int32.
__device__ __forceinline__ int cell_i32(float v) { return max(__float2int_rd(v), 0); }
__device__ __forceinline__ int cell_i32(double v) { return max(__double2int_rd(v), 0); }

// Origin, inverse cell size and id of the cloud a thread's points are in
// (without a batch: of the point set), looked up when a point lies outside the
// one before.  A thread's points are in input order and a few hundred apart at
// most, so a search per thread serves nearly all of them (5.2M points in 512
// clouds: counts and first pass 87 us, 112 with a search per point).
template <class T>
struct CloudCursor {
    T o[3];
    T inv_cs;
    int32_t begin = 0, end = 0;  // its positions; none before the first look-up
    int32_t cloud = 0;
    __device__ __forceinline__ explicit CloudCursor(const EncodeParams<T>& ep)
        : o{ep.o[0], ep.o[1], ep.o[2]}, inv_cs(ep.inv_cs) {}
    __device__ __forceinline__ void seek(const Batch& bt, int64_t i) {
        if (i >= begin && i < end) return;
        cloud = cloud_of_position(bt, i);
        begin = (int32_t)bt.coff[cloud];
        end = (int32_t)bt.coff[cloud + 1];
        const double* cp = bt.cparam + (size_t)cloud * kCloudParams;
#pragma unroll
        for (int d = 0; d < 3; ++d) o[d] = (T)cp[d];
        inv_cs = (T)cp[3];
    }
};

// Morton key of one point's cell (src/cpu/bin_cpu.jl:12-31,
// src/morton.jl:13-60): floor((x - origin) * inv_cs) per axis, clamped to the
// key's bits per axis, bit-interleaved with x in the lowest bit; in a batch,
// (cloud << kbits) | morton with the cloud's own origin and cell size.
// A 32-bit key K means that the host found every cell index below 2^10 (3D)
// or 2^16 (2D), so the interleave runs on 32-bit words.
template <class T, int D, class K>
__device__ __forceinline__ K point_key(const T* x, int64_t i, const EncodeParams<T>& ep, CloudCursor<T>& cur) {
    constexpr int64_t cmax = (1LL << Dims<D>::bits) - 1;
    if (ep.bt.n_clouds) cur.seek(ep.bt, i);
    const T* o = cur.o;
    const T inv_cs = cur.inv_cs;
    const int cloud = cur.cloud;
    if constexpr (sizeof(K) == 4) {
        uint32_t c[3] = {0, 0, 0};
#pragma unroll
        for (int d = 0; d < D; ++d) c[d] = (uint32_t)cell_i32(mul_rn(sub_rn(x[d], o[d]), inv_cs));
        const uint32_t m = (D == 3) ? ((spread3_32(c[2]) << 2) | (spread3_32(c[1]) << 1) | spread3_32(c[0]))
                                    : ((spread2_32(c[1]) << 1) | spread2_32(c[0]));
        return ep.bt.n_clouds ? (((uint32_t)cloud << ep.bt.kbits) | m) : m;
    }
    uint64_t c[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const T v = mul_rn(sub_rn(x[d], o[d]), inv_cs);
        int64_t ci = (int64_t)floor(v);
        ci = ci < 0 ? 0 : (ci > cmax ? cmax : ci);
        c[d] = (uint64_t)ci;
    }
    const uint64_t m = (D == 3) ? ((split_by_3(c[2]) << 2) | (split_by_3(c[1]) << 1) | split_by_3(c[0]))
                                : ((split_by_2(c[1]) << 1) | split_by_2(c[0]));
    return (K)(ep.bt.n_clouds ? (((uint64_t)cloud << ep.bt.kbits) | m) : m);
}

constexpr int kLook = 4;  // look-back words per round trip

// Every pass's digit counts in one read of the coordinates.
template <class T, int D, class K>
__global__ void __launch_bounds__(kSortThreads) k_point_counts(const T* __restrict__ coords, int64_t n, int passes,
                                                               EncodeParams<T> ep, uint32_t* __restrict__ counts) {
    pdl_wait();
    pdl_trigger();
    __shared__ uint32_t c[kOnesweepMaxPasses][256];
    for (int p = 0; p < passes; ++p) c[p][threadIdx.x] = 0;
    __syncthreads();
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nthr = (int64_t)gridDim.x * blockDim.x;
    CloudCursor<T> cur(ep);
    auto take = [&](const T* x, int64_t i) {
        const K k = point_key<T, D, K>(x, i, ep, cur);
        for (int p = 0; p < passes; ++p) atomicAdd(&c[p][(unsigned)(k >> (8 * p)) & 255u], 1u);
    };
    int64_t done = 0;  // points counted by the vector loop
    if constexpr (sizeof(T) == 4) {
        if (((uintptr_t)coords & 15) == 0) {
            // four points = D float4
            const float4* v = reinterpret_cast<const float4*>(coords);
            for (int64_t g = tid; g < n / 4; g += nthr) {
                float4 q[D];
#pragma unroll
                for (int d = 0; d < D; ++d) q[d] = v[D * g + d];
                const float* x = reinterpret_cast<const float*>(q);
#pragma unroll
                for (int j = 0; j < 4; ++j) take(x + D * j, 4 * g + j);
            }
            done = n / 4 * 4;
        }
    }
    for (int64_t i = done + tid; i < n; i += nthr) {
        T x[D];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = coords[(int64_t)D * i + d];
        take(x, i);
    }
    __syncthreads();
    for (int p = 0; p < passes; ++p)
        if (c[p][threadIdx.x]) atomicAdd(&counts[(size_t)p * 257 + threadIdx.x], c[p][threadIdx.x]);
}

// 16 bytes from global to shared memory without passing through registers.
__device__ __forceinline__ void copy_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(sdst)), "l"(gsrc)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shared memory of one k_point_pass block.  The tile's points stay in input
// order (in the first pass their bare coordinates), `order` lists them in
// digit order.
template <class T, int D, class K, bool FIRST>
struct PointPassSmem {
    static constexpr int kRec = FIRST ? D * sizeof(T) : sizeof(SPt<T, D>);  // bytes per point
    alignas(16) unsigned char pts[kSortTile * kRec];
    K key[kSortTile];
    int32_t wc[kSortThreads / 32][256];
    int32_t tstart[256];
    int32_t gstart[256];
    uint16_t order[kSortTile];
    int32_t scan_sm[kSortThreads / 32 + 1];
    int tile;
};

template <class T, int D, class K, bool FIRST>
constexpr size_t point_pass_smem() { return sizeof(PointPassSmem<T, D, K, FIRST>); }

// One pass on digit `pass`.  FIRST: the points come from `coords` (key
// encoded here, value = the point and its index); otherwise from (kin, pin).
// LAST: writes kout, pout (the sorted points) and perm[dst] = original index.
// The tile's points travel to shared memory by asynchronous copies while its
// keys are ranked and the tiles before it are waited for.  Bound by the
// instructions of the ranking and by shared memory (random 16-byte reads in
// digit order), not by DRAM: a pass over 16M points moves 640 MB in 226 us
// (2.8 TB/s; 236 us with the points staged in digit order through registers).
// Not faster: 4096-point tiles, look-back over 8 to 32 tiles per round trip.
template <class T, int D, class K, bool FIRST, bool LAST>
__global__ void __launch_bounds__(kSortThreads) k_point_pass(
    const T* __restrict__ coords, EncodeParams<T> ep, const K* __restrict__ kin, const SPt<T, D>* __restrict__ pin,
    K* __restrict__ kout, SPt<T, D>* __restrict__ pout, int32_t* __restrict__ perm, int64_t n, int pass, int ntiles, uint32_t* __restrict__ scratch, int* __restrict__ status, int64_t spin_limit,
    int withhold_tile) {
    pdl_wait();
    pdl_trigger();
    using Smem = PointPassSmem<T, D, K, FIRST>;
    extern __shared__ __align__(16) unsigned char pp_smem[];
    Smem& sm = *reinterpret_cast<Smem*>(pp_smem);
    const int shift = 8 * pass;
    uint32_t* counts = scratch + (size_t)pass * 257;
    uint32_t* look = scratch + (size_t)kOnesweepMaxPasses * 257 + (size_t)pass * ntiles * 256;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) sm.tile = (int)atomicAdd(&counts[256], 1u);
#pragma unroll
    for (int j = 0; j < kSortThreads / 32; ++j) sm.wc[j][threadIdx.x] = 0;
    __syncthreads();
    const int t = sm.tile;
    const int64_t tbase = (int64_t)t * kSortTile;
    const int tcnt = (int)(n - tbase < kSortTile ? n - tbase : kSortTile);  // points of this tile
    {
        // a tile's first byte is a multiple of 16 from the array's
        const unsigned char* g = FIRST ? reinterpret_cast<const unsigned char*>(coords) + tbase * Smem::kRec
                                       : reinterpret_cast<const unsigned char*>(pin + tbase);
        const int bytes = tcnt * Smem::kRec;
        const bool vec = !FIRST || ((uintptr_t)coords & 15) == 0;
        const int whole = vec ? bytes & ~15 : 0;
        for (int b = threadIdx.x * 16; b < whole; b += kSortThreads * 16) copy_async16(sm.pts + b, g + b);
        if (FIRST)
            for (int b = whole + threadIdx.x * (int)sizeof(T); b < bytes; b += kSortThreads * (int)sizeof(T))
                *reinterpret_cast<T*>(sm.pts + b) = *reinterpret_cast<const T*>(g + b);
    }
    const int lbase = w * (32 * kSortItems);  // this warp's part of the tile
    K key[kSortItems];
    CloudCursor<T> cur(ep);
    if (FIRST) {
        copy_async_wait();
        __syncthreads();
    }
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const int l = lbase + it * 32 + lane;
        key[it] = K(0);
        if (l < tcnt)
            key[it] = FIRST ? point_key<T, D, K>(reinterpret_cast<const T*>(sm.pts) + D * l, tbase + l, ep, cur)
                            : kin[tbase + l];
    }
    // Rank of each key among the tile's keys of its digit that come before it:
    // the lanes sharing a digit by match, the first of them advances the
    // warp's counter (in item order: the counters' old values return while the
    // next items' updates are issued).
    unsigned peers[kSortItems];
    int32_t rk[kSortItems];
#pragma unroll
    for (int it = 0; it < kSortItems; ++it)
        peers[it] = __match_any_sync(
            0xffffffffu, lbase + it * 32 + lane < tcnt ? (int)((unsigned)(key[it] >> shift) & 255u) : 256);
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        rk[it] = 0;
        if (lbase + it * 32 + lane < tcnt && (peers[it] & lanemask_lt()) == 0)
            rk[it] = atomicAdd(&sm.wc[w][(unsigned)(key[it] >> shift) & 255u], __popc(peers[it]));
        __syncwarp();
    }
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        rk[it] = __shfl_sync(0xffffffffu, rk[it], __ffs(peers[it]) - 1) + __popc(peers[it] & lanemask_lt());
        const int l = lbase + it * 32 + lane;
        if (l < tcnt) sm.key[l] = key[it];
    }
    __syncthreads();
    // thread = digit: warp offsets within the tile's run, the tile's count
    const int d = threadIdx.x;
    int32_t run = 0;
#pragma unroll
    for (int j = 0; j < kSortThreads / 32; ++j) {
        const int32_t c = sm.wc[j][d];
        sm.wc[j][d] = run;
        run += c;
    }
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> mine(look[(size_t)t * 256 + d]);
    // A withheld tile (a test aid: pass 0, tile `withhold_tile`) never
    // publishes, so the waits of the tiles after it run out.
    const bool publish = !(pass == 0 && t == withhold_tile);
    if (publish) mine.store((t == 0 ? kLookPrefix : kLookAggregate) | (uint32_t)run, cuda::memory_order_relaxed);
    uint32_t excl = 0;
    bool timed_out = false;
    if (t > 0) {
        // kLook predecessors per round trip, added in order up to the first
        // inclusive prefix; a word not yet published stops the round.
        int j = t - 1;
        int64_t spins = 0;
        while (true) {
            uint32_t v[kLook];
#pragma unroll
            for (int u = 0; u < kLook; ++u)
                v[u] = j - u >= 0 ? cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(look[(size_t)(j - u) * 256 + d])
                                        .load(cuda::memory_order_relaxed)
                                  : kLookPrefix;
            int u = 0;
            bool done = false;
            for (; u < kLook; ++u) {
                if ((v[u] & ~kLookValue) == 0) break;
                excl += v[u] & kLookValue;
                if ((v[u] & ~kLookValue) == kLookPrefix) {
                    done = true;
                    break;
                }
            }
            if (done) break;
            j -= u;
            if (u < kLook) {
                if (++spins > spin_limit) {
                    timed_out = true;
                    break;
                }
                __nanosleep(32);
            }
        }
        if (publish) mine.store(kLookPrefix | (excl + (uint32_t)run), cuda::memory_order_relaxed);
    }
    int32_t tile_total, all;
    const int32_t tst = block_exclusive_scan<int32_t>(run, sm.scan_sm, &tile_total);
    const int32_t base = block_exclusive_scan<int32_t>((int32_t)counts[d], sm.scan_sm, &all);
    sm.tstart[d] = tst;
    sm.gstart[d] = (int32_t)(base + excl);
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
        const int l = lbase + it * 32 + lane;
        const unsigned dg = (unsigned)(key[it] >> shift) & 255u;
        if (l < tcnt) sm.order[sm.tstart[dg] + sm.wc[w][dg] + rk[it]] = (uint16_t)l;
    }
    if (!FIRST) copy_async_wait();
    __syncthreads();
    // Each digit's run contiguously, in digit order.
    for (int i = threadIdx.x; i < tile_total; i += kSortThreads) {
        const int l = sm.order[i];
        const K k = sm.key[l];
        const int dd = (int)((unsigned)(k >> shift) & 255u);
        const int64_t dst = (int64_t)sm.gstart[dd] + (i - sm.tstart[dd]);
        if (dst >= 0 && dst < n) {  // always, unless a wait ran out and left a prefix short
            SPt<T, D> p;
            if (FIRST) {
                const T* x = reinterpret_cast<const T*>(sm.pts) + D * l;
#pragma unroll
                for (int c = 0; c < D; ++c) p.x[c] = x[c];
                p.idx = (int32_t)(tbase + l);
            } else {
                p = reinterpret_cast<const SPt<T, D>*>(sm.pts)[l];
            }
            kout[dst] = k;
            pout[dst] = p;
            if (LAST) perm[dst] = p.idx;
        } else {
            timed_out = true;
        }
    }
    if (timed_out) atomicOr(status, (int)DF_TIMEOUT);
}

// iperm[perm[k]] = k: after the last pass, in a pass of its own, so that the
// random 4-byte stores land in a 4n-byte target that L2 holds while nothing
// else streams.  An entry outside [0, n) can only be stale after a look-back
// wait ran out (DF_TIMEOUT is then set already) and is skipped.
__global__ void __launch_bounds__(kSortThreads) k_inverse_perm(const int32_t* __restrict__ perm, int64_t n,
                                                               int32_t* __restrict__ iperm, int* __restrict__ status) {
    pdl_wait();
    pdl_trigger();
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int32_t j = perm[k];
    if ((uint64_t)(uint32_t)j < (uint64_t)n)
        iperm[j] = (int32_t)k;
    else
        atomicOr(status, (int)DF_TIMEOUT);
}

template <class T, int D, class K, bool FIRST, bool LAST>
cudaError_t launch_point_pass(const T* coords, const EncodeParams<T>& ep, const K* kin, const SPt<T, D>* pin, K* kout,
                              SPt<T, D>* pout, int32_t* perm, int64_t n, int pass, int ntiles, uint32_t* scratch,
                              int* status, int64_t spin_limit, int withhold, cudaStream_t s) {
    constexpr size_t smem = point_pass_smem<T, D, K, FIRST>();
    auto kern = k_point_pass<T, D, K, FIRST, LAST>;
    static bool attr_set = false;  // per instantiation
    if (!attr_set) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    launch_pdl(kern, ntiles, kSortThreads, smem, s, coords, ep, kin, pin, kout, pout, perm, n, pass, ntiles,
        scratch, status, spin_limit, withhold);
    return cudaGetLastError();
}

// Sorts the n points of `coords` by Morton key (passes 8-bit digits, 1..8):
// on return keys_out holds the sorted keys, spts the sorted points and perm the
// original index of each sorted position.  kt and ptmp are scratch of n keys /
// points (used when passes > 1); `scratch` holds onesweep_words(n,
// kOnesweepMaxPasses) words.  Launches 1 + passes kernels.
template <class T, int D, class K>
cudaError_t point_sort(const T* coords, const EncodeParams<T>& ep, int64_t n, int passes, K* keys_out, K* kt,
                       SPt<T, D>* spts, SPt<T, D>* ptmp, int32_t* perm, uint32_t* scratch, int* status,
                       int sms, int64_t spin_limit, int withhold, cudaStream_t s, int64_t* launches) {
    const int ntiles = sort_tiles(n);
    cudaError_t e = cudaMemsetAsync(scratch, 0, onesweep_words(n, passes) * 4, s);
    if (e != cudaSuccess) return e;
    const int hblocks = (int)std::min<int64_t>(ntiles, (int64_t)4 * std::max(sms, 1));
    launch_pdl(k_point_counts<T, D, K>, hblocks, kSortThreads, 0, s, coords, n, passes, ep, scratch);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *launches += 1 + passes;
    // Pass p writes the final buffers when passes - 1 - p is even, so the
    // last pass lands in (keys_out, spts).
    auto kb = [&](int p) { return ((passes - 1 - p) & 1) == 0 ? keys_out : kt; };
    auto pb = [&](int p) { return ((passes - 1 - p) & 1) == 0 ? spts : ptmp; };
    if (passes == 1) {
        if ((e = launch_point_pass<T, D, K, true, true>(coords, ep, nullptr, nullptr, keys_out, spts, perm, n, 0,
                                                        ntiles, scratch, status, spin_limit, withhold, s)))
            return e;
    } else {
        if ((e = launch_point_pass<T, D, K, true, false>(coords, ep, nullptr, nullptr, kb(0), pb(0), nullptr, n, 0,
                                                         ntiles, scratch, status, spin_limit, withhold, s)))
            return e;
        for (int p = 1; p < passes - 1; ++p)
            if ((e = launch_point_pass<T, D, K, false, false>(coords, ep, kb(p - 1), pb(p - 1), kb(p), pb(p), nullptr,
                                                              n, p, ntiles, scratch, status, spin_limit,
                                                              withhold, s)))
                return e;
        if ((e = launch_point_pass<T, D, K, false, true>(coords, ep, kb(passes - 2), pb(passes - 2), keys_out, spts,
                                                         perm, n, passes - 1, ntiles, scratch, status,
                                                         spin_limit, withhold, s)))
            return e;
    }
    return cudaGetLastError();
}

}  // namespace oct
