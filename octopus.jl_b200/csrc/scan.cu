// Device-wide exclusive scan, reduce-then-scan in two launches (three above
// kInlineTiles tiles).  No kernel waits on another block, so there is nothing
// to spin on.
#include "scan.cuh"

namespace oct {

// A thread's eight consecutive items, from `first` on (a multiple of eight):
// one 32-byte load and two 32-byte stores where the array starts on such a
// boundary (vec) and the items lie inside it.  Through shared memory and with
// one store per item, the lanes 64 bytes apart, the scan of 1M counts took 21 us,
// now 10.5.
static_assert(kScanItems == 8 && kSmallItems == 8, "");
__device__ __forceinline__ void load_items(const int32_t* in, int64_t first, int64_t n, bool vec,
                                           int32_t* v) {
    if (vec && first + 8 <= n) {
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
            : "l"(in + first)
            : "memory");
    } else {
#pragma unroll
        for (int it = 0; it < 8; ++it) v[it] = first + it < n ? in[first + it] : 0;
    }
}
// out[first + it] = run + the items before it
template <class Out>
__device__ __forceinline__ void store_items(Out* out, int64_t first, int64_t n, bool vec, const int32_t* v,
                                            int64_t run) {
    Out o[8];
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        o[it] = (Out)run;
        run += v[it];
    }
    if (vec && first + 8 <= n) {
        if constexpr (sizeof(Out) == 8) {
#pragma unroll
            for (int h = 0; h < 8; h += 4)
                asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(out + first + h), "l"(o[h]),
                             "l"(o[h + 1]), "l"(o[h + 2]), "l"(o[h + 3])
                             : "memory");
        } else {
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + first), "r"(o[0]),
                         "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                         : "memory");
        }
    } else {
#pragma unroll
        for (int it = 0; it < 8; ++it)
            if (first + it < n) out[first + it] = o[it];
    }
}
__device__ __forceinline__ bool on_32_bytes(const void* p) { return ((uintptr_t)p & 31) == 0; }

// Per-tile sums of kScanTile consecutive inputs.
template <class In>
__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(const In* __restrict__ in, int64_t n,
                                                                 int64_t* __restrict__ tile_sums) {
    pdl_wait();
    pdl_trigger();
    __shared__ int64_t sm[kScanThreads / 32 + 1];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    int64_t s = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) {
        const int64_t i = base + (int64_t)it * kScanThreads + threadIdx.x;
        if (i < n) s += in[i];
    }
    int64_t tot;
    block_exclusive_scan<int64_t>(s, sm, &tot);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

// Exclusive scan of the tile sums by one block, carrying across chunks.
__global__ void __launch_bounds__(1024) k_scan_tiles(int64_t* __restrict__ tile_sums, int64_t ntiles,
                                                     int64_t* __restrict__ d_total) {
    pdl_wait();
    pdl_trigger();
    __shared__ int64_t sm[1024 / 32 + 1];
    int64_t carry = 0;
    for (int64_t base = 0; base < ntiles; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const int64_t v = i < ntiles ? tile_sums[i] : 0;
        int64_t tot;
        const int64_t ex = block_exclusive_scan<int64_t>(v, sm, &tot);
        if (i < ntiles) tile_sums[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0 && d_total) *d_total = carry;
}

// Final pass: each tile scans its items in order (blocked per thread) and
// adds the tile offset.  SUMS: tile_off holds the tiles' sums (not yet
// scanned) and each block adds up those before its own (at most
// kInlineTiles of them, a few loads per thread), so no separate launch scans
// them; the last block also writes the total to *d_total.
template <class In, class Out, bool SUMS>
__global__ void __launch_bounds__(kScanThreads) k_scan_final(const In* in, int64_t n,
                                                             const int64_t* __restrict__ tile_off, Out* out,
                                                             int64_t* __restrict__ d_total) {
    pdl_wait();
    pdl_trigger();
    __shared__ int64_t sm[kScanThreads / 32 + 1];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    const int64_t first = base + (int64_t)threadIdx.x * kScanItems;
    In v[kScanItems];
    load_items(in, first, n, on_32_bytes(in), v);
    int64_t toff;
    if (SUMS) {
        int64_t part = 0;
        for (int j = threadIdx.x; j < (int)blockIdx.x; j += kScanThreads) part += tile_off[j];
        int64_t before;
        block_exclusive_scan<int64_t>(part, sm, &before);
        toff = before;
    } else {
        toff = tile_off[blockIdx.x];
    }
    int64_t s = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) s += v[it];
    int64_t tot;
    const int64_t run = block_exclusive_scan<int64_t>(s, sm, &tot) + toff;
    store_items(out, first, n, on_32_bytes(out), v, run);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        out[n] = (Out)(toff + tot);
        if (SUMS && d_total) *d_total = toff + tot;
    }
}

// Short inputs in one launch of one block, each thread's kSmallItems
// consecutive ones (all read before any is written, so `in` and `out` may
// alias).
template <class In, class Out>
__global__ void __launch_bounds__(kSmallScanThreads) k_scan_small(const In* in, int n, Out* out,
                                                                  int64_t* __restrict__ d_total) {
    pdl_wait();
    pdl_trigger();
    __shared__ int64_t sm[kSmallScanThreads / 32 + 1];
    const int64_t first = (int64_t)threadIdx.x * kSmallItems;
    In v[kSmallItems];
    load_items(in, first, n, on_32_bytes(in), v);
    int64_t sum = 0;
#pragma unroll
    for (int it = 0; it < kSmallItems; ++it) sum += v[it];
    int64_t tot;
    const int64_t run = block_exclusive_scan<int64_t>(sum, sm, &tot);
    store_items(out, first, n, on_32_bytes(out), v, run);
    if (threadIdx.x == 0) {
        out[n] = (Out)tot;
        if (d_total) *d_total = tot;
    }
}

// out[0..n] = exclusive scan of in[0..n-1]; out[n] = total (also *d_total).
// `in` and `out` may alias: each tile's block reads its inputs before it writes.
template <class In, class Out>
int exclusive_scan(const In* in, Out* out, int64_t n, int64_t* d_total, int64_t* tile_tmp, cudaStream_t s) {
    if (n <= 0) {
        cudaMemsetAsync(out, 0, sizeof(Out), s);
        if (d_total) cudaMemsetAsync(d_total, 0, sizeof(int64_t), s);
        return 0;
    }
    if (n <= kSmallScan) {
        launch_pdl(k_scan_small<In, Out>, 1, kSmallScanThreads, 0, s, in, (int)n, out, d_total);
        return 1;
    }
    const int ntiles = div_up(n, kScanTile);
    launch_pdl(k_scan_tile_sums<In>, ntiles, kScanThreads, 0, s, in, n, tile_tmp);
    if (ntiles <= kInlineTiles) {
        launch_pdl(k_scan_final<In, Out, true>, ntiles, kScanThreads, 0, s, in, n, tile_tmp, out, d_total);
        return 2;
    }
    launch_pdl(k_scan_tiles, 1, 1024, 0, s, tile_tmp, ntiles, d_total);
    launch_pdl(k_scan_final<In, Out, false>, ntiles, kScanThreads, 0, s, in, n, tile_tmp, out, nullptr);
    return 3;
}

int exclusive_scan_i32_i64(const int32_t* in, int64_t* out, int64_t n, int64_t* d_total, int64_t* tile_tmp,
                           cudaStream_t s) {
    return exclusive_scan<int32_t, int64_t>(in, out, n, d_total, tile_tmp, s);
}

int exclusive_scan_i32_i32(const int32_t* in, int32_t* out, int64_t n, int64_t* tile_tmp, cudaStream_t s) {
    return exclusive_scan<int32_t, int32_t>(in, out, n, nullptr, tile_tmp, s);
}

}  // namespace oct
