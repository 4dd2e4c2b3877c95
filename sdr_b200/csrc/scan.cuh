// Exclusive prefix sums over u32 arrays (tile = 4096 items per 1024-thread block).
// Used for the counting-sort cell starts, order-preserving particle compaction
// (ParticleSet::retain, src/particles.rs:38-49) and the fluid-cell lists.
#pragma once
#include "common.cuh"

namespace sdr {

constexpr int kScanBS = 1024;
constexpr int kScanIPT = 4;
constexpr int kScanTile = kScanBS * kScanIPT;

// Tiles from which their sums are scanned by a kernel of their own; below, every
// block of the last kernel adds up the sums before it (1,800 to 2,300 tiles, the sort,
// set-up and compaction of a 0.2 mm pool: 876 us against 893 with that kernel).
constexpr uint32_t kScanManyTiles = 4096;
// Tiles up to which there are no sums at all: every block adds up the items before
// its tile. Not in place, where other blocks have overwritten them (one tile apart).
// With two tiles, a 2 mm scene's sort 47 -> 39 us; with fifteen, a jet's, no gain left.
constexpr uint32_t kScanFewTiles = 8;

// A thread's items of a tile, zero past the end.
__device__ __forceinline__ void scan_load(const uint32_t* __restrict__ in, size_t base, uint32_t n, uint32_t (&v)[kScanIPT]) {
    static_assert(kScanIPT == 4, "a 16-byte load");
    if (base + kScanIPT <= n && ((uintptr_t)in & 15) == 0) {
        const uint4 x = *reinterpret_cast<const uint4*>(in + base);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
        return;
    }
#pragma unroll
    for (int q = 0; q < kScanIPT; ++q) v[q] = base + q < n ? in[base + q] : 0u;
}
__device__ __forceinline__ void scan_store(uint32_t* __restrict__ out, size_t base, uint32_t n, const uint32_t (&v)[kScanIPT]) {
    if (base + kScanIPT <= n && ((uintptr_t)out & 15) == 0) {
        *reinterpret_cast<uint4*>(out + base) = make_uint4(v[0], v[1], v[2], v[3]);
        return;
    }
#pragma unroll
    for (int q = 0; q < kScanIPT; ++q)
        if (base + q < n) out[base + q] = v[q];
}

// Block-wide exclusive scan of one value per thread and sum of another: returns
// the scan, the block's total of the values and the sum of `add`.
__device__ __forceinline__ uint32_t block_exscan_u32(uint32_t v, uint32_t add, uint32_t& total, uint32_t& sum) {
    __shared__ uint32_t sh[34], sh_add[kScanBS / 32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (l >= o) x += y;
    }
    add = __reduce_add_sync(0xffffffffu, add);
    if (l == 31) {
        sh[w] = x;
        sh_add[w] = add;
    }
    __syncthreads();
    if (w == 0) {
        const uint32_t s = sh[l], all = __reduce_add_sync(0xffffffffu, sh_add[l]);
        uint32_t t = s;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (l >= o) t += y;
        }
        sh[l] = t - s;  // exclusive warp offsets
        if (l == 31) {
            sh[32] = t;  // block total
            sh[33] = all;
        }
    }
    __syncthreads();
    const uint32_t excl = sh[w] + x - v;
    total = sh[32];
    sum = sh[33];
    __syncthreads();
    return excl;
}

__device__ __forceinline__ void k_scan_tiles_body(VB vb_, const uint32_t* __restrict__ in, uint32_t n,
                                                       uint32_t* __restrict__ tile_sums) {
    uint32_t v[kScanIPT], total, sum;
    scan_load(in, (size_t)vb_.bid * kScanTile + (size_t)threadIdx.x * kScanIPT, n, v);
    block_exscan_u32(0u, v[0] + v[1] + v[2] + v[3], total, sum);
    if (threadIdx.x == 0) tile_sums[vb_.bid] = sum;
}
__global__ void __launch_bounds__(kScanBS) k_scan_tiles(const uint32_t* __restrict__ in, uint32_t n,
                                                       uint32_t* __restrict__ tile_sums) { pdl_begin(); k_scan_tiles_body(VB{blockIdx.x, gridDim.x}, in, n, tile_sums); }

// One block scans all tile sums (exclusive) in order.
__device__ __forceinline__ void k_scan_sums_body(VB vb_, uint32_t* __restrict__ sums, uint32_t nt) {
    uint32_t carry = 0;
    for (uint32_t b = 0; b < nt; b += kScanBS) {
        const uint32_t i = b + threadIdx.x;
        uint32_t tot, none;
        const uint32_t ex = block_exscan_u32(i < nt ? sums[i] : 0u, 0u, tot, none);
        if (i < nt) sums[i] = carry + ex;
        carry += tot;
    }
}
__global__ void __launch_bounds__(kScanBS) k_scan_sums(uint32_t* __restrict__ sums, uint32_t nt) { pdl_begin(); k_scan_sums_body(VB{blockIdx.x, gridDim.x}, sums, nt); }

// A tile of the scan. What comes before it: `sums` scanned, the tiles' sums, or
// (none) the items themselves.
__device__ __forceinline__ void k_scan_apply_body(VB vb_, const uint32_t* in, uint32_t n, const uint32_t* __restrict__ sums,
                                                  int scanned, uint32_t* out, uint32_t* __restrict__ out2,
                                                  uint32_t* __restrict__ total) {
    const size_t base = (size_t)vb_.bid * kScanTile + (size_t)threadIdx.x * kScanIPT;
    uint32_t v[kScanIPT], before = 0;
    scan_load(in, base, n, v);
    if (!sums) {
        for (uint32_t t = 0; t < vb_.bid; ++t) {
            uint32_t x[kScanIPT];
            scan_load(in, (size_t)t * kScanTile + (size_t)threadIdx.x * kScanIPT, n, x);
            before += x[0] + x[1] + x[2] + x[3];
        }
    } else if (!scanned) {
        for (uint32_t t = threadIdx.x; t < vb_.bid; t += kScanBS) before += sums[t];
    } else if (threadIdx.x == 0) {
        before = sums[vb_.bid];
    }
    uint32_t tot, sum;
    uint32_t run = block_exscan_u32(v[0] + v[1] + v[2] + v[3], before, tot, sum) + sum;
#pragma unroll
    for (int q = 0; q < kScanIPT; ++q) {
        const uint32_t x = v[q];
        v[q] = run;
        run += x;
    }
    scan_store(out, base, n, v);
    if (out2) scan_store(out2, base, n, v);
    if (total && vb_.bid + 1 == vb_.nb && threadIdx.x == 0) *total = sum + tot;
}
__global__ void __launch_bounds__(kScanBS) k_scan_apply(const uint32_t* in, uint32_t n, const uint32_t* __restrict__ sums,
                                                        int scanned, uint32_t* out, uint32_t* __restrict__ out2,
                                                        uint32_t* __restrict__ total) { pdl_begin(); k_scan_apply_body(VB{blockIdx.x, gridDim.x}, in, n, sums, scanned, out, out2, total); }

}  // namespace sdr
