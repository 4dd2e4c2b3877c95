// pcg (src/pressure.rs:341-397) over tiles of the grid: on one cluster of SMs for
// small grids, over the whole GPU for large ones. Every solve on a GPU of its own.
//
// The MIC(0) factor (pressure.rs:442-513) and its two triangular sweeps
// (pressure.rs:517-570) are recurrences along i+j+k. Here the grid's (j, k)
// lines are cut into tiles of kTwJ x kTwK lines, one CTA per tile and one
// thread per line. A tile walks the levels L = i+j+k of its cells in order;
// within a level every line has at most one cell (i = L - j - k), whose -x
// predecessor is the thread's own previous cell (a register) and whose -y and
// -z predecessors are the neighbouring lines' cells of level L-1. Those live
// in a shared-memory window of two levels, one slot per line plus a halo
// row and column for the cells of the neighbouring tiles. So a level costs one
// barrier of the tile's threads, and tiles synchronise only with their two
// upstream neighbours through exchange entries that mark their own readiness:
// a tile runs as soon as its neighbours are one level ahead, and a sweep takes
// about (levels x the level step) + (tile hops x the hand-off latency) instead
// of one grid-wide barrier per level. The backward sweep mirrors it (tiles
// wait on their +y / +z neighbours, levels in decreasing order): thread t then
// takes line 255 - t, so both sweeps read the same two slots.
//
// The level step is a chain of latencies (cycles on a B200: shared load 29,
// add 12, multiply 8, barrier of 8 warps 40; a bare step, the window's loads, the
// sums and products, the store and the barrier, takes 103 with 8 or 11 warps at the
// barrier, 146 with the operands' loads and the result's store) and of issue
// slots (two warps per scheduler), so it holds as few instructions as it can. A
// tile that waits for no other takes 290 to 365 a level, the others on average 349
// (a 2 mm scene) to 620 (a 0.4 mm pool) and 825 (0.2 mm).
// A branch per neighbour, 64-bit addresses and the operands' arrival took it to
// about 1,400 cycles. The step now has no branch: a line without a fluid cell
// at a level leaves -0.0 in its slot, and t + (-0.0) is t for every t, so each
// cell adds its three predecessors unconditionally and no neighbour mask is
// read. The operands (residual or forward result, factor, z's places) are rows
// brought to shared memory by the bulk-copy engine, four levels to a copy, and
// each thread reads its own of level s+1 while it computes level s. The loop is
// unrolled over a copy's four levels, so that addresses are a constant away
// from a register (unrolled over 16 levels, a step took 700 cycles on sweeps of
// 15 levels: the instructions themselves had to be fetched).
//
// Per cell the arithmetic is that of k_pcg / k_pcg_cluster (the same operands
// in the same order), so the factor and both sweeps give the same bits, and so
// does the solve: the matvec, the updates and the dots run in the wavefront
// order and tiling of the other kernels, spread over the grid. The sweeps'
// operands live in rows: per tile one row of kTwLines entries per level of its
// range, so a level is contiguous. The update phase writes the residual into
// its row; z goes straight to its place in wavefront order (the cells of a
// tile row are neighbours there too, so a level's stores are runs of 128 bytes).
//
// Synchronisation, grid form: one cooperative launch (every CTA resident),
// phases separated by a grid barrier (an arrival counter and a generation word,
// release/acquire at GPU scope), neighbour values through exchange planes in
// global memory, polled by a progress warp per face. Cluster form, where the
// grid has at most 16 tiles: one thread-block cluster, the hardware barrier,
// neighbour values stored straight into the consumer's shared memory
// (distributed shared memory, about a third of the hand-off through L2). In a
// sweep the 8 compute warps share a named barrier per level with three clerk
// warps, which have the level's y values, z values and operands ready before
// they join: a release store, a try_wait or a poll on a compute warp cost
// 90 cycles of every other level. Only tiles with fluid cells take a CTA.
// Every wait gives up after about a second (2^31 SM cycles) or soon after
// another CTA has given up, sets an error bit and lets the kernel wind down.
#pragma once
#include "pressure.cuh"

namespace sdr {

constexpr int kTwJ = 16;                     // lines per tile along y
constexpr int kTwK = 16;                     // lines per tile along z
constexpr int kTwLines = kTwJ * kTwK;        // compute threads: one per line
// Threads: the compute warps, three clerk warps (kTwBarrier threads share a
// level's barrier), the operand warp, on the grid a progress warp per upstream
// face, and more for
// the grid-wide phases (24 warps per SM keep enough loads in flight; one CTA
// per SM makes the grid barrier half of what two cost).
constexpr int kTwBS = 768;
constexpr int kTwBarrier = kTwLines + 96;
constexpr int kTwWarps = kTwBS / 32;
constexpr int kTwPitch = kTwJ + 1;           // window slots per line row: the halo, then the tile's lines
constexpr int kTwSlots = (kTwK + 1) * kTwPitch;  // window slots per level
constexpr int kTwDepth = 16;                 // levels of operands in shared memory
constexpr int kTwGroup = 4;                  // levels per bulk copy
constexpr int kTwGroups = kTwDepth / kTwGroup;
constexpr int kTwRing = 16;                  // levels of neighbour values staged ahead on the grid (a power of two)
constexpr long long kTwWaitCycles = 1ll << 31;  // ~1.1 s at 1965 MHz
constexpr uint32_t kTwErrWait = 16u;         // error bit: a sweep or barrier wait gave up
constexpr uint16_t kTwNoCell = 0xFFFFu;      // a row entry without a fluid cell
constexpr int kTwFace = 16;                  // lines of a tile face (either face)
// Levels a progress-warp poll covers: two per load (the half-warps take
// neighbouring levels), kTwPoll loads in flight.
constexpr int kTwPoll = 2;
constexpr int kTwThirds = kTwBS / kTwLines;  // 256-thread groups of a CTA in the matvec
constexpr int kTwBatch = 2 * kTwThirds;      // 256-cell dot tiles of the matvec a CTA has in flight
constexpr int kTwScratch = 4096;             // doubles of scratch of the grid-wide phases
constexpr int kTwClusterCtas = 16;           // most tiles the cluster form takes: one per CTA
static_assert(kTwJ == kTwFace && kTwK == kTwFace, "both tile faces hold kTwFace lines");
static_assert((kTwRing & (kTwRing - 1)) == 0, "the ring's level is taken by a mask");
static_assert(kTile == kTwLines, "the matvec takes one cell of a dot tile per compute thread");
static_assert(kTwScratch >= kTwBatch * kTile && kTwScratch % 32 == 0 && kTwScratch <= kTwDepth * kTwLines, "scratch");

struct TwArgs {
    PcgArgs a;                   // wavefront-order vectors, tables and dots (as k_pcg)
    int nx, ny, nz;
    int tj, tk, ntiles;          // tiles along y and z
    // Rows: per tile, one row of kTwLines entries per level of its range
    // (entry = rbase[tile] + (L - tlo[tile]) * kTwLines + line).
    uint16_t* word;              // rows: fluid-neighbour bits (NB_*) | non-solid count << 8, or kTwNoCell
    uint32_t* idx;               // rows: the cell's wavefront index (cells only)
    double* rr;                  // rows: residual (cells only)
    double* pc;                  // rows: MIC(0) factor; -0.0, which no factor is, where there is no cell
    double* qr;                  // rows: forward sweep result (cells only)
    uint32_t* tpos;              // wavefront index -> row entry of its cell
    uint32_t* rbase;             // per tile: its first row entry (ntiles + 1 entries)
    int* tlist;                  // the tiles with fluid cells in increasing order, after their number
    int* trank;                  // per tile: its place in that list (-1: no fluid cell)
    size_t rows_cap;             // row entries allocated
    // Exchange planes, level-major like the rows: a tile's boundary values of
    // its q-th level (sweep order) at rbase[tile] / kTwFace + q * kTwFace + l,
    // l the line along the face; the z face plane follows the y face plane
    // (rows_cap / kTwFace entries each). A level's values are one 128-byte line.
    double* exf;                 // forward sweeps: the +y face, then the +z face
    double* exb;                 // backward sweeps: the -y face, then the -z face
    int* tlo;                    // per tile: first and last level of its fluid cells
    int* thi;
    unsigned* bar;               // grid barrier: [0] arrivals, [1] generation
    double* gslots;              // 2 x gridDim CTA partials of grid maxima
    // Tile sums of the tree-order dots, an array for each of the two dots:
    double* sums_as;             // s*As, written by the matvec
    double* sums_zr;             // z*r, written behind the sweeps
    uint32_t* err;               // error bits
    uint32_t* out_tiles;         // number of tiles with fluid cells
    int plane;                   // cluster form: levels of a halo plane (no tile has more)
};

// ---------------------------------------------------------------- memory-order helpers
// Exchange-plane entries: written and polled with relaxed GPU-scope accesses.
// kTwEmpty is a signalling-NaN pattern no arithmetic produces (IEEE results
// are quiet NaNs), so it can mark an entry not yet written.
constexpr unsigned long long kTwEmpty = 0x7FF4DEADBEEF0001ull;
__device__ __forceinline__ double ld_relaxed_gpu_f64(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu_f64(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_gpu_u64(double* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ bool tw_failed(const TwArgs& t) { return *(volatile uint32_t*)t.err != 0u; }
// Barrier of the compute and clerk warps (named barrier 1).
__device__ __forceinline__ void tw_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kTwBarrier) : "memory"); }

// A tile and its neighbours (-y, +y, -z, +z): level range, first row entry and
// place in the tile list; an empty range where there is no fluid cell or no tile.
struct TwSpan {
    int lo, hi, rank;
    uint32_t row0;
};
struct TwShared {
    double win[2][kTwSlots];          // the last two levels' values by window slot
    // operand rows by level of the sweep mod kTwDepth (backward: the levels of a
    // group in decreasing place, as they lie in memory):
    double op_a[kTwDepth][kTwLines];  // residual or forward result (and scratch of the grid-wide phases),
    double op_b[kTwDepth][kTwLines];  // factor,
    uint32_t op_i[kTwDepth][kTwLines];  // and wavefront index (backward)
    uint64_t op_full[kTwGroups];      // mbarriers: the group's rows have arrived
    double ring[2][kTwRing][kTwFace];  // grid form: the upstream tiles' values by level (kTwEmpty: none yet)
    double red[kTwWarps];
    int ok;
    int passed;                       // the last level of a group whose barrier this tile has passed
    int ntile, first;                 // tiles with fluid cells, and the first of this CTA's
    int tile;                         // the tile `span` describes (-1: none)
    TwSpan span[5];                   // it, then its -y, +y, -z, +z neighbours
    uint8_t m[2][kTwSlots];           // the factorisation's neighbour masks of the last two levels, by window slot
};
// In the cluster form the upstream tiles write their boundary values straight
// into this CTA's halo planes, behind TwShared: [direction][face][level][line].
constexpr size_t kTwSmem = (sizeof(TwShared) + 127) / 128 * 128;
constexpr size_t kTwMaxSmem = 227 * 1024;
constexpr size_t tw_cluster_smem(int plane) { return kTwSmem + (size_t)4 * plane * kTwFace * sizeof(double); }
extern __shared__ __align__(128) unsigned char tw_smem[];
#define TW_SH (*reinterpret_cast<TwShared*>(tw_smem))
__device__ __forceinline__ double* tw_plane(const TwArgs& t, int dir, int face) {
    return reinterpret_cast<double*>(tw_smem + kTwSmem) + (size_t)(dir * 2 + face) * t.plane * kTwFace;
}
__device__ __forceinline__ double* tw_scratch() { return &TW_SH.op_a[0][0]; }
__device__ __forceinline__ double lds_volatile(uint32_t a) {
    double v;
    asm volatile("ld.relaxed.cluster.shared::cta.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts_volatile(uint32_t a, unsigned long long v) {
    asm volatile("st.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ bool tw_empty(double v) { return __double_as_longlong(v) == (long long)kTwEmpty; }

// Barrier over every CTA of the solve. Grid form: false if the wait gave up or
// another CTA has (the error bit is set). Cluster form: the hardware barrier;
// a solve whose sweeps gave up runs on to its end, in step, with the bit set.
template <bool CL>
__device__ bool tw_grid_sync(const TwArgs& t) {
    if (CL) {
        cluster_sync_all();
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned gen = ld_acquire_gpu_u32(t.bar + 1);
        const unsigned arrived = atom_add_acqrel_gpu(t.bar, 1u) + 1u;
        if (arrived == gridDim.x) {
            t.bar[0] = 0u;  // ordered before the release of the next generation
            st_release_gpu_u32(t.bar + 1, gen + 1u);
        } else {
            const long long t0 = clock64();
            while (ld_acquire_gpu_u32(t.bar + 1) == gen) {
                if (tw_failed(t)) {
                    ok = 0;
                    break;
                }
                if (clock64() - t0 > kTwWaitCycles) {
                    atomicOr(t.err, kTwErrWait);
                    ok = 0;
                    break;
                }
            }
        }
        if (ok && tw_failed(t)) ok = 0;  // another CTA gave up: wind down
        TW_SH.ok = ok;
    }
    __syncthreads();
    return TW_SH.ok != 0;
}

// Maximum over a warp of values that are not negative (so ordered like their bits).
__device__ __forceinline__ double tw_warp_max(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)__double2loint(v) : 0u);
    return __hiloint2double((int)mh, (int)ml);
}

// Maximum over the grid (order-free) of values that are not negative: CTA maxima
// through a double-buffered slot array.
template <bool CL>
__device__ bool tw_grid_max(const TwArgs& t, double v, int& parity, double& out) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = tw_warp_max(v);
    if (lane == 0) TW_SH.red[w] = v;
    __syncthreads();
    double* sl = t.gslots + (size_t)parity * gridDim.x;
    parity ^= 1;
    if (w == 0) {
        v = tw_warp_max(lane < kTwWarps ? TW_SH.red[lane] : 0.0);
        if (lane == 0) sl[blockIdx.x] = v;
    }
    if (!tw_grid_sync<CL>(t)) return false;
    if (CL) {  // at most 16: every warp reads them itself
        out = tw_warp_max(lane < (int)gridDim.x ? __ldcg(sl + lane) : 0.0);
        return true;
    }
    if (w == 0) {
        double m = 0.0;
        for (unsigned q = lane; q < gridDim.x; q += 32) m = fmax(m, __ldcg(sl + q));
        m = tw_warp_max(m);
        if (lane == 0) TW_SH.red[0] = m;
    }
    __syncthreads();
    out = TW_SH.red[0];
    __syncthreads();
    return true;
}

// Total of the tree-order tile sums (the lane pattern and xor tree of
// pcg_tile_total): the CTA brings them to shared memory, warp 0 adds them.
// One warp loading them from L2 itself took 7 us for the 4,650 sums of a
// 1.19 M-cell pool, twice per iteration. Where the loads of every warp are few
// (the cluster form's scenes) each adds them itself, without the CTA's barriers.
// Every CTA reads all of the sums, and may be late: between its read and the
// next write of the same array there has to be a barrier of all CTAs. With an
// array per dot the barriers of the other dot are that: sums_as is written by
// the next matvec, behind the barriers of the residual's maximum and around
// the z*r sums; sums_zr behind the next sweeps, after the barrier of the s*As
// sums. (In one array, the cluster form, whose direction has no barrier of its
// own, stored a matvec's sums while a late CTA still read those of z*r.)
__device__ double tw_tile_total(const double* sums, uint32_t ntile) {
    if (gridDim.x * ntile <= 4096) {
        double s = 0.0;
#pragma unroll 4
        for (uint32_t q = threadIdx.x & 31; q < ntile; q += 32) s = dadd(s, __ldcg(sums + q));
        return warp_tree_sum(s);
    }
    double* const scratch = tw_scratch();
    constexpr uint32_t kChunk = kTwScratch;
    double s = 0.0;
    for (uint32_t c0 = 0; c0 < ntile; c0 += kChunk) {
        const uint32_t n = min(kChunk, ntile - c0);
        __syncthreads();
        for (uint32_t q = threadIdx.x; q < n; q += kTwBS) scratch[q] = __ldcg(sums + c0 + q);
        __syncthreads();
        if (threadIdx.x < 32) {
#pragma unroll 8
            for (uint32_t q = threadIdx.x; q < n; q += 32) s = dadd(s, scratch[q]);
        }
    }
    if (threadIdx.x < 32) {
        s = warp_tree_sum(s);
        if (threadIdx.x == 0) TW_SH.red[0] = s;
    }
    __syncthreads();
    const double r = TW_SH.red[0];
    __syncthreads();
    return r;
}

// The reference's chunked dot (pressure.rs:588-603) over `prod` in cell
// order: one warp per 4096-cell chunk across the grid, then the chunk sums in
// chunk order (as pcg_exact_dot).
template <bool CL>
__device__ bool tw_exact_dot(const TwArgs& t, double& out) {
    const PcgArgs& a = t.a;
    if (!tw_grid_sync<CL>(t)) return false;  // products complete
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * kTwWarps + (threadIdx.x >> 5), nw = gridDim.x * kTwWarps;
    for (int ch = gw; ch < a.nchunks; ch += nw) {
        int q = a.chunk_start[ch];
        const int e = a.chunk_start[ch + 1];
        double acc = 0.0;
        for (; q < e; q += 512) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int idx = q + u * 32 + lane;
                v[u] = idx < e ? __ldcg(a.prod + idx) : 0.0;
            }
            const int cnt = min(512, e - q);
#pragma unroll
            for (int u = 0; u < 16; ++u) {
#pragma unroll 8
                for (int src = 0; src < 32; ++src) {
                    const double x = __shfl_sync(0xffffffffu, v[u], src);
                    if (u * 32 + src < cnt) acc = dadd(acc, x);
                }
            }
        }
        if (lane == 0) a.partials[ch] = acc;
    }
    if (!tw_grid_sync<CL>(t)) return false;
    if (threadIdx.x == 0) {
        double s = -0.0;
        for (int ch = 0; ch < a.nchunks; ++ch) s = dadd(s, __ldcg(a.partials + ch));
        TW_SH.red[0] = s;
    }
    __syncthreads();
    out = TW_SH.red[0];
    __syncthreads();
    return true;
}

// ---------------------------------------------------------------- the tile sweeps
enum { TW_BUILD = 0, TW_FORWARD = 1, TW_BACKWARD = 2 };

// Line of window slot order `l` of a face: the backward sweep runs mirrored.
__device__ __forceinline__ int tw_mirror(bool fwd, int l) { return fwd ? l : kTwFace - 1 - l; }

// Which of a tile's levels take values from the upstream tile of a face, and
// from where: level q (of the sweep, from 0) in [qa, qb) takes the upstream
// tile's level q + shift.
struct TwFeed {
    int qa, qb, shift;
    const TwSpan* up;
};
template <int MODE>
__device__ __forceinline__ TwFeed tw_feed(int face) {
    constexpr bool fwd = MODE != TW_BACKWARD;
    const TwSpan& me = TW_SH.span[0];
    TwFeed f;
    f.up = &TW_SH.span[1 + 2 * face + (fwd ? 0 : 1)];
    f.shift = (fwd ? me.lo - f.up->lo : f.up->hi - me.hi) - 1;
    const int nlev = me.hi - me.lo + 1, np = f.up->hi - f.up->lo + 1;
    f.qa = max(0, -f.shift);
    f.qb = np > 0 ? min(nlev, np - f.shift) : 0;
    return f;
}

// Grid form: the progress warp of one face (0: y, 1: z) of a tile's sweep. It
// brings the upstream tile's boundary values into the shared ring, from which
// the face's clerk takes them. The values carry their own readiness: every
// entry of an exchange plane holds kTwEmpty until its producer writes it (the
// planes are filled when the solve lays out its rows), a lane polls the entries
// the next levels need (relaxed loads; lane l takes line l % 16, the upper
// half-warp one level further), and resets each entry it staged to kTwEmpty
// (the producer writes it again only in the next sweep of this direction,
// after a grid barrier). Ring entries work the same way: kTwEmpty until staged,
// and again once the clerk has taken them. So a hand-off costs the producer's
// store reaching L2 and one poll, with no progress flags and no fences.
template <int MODE>
__device__ void tw_progress_warp(const TwArgs& t, int face) {
    constexpr bool fwd = MODE != TW_BACKWARD;
    const TwFeed f = tw_feed<MODE>(face);
    const int lane = threadIdx.x & 31, l = lane & 15, half = lane >> 4;
    const int J = TW_SH.tile % t.tj, K = TW_SH.tile / t.tj;
    const bool line_ok = face == 0 ? K * kTwK + l < t.nz : J * kTwJ + l < t.ny;
    // the upstream tile's entries of this line: level q's at src + q * kTwFace
    double* const src = (fwd ? t.exf : t.exb) + (face == 0 ? 0 : t.rows_cap / kTwFace) + f.up->row0 / kTwFace + l +
                        (ptrdiff_t)f.shift * kTwFace;
    const uint32_t ring = smem_addr(&TW_SH.ring[face][0][l]);
    int next = f.qa;
    const long long t0 = clock64();
    for (unsigned polls = 1; next < f.qb; ++polls) {
        // entries of levels next + half, next + 2 + half, ..., loaded at once
        double v[kTwPoll], room[kTwPoll];
        bool need[kTwPoll];
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u) {
            const int q = next + 2 * u + half;
            need[u] = line_ok && q < f.qb;
            v[u] = need[u] ? ld_relaxed_gpu_f64(src + (ptrdiff_t)q * kTwFace) : -0.0;
        }
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u)
            room[u] = lds_volatile(ring + ((next + 2 * u + half) & (kTwRing - 1)) * (kTwFace * 8));
        int nr = 0;  // levels that are ready and have room, in order: all 16 lines of each
        bool open = true;
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u) {
            const int q = next + 2 * u + half;
            const bool ok = q < f.qb && (!need[u] || (!tw_empty(v[u]) && tw_empty(room[u])));
            const unsigned b = __ballot_sync(0xffffffffu, ok);
            if (open && (b & 0xffffu) == 0xffffu) {
                ++nr;
                open = (b >> 16) == 0xffffu;
                nr += open ? 1 : 0;
            } else {
                open = false;
            }
        }
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u)
            if (2 * u + half < nr && need[u])
                sts_volatile(ring + ((next + 2 * u + half) & (kTwRing - 1)) * (kTwFace * 8),
                             (unsigned long long)__double_as_longlong(v[u]));
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u)
            if (2 * u + half < nr && need[u])
                st_relaxed_gpu_u64(src + (ptrdiff_t)(next + 2 * u + half) * kTwFace, kTwEmpty);
        next += nr;
        if ((polls & 63u) == 0u && __shfl_sync(0xffffffffu, (int)(tw_failed(t) || clock64() - t0 > kTwWaitCycles), 0)) {
            if (lane == 0) atomicOr(t.err, kTwErrWait);  // the clerk gives up by itself
            break;
        }
    }
}

// The clerk of one face: before each level's barrier it puts the upstream
// tile's values of the level into the window's halo (-0.0 where there are
// none: beyond the upstream tile's levels or the grid's edge), from the ring or
// the halo plane, and marks them taken. The wait is bounded; after it has given
// up the halo gets whatever is there. The factorisation's neighbour masks come
// from the upstream tile's rows.
template <int MODE, bool CL>
__device__ void tw_face_clerk(const TwArgs& t, int face) {
    constexpr bool fwd = MODE != TW_BACKWARD;
    const TwFeed f = tw_feed<MODE>(face);
    const int nlev = TW_SH.span[0].hi - TW_SH.span[0].lo + 1;
    const int lane = threadIdx.x & 31, l = lane & 15;
    const int J = TW_SH.tile % t.tj, K = TW_SH.tile / t.tj;
    const bool mine = lane < kTwFace && (face == 0 ? K * kTwK + l < t.nz : J * kTwJ + l < t.ny);
    const int lm = tw_mirror(fwd, l);
    const int slot = face == 0 ? (lm + 1) * kTwPitch : lm + 1;
    const uint32_t halo = smem_addr(&TW_SH.win[0][slot]);
    const uint32_t src = CL ? smem_addr(tw_plane(t, fwd ? 0 : 1, face) + l) : smem_addr(&TW_SH.ring[face][0][l]);
    const uint16_t* const words = t.word + (size_t)f.up->row0 + (ptrdiff_t)f.shift * kTwLines +
                                  (face == 0 ? l * kTwJ + kTwJ - 1 : (kTwK - 1) * kTwJ + l);
    bool given_up = false;
    uint16_t wd[kTwGroup], wn[kTwGroup];
    if (MODE == TW_BUILD) {
#pragma unroll
        for (int u = 0; u < kTwGroup; ++u) wd[u] = mine && u >= f.qa && u < f.qb ? __ldcg(words + u * kTwLines) : 0;
    }
    for (int q0 = 0; q0 < nlev; q0 += kTwGroup) {
        if (MODE == TW_BUILD) {
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) {
                const int q = q0 + kTwGroup + u;
                wn[u] = mine && q >= f.qa && q < f.qb ? __ldcg(words + (ptrdiff_t)q * kTwLines) : 0;
            }
        }
#pragma unroll
        for (int u = 0; u < kTwGroup; ++u) {
            const int q = q0 + u;
            if (u > 0 && q >= nlev) break;
            double v = -0.0;
            if (q >= f.qa && q < f.qb) {
                const uint32_t at = src + (CL ? q : q & (kTwRing - 1)) * (kTwFace * 8);
                if (mine) v = lds_volatile(at);
                if (!given_up && __any_sync(0xffffffffu, tw_empty(v))) {
                    const long long t0 = clock64();
                    for (unsigned spin = 1;; ++spin) {
                        if (mine) v = lds_volatile(at);
                        if (!__any_sync(0xffffffffu, tw_empty(v))) break;
                        if ((spin & 255u) == 0u &&
                            __shfl_sync(0xffffffffu, (int)(tw_failed(t) || clock64() - t0 > kTwWaitCycles), 0)) {
                            if (lane == 0) atomicOr(t.err, kTwErrWait);
                            given_up = true;
                            break;
                        }
                    }
                }
                if (mine) sts_volatile(at, kTwEmpty);
            }
            if (lane < kTwFace) {
                sts_f64(halo + ((u + 1) & 1) * (kTwSlots * 8), v);
                if (MODE == TW_BUILD) TW_SH.m[(u + 1) & 1][slot] = wd[u] == kTwNoCell ? (uint8_t)0 : (uint8_t)wd[u];
            }
            tw_bar();
        }
        if (MODE == TW_BUILD) {
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) wd[u] = wn[u];
        }
    }
}

// Wait until group g of the operands has arrived; parity: of the group's use (bounded).
__device__ __forceinline__ void tw_op_wait(const TwArgs& t, int g, uint32_t parity) {
    const uint32_t bar = smem_addr(&TW_SH.op_full[g]);
    long long t0 = 0;
    for (unsigned spin = 0;; ++spin) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return;
        if (spin == 0) t0 = clock64();
        else if (clock64() - t0 > 2 * kTwWaitCycles) {
            atomicOr(t.err, kTwErrWait);
            return;
        }
    }
}

// The operand warp (one lane): the rows of the sweep's levels, a group per
// bulk copy, completing on the group's mbarrier. A group's place is free once
// the barrier of its last level has been passed (those operands were read
// before it). Groups past the last level arrive without a copy, so that every
// sweep uses each mbarrier equally often. The compute warps and the operand
// clerk wait for every group that has a copy, so none is in flight when the
// sweep ends, also while the kernel winds down.
template <int MODE>
__device__ void tw_operand_warp(const TwArgs& t) {
    constexpr bool fwd = MODE != TW_BACKWARD;
    const int nlev = TW_SH.span[0].hi - TW_SH.span[0].lo + 1;
    const size_t row0 = TW_SH.span[0].row0;
    asm volatile("fence.proxy.async;" ::: "memory");  // the rows were written by ordinary stores
    const long long t0 = clock64();
    int passed = -1;  // levels whose barrier has been passed, told by the operand clerk group by group
    for (int q = 0; q < nlev || (q & (kTwDepth - 1)) != 0; q += kTwGroup) {
        for (unsigned spin = 1; passed < q - kTwDepth + kTwGroup - 1; ++spin) {
            asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(passed) : "r"(smem_addr(&TW_SH.passed)) : "memory");
            if ((spin & 255u) == 0u && clock64() - t0 > 2 * kTwWaitCycles) {  // cannot happen: every level is passed
                atomicOr(t.err, kTwErrWait);
                return;
            }
        }
        const uint32_t bar = smem_addr(&TW_SH.op_full[(q / kTwGroup) % kTwGroups]);
        if (q >= nlev) {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
            continue;
        }
        const int n = min(kTwGroup, nlev - q);
        const int at = (q & (kTwDepth - 1)) + (fwd ? 0 : kTwGroup - n);
        const size_t e = row0 + (size_t)(fwd ? q : nlev - q - n) * kTwLines;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"((uint32_t)(n * kTwLines * (fwd ? 16 : 20)))
                     : "memory");
        auto copy = [&](void* dst, const void* src, uint32_t bytes) {
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_addr(dst)),
                "l"(src), "r"(bytes), "r"(bar)
                : "memory");
        };
        copy(TW_SH.op_a[at], (fwd ? t.rr : t.qr) + e, (uint32_t)(n * kTwLines * 8));
        copy(TW_SH.op_b[at], t.pc + e, (uint32_t)(n * kTwLines * 8));
        if (!fwd) copy(TW_SH.op_i[at], t.idx + e, (uint32_t)(n * kTwLines * 4));
    }
}

// The operand clerk: it joins a level's barrier once the operands of the level
// after it are there, and tells the operand warp of each group passed.
template <int MODE>
__device__ void tw_operand_clerk(const TwArgs& t, uint32_t parity0) {
    const int nlev = TW_SH.span[0].hi - TW_SH.span[0].lo + 1;
    for (int q = 0; q < nlev; ++q) {
        const bool group = MODE != TW_BUILD && (q + 1) % kTwGroup == 0;  // level q ends one
        if (group && q + 1 < nlev)
            tw_op_wait(t, (q + 1) / kTwGroup % kTwGroups, (parity0 + (uint32_t)(q + 1) / kTwDepth) & 1u);
        tw_bar();
        if (group && (threadIdx.x & 31) == 0)
            asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_addr(&TW_SH.passed)), "r"(q) : "memory");
    }
}

// The factor of one cell (build_mic0, pressure.rs:442-513).
__device__ __forceinline__ double tw_factor(uint8_t m, double diag, double pxi, uint8_t mx_, double pyj, uint8_t my_,
                                            double pzk, uint8_t mz_) {
    const double TAU = 0.97, SIGMA = 0.25;
    double axi = 0, axi_y = 0, axi_z = 0, ayj = 0, ayj_x = 0, ayj_z = 0, azk = 0, azk_x = 0, azk_y = 0;
    if (m >> NB_MX & 1) {
        axi = -1.0;
        axi_y = (mx_ >> NB_PY & 1) ? -1.0 : 0.0;
        axi_z = (mx_ >> NB_PZ & 1) ? -1.0 : 0.0;
    } else {
        pxi = 0.0;
    }
    if (m >> NB_MY & 1) {
        ayj = -1.0;
        ayj_x = (my_ >> NB_PX & 1) ? -1.0 : 0.0;
        ayj_z = (my_ >> NB_PZ & 1) ? -1.0 : 0.0;
    } else {
        pyj = 0.0;
    }
    if (m >> NB_MZ & 1) {
        azk = -1.0;
        azk_x = (mz_ >> NB_PX & 1) ? -1.0 : 0.0;
        azk_y = (mz_ >> NB_PY & 1) ? -1.0 : 0.0;
    } else {
        pzk = 0.0;
    }
    const double tx = dmul(axi, pxi), ty = dmul(ayj, pyj), tz = dmul(azk, pzk);
    const double mx = dmul(dmul(dmul(axi, dadd(axi_y, axi_z)), pxi), pxi);
    const double my = dmul(dmul(dmul(ayj, dadd(ayj_x, ayj_z)), pyj), pyj);
    const double mz = dmul(dmul(dmul(azk, dadd(azk_x, azk_y)), pzk), pzk);
    double e = dsub(dsub(dsub(dsub(diag, dmul(tx, tx)), dmul(ty, ty)), dmul(tz, tz)),
                    dmul(TAU, dadd(dadd(mx, my), mz)));
    if (e < dmul(SIGMA, diag)) e = diag;
    return e > 0.0 ? ddiv(1.0, __dsqrt_rn(e)) : 0.0;
}

// One tile's sweep. BUILD: the MIC(0) factor into pc (forward order). FORWARD:
// q = L^-1 r into qr. BACKWARD: z = L^-T q, plus the z*r products in cell
// order for the reference dot order. `uses` counts the rounds of the operand
// ring this CTA has consumed (the same in every thread).
template <int MODE, bool CL>
__device__ __forceinline__ void tw_sweep(const TwArgs& t, int tile, uint32_t& uses) {
    const PcgArgs& a = t.a;
    const int tid = threadIdx.x;
    constexpr bool fwd = MODE != TW_BACKWARD;
    if (TW_SH.tile != tile) {  // the same in every thread; a CTA with one tile comes here once
        __syncthreads();
        if (tid < 5) {
            const int J = tile % t.tj, K = tile / t.tj;
            const int nb = tid == 0   ? tile
                           : tid == 1 ? (J > 0 ? tile - 1 : -1)
                           : tid == 2 ? (J + 1 < t.tj ? tile + 1 : -1)
                           : tid == 3 ? (K > 0 ? tile - t.tj : -1)
                                      : (K + 1 < t.tk ? tile + t.tj : -1);
            TwSpan sp{1, 0, -1, 0u};
            if (nb >= 0 && __ldcg(t.thi + nb) >= __ldcg(t.tlo + nb))
                sp = TwSpan{__ldcg(t.tlo + nb), __ldcg(t.thi + nb), __ldcg(t.trank + nb), __ldcg(t.rbase + nb)};
            TW_SH.span[tid] = sp;
            if (tid == 0) TW_SH.tile = tile;
        }
        __syncthreads();
    }
    const int nlev = TW_SH.span[0].hi - TW_SH.span[0].lo + 1;
    const size_t row0 = TW_SH.span[0].row0;
    // window slot of this thread's line; its predecessors are at slot - 1 and slot - kTwPitch
    const int lj = tid % kTwJ, lk = (tid / kTwJ) & (kTwK - 1);
    const int slot = (lk + 1) * kTwPitch + lj + 1;
    if (tid == 0) TW_SH.passed = -1;
    if (tid < kTwLines) {  // no value before the first level
        TW_SH.win[1][slot] = -0.0;
        if (MODE == TW_BUILD) TW_SH.m[1][slot] = 0;
    }
    __syncthreads();
    const uint32_t parity0 = uses & 1u;
    if (MODE != TW_BUILD) uses += (uint32_t)(nlev + kTwDepth - 1) / kTwDepth;
    if (tid >= kTwLines) {
        const int w = (tid - kTwLines) >> 5;
        if (w < 2) tw_face_clerk<MODE, CL>(t, w);
        else if (w == 2) tw_operand_clerk<MODE>(t, parity0);
        else if (MODE != TW_BUILD && tid == kTwLines + 96) tw_operand_warp<MODE>(t);
        else if (!CL && (w == 4 || w == 5)) tw_progress_warp<MODE>(t, w - 4);
        __syncthreads();
        return;
    }
    const int line = fwd ? tid : kTwLines - 1 - tid;  // the line this thread takes
    const int j = TW_SH.tile % t.tj * kTwJ + line % kTwJ, k = TW_SH.tile / t.tj * kTwK + line / kTwJ;
    // The lines on the downstream faces pass every level's value on where the
    // downstream tile has the level after it (-0.0 where the line has no fluid
    // cell, so every entry that is waited for gets written): into their
    // exchange plane, or into the downstream CTA's halo plane. Level q's entry
    // of face line l is ex + q * kTwFace, for q in [xa, xa + xn).
    const bool in_grid = j < t.ny && k < t.nz;
    const TwSpan& dy = TW_SH.span[fwd ? 2 : 1];
    const TwSpan& dz = TW_SH.span[fwd ? 4 : 3];
    const int sy = fwd ? TW_SH.span[0].lo - dy.lo : dy.hi - TW_SH.span[0].hi;  // level q is its level q + sy
    const int sz = fwd ? TW_SH.span[0].lo - dz.lo : dz.hi - TW_SH.span[0].hi;
    const int ya = max(0, -1 - sy), yn = in_grid && lj == kTwJ - 1 ? max(min(nlev, dy.hi - dy.lo - sy) - ya, 0) : 0;
    const int za = max(0, -1 - sz), zn = in_grid && lk == kTwK - 1 ? max(min(nlev, dz.hi - dz.lo - sz) - za, 0) : 0;
    double *ex_y = nullptr, *ex_z = nullptr;
    uint32_t rx_y = 0u, rx_z = 0u;
    if (CL) {
        auto remote = [&](const TwSpan& d, int face, int l, int sh) {
            const uint32_t own = smem_addr(tw_plane(t, fwd ? 0 : 1, face) + l) + (uint32_t)((sh + 1) * (kTwFace * 8));
            uint32_t r;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(own), "r"(max(d.rank, 0)));
            return r;
        };
        rx_y = remote(dy, 0, line / kTwJ, sy);
        rx_z = remote(dz, 1, line % kTwJ, sz);
    } else {
        double* const ex_own = (fwd ? t.exf : t.exb) + row0 / kTwFace;
        ex_y = ex_own + (size_t)(line / kTwJ);
        ex_z = ex_own + t.rows_cap / kTwFace + (size_t)(line % kTwJ);
    }
    // bit u of the masks: the group's level u is in the range
    auto in_range = [](int q0, int first, int n) -> unsigned {
        const int lo = min(max(first - q0, 0), kTwGroup), hi = min(max(first + n - q0, 0), kTwGroup);
        return (1u << hi) - (1u << lo);
    };
    unsigned my_ = 0u, mz_ = 0u;
    auto pass_on = [&](int u, double v) {
        if (my_ >> u & 1u) {
            if (CL) asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(rx_y + u * (kTwFace * 8)), "d"(v) : "memory");
            else st_relaxed_gpu_f64(ex_y + u * kTwFace, v);
        }
        if (mz_ >> u & 1u) {
            if (CL) asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(rx_z + u * (kTwFace * 8)), "d"(v) : "memory");
            else st_relaxed_gpu_f64(ex_z + u * kTwFace, v);
        }
    };
    auto next_group = [&] {
        if (CL) {
            rx_y += kTwGroup * kTwFace * 8;
            rx_z += kTwGroup * kTwFace * 8;
        } else {
            ex_y += kTwGroup * kTwFace;
            ex_z += kTwGroup * kTwFace;
        }
    };
    double carry = -0.0;  // the value of this line's previous cell (the -x / +x predecessor)
    const long long t_loop = a.timing && tid == 0 ? clock64() : 0;
    const uint32_t w0 = smem_addr(&TW_SH.win[0][slot]);
    constexpr int kWin = kTwSlots * 8;  // level u of a group writes window u % 2 and reads the other
    if (MODE == TW_BUILD) {
        uint8_t carry_m = 0;
        const uint16_t* words = t.word + row0 + line;
        double* pout = t.pc + row0 + line;
        uint16_t wd[kTwGroup], wn[kTwGroup];
#pragma unroll
        for (int u = 0; u < kTwGroup; ++u) wd[u] = u < nlev ? __ldcg(words + u * kTwLines) : kTwNoCell;
        for (int q0 = 0; q0 < nlev; q0 += kTwGroup) {
            my_ = in_range(q0, ya, yn);
            mz_ = in_range(q0, za, zn);
            words += kTwGroup * kTwLines;
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u)
                wn[u] = q0 + kTwGroup + u < nlev ? __ldcg(words + u * kTwLines) : kTwNoCell;
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) {
                const int q = q0 + u;
                if (q >= nlev) break;  // the same in every thread
                const uint8_t m = (uint8_t)wd[u];
                tw_bar();
                const uint32_t wr = w0 + ((u + 1) & 1) * kWin;
                const double vy = lds_f64<-8>(wr), vz = lds_f64<-8 * kTwPitch>(wr);
                double pc = -0.0;
                if (wd[u] != kTwNoCell)
                    pc = tw_factor(m, (double)(wd[u] >> 8), carry, carry_m, vy, TW_SH.m[(u + 1) & 1][slot - 1], vz,
                                   TW_SH.m[(u + 1) & 1][slot - kTwPitch]);
                sts_f64(w0 + (u & 1) * kWin, pc);
                TW_SH.m[u & 1][slot] = wd[u] != kTwNoCell ? m : (uint8_t)0;
                pass_on(u, pc);
                pout[u * kTwLines] = pc;
                carry = pc;
                carry_m = m;
            }
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) wd[u] = wn[u];
            pout += kTwGroup * kTwLines;
            next_group();
        }
    } else {
        tw_op_wait(t, 0, parity0);
        // place of level u's operands within its group (backward: decreasing)
        constexpr int kRev = fwd ? 0 : kTwGroup - 1;
        constexpr uint32_t kRow = kTwLines * 8;  // bytes of a level's row; op_b follows op_a
        const uint32_t o_first = smem_addr(TW_SH.op_a) + (uint32_t)line * 8;
        const uint32_t oi_first = smem_addr(TW_SH.op_i) + (uint32_t)line * 4;
        uint32_t o = o_first, oi = oi_first;
        double ra = lds_f64<kRev * kRow>(o), pc = lds_f64<kRev * kRow + kTwDepth * kRow>(o);
        uint32_t at = fwd ? 0u : lds_u32<kRev * kRow / 2>(oi);
        double* qout = t.qr + row0 + line;
        for (int q0 = 0; q0 < nlev; q0 += kTwGroup) {
            // the next group's operands
            const uint32_t gn = (uint32_t)(q0 / kTwGroup + 1) & (kTwGroups - 1);
            const uint32_t on = o_first + gn * (kTwGroup * kRow), oin = oi_first + gn * (kTwGroup * kRow / 2);
            const int left = nlev - q0;
            my_ = in_range(q0, ya, yn);
            mz_ = in_range(q0, za, zn);
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) {
                if (u > 0 && u >= left) break;  // the same in every thread
                tw_bar();
                const uint32_t wr = w0 + ((u + 1) & 1) * kWin;
                const double vy = lds_f64<-8>(wr), vz = lds_f64<-8 * kTwPitch>(wr);
                const bool cell = __double2hiint(pc) >= 0;
                double out, result;
                if (MODE == TW_FORWARD) {
                    // t = r + pq[-x] + pq[-y] + pq[-z]; q = t * pc (pcg_apply_mic0, forward)
                    result = dmul(dadd(dadd(dadd(ra, carry), vy), vz), pc);
                    out = cell ? dmul(pc, result) : -0.0;
                } else {
                    // t = q + pc z[+x] + pc z[+y] + pc z[+z]; z = t * pc (pcg_apply_mic0, backward)
                    result = dmul(dadd(dadd(dadd(ra, dmul(pc, carry)), dmul(pc, vy)), dmul(pc, vz)), pc);
                    out = cell ? result : -0.0;
                }
                sts_f64(w0 + (u & 1) * kWin, out);
                pass_on(u, out);
                carry = out;
                // off the chain: level q + 1's operands (past the last level values
                // nobody uses) and the result
                constexpr int kM = kTwGroup - 1;
                const uint32_t os = (u < kM ? o : on) + (uint32_t)(((u + 1) & kM) ^ kRev) * kRow;
                ra = lds_f64<0>(os);
                pc = lds_f64<kTwDepth * kRow>(os);
                if (MODE == TW_FORWARD) {
                    if (cell) qout[u * kTwLines] = result;
                } else {
                    if (cell) {
                        a.z[at] = result;
                        if (a.exact_dots)  // the reference dot order is over cells in cell order
                            a.prod[a.cinv[at]] = dmul(result, __ldcg(a.r + at));
                    }
                    at = lds_u32<0>((u < kM ? oi : oin) + (uint32_t)(((u + 1) & kM) ^ kRev) * (kRow / 2));
                }
            }
            o = on;
            oi = oin;
            qout += kTwGroup * kTwLines;
            next_group();
        }
    }
    if (MODE != TW_BUILD && a.timing && tid == 0) {  // per tile: level-loop cycles, levels, sweeps
        const unsigned long long loop = (unsigned long long)(clock64() - t_loop);
        atomicAdd(a.timing + 9, loop);
        atomicAdd(a.timing + 10, (unsigned long long)nlev);
        atomicAdd(a.timing + 11, 1ull);
        if (TW_SH.span[fwd ? 1 : 2].rank < 0 && TW_SH.span[fwd ? 3 : 4].rank < 0) {  // it never waits: the bare level step
            atomicAdd(a.timing + 12, loop);
            atomicAdd(a.timing + 13, (unsigned long long)nlev);
        }
    }
    __syncthreads();  // the clerks and progress warps are done
}

// Every tile of this CTA: entries blockIdx.x, blockIdx.x + gridDim.x, ... of
// the tile list, in increasing order forward (each tile after its -y and -z
// neighbours) and in decreasing order backward, so waits always point to tiles
// earlier in some CTA's order and the earliest unfinished tile can always run.
template <int MODE, bool CL>
__device__ bool tw_sweep_all(const TwArgs& t, uint32_t& uses) {
    const int G = (int)gridDim.x, b = (int)blockIdx.x;
    if (TW_SH.ntile <= G) {  // at most one tile each (always so in the cluster form)
        if (b < TW_SH.ntile) tw_sweep<MODE, CL>(t, TW_SH.first, uses);
        return CL || !tw_failed(t);
    }
    const int n = TW_SH.ntile;
    if (MODE == TW_BACKWARD) {
        if (b < n)
            for (int q = b + ((n - 1 - b) / G) * G; q >= 0; q -= G) tw_sweep<MODE, CL>(t, __ldcg(t.tlist + 1 + q), uses);
    } else {
        for (int q = b; q < n; q += G) tw_sweep<MODE, CL>(t, __ldcg(t.tlist + 1 + q), uses);
    }
    return CL || !tw_failed(t);
}

// ---------------------------------------------------------------- the solve
// s*As and As (apply_a, pressure.rs:400-439) of the dot tiles of this CTA: a
// contiguous share, kTwBatch tiles at a time. Each third of the CTA takes
// kTwBatch / 3 of them, a thread one cell of each (their loads are
// independent); the products meet in shared memory and a warp per tile adds
// them in the tree order (lane l: cells l, l+32, ...; then the xor tree).
// kPer: tiles of a third at a time; of a share of a tile per third one, as the
// places without a tile cost their instructions too.
// TURN: the direction is formed on the way, next = z + beta s for the cell and its
// neighbours, and p takes alpha s: no pass of its own and no barrier behind it,
// for twice the gathers. In the cluster form, where a barrier is a tenth of what is
// between two sweeps (2 mm 340 -> 326 us a solve, 0.5 mm jet 1033 -> 1017); the
// grid form, on an earlier version, lost by it (a 0.2 mm pool 76.8 -> 82.8 ms).
template <int kPer, bool TURN>
__device__ __forceinline__ void tw_matvec_by(const TwArgs& t, uint32_t nf, uint32_t ntile, const double* s, double* next,
                                             double alpha, double beta) {
    constexpr int kBatch = kPer * kTwThirds;
    const PcgArgs& a = t.a;
    double* const scratch = tw_scratch();
    const uint32_t per = (ntile + gridDim.x - 1) / gridDim.x;
    const uint32_t t0 = min(blockIdx.x * per, ntile), t1 = min(t0 + per, ntile);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int third = threadIdx.x / kTile, tc = threadIdx.x % kTile;
    for (uint32_t tb = t0; tb < t1; tb += kBatch) {
        int2 nb[kPer][3];
        double sv[kPer], dg[kPer], zv[kPer], pv[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t tl = tb + third + q * kTwThirds, i = tl * kTile + tc;
            const bool live = tl < t1 && i < nf;
            const int2* nb2 = reinterpret_cast<const int2*>(a.nbr + (size_t)(live ? i : 0) * 6);
#pragma unroll
            for (int d = 0; d < 3; ++d) nb[q][d] = live ? nb2[d] : make_int2(-1, -1);
            sv[q] = live ? __ldcg(s + i) : 0.0;
            if (TURN) {
                zv[q] = live ? __ldcg(a.z + i) : 0.0;
                pv[q] = live ? __ldcg(a.p + i) : 0.0;
            }
            dg[q] = live ? (double)a.diag[i] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t tl = tb + third + q * kTwThirds, i = tl * kTile + tc;
            const int nbv[6] = {nb[q][0].x, nb[q][0].y, nb[q][1].x, nb[q][1].y, nb[q][2].x, nb[q][2].y};
            double nsv[6];
#pragma unroll
            for (int d = 0; d < 6; ++d) nsv[d] = nbv[d] >= 0 ? __ldcg(s + nbv[d]) : 0.0;
            if (TURN) {
                double nz[6];
#pragma unroll
                for (int d = 0; d < 6; ++d) nz[d] = nbv[d] >= 0 ? __ldcg(a.z + nbv[d]) : 0.0;
#pragma unroll
                for (int d = 0; d < 6; ++d) nsv[d] = dadd(nz[d], dmul(beta, nsv[d]));
                if (tl < t1 && i < nf) a.p[i] = dadd(pv[q], dmul(alpha, sv[q]));
                sv[q] = dadd(zv[q], dmul(beta, sv[q]));
                if (tl < t1 && i < nf) next[i] = sv[q];
            }
            double v = dmul(dg[q], sv[q]);
            v = nbv[NB_PX] >= 0 ? dsub(v, nsv[NB_PX]) : v;
            v = nbv[NB_MX] >= 0 ? dsub(v, nsv[NB_MX]) : v;
            v = nbv[NB_PY] >= 0 ? dsub(v, nsv[NB_PY]) : v;
            v = nbv[NB_MY] >= 0 ? dsub(v, nsv[NB_MY]) : v;
            v = nbv[NB_PZ] >= 0 ? dsub(v, nsv[NB_PZ]) : v;
            v = nbv[NB_MZ] >= 0 ? dsub(v, nsv[NB_MZ]) : v;
            if (tl < t1 && i < nf) {
                a.as[i] = v;
                if (a.exact_dots) a.prod[a.cinv[i]] = dmul(sv[q], v);
            }
            scratch[(tl - tb) * kTile + tc] = dmul(sv[q], v);
        }
        if (a.exact_dots) continue;
        __syncthreads();
        if (w < kBatch && tb + w < t1) {
            double acc = 0.0;
#pragma unroll
            for (int u = 0; u < kTile / 32; ++u)
                if ((tb + w) * kTile + u * 32 + lane < nf) acc = dadd(acc, scratch[w * kTile + u * 32 + lane]);
            acc = warp_tree_sum(acc);
            if (lane == 0) t.sums_as[tb + w] = acc;
        }
        __syncthreads();
    }
}

template <bool TURN>
__device__ __forceinline__ void tw_matvec(const TwArgs& t, uint32_t nf, uint32_t ntile, const double* s, double* next,
                                          double alpha, double beta) {
    if (ntile <= kTwThirds * gridDim.x) tw_matvec_by<1, TURN>(t, nf, ntile, s, next, alpha, beta);
    else tw_matvec_by<kTwBatch / kTwThirds, TURN>(t, nf, ntile, s, next, alpha, beta);
}

// dot(z, r) by the tiles of the tree order, a warp per tile.
__device__ __forceinline__ void tw_dot_zr(const TwArgs& t, uint32_t nf, uint32_t ntile) {
    const PcgArgs& a = t.a;
    const int lane = threadIdx.x & 31;
    for (uint32_t tl = blockIdx.x * kTwWarps + (threadIdx.x >> 5); tl < ntile; tl += gridDim.x * kTwWarps) {
        double zv[kTile / 32], rv[kTile / 32];
#pragma unroll
        for (int u = 0; u < kTile / 32; ++u) {
            const uint32_t i = tl * kTile + lane + 32u * u;
            zv[u] = i < nf ? __ldcg(a.z + i) : 0.0;
            rv[u] = i < nf ? __ldcg(a.r + i) : 0.0;
        }
        double acc = 0.0;
#pragma unroll
        for (int u = 0; u < kTile / 32; ++u)
            if (tl * kTile + lane + 32u * u < nf) acc = dadd(acc, dmul(zv[u], rv[u]));
        acc = warp_tree_sum(acc);
        if (lane == 0) t.sums_zr[tl] = acc;
    }
}

template <bool CL>
__device__ __forceinline__ void tw_solve(const TwArgs& t) {
    const PcgArgs& a = t.a;
    const uint32_t nf = *a.nf;
    const uint32_t ntile = (nf + kTile - 1) / kTile;
    const uint32_t G = gridDim.x * kTwBS, gt = blockIdx.x * kTwBS + threadIdx.x;
    const int lane = threadIdx.x & 31;
    constexpr int kU = 4;  // cells a thread of the elementwise phases has in flight
    int parity = 0;
    double residual = 0.0, sigma = 0.0, alpha = 0.0, beta = 0.0;
    double *s = a.s, *next = a.q;  // the cluster form turns the direction from one to the other
    bool owed = false;  // p has not had the last step's alpha * s
    // phase timers of CTA 0 (between grid barriers every CTA passes together)
    const bool timed = a.timing != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
    long long tck = timed ? clock64() : 0;
#define TW_SECTION(idx)                                              \
    do {                                                             \
        if (timed) {                                                 \
            const long long now_ = clock64();                        \
            atomicAdd(a.timing + (idx), (unsigned long long)(now_ - tck)); \
            tck = now_;                                              \
        }                                                            \
    } while (0)
    int iters = 0;
    uint32_t uses = 0;  // rounds of the operand ring consumed (phases of op_full)
    if (threadIdx.x < kTwGroups)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&TW_SH.op_full[threadIdx.x])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");  // before the first barrier below
    if (threadIdx.x == 0) TW_SH.tile = -1;
    if (CL) {  // nobody's values yet (before the barriers of the set-up)
        unsigned long long* const pl = reinterpret_cast<unsigned long long*>(tw_plane(t, 0, 0));
        for (int q = threadIdx.x; q < 4 * t.plane * kTwFace; q += kTwBS) pl[q] = kTwEmpty;
    } else if (threadIdx.x < 2 * kTwRing * kTwFace) {
        reinterpret_cast<unsigned long long*>(TW_SH.ring)[threadIdx.x] = kTwEmpty;
    }
    double mx = 0.0;
    for (uint32_t i = gt; i < nf; i += G) mx = fmax(mx, fabs(a.b[i]));
    for (uint32_t q = gt; q < (uint32_t)t.ntiles; q += G) {
        t.tlo[q] = INT32_MAX;
        t.thi[q] = -1;
    }
    if (!tw_grid_max<CL>(t, mx, parity, residual)) goto out;
    if (residual > a.tol) {
        // r and p, and the tiles' level ranges
        for (uint32_t i = gt; i < nf; i += G) {
            const uint32_t cell = a.lv_cell[i];
            const int ii = (int)(cell % (uint32_t)t.nx), jj = (int)((cell / (uint32_t)t.nx) % (uint32_t)t.ny),
                      kk = (int)(cell / ((uint32_t)t.nx * (uint32_t)t.ny));
            a.r[i] = a.b[i];
            a.p[i] = 0.0;
            const int tile = jj / kTwJ + (kk / kTwK) * t.tj;
            atomicMin(t.tlo + tile, ii + jj + kk);
            atomicMax(t.thi + tile, ii + jj + kk);
        }
        if (!tw_grid_sync<CL>(t)) goto out;
        // each tile's first row entry: a prefix over the tiles' level counts (one warp)
        if (blockIdx.x == 0 && threadIdx.x < 32) {
            unsigned long long run = 0;
            int listed = 0;
            for (int b0 = 0; b0 < t.ntiles; b0 += 32) {
                const int q = b0 + lane;
                unsigned long long n = 0;
                if (q < t.ntiles) {
                    const int lo = __ldcg(t.tlo + q), hi = __ldcg(t.thi + q);
                    n = hi >= lo ? (unsigned long long)(hi - lo + 1) * kTwLines : 0ull;
                }
                unsigned long long x = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (q < t.ntiles) t.rbase[q] = (uint32_t)(run + x - n);
                const unsigned some = __ballot_sync(0xffffffffu, n > 0);
                const int at = listed + __popc(some & ((1u << lane) - 1u));
                if (n > 0) t.tlist[1 + at] = q;
                if (q < t.ntiles) t.trank[q] = n > 0 ? at : -1;
                listed += __popc(some);
                run += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) {
                t.tlist[0] = listed;
                *t.out_tiles = (uint32_t)listed;
                t.rbase[t.ntiles] = (uint32_t)min(run, (unsigned long long)t.rows_cap);
                if (run > (unsigned long long)t.rows_cap) atomicOr(t.err, kTwErrWait);  // cannot happen: sized per tile
            }
        }
        if (!tw_grid_sync<CL>(t)) goto out;
        {  // rows: every entry without a cell, then every cell's entry; every exchange entry unwritten
            const size_t nrow = __ldcg(t.rbase + t.ntiles);
            {
                uint32_t* w2 = reinterpret_cast<uint32_t*>(t.word);  // two entries a store; nrow is a multiple of 256
                for (size_t q = gt; q < nrow / 2; q += G) w2[q] = kTwNoCell | (uint32_t)kTwNoCell << 16;
            }
            if (threadIdx.x == 0) {
                TW_SH.ntile = __ldcg(t.tlist);
                TW_SH.first = (int)blockIdx.x < TW_SH.ntile ? __ldcg(t.tlist + 1 + blockIdx.x) : -1;
            }
            const size_t nex = nrow / kTwFace, xf = t.rows_cap / kTwFace;
            unsigned long long* ef = reinterpret_cast<unsigned long long*>(t.exf);
            unsigned long long* eb = reinterpret_cast<unsigned long long*>(t.exb);
            for (size_t q = gt; !CL && q < nex; q += G) {
                ef[q] = kTwEmpty;
                ef[xf + q] = kTwEmpty;
                eb[q] = kTwEmpty;
                eb[xf + q] = kTwEmpty;
            }
        }
        if (!tw_grid_sync<CL>(t)) goto out;
        for (uint32_t i = gt; i < nf; i += G) {
            const uint32_t cell = a.lv_cell[i];
            const int ii = (int)(cell % (uint32_t)t.nx), jj = (int)((cell / (uint32_t)t.nx) % (uint32_t)t.ny),
                      kk = (int)(cell / ((uint32_t)t.nx * (uint32_t)t.ny));
            const int tile = jj / kTwJ + (kk / kTwK) * t.tj;
            const size_t e = (size_t)__ldcg(t.rbase + tile) +
                             (size_t)(ii + jj + kk - __ldcg(t.tlo + tile)) * kTwLines +
                             (size_t)((kk % kTwK) * kTwJ + jj % kTwJ);
            if (e >= t.rows_cap) continue;  // cannot happen: the ranges were sized above
            t.word[e] = (uint16_t)(a.nmask[i] | a.diag[i] << 8);
            t.idx[e] = i;
            t.rr[e] = a.b[i];
            t.tpos[i] = (uint32_t)e;
        }
        if (!tw_grid_sync<CL>(t)) goto out;
        if (!tw_sweep_all<TW_BUILD, CL>(t, uses)) goto out;
        if (!tw_grid_sync<CL>(t)) goto out;  // the factor's exchange planes are reused by the sweeps
        TW_SECTION(0);
        if (!tw_sweep_all<TW_FORWARD, CL>(t, uses)) goto out;
        if (!tw_sweep_all<TW_BACKWARD, CL>(t, uses)) goto out;
        // dot(z, r)
        if (a.exact_dots) {
            if (!tw_exact_dot<CL>(t, sigma)) goto out;
        } else {
            if (!tw_grid_sync<CL>(t)) goto out;
            tw_dot_zr(t, nf, ntile);
            if (!tw_grid_sync<CL>(t)) goto out;
            sigma = tw_tile_total(t.sums_zr, ntile);
        }
        for (uint32_t i = gt; i < nf; i += G) a.s[i] = __ldcg(a.z + i);
        if (!tw_grid_sync<CL>(t)) goto out;
        for (int it = 0; it < a.max_iters; ++it) {
            iters = it + 1;
            if (CL && it > 0) {
                tw_matvec<true>(t, nf, ntile, s, next, alpha, beta);
                double* const x = s;
                s = next;
                next = x;
                owed = false;
            } else {
                tw_matvec<false>(t, nf, ntile, s, nullptr, 0.0, 0.0);
            }
            double denom;  // dot(s, As)
            if (a.exact_dots) {
                if (!tw_exact_dot<CL>(t, denom)) goto out;
            } else {
                if (!tw_grid_sync<CL>(t)) goto out;
                denom = tw_tile_total(t.sums_as, ntile);
            }
            TW_SECTION(3);
            if (fabs(denom) < 1e-30) break;
            alpha = ddiv(sigma, denom);
            double mr = 0.0;
            for (uint32_t i0 = gt; i0 < nf; i0 += kU * G) {
                double rv[kU], av[kU];
                uint32_t e[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const uint32_t i = i0 + u * G;
                    rv[u] = i < nf ? a.r[i] : 0.0;  // this thread's own store
                    av[u] = i < nf ? __ldcg(a.as + i) : 0.0;
                    e[u] = i < nf ? t.tpos[i] : 0u;
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const uint32_t i = i0 + u * G;
                    if (i >= nf) break;
                    const double nr = dsub(rv[u], dmul(alpha, av[u]));
                    a.r[i] = nr;
                    t.rr[e[u]] = nr;
                    mr = fmax(mr, fabs(nr));
                }
            }
            owed = true;  // p takes alpha * s with the next direction, which reads s too
            if (!tw_grid_max<CL>(t, mr, parity, residual)) goto out;  // also publishes the residual rows
            TW_SECTION(5);
            if (residual <= a.tol) break;
            if (!tw_sweep_all<TW_FORWARD, CL>(t, uses)) goto out;
            if (!tw_sweep_all<TW_BACKWARD, CL>(t, uses)) goto out;
            double sigma_new;  // dot(z, r)
            if (a.exact_dots) {
                if (!tw_exact_dot<CL>(t, sigma_new)) goto out;
            } else {
                if (!tw_grid_sync<CL>(t)) goto out;
                TW_SECTION(1);  // the sweeps end at this barrier
                tw_dot_zr(t, nf, ntile);
                if (!tw_grid_sync<CL>(t)) goto out;
                sigma_new = tw_tile_total(t.sums_zr, ntile);
                TW_SECTION(4);
            }
            beta = ddiv(sigma_new, sigma);
            sigma = sigma_new;
            if (!CL) {  // in the cluster form the next matvec turns s
                for (uint32_t i0 = gt; i0 < nf; i0 += kU * G) {
                    double sv[kU], pv[kU], zv[kU];
#pragma unroll
                    for (int u = 0; u < kU; ++u) {
                        const uint32_t i = i0 + u * G;
                        sv[u] = i < nf ? a.s[i] : 0.0;
                        pv[u] = i < nf ? a.p[i] : 0.0;
                        zv[u] = i < nf ? __ldcg(a.z + i) : 0.0;
                    }
#pragma unroll
                    for (int u = 0; u < kU; ++u) {
                        const uint32_t i = i0 + u * G;
                        if (i >= nf) break;
                        a.p[i] = dadd(pv[u], dmul(alpha, sv[u]));
                        a.s[i] = dadd(zv[u], dmul(beta, sv[u]));
                    }
                }
                owed = false;
                if (!tw_grid_sync<CL>(t)) goto out;  // s complete before the next matvec reads neighbours
                TW_SECTION(6);
            }
        }
        if (CL) pdl_next();
        for (uint32_t i = gt; i < nf; i += G)
            a.p_dense[a.lv_cell[i]] = owed ? dadd(__ldcg(a.p + i), dmul(alpha, __ldcg(s + i))) : __ldcg(a.p + i);
    }
out:
    TW_SECTION(7);
#undef TW_SECTION
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iters = iters;
        *a.out_residual = residual;
        if (a.timing) a.timing[14] += 1;
    }
    if (CL) cluster_sync_all();  // no CTA leaves while another may still write into its planes
}

// Launched cooperatively (every CTA resident at once), at most one CTA per SM.
__global__ void __launch_bounds__(kTwBS, 1) k_pcg_tiles(TwArgs t) { tw_solve<false>(t); }
// Launched as one cluster with a CTA per tile of the grid.
__global__ void __launch_bounds__(kTwBS, 1) k_pcg_tiles_cluster(TwArgs t) {
    pdl_wait();
    tw_solve<true>(t);
}

}  // namespace sdr
