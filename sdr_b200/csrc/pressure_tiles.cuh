// pcg (src/pressure.rs:341-397) over the whole GPU, for large fluid regions.
//
// The MIC(0) factor (pressure.rs:442-513) and its two triangular sweeps
// (pressure.rs:517-570) are recurrences along i+j+k. Here the grid's (j, k)
// lines are cut into tiles of kTwJ x kTwK lines, one CTA per tile and one
// thread per line. A tile walks the levels L = i+j+k of its cells in order;
// within a level every line has at most one cell (i = L - j - k), whose -x
// predecessor is the thread's own previous cell (a register) and whose -y and
// -z predecessors are the neighbouring lines' cells of level L-1. Those live
// in a shared-memory window of kTwRing levels, one slot per line plus a halo
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
// add 12, multiply 8, barrier of 8 warps 40; 132 for a bare step) and of issue
// slots (two warps per scheduler), so it holds as few instructions as it can.
// A branch per neighbour, 64-bit addresses and the operands' arrival took it to
// about 1,400 cycles. The step now has no branch: a line without a fluid cell
// at a level leaves -0.0 in its slot, and t + (-0.0) is t for every t, so each
// cell adds its three predecessors unconditionally and no neighbour mask is
// read. The operands (residual or forward result, factor, z's places) are rows
// brought to shared memory by the bulk-copy engine, four levels to a copy, and
// each thread reads its own of level s+1 while it computes level s. The loop is
// unrolled over a copy's four levels, so most addresses are a constant away
// from a register (unrolled over the whole window, a step took 700 cycles on
// sweeps of 15 levels: the instructions themselves had to be fetched).
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
// Synchronisation: one cooperative launch (every CTA resident). Phases are
// separated by a grid barrier (an arrival counter and a generation word,
// release/acquire at GPU scope). In a sweep the 8 compute warps of a CTA share
// a named barrier per level; two more warps, one per upstream face, poll the
// upstream tiles' exchange entries and copy their values into the window's
// halo, and one issues the operand copies, so compute threads never wait on a
// global load. Only tiles with fluid cells take a CTA. Every wait gives up
// after about a second (2^31 SM cycles) or as soon as another CTA has given
// up, sets an error bit and lets the kernel wind down. The waits of a level (y
// values, z values, operands) and the published progress belong to three clerk
// warps that join its barrier: one release store or one try_wait on a compute
// warp cost 90 cycles of every other level.
#pragma once
#include "pressure.cuh"

namespace sdr {

constexpr int kTwJ = 16;                     // lines per tile along y
constexpr int kTwK = 16;                     // lines per tile along z
constexpr int kTwLines = kTwJ * kTwK;        // compute threads: one per line
// Threads: the compute warps, a progress warp per upstream face, the operand
// warp, three clerk warps (kTwBarrier threads share a level's barrier), and
// more for the grid-wide phases (24 warps per SM keep enough loads in
// flight; one CTA per SM makes the grid barrier half of what two cost).
constexpr int kTwBS = 768;
constexpr int kTwBarrier = kTwLines + 96;
constexpr int kTwWarps = kTwBS / 32;
constexpr int kTwRing = 16;                  // levels the window holds (a power of two)
constexpr int kTwPitch = kTwJ + 1;           // window slots per line row: the halo, then the tile's lines
constexpr int kTwSlots = (kTwK + 1) * kTwPitch;  // window slots per level
constexpr int kTwDepth = kTwRing;            // levels of operands in shared memory
constexpr int kTwGroup = 4;                  // levels per bulk copy
constexpr int kTwGroups = kTwDepth / kTwGroup;
constexpr long long kTwWaitCycles = 1ll << 31;  // ~1.1 s at 1965 MHz
constexpr uint32_t kTwErrWait = 16u;         // error bit: a sweep or barrier wait gave up
constexpr uint16_t kTwNoCell = 0xFFFFu;      // a row entry without a fluid cell
constexpr int kTwFace = 16;                  // lines of a tile face (either face)
// Levels a progress-warp poll covers: two per load (the half-warps take
// neighbouring levels), kTwPoll loads in flight.
constexpr int kTwPoll = 3;
constexpr int kTwThirds = kTwBS / kTwLines;  // 256-thread groups of a CTA in the matvec
constexpr int kTwBatch = 2 * kTwThirds;      // 256-cell dot tiles of the matvec a CTA has in flight
static_assert(kTwJ == kTwFace && kTwK == kTwFace, "both tile faces hold kTwFace lines");
static_assert((kTwRing & (kTwRing - 1)) == 0, "the window's level is taken by a mask");
static_assert(kTile == kTwLines, "the matvec takes one cell of a dot tile per compute thread");
static_assert(kTwRing * kTwSlots >= kTwBatch * kTile, "the grid-wide phases use the window as scratch");

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
    uint32_t* err;               // error bits
};

// ---------------------------------------------------------------- memory-order helpers
__device__ __forceinline__ unsigned long long ld_acquire_cta_sh(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.cta.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta_sh(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.cta.shared::cta.u64 [%0], %1;" ::"r"(smem_addr(p)), "l"(v) : "memory");
}
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
// Shared-memory accesses at a constant offset from a 32-bit address, in program
// order with the barriers around them.
template <int OFF>
__device__ __forceinline__ double lds_f64(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1+%2];" : "=d"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF>
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF));
    return v;
}
__device__ __forceinline__ void sts_f64(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ bool tw_failed(const TwArgs& t) { return *(volatile uint32_t*)t.err != 0u; }
// Barrier of the compute and clerk warps (named barrier 1).
__device__ __forceinline__ void tw_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kTwBarrier) : "memory"); }

struct TwShared {
    double win[kTwRing * kTwSlots];   // the last levels' values by window slot; scratch of the grid-wide phases
    // operand rows by level of the sweep mod kTwDepth (backward: the levels of a
    // group in decreasing place, as they lie in memory):
    double op_a[kTwDepth][kTwLines];  // residual or forward result,
    double op_b[kTwDepth][kTwLines];  // factor,
    uint32_t op_i[kTwDepth][kTwLines];  // and wavefront index (backward)
    uint64_t op_full[kTwGroups];      // mbarriers: the group's rows have arrived
    unsigned long long avail[2];      // levels (of the sweep) whose y / z neighbour values are in the window
    long long mine;                   // the last level (of the sweep, from 0) whose barrier this tile has passed
    double red[kTwWarps];
    int ok;
    uint8_t m[2][kTwSlots];           // the factorisation's neighbour masks of the last two levels, by window slot
    uint8_t ringm[2][kTwRing][kTwFace];  // the upstream neighbours' masks by level (factorisation)
};
constexpr size_t kTwSmem = sizeof(TwShared);
extern __shared__ __align__(128) unsigned char tw_smem[];
#define TW_SH (*reinterpret_cast<TwShared*>(tw_smem))

// Grid barrier; false if the wait gave up or another CTA has (the error bit is set).
__device__ bool tw_grid_sync(const TwArgs& t) {
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

__device__ __forceinline__ double tw_block_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) TW_SH.red[threadIdx.x >> 5] = v;
    __syncthreads();
    double m = TW_SH.red[0];
    for (int w = 1; w < kTwWarps; ++w) m = fmax(m, TW_SH.red[w]);
    __syncthreads();
    return m;
}

// Maximum over the grid (order-free): CTA maxima through a double-buffered slot array.
__device__ bool tw_grid_max(const TwArgs& t, double v, int& parity, double& out) {
    const double bm = tw_block_max(v);
    double* sl = t.gslots + (size_t)parity * gridDim.x;
    parity ^= 1;
    if (threadIdx.x == 0) sl[blockIdx.x] = bm;
    if (!tw_grid_sync(t)) return false;
    if (threadIdx.x < 32) {
        double m = 0.0;
        for (unsigned q = threadIdx.x; q < gridDim.x; q += 32) m = fmax(m, __ldcg(sl + q));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) TW_SH.red[0] = m;
    }
    __syncthreads();
    out = TW_SH.red[0];
    __syncthreads();
    return true;
}

// Total of the tree-order tile sums (the lane pattern and xor tree of
// pcg_tile_total): the CTA brings them to shared memory, warp 0 adds them.
// One warp loading them from L2 itself took 7 us for the 4,650 sums of a
// 1.19 M-cell pool, twice per iteration.
__device__ double tw_tile_total(const TwArgs& t, uint32_t ntile) {
    double* const scratch = TW_SH.win;
    constexpr uint32_t kChunk = kTwRing * kTwSlots / 32 * 32;
    double s = 0.0;
    for (uint32_t c0 = 0; c0 < ntile; c0 += kChunk) {
        const uint32_t n = min(kChunk, ntile - c0);
        __syncthreads();
        for (uint32_t q = threadIdx.x; q < n; q += kTwBS) scratch[q] = __ldcg(t.a.tpart + c0 + q);
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
__device__ bool tw_exact_dot(const TwArgs& t, double& out) {
    const PcgArgs& a = t.a;
    if (!tw_grid_sync(t)) return false;  // products complete
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
    if (!tw_grid_sync(t)) return false;
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
// Window slots of the sweep's level q.
__device__ __forceinline__ double* tw_win(int q) { return TW_SH.win + (q & (kTwRing - 1)) * kTwSlots; }

// The progress warp of one face (0: y, 1: z) of a tile's sweep: it brings the
// upstream tile's boundary values into the window's halo and publishes how
// many levels are there. The values carry their own readiness: every
// entry of an exchange plane holds kTwEmpty until its producer writes it (the
// planes are filled when the solve lays out its rows), a lane polls the entries
// the next levels need (relaxed loads; lane l takes line l % 16, the upper
// half-warp one level further), and resets each entry it staged to kTwEmpty
// (the producer writes it again only in the next sweep of this direction,
// after a grid barrier). So a hand-off costs the producer's store reaching L2
// and one poll, with no progress flags and no GPU-scope fences. A level needs
// no entry where the producer tile has no level before it (its range is in
// tlo/thi) or the line lies outside the grid: the halo gets -0.0 there. The
// factorisation also stages the upstream cell's neighbour mask from its row.
template <int MODE>
__device__ void tw_progress_warp(const TwArgs& t, int face, int tile, int nb, int s_first, int nlev, int nlevels) {
    constexpr bool fwd = MODE != TW_BACKWARD;
    const int lane = threadIdx.x & 31;
    const int J = tile % t.tj, K = tile / t.tj;
    const int j0 = J * kTwJ, k0 = K * kTwK;
    const int l = lane & 15, half = lane >> 4;
    // this tile's boundary line
    const int jl = face == 0 ? (fwd ? j0 : j0 + kTwJ - 1) : j0 + l;
    const int kl = face == 0 ? k0 + l : (fwd ? k0 : k0 + kTwK - 1);
    const bool line_ok = jl < t.ny && kl < t.nz;
    const int lm = tw_mirror(fwd, l);
    const int slot = face == 0 ? (lm + 1) * kTwPitch : lm + 1;
    // the producer's entries of this line: level q of its sweep at src + q * kTwFace
    double* src = (fwd ? t.exf : t.exb) + (face == 0 ? 0 : t.rows_cap / kTwFace) +
                  (size_t)__ldcg(t.rbase + nb) / kTwFace + (size_t)l;
    // the producer's levels before this tile's level q: its level q - 1 + shift, if within [0, np)
    int np = 0, shift = 0;
    if (line_ok) {
        const int lo = __ldcg(t.tlo + nb), hi = __ldcg(t.thi + nb);
        if (hi >= lo) {
            np = hi - lo + 1;
            shift = s_first - (fwd ? lo : nlevels - 1 - hi);
        }
    }
    src += (ptrdiff_t)(shift - 1) * kTwFace;  // level q's entry: src + q * kTwFace
    // and the upstream cell's word (forward: the producer's last line row or column)
    const uint16_t* const words = t.word + (size_t)__ldcg(t.rbase + nb) + (ptrdiff_t)(shift - 1) * kTwLines +
                                  (face == 0 ? l * kTwJ + kTwJ - 1 : (kTwK - 1) * kTwJ + l);
    int next = 0;  // next level to stage
    const long long t0 = clock64();
    for (unsigned polls = 1; next < nlev; ++polls) {
        const int mine = (int)(long long)ld_acquire_cta_sh(reinterpret_cast<unsigned long long*>(&TW_SH.mine));
        const int lim = min(nlev, mine + kTwRing);  // window room: levels below lim
        // entries of levels next + half, next + 2 + half, ..., loaded at once
        double v[kTwPoll];
        uint16_t mk[kTwPoll];
        bool need[kTwPoll];
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u) {
            const int q = next + 2 * u + half;
            need[u] = q < lim && (unsigned)(q - 1 + shift) < (unsigned)np;
            if (MODE == TW_BUILD) mk[u] = need[u] ? __ldcg(words + (ptrdiff_t)q * kTwLines) : (uint16_t)0;
            v[u] = need[u] ? ld_relaxed_gpu_f64(src + (ptrdiff_t)q * kTwFace) : -0.0;
        }
        int nr = 0;  // levels that are ready, in order: all 16 lines of each
        bool open = true;
#pragma unroll
        for (int u = 0; u < kTwPoll; ++u) {
            const bool ok = next + 2 * u + half < lim &&
                            !(need[u] && __double_as_longlong(v[u]) == (long long)kTwEmpty);
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
        for (int u = 0; u < kTwPoll; ++u) {
            if (2 * u + half < nr) {
                const int q = next + 2 * u + half;
                tw_win(q - 1)[slot] = v[u];
                if (MODE == TW_BUILD) TW_SH.ringm[face][q & (kTwRing - 1)][l] = (uint8_t)mk[u];
            }
        }
        if (nr) {
            __syncwarp();
            if (lane == 0) st_release_cta_sh(&TW_SH.avail[face], (unsigned long long)(next + nr));
#pragma unroll
            for (int u = 0; u < kTwPoll; ++u)
                if (2 * u + half < nr && need[u])
                    st_relaxed_gpu_u64(src + (ptrdiff_t)(next + 2 * u + half) * kTwFace, kTwEmpty);
            next += nr;
        }
        if ((polls & 63u) == 0u && __shfl_sync(0xffffffffu, (int)(tw_failed(t) || clock64() - t0 > kTwWaitCycles), 0)) {
            if (lane == 0) {
                atomicOr(t.err, kTwErrWait);
                st_release_cta_sh(&TW_SH.avail[face], ~0ull >> 1);  // release this tile's compute warps
            }
            break;
        }
    }
}

// The operand warp (one lane): the rows of the sweep's levels, a group per
// bulk copy, completing on the group's mbarrier. A group's place is free once
// the barrier of its old last level has been passed (those operands were read
// before it). Every group is issued even while the kernel winds down (groups
// past the last level arrive without a copy, so that every sweep uses each
// mbarrier equally often), and the compute threads wait for every group, so no
// copy is in flight when the sweep ends.
template <int MODE>
__device__ void tw_operand_warp(const TwArgs& t, size_t row0, int nlev) {
    asm volatile("fence.proxy.async;" ::: "memory");  // the rows were written by ordinary stores
    constexpr bool fwd = MODE != TW_BACKWARD;
    const long long t0 = clock64();
    int passed = -1;
    for (int q = 0; q < nlev || (q & (kTwDepth - 1)) != 0; q += kTwGroup) {
        const uint32_t bar = smem_addr(&TW_SH.op_full[(q / kTwGroup) % kTwGroups]);
        // a group past the last level only waits until its old use has been seen
        const int until = q - kTwDepth + (q < nlev ? kTwGroup - 1 : 0);
        for (unsigned spin = 1; passed < until; ++spin) {
            passed = (int)(long long)ld_acquire_cta_sh(reinterpret_cast<unsigned long long*>(&TW_SH.mine));
            if ((spin & 255u) == 0u && clock64() - t0 > 2 * kTwWaitCycles) {  // cannot happen: every level is passed
                atomicOr(t.err, kTwErrWait);
                return;
            }
        }
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

// A clerk's wait until the window holds the neighbour values of level s;
// returns the levels it holds.
__device__ __forceinline__ int tw_wait(const TwArgs& t, int which, int s) {
    unsigned long long have = ld_acquire_cta_sh(&TW_SH.avail[which]);
    if (have <= (unsigned long long)s) {
        const long long t0 = clock64();
        for (unsigned spin = 1; (have = ld_acquire_cta_sh(&TW_SH.avail[which])) <= (unsigned long long)s; ++spin) {
            if ((spin & 255u) == 0u && (tw_failed(t) || clock64() - t0 > kTwWaitCycles)) {
                atomicOr(t.err, kTwErrWait);
                return INT32_MAX;
            }
        }
    }
    return (int)min(have, (unsigned long long)INT32_MAX);
}

// A clerk warp: it joins the barrier of every level once the level may begin.
// Clerk 0 waits for the y neighbour's values, clerk 1 for the z neighbour's
// and publishes the level passed, clerk 2 waits for the operand group of the
// level after.
template <int MODE>
__device__ void tw_clerk_warp(const TwArgs& t, int clerk, int nb, int nlev, uint32_t parity0) {
    int have = nb >= 0 ? 0 : INT32_MAX;
    for (int q = 0; q < nlev; ++q) {
        if (clerk < 2) {
            if (have <= q) have = tw_wait(t, clerk, q);
        } else if (MODE != TW_BUILD && (q + 1) % kTwGroup == 0 && q + 1 < nlev) {
            tw_op_wait(t, (q + 1) / kTwGroup % kTwGroups, (parity0 + (uint32_t)(q + 1) / kTwDepth) & 1u);
        }
        tw_bar();
        if (clerk == 1 && (threadIdx.x & 31) == 0)
            st_release_cta_sh(reinterpret_cast<unsigned long long*>(&TW_SH.mine), (unsigned long long)(long long)q);
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
template <int MODE>
__device__ __forceinline__ void tw_sweep(const TwArgs& t, int tile, int nlevels, uint32_t& uses) {
    const PcgArgs& a = t.a;
    const int tid = threadIdx.x;
    const int J = tile % t.tj, K = tile / t.tj;
    constexpr bool fwd = MODE != TW_BACKWARD;
    // upstream neighbours of this sweep
    const int nby = fwd ? (J > 0 ? tile - 1 : -1) : (J + 1 < t.tj ? tile + 1 : -1);
    const int nbz = fwd ? (K > 0 ? tile - t.tj : -1) : (K + 1 < t.tk ? tile + t.tj : -1);
    const int lo = __ldcg(t.tlo + tile), hi = __ldcg(t.thi + tile);
    const int s_first = fwd ? lo : nlevels - 1 - hi;  // the sweep's level 0
    const int nlev = hi - lo + 1;
    // window slot of this thread's line; its predecessors are at slot - 1 and slot - kTwPitch
    const int lj = tid % kTwJ, lk = (tid / kTwJ) & (kTwK - 1);
    const int slot = (lk + 1) * kTwPitch + lj + 1;
    if (tid == 0) {
        TW_SH.mine = -1;
        TW_SH.avail[0] = TW_SH.avail[1] = 0ull;
    }
    if (tid < kTwLines) {  // no value before the first level, nor beyond the grid's edge
        tw_win(-1)[slot] = -0.0;
        if (MODE == TW_BUILD) TW_SH.m[1][slot] = 0;
        if (nby < 0)
            TW_SH.win[lj * kTwSlots + (lk + 1) * kTwPitch] = -0.0;  // (level, line) of kTwRing x kTwK
        if (nbz < 0)
            TW_SH.win[lk * kTwSlots + lj + 1] = -0.0;
    }
    __syncthreads();
    const size_t row0 = (size_t)__ldcg(t.rbase + tile);
    const uint32_t parity0 = uses & 1u;
    if (MODE != TW_BUILD) uses += (uint32_t)(nlev + kTwDepth - 1) / kTwDepth;
    if (tid >= kTwLines) {
        const int w = (tid - kTwLines) >> 5;
        if (w < 2) {
            const int nb = w == 0 ? nby : nbz;
            if (nb >= 0) tw_progress_warp<MODE>(t, w, tile, nb, s_first, nlev, nlevels);
        } else if (w == 2) {
            if (MODE != TW_BUILD && tid == kTwLines + 64) tw_operand_warp<MODE>(t, row0, nlev);
        } else if (w < 6) {
            tw_clerk_warp<MODE>(t, w - 3, w == 3 ? nby : w == 4 ? nbz : -1, nlev, parity0);
        }
        __syncthreads();
        return;
    }
    const int line = fwd ? tid : kTwLines - 1 - tid;  // the line this thread takes
    const int j = J * kTwJ + line % kTwJ, k = K * kTwK + line / kTwJ;
    // the lines on the downstream faces write an exchange entry at every level
    // (-0.0 where the line has no fluid cell), so the downstream tile's
    // progress warp finds every entry it polls written; level q's entry of
    // face line l is ex + q * kTwFace
    double* const ex_own = (fwd ? t.exf : t.exb) + row0 / kTwFace;
    const bool in_grid = j < t.ny && k < t.nz;
    const bool on_y = in_grid && lj == kTwJ - 1, on_z = in_grid && lk == kTwK - 1;
    double* ex_y = ex_own + (size_t)(line / kTwJ);
    double* ex_z = ex_own + t.rows_cap / kTwFace + (size_t)(line % kTwJ);
    double carry = -0.0;  // the value of this line's previous cell (the -x / +x predecessor)
    const long long t_loop = a.timing && tid == 0 ? clock64() : 0;
    // Shared-memory addresses: this line's place in the window by level of the
    // ring, as byte offsets from one register.
    constexpr uint32_t kLevel = kTwSlots * 8;
    const uint32_t w_first = smem_addr(TW_SH.win) + (uint32_t)slot * 8;
    uint32_t w = w_first, w_prev = w_first + (kTwRing - 1) * kLevel;
    if (MODE == TW_BUILD) {
        uint8_t carry_m = 0;
        const uint16_t* words = t.word + row0 + line;
        double* pout = t.pc + row0 + line;
        uint16_t wd[kTwGroup], wn[kTwGroup];
#pragma unroll
        for (int u = 0; u < kTwGroup; ++u) wd[u] = u < nlev ? __ldcg(words + u * kTwLines) : kTwNoCell;
        for (int q0 = 0; q0 < nlev; q0 += kTwGroup) {
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
                const double vy = lds_f64<-8>(w_prev), vz = lds_f64<-8 * kTwPitch>(w_prev);
                double pc = -0.0;
                if (wd[u] != kTwNoCell) {
                    const uint8_t my = lj == 0 ? TW_SH.ringm[0][q & (kTwRing - 1)][lk] : TW_SH.m[(u + 1) & 1][slot - 1];
                    const uint8_t mz =
                        lk == 0 ? TW_SH.ringm[1][q & (kTwRing - 1)][lj] : TW_SH.m[(u + 1) & 1][slot - kTwPitch];
                    pc = tw_factor(m, (double)(wd[u] >> 8), carry, carry_m, vy, my, vz, mz);
                }
                sts_f64(w, pc);
                TW_SH.m[u & 1][slot] = wd[u] != kTwNoCell ? m : (uint8_t)0;
                if (on_y) st_relaxed_gpu_f64(ex_y + u * kTwFace, pc);
                if (on_z) st_relaxed_gpu_f64(ex_z + u * kTwFace, pc);
                pout[u * kTwLines] = pc;
                carry = pc;
                carry_m = m;
                w_prev = w;
                w += kLevel;
                if (u == kTwGroup - 1 && w == w_first + kTwRing * kLevel) w = w_first;
            }
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) wd[u] = wn[u];
            pout += kTwGroup * kTwLines;
            ex_y += kTwGroup * kTwFace;
            ex_z += kTwGroup * kTwFace;
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
        double result = 0.0;  // the level before's q or z,
        bool owed = false;    // if the line had a cell there,
        uint32_t at_p = 0u;   // and z's place
        for (int q0 = 0; q0 < nlev; q0 += kTwGroup) {
            // the next group's operands
            const uint32_t gn = (uint32_t)(q0 / kTwGroup + 1) & (kTwGroups - 1);
            const uint32_t on = o_first + gn * (kTwGroup * kRow), oin = oi_first + gn * (kTwGroup * kRow / 2);
            const int left = nlev - q0;
#pragma unroll
            for (int u = 0; u < kTwGroup; ++u) {
                if (u > 0 && u >= left) break;  // the same in every thread
                tw_bar();
                const double vy = lds_f64<-8>(w_prev), vz = lds_f64<-8 * kTwPitch>(w_prev);
                // level q + 1's operands (past the last level: values nobody uses)
                constexpr int kM = kTwGroup - 1;
                const uint32_t os = (u < kM ? o : on) + (uint32_t)(((u + 1) & kM) ^ kRev) * kRow;
                const double ra_n = lds_f64<0>(os), pc_n = lds_f64<kTwDepth * kRow>(os);
                const uint32_t at_n =
                    fwd ? 0u : lds_u32<0>((u < kM ? oi : oin) + (uint32_t)(((u + 1) & kM) ^ kRev) * (kRow / 2));
                // the level before's result goes out while these loads run
                if (MODE == TW_FORWARD) {
                    if (owed) qout[(u - 1) * kTwLines] = result;
                } else if (owed) {
                    a.z[at_p] = result;
                    if (a.exact_dots)  // the reference dot order is over cells in cell order
                        a.prod[a.cinv[at_p]] = dmul(result, __ldcg(a.r + at_p));
                }
                const bool cell = __double2hiint(pc) >= 0;
                double out;
                if (MODE == TW_FORWARD) {
                    // t = r + pq[-x] + pq[-y] + pq[-z]; q = t * pc (pcg_apply_mic0, forward)
                    const double qv = dmul(dadd(dadd(dadd(ra, carry), vy), vz), pc);
                    out = cell ? dmul(pc, qv) : -0.0;
                    result = qv;
                } else {
                    // t = q + pc z[+x] + pc z[+y] + pc z[+z]; z = t * pc (pcg_apply_mic0, backward)
                    const double zv = dmul(dadd(dadd(dadd(ra, dmul(pc, carry)), dmul(pc, vy)), dmul(pc, vz)), pc);
                    out = cell ? zv : -0.0;
                    result = zv;
                    at_p = at;
                }
                sts_f64(w, out);
                owed = cell;
                if (on_y) st_relaxed_gpu_f64(ex_y + u * kTwFace, out);
                if (on_z) st_relaxed_gpu_f64(ex_z + u * kTwFace, out);
                w_prev = w;
                w += kLevel;
                if (u == kTwGroup - 1 && w == w_first + kTwRing * kLevel) w = w_first;
                carry = out;
                ra = ra_n;
                pc = pc_n;
                at = at_n;
            }
            o = on;
            oi = oin;
            qout += kTwGroup * kTwLines;
            ex_y += kTwGroup * kTwFace;
            ex_z += kTwGroup * kTwFace;
        }
        const int last = (nlev - 1) % kTwGroup - kTwGroup;  // qout is a group past the last level's
        if (owed && MODE == TW_FORWARD) qout[last * kTwLines] = result;
        if (owed && MODE == TW_BACKWARD) {
            a.z[at_p] = result;
            if (a.exact_dots) a.prod[a.cinv[at_p]] = dmul(result, __ldcg(a.r + at_p));
        }
    }
    if (MODE != TW_BUILD && a.timing && tid == 0) {  // per tile: level-loop cycles, levels, sweeps
        const unsigned long long loop = (unsigned long long)(clock64() - t_loop);
        atomicAdd(a.timing + 9, loop);
        atomicAdd(a.timing + 10, (unsigned long long)nlev);
        atomicAdd(a.timing + 11, 1ull);
        if (nby < 0 && nbz < 0) {  // a tile that never waits: the bare level step
            atomicAdd(a.timing + 12, loop);
            atomicAdd(a.timing + 13, (unsigned long long)nlev);
        }
    }
    __syncthreads();  // the progress warps have published the final counts and left
}

// Every tile of this CTA: entries blockIdx.x, blockIdx.x + gridDim.x, ... of
// the tile list, in increasing order forward (each tile after its -y and -z
// neighbours) and in decreasing order backward, so waits always point to tiles
// earlier in some CTA's order and the earliest unfinished tile can always run.
template <int MODE>
__device__ bool tw_sweep_all(const TwArgs& t, int nlevels, uint32_t& uses) {
    const int G = (int)gridDim.x, b = (int)blockIdx.x, n = __ldcg(t.tlist);
    if (MODE == TW_BACKWARD) {
        if (b < n)
            for (int q = b + ((n - 1 - b) / G) * G; q >= 0; q -= G) tw_sweep<MODE>(t, __ldcg(t.tlist + 1 + q), nlevels, uses);
    } else {
        for (int q = b; q < n; q += G) tw_sweep<MODE>(t, __ldcg(t.tlist + 1 + q), nlevels, uses);
    }
    return !tw_failed(t);
}

// ---------------------------------------------------------------- the solve
// s*As and As (apply_a, pressure.rs:400-439) of the dot tiles of this CTA: a
// contiguous share, kTwBatch tiles at a time. Each third of the CTA takes
// kTwBatch / 3 of them, a thread one cell of each (their loads are
// independent); the products meet in shared memory and a warp per tile adds
// them in the tree order (lane l: cells l, l+32, ...; then the xor tree).
__device__ void tw_matvec(const TwArgs& t, uint32_t nf, uint32_t ntile) {
    constexpr int kPer = kTwBatch / kTwThirds;
    const PcgArgs& a = t.a;
    double* const scratch = TW_SH.win;
    const uint32_t per = (ntile + gridDim.x - 1) / gridDim.x;
    const uint32_t t0 = min(blockIdx.x * per, ntile), t1 = min(t0 + per, ntile);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int third = threadIdx.x / kTile, tc = threadIdx.x % kTile;
    for (uint32_t tb = t0; tb < t1; tb += kTwBatch) {
        int2 nb[kPer][3];
        double sv[kPer], dg[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t tl = tb + third + q * kTwThirds, i = tl * kTile + tc;
            const bool live = tl < t1 && i < nf;
            const int2* nb2 = reinterpret_cast<const int2*>(a.nbr + (size_t)(live ? i : 0) * 6);
#pragma unroll
            for (int d = 0; d < 3; ++d) nb[q][d] = live ? nb2[d] : make_int2(-1, -1);
            sv[q] = live ? __ldcg(a.s + i) : 0.0;
            dg[q] = live ? (double)a.diag[i] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t tl = tb + third + q * kTwThirds, i = tl * kTile + tc;
            const int nbv[6] = {nb[q][0].x, nb[q][0].y, nb[q][1].x, nb[q][1].y, nb[q][2].x, nb[q][2].y};
            double nsv[6];
#pragma unroll
            for (int d = 0; d < 6; ++d) nsv[d] = nbv[d] >= 0 ? __ldcg(a.s + nbv[d]) : 0.0;
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
        if (w < kTwBatch && tb + w < t1) {
            double acc = 0.0;
#pragma unroll
            for (int u = 0; u < kTile / 32; ++u)
                if ((tb + w) * kTile + u * 32 + lane < nf) acc = dadd(acc, scratch[w * kTile + u * 32 + lane]);
            acc = warp_tree_sum(acc);
            if (lane == 0) a.tpart[tb + w] = acc;
        }
        __syncthreads();
    }
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
        if (lane == 0) a.tpart[tl] = acc;
    }
}

// Launched cooperatively (every CTA resident at once).
__global__ void __launch_bounds__(kTwBS, 1) k_pcg_tiles(TwArgs t) {
    const PcgArgs& a = t.a;
    const uint32_t nf = *a.nf;
    const uint32_t ntile = (nf + kTile - 1) / kTile;
    const uint32_t G = gridDim.x * kTwBS, gt = blockIdx.x * kTwBS + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int nlevels = a.nlevels;
    constexpr int kU = 4;  // cells a thread of the elementwise phases has in flight
    int parity = 0;
    double residual = 0.0, sigma = 0.0, alpha = 0.0;
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
    double mx = 0.0;
    for (uint32_t i = gt; i < nf; i += G) mx = fmax(mx, fabs(a.b[i]));
    for (uint32_t q = gt; q < (uint32_t)t.ntiles; q += G) {
        t.tlo[q] = INT32_MAX;
        t.thi[q] = -1;
    }
    if (!tw_grid_max(t, mx, parity, residual)) goto out;
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
        if (!tw_grid_sync(t)) goto out;
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
                if (n > 0) t.tlist[1 + listed + __popc(some & ((1u << lane) - 1u))] = q;
                listed += __popc(some);
                run += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) {
                t.tlist[0] = listed;
                t.rbase[t.ntiles] = (uint32_t)min(run, (unsigned long long)t.rows_cap);
                if (run > (unsigned long long)t.rows_cap) atomicOr(t.err, kTwErrWait);  // cannot happen: sized per tile
            }
        }
        if (!tw_grid_sync(t)) goto out;
        {  // rows: every entry without a cell, then every cell's entry; every exchange entry unwritten
            const size_t nrow = __ldcg(t.rbase + t.ntiles);
            {
                uint32_t* w2 = reinterpret_cast<uint32_t*>(t.word);  // two entries a store; nrow is a multiple of 256
                for (size_t q = gt; q < nrow / 2; q += G) w2[q] = kTwNoCell | (uint32_t)kTwNoCell << 16;
            }
            const size_t nex = nrow / kTwFace, xf = t.rows_cap / kTwFace;
            unsigned long long* ef = reinterpret_cast<unsigned long long*>(t.exf);
            unsigned long long* eb = reinterpret_cast<unsigned long long*>(t.exb);
            for (size_t q = gt; q < nex; q += G) {
                ef[q] = kTwEmpty;
                ef[xf + q] = kTwEmpty;
                eb[q] = kTwEmpty;
                eb[xf + q] = kTwEmpty;
            }
        }
        if (!tw_grid_sync(t)) goto out;
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
        if (!tw_grid_sync(t)) goto out;
        if (!tw_sweep_all<TW_BUILD>(t, nlevels, uses)) goto out;
        if (!tw_grid_sync(t)) goto out;  // the factor's exchange planes are reused by the sweeps
        TW_SECTION(0);
        if (!tw_sweep_all<TW_FORWARD>(t, nlevels, uses)) goto out;
        if (!tw_sweep_all<TW_BACKWARD>(t, nlevels, uses)) goto out;
        // dot(z, r)
        if (a.exact_dots) {
            if (!tw_exact_dot(t, sigma)) goto out;
        } else {
            if (!tw_grid_sync(t)) goto out;
            tw_dot_zr(t, nf, ntile);
            if (!tw_grid_sync(t)) goto out;
            sigma = tw_tile_total(t, ntile);
        }
        for (uint32_t i = gt; i < nf; i += G) a.s[i] = __ldcg(a.z + i);
        if (!tw_grid_sync(t)) goto out;
        for (int it = 0; it < a.max_iters; ++it) {
            iters = it + 1;
            tw_matvec(t, nf, ntile);
            double denom;  // dot(s, As)
            if (a.exact_dots) {
                if (!tw_exact_dot(t, denom)) goto out;
            } else {
                if (!tw_grid_sync(t)) goto out;
                denom = tw_tile_total(t, ntile);
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
            if (!tw_grid_max(t, mr, parity, residual)) goto out;  // also publishes the residual rows
            TW_SECTION(5);
            if (residual <= a.tol) break;
            if (!tw_sweep_all<TW_FORWARD>(t, nlevels, uses)) goto out;
            if (!tw_sweep_all<TW_BACKWARD>(t, nlevels, uses)) goto out;
            double sigma_new;  // dot(z, r)
            if (a.exact_dots) {
                if (!tw_exact_dot(t, sigma_new)) goto out;
            } else {
                if (!tw_grid_sync(t)) goto out;
                TW_SECTION(1);  // the sweeps end at this barrier
                tw_dot_zr(t, nf, ntile);
                if (!tw_grid_sync(t)) goto out;
                sigma_new = tw_tile_total(t, ntile);
                TW_SECTION(4);
            }
            const double beta = ddiv(sigma_new, sigma);
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
            if (!tw_grid_sync(t)) goto out;  // s complete before the next matvec reads neighbours
            TW_SECTION(6);
            sigma = sigma_new;
        }
        for (uint32_t i = gt; i < nf; i += G)
            a.p_dense[a.lv_cell[i]] = owed ? dadd(a.p[i], dmul(alpha, a.s[i])) : a.p[i];
    }
out:
    TW_SECTION(7);
#undef TW_SECTION
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iters = iters;
        *a.out_residual = residual;
        if (a.timing) a.timing[14] += 1;
    }
}

}  // namespace sdr
