// Preview rendering (src/render.rs:139-308) on the device: the cavity
// cross-section or silhouette from the f64 SDF, then the fluid as
// speed-coloured dots or as the translucent amber pool. Pixels equal the
// reference's, which draws sequentially:
//  * dots: a later particle overwrites an earlier one, so each pixel takes the
//    colour of the highest-index particle whose disk covers it (atomicMax on
//    index + 1, then one colouring pass);
//  * amber: the coverage update cov += (1 - cov) * a is order-dependent in
//    f64, so particles are binned by image tile in index order (the stable
//    counting sort of the particle pipeline) and a block per 8 x 8 pixels
//    merges the nine neighbouring tiles' lists in index order, each pixel
//    applying exactly the reference's sequence of updates.
// The needle overlay is drawn on the host afterwards (a few dozen pixels).
#pragma once
#include "grid.cuh"

namespace sdr {

struct RenderView {
    int hax, vax, oax, flip_v, project, amber;
    double slice, slab;
    double mn[3], mx[3];
    double wm, hm;
    uint32_t w, h;
};

__device__ __forceinline__ double rv_comp(double x, double y, double z, int a) {
    return a == 0 ? x : (a == 1 ? y : z);
}

__device__ __forceinline__ long long rv_as_i64(double f) {  // Rust `as i64`: truncate, saturate, NaN -> 0
    if (isnan(f)) return 0;
    if (f >= 9223372036854775807.0) return 9223372036854775807LL;
    if (f <= -9223372036854775808.0) return (-9223372036854775807LL - 1);
    return (long long)f;
}

__device__ __forceinline__ uint8_t rv_as_u8(double f) {
    if (isnan(f) || f <= 0.0) return 0;
    if (f >= 255.0) return 255;
    return (uint8_t)f;
}

__device__ __forceinline__ double rv_clamp01(double t) { return t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t); }

// to_px (render.rs:181-191)
__device__ __forceinline__ void rv_to_px(const RenderView& v, float4 p, long long& cx, long long& cy) {
    const double a = rv_comp(p.x, p.y, p.z, v.hax), b = rv_comp(p.x, p.y, p.z, v.vax);
    const double fx = dmul(ddiv(dsub(a, v.mn[v.hax]), v.wm), (double)v.w);
    const double fy = v.flip_v ? dmul(ddiv(dsub(v.mx[v.vax], b), v.hm), (double)v.h)
                               : dmul(ddiv(dsub(b, v.mn[v.vax]), v.hm), (double)v.h);
    cx = rv_as_i64(fx);
    cy = rv_as_i64(fy);
}

__device__ __forceinline__ bool rv_in_slab(const RenderView& v, float4 p) {
    return !(fabs(dsub(rv_comp(p.x, p.y, p.z, v.oax), v.slice)) > v.slab);
}

// Background (render.rs:159-178): interior where the SDF is negative on the
// plane, or at any of 96 depths for a projection.
__global__ void k_render_bg(RenderView v, SdfD s, uint8_t* __restrict__ rgb) {
    __shared__ int depth_i[96];
    __shared__ double depth_f[96];
    if (v.project && threadIdx.x < 96) {
        const double lo = v.mn[v.oax], span = fmax(dsub(v.mx[v.oax], v.mn[v.oax]), 1e-9);
        const double d = dadd(lo, dmul(ddiv((double)threadIdx.x + 0.5, 96.0), span));
        int i;
        double f;
        clamp_base_d(ddiv(dsub(d, rv_comp(s.ox, s.oy, s.oz, v.oax)), s.dx), v.oax == 0 ? s.nx : (v.oax == 1 ? s.ny : s.nz), i, f);
        depth_i[threadIdx.x] = i;
        depth_f[threadIdx.x] = f;
    }
    __syncthreads();
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)v.w * v.h) return;
    const uint32_t px = (uint32_t)(q % v.w), py = (uint32_t)(q / v.w);
    // in_plane_world (render.rs:319-338)
    const double wx = dadd(v.mn[v.hax], dmul(ddiv((double)px + 0.5, (double)v.w), v.wm));
    const double fyv = dmul(ddiv((double)py + 0.5, (double)v.h), v.hm);
    const double wy = v.flip_v ? dsub(v.mx[v.vax], fyv) : dadd(v.mn[v.vax], fyv);
    bool interior = false;
    if (v.project) {
        // The samples of a ray differ along one axis only: the grid places of
        // the other two are taken once, those of the 96 depths once per block
        // (shared memory). Sdf::sample with its operations in order
        // (sdf_sample_d): 103 us per 600 px image before, a quarter of it now.
        const double p[3] = {v.hax == 0 ? wx : (v.vax == 0 ? wy : 0.0), v.hax == 1 ? wx : (v.vax == 1 ? wy : 0.0),
                             v.hax == 2 ? wx : (v.vax == 2 ? wy : 0.0)};
        int ia, ib;
        double fa, fb;  // the in-plane axes in x, y, z order
        const int A = v.oax == 0 ? 1 : 0, B = v.oax == 2 ? 1 : 2;
        clamp_base_d(ddiv(dsub(p[A], A == 0 ? s.ox : s.oy), s.dx), A == 0 ? s.nx : s.ny, ia, fa);
        clamp_base_d(ddiv(dsub(p[B], B == 1 ? s.oy : s.oz), s.dx), B == 1 ? s.ny : s.nz, ib, fb);
        for (int k = 0; k < 96 && !interior; ++k) {
            const int io = depth_i[k];
            const double fo = depth_f[k];
            const int i = v.oax == 0 ? io : ia, j = v.oax == 1 ? io : (v.oax == 0 ? ia : ib), l = v.oax == 2 ? io : ib;
            const double fx = v.oax == 0 ? fo : fa, fy = v.oax == 1 ? fo : (v.oax == 0 ? fa : fb), fz = v.oax == 2 ? fo : fb;
            interior = sdf_lerp_d(s, i, j, l, fx, fy, fz) < 0.0;
        }
    } else {
        double c[3] = {0.0, 0.0, 0.0};
        c[v.hax] = wx;
        c[v.vax] = wy;
        c[v.oax] = v.slice;
        interior = sdf_sample_d(s, c[0], c[1], c[2]) < 0.0;
    }
    uint8_t* o = rgb + 3 * q;
    if (interior) {
        o[0] = 232; o[1] = 236; o[2] = 244;
    } else {
        o[0] = 44; o[1] = 44; o[2] = 54;
    }
}

// Peak particle speed (solver.rs:884-890) as the bit pattern of a
// non-negative double, which orders like the value.
__global__ void k_render_max_speed(const float4* __restrict__ vel, uint32_t n, unsigned long long* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    if (i < n) {
        const float4 u = vel[i];
        m = __dsqrt_rn(dadd(dadd(dmul(u.x, u.x), dmul(u.y, u.y)), dmul(u.z, u.z)));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// Speed dots (render.rs:201-221): radius-2 disks; the highest index wins.
__global__ void k_render_dots_mark(RenderView v, const float4* __restrict__ pos, uint32_t n,
                                   uint32_t* __restrict__ owner) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    if (!rv_in_slab(v, p)) return;
    long long cx, cy;
    rv_to_px(v, p, cx, cy);
    for (int dy = -2; dy <= 2; ++dy)
        for (int dx = -2; dx <= 2; ++dx) {
            if (dx * dx + dy * dy > 4) continue;
            const long long x = cx + dx, y = cy + dy;
            if (x < 0 || y < 0 || x >= (long long)v.w || y >= (long long)v.h) continue;
            atomicMax(owner + (size_t)y * v.w + x, i + 1);
        }
}

// speed_color (render.rs:417-428) of the winning particle.
__global__ void k_render_dots_color(RenderView v, const float4* __restrict__ vel, const uint32_t* __restrict__ owner,
                                    const unsigned long long* __restrict__ peak_bits, double vmax,
                                    uint8_t* __restrict__ rgb) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (size_t)v.w * v.h) return;
    const uint32_t o = owner[q];
    if (!o) return;
    const double vm = vmax > 0.0 ? vmax : fmax(__longlong_as_double((long long)*peak_bits), 1e-6);
    const float4 u = vel[o - 1];
    const double sp = __dsqrt_rn(dadd(dadd(dmul(u.x, u.x), dmul(u.y, u.y)), dmul(u.z, u.z)));
    const double t = rv_clamp01(rv_clamp01(ddiv(sp, vm)));
    double r, g, b;
    if (t < 0.5) {
        const double uu = ddiv(t, 0.5);
        r = 0.0; g = uu; b = dsub(1.0, uu);
    } else {
        const double uu = ddiv(dsub(t, 0.5), 0.5);
        r = uu; g = dsub(1.0, uu); b = 0.0;
    }
    uint8_t* c = rgb + 3 * q;
    c[0] = rv_as_u8(dmul(r, 255.0));
    c[1] = rv_as_u8(dmul(g, 255.0));
    c[2] = rv_as_u8(dmul(b, 255.0));
}

// Amber pool, binning: the tile (side T = splat radius) of each particle's
// centre pixel on a grid with one tile of margin; particles outside it (or
// the slab) go to the last bin, which no pixel reads.
__global__ void k_render_amber_keys(RenderView v, const float4* __restrict__ pos, uint32_t n, int T, int ntx,
                                    int nty, uint32_t* __restrict__ key, int2* __restrict__ cxy,
                                    uint32_t* __restrict__ hist) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t dump = (uint32_t)(ntx + 2) * (uint32_t)(nty + 2);
    const float4 p = pos[i];
    uint32_t k = dump;
    if (rv_in_slab(v, p)) {
        long long cx, cy;
        rv_to_px(v, p, cx, cy);
        const long long tx = (cx >= 0 ? cx / T : -((-cx + T - 1) / T)) + 1;
        const long long ty = (cy >= 0 ? cy / T : -((-cy + T - 1) / T)) + 1;
        if (tx >= 0 && ty >= 0 && tx <= ntx + 1 && ty <= nty + 1) {
            k = (uint32_t)(ty * (ntx + 2) + tx);
            cxy[i] = make_int2((int)cx, (int)cy);
        }
    }
    key[i] = k;
    // particles of a warp are near each other: one add per bin and warp
    const unsigned same = __match_any_sync(__activemask(), k);
    if ((int)(threadIdx.x & 31) == __ffs((int)same) - 1) atomicAdd(hist + k, (uint32_t)__popc(same));
}

__device__ __forceinline__ uint8_t rv_lerp(uint8_t a, uint8_t b, double t) {  // lerp_u8, render.rs:311-316
    t = rv_clamp01(t);
    double x = round(dadd(dmul((double)a, dsub(1.0, t)), dmul((double)b, t)));
    x = x < 0.0 ? 0.0 : (x > 255.0 ? 255.0 : x);
    return (uint8_t)x;
}

// Amber pool, compositing (render.rs:261-307): every pixel replays, in
// particle order, the splats of the particles binned in its 3x3 tiles. A block
// takes up to 8 x 8 pixels of a tile: it brings the next kAmTake particles of
// each of the nine lists to shared memory, those below the least last index of
// the lists that go on are the next ones in order, each finds its place by
// binary searches in the other lists, and every pixel walks the merged piece.
// A pixel is done once no splat can change its coverage any more (the update
// rounds to the same value even for the largest a, 0.22). Each pixel merging
// the nine lists by itself from global memory took 18 ms for 2.8 M particles
// on 600 px and 0.56 ms for 77,000. A tile is as wide as a splat's radius, 8 px at
// 600 px of image but 3 below 280, where a block has 9 pixels for its 64 threads and
// still wins: a preview of 77,000 particles takes 351 us at 300 px (663 before), 326
// at 260 (577), 332 at 200 (751) and 1.2 ms at 40 (12.6).
constexpr int kAmPx = 8;              // pixels of a block along each axis
constexpr int kAmBS = kAmPx * kAmPx;  // 64
constexpr int kAmTake = 128;          // particles of each list at a time
constexpr int kAmTable = 1024;        // splat weights by squared distance (radius up to 31 px), else computed

__global__ void __launch_bounds__(kAmBS) k_render_amber_pixels(RenderView v, int r, int T, int ntx,
                                                               const uint32_t* __restrict__ start,
                                                               const uint32_t* __restrict__ perm,
                                                               const int2* __restrict__ cxy, uint8_t* __restrict__ rgb) {
    __shared__ uint32_t s_idx[9][kAmTake];
    __shared__ int s_n[9];
    __shared__ short2 s_xy[9 * kAmTake];
    __shared__ double s_a[kAmTable];
    const int tid = threadIdx.x;
    const int per = (T + kAmPx - 1) / kAmPx;  // blocks of a tile along each axis
    const int tile = blockIdx.x / (per * per), part = blockIdx.x % (per * per);
    const int tx = tile % ntx + 1, ty = tile / ntx + 1;  // with the margin tile
    const int lx = part % per * kAmPx + tid % kAmPx, ly = part / per * kAmPx + tid / kAmPx;
    const int x0 = (tx - 1) * T, y0 = (ty - 1) * T;
    const int x = x0 + lx, y = y0 + ly;
    const bool live = lx < T && ly < T && x < (int)v.w && y < (int)v.h;
    const int rr_i = r * r;
    const double rr = (double)((long long)r * r);
    auto weight = [&](int d2) { return dmul(0.22, dsub(1.0, ddiv((double)d2, rr))); };
    const bool table = rr_i < kAmTable;
    if (table)
        for (int d2 = tid; d2 <= rr_i; d2 += kAmBS) s_a[d2] = weight(d2);
    uint32_t cur[9], end[9];  // the same in every thread
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const uint32_t bin = (uint32_t)(ty + b / 3 - 1) * (uint32_t)(ntx + 2) + (uint32_t)(tx + b % 3 - 1);
        cur[b] = start[bin];
        end[b] = start[bin + 1];
    }
    double cov = 0.0;
    bool done = !live;
    for (;;) {
        uint32_t left = 0, pivot = 0xFFFFFFFFu;
#pragma unroll
        for (int b = 0; b < 9; ++b) {
            left += end[b] - cur[b];
            for (uint32_t q = tid; q < kAmTake && cur[b] + q < end[b]; q += kAmBS) s_idx[b][q] = perm[cur[b] + q];
        }
        if (left == 0) break;
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 9; ++b)
            if (end[b] - cur[b] > (uint32_t)kAmTake) pivot = min(pivot, s_idx[b][kAmTake - 1]);
        if (tid < 9) {  // entries of list tid up to the pivot
            uint32_t c = 0, e = 0;
#pragma unroll
            for (int b = 0; b < 9; ++b)
                if (b == tid) {
                    c = cur[b];
                    e = end[b];
                }
            int lo = 0, hi = (int)min(e - c, (uint32_t)kAmTake);
            while (lo < hi) {
                const int m = (lo + hi) / 2;
                if (s_idx[tid][m] <= pivot) lo = m + 1;
                else hi = m;
            }
            s_n[tid] = lo;
        }
        __syncthreads();
        int total = 0;
#pragma unroll
        for (int b = 0; b < 9; ++b) {
            const int n = s_n[b];
            total += n;
            for (int q = tid; q < n; q += kAmBS) {
                const uint32_t p = s_idx[b][q];
                int at = q;
                for (int o = 0; o < 9; ++o) {
                    if (o == b) continue;
                    int lo = 0, hi = s_n[o];
                    while (lo < hi) {
                        const int m = (lo + hi) / 2;
                        if (s_idx[o][m] < p) lo = m + 1;
                        else hi = m;
                    }
                    at += lo;
                }
                const int2 c = cxy[p];
                s_xy[at] = make_short2((short)(c.x - x0), (short)(c.y - y0));  // within two tiles of this one
            }
            cur[b] += (uint32_t)n;
        }
        __syncthreads();
        if (!done) {
            for (int e = 0; e < total; ++e) {
                const short2 c = s_xy[e];
                const int dx = lx - c.x, dy = ly - c.y, d2 = dx * dx + dy * dy;
                if (d2 > rr_i) continue;
                cov = dadd(cov, dmul(dsub(1.0, cov), table ? s_a[d2] : weight(d2)));
            }
            done = dadd(cov, dmul(dsub(1.0, cov), 0.22)) == cov;
        }
        if (__syncthreads_and(done)) break;
    }
    if (!live) return;
    const size_t q = (size_t)y * v.w + x;
    const double cc = rv_clamp01(cov);
    if (cc <= 1.0 / 255.0) return;
    uint8_t* o = rgb + 3 * q;
    const uint8_t film[3] = {242, 178, 92}, deep[3] = {150, 78, 18};
    for (int k = 0; k < 3; ++k) {
        const uint8_t amber = rv_lerp(film[k], deep[k], cc);
        o[k] = rv_lerp(o[k], amber, cc);
    }
}

}  // namespace sdr
