// Grid-side kernels: static cavity mask and base labels (solver.rs:184-222,
// 342-361), velocity extrapolation (solver.rs:608-647, 960-1009) and the
// face max-reduction behind cfl_dt (grid.rs:202-206).
#pragma once
#include "common.cuh"
#include "particles.cuh"

namespace sdr {

// Sdf::sample (sdf.rs:134-166) in f64 with the reference's operation order.
__device__ __forceinline__ void clamp_base_d(double g, int n, int& i, double& f) {
    if (g <= 0.0) {
        i = 0;
        f = 0.0;
    } else if (g >= (double)(n - 1)) {
        i = n - 2;
        f = 1.0;
    } else {
        double fl = floor(g);
        i = (int)fl;
        f = dsub(g, fl);
    }
}

struct SdfD {
    int nx, ny, nz;
    double dx, ox, oy, oz;
    const double* data;
};

__device__ __forceinline__ double sdf_lerp_d(const SdfD& s, int i, int j, int k, double fx, double fy, double fz) {
    auto at = [&](int a, int b, int c) { return s.data[((size_t)c * s.ny + b) * s.nx + a]; };
    double gx = dsub(1.0, fx), gy = dsub(1.0, fy), gz = dsub(1.0, fz);
    double c00 = dadd(dmul(at(i, j, k), gx), dmul(at(i + 1, j, k), fx));
    double c10 = dadd(dmul(at(i, j + 1, k), gx), dmul(at(i + 1, j + 1, k), fx));
    double c01 = dadd(dmul(at(i, j, k + 1), gx), dmul(at(i + 1, j, k + 1), fx));
    double c11 = dadd(dmul(at(i, j + 1, k + 1), gx), dmul(at(i + 1, j + 1, k + 1), fx));
    double c0 = dadd(dmul(c00, gy), dmul(c10, fy));
    double c1 = dadd(dmul(c01, gy), dmul(c11, fy));
    return dadd(dmul(c0, gz), dmul(c1, fz));
}
__device__ __forceinline__ double sdf_sample_d(const SdfD& s, double px, double py, double pz) {
    double lx = ddiv(dsub(px, s.ox), s.dx), ly = ddiv(dsub(py, s.oy), s.dx),
           lz = ddiv(dsub(pz, s.oz), s.dx);
    int i, j, k;
    double fx, fy, fz;
    clamp_base_d(lx, s.nx, i, fx);
    clamp_base_d(ly, s.ny, j, fy);
    clamp_base_d(lz, s.nz, k, fz);
    return sdf_lerp_d(s, i, j, k, fx, fy, fz);
}

// cavity_mask (solver.rs:194-199) and the static half of classify
// (solver.rs:344-361): outlet cells are Air, non-cavity Solid, the rest Air.
__device__ __forceinline__ void k_cavity_and_base_body(VB vb_, Grid g, SdfD s, int has_outlet, Aabb outlet,
                                  uint8_t* __restrict__ cavity, uint8_t* __restrict__ base,
                                  int recompute_cavity) {
    size_t c = (size_t)vb_.bid * blockDim.x + threadIdx.x;
    size_t n = (size_t)g.nx * g.ny * g.nz;
    if (c >= n) return;
    int i = c % g.nx, j = (c / g.nx) % g.ny, k = c / ((size_t)g.nx * g.ny);
    double cx = dadd(g.ox, dmul((double)i + 0.5, g.dx));
    double cy = dadd(g.oy, dmul((double)j + 0.5, g.dx));
    double cz = dadd(g.oz, dmul((double)k + 0.5, g.dx));
    uint8_t cav;
    if (recompute_cavity) {
        cav = sdf_sample_d(s, cx, cy, cz) < 0.0 ? 1 : 0;
        cavity[c] = cav;
    } else {
        cav = cavity[c];
    }
    bool out = has_outlet && aabb_contains(outlet, cx, cy, cz);
    base[c] = out ? AIR : (!cav ? SOLID : AIR);
}
__global__ void k_cavity_and_base(Grid g, SdfD s, int has_outlet, Aabb outlet,
                                  uint8_t* __restrict__ cavity, uint8_t* __restrict__ base,
                                  int recompute_cavity) { pdl_begin(); k_cavity_and_base_body(VB{blockIdx.x, gridDim.x}, g, s, has_outlet, outlet, cavity, base, recompute_cavity); }

// Validity for extrapolation: the face borders a Fluid cell (solver.rs:612-642).
// Bricks of nodes that four sweeps can reach from a fluid cell (four nodes before
// it to five behind it, so at most two a direction) get this extrapolation's number.
__device__ __forceinline__ void k_extrap_valid_body(VB vb_, Grid g, const uint8_t* __restrict__ cells, uint8_t* __restrict__ ku,
                               uint8_t* __restrict__ kv, uint8_t* __restrict__ kw, uint32_t* __restrict__ brick, uint32_t epoch,
                               unsigned int* __restrict__ maxbits) {
    if (vb_.bid == 0 && threadIdx.x < 3) maxbits[threadIdx.x] = 0u;  // of k_face_max
    int i, j, k;
    if (!node_of(g, (size_t)vb_.bid * blockDim.x + threadIdx.x, i, j, k)) return;
    auto fl = [&](int a, int b, int c) {
        return cells[((size_t)c * g.ny + b) * g.nx + a] == FLUID;
    };
    const bool own = i < g.nx && j < g.ny && k < g.nz && fl(i, j, k);
    if (j < g.ny && k < g.nz) ku[((size_t)k * g.ny + j) * (g.nx + 1) + i] = own || (i > 0 && fl(i - 1, j, k));
    if (i < g.nx && k < g.nz) kv[((size_t)k * (g.ny + 1) + j) * g.nx + i] = own || (j > 0 && fl(i, j - 1, k));
    if (i < g.nx && j < g.ny) kw[((size_t)k * g.ny + j) * g.nx + i] = own || (k > 0 && fl(i, j, k - 1));
    if (own) {
        const int bx = brick_dim(g.nx), by = brick_dim(g.ny), bz = brick_dim(g.nz);
        const int i0 = max(i - 4, 0) / kBrick, j0 = max(j - 4, 0) / kBrick, k0 = max(k - 4, 0) / kBrick;
        const int i1 = min((i + 5) / kBrick, bx - 1), j1 = min((j + 5) / kBrick, by - 1), k1 = min((k + 5) / kBrick, bz - 1);
        for (int c = k0; c <= k1; ++c)
            for (int b = j0; b <= j1; ++b)
                for (int a = i0; a <= i1; ++a) {
                    uint32_t* const f = brick + ((size_t)c * by + b) * bx + a;
                    if (*f != epoch) *f = epoch;
                }
    }
}
__global__ void k_extrap_valid(Grid g, const uint8_t* __restrict__ cells, uint8_t* __restrict__ ku,
                               uint8_t* __restrict__ kv, uint8_t* __restrict__ kw, uint32_t* __restrict__ brick,
                               uint32_t epoch, unsigned int* __restrict__ maxbits) { pdl_begin(); k_extrap_valid_body(VB{blockIdx.x, gridDim.x}, g, cells, ku, kv, kw, brick, epoch, maxbits); }

// One snapshot sweep of extrapolate (solver.rs:964-1007) on one unknown face,
// in place. kn holds 0 for unknown, 1 for known from the start and s + 2 for
// a face that became known in sweep s; sweep s reads only faces known before
// it, whose values no longer change, so every face sees the snapshot the
// reference's copy-then-update sweep gives it. Unknown entries take the mean
// of their known neighbours, summed in the order -x,+x,-y,+y,-z,+z; everything
// else is left as it is (the reference copies it unchanged).
__device__ __forceinline__ void extrap_one(float* __restrict__ f, uint8_t* __restrict__ kn, int sweep, int nx,
                                           int ny, int nz, int i, int j, int k) {
    const size_t c = ((size_t)k * ny + j) * nx + i;
    // The six bytes side by side, then the values: one after another, as the
    // conditions come, a face is a chain of up to twelve round trips.
    const size_t sy = nx, sz = (size_t)nx * ny;
    const bool in[6] = {i > 0, i + 1 < nx, j > 0, j + 1 < ny, k > 0, k + 1 < nz};
    const size_t at[6] = {c - 1, c + 1, c - sy, c + sy, c - sz, c + sz};
    uint8_t nk[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) nk[q] = in[q] ? kn[at[q]] : (uint8_t)0;
    float fv[6];
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        // in [1, sweep + 1]: known before this sweep
        const bool known = nk[q] != 0 && nk[q] <= sweep + 1;
        fv[q] = known ? f[at[q]] : 0.0f;  // a sum from +0 is never -0: adding +0 changes no bit
        cnt += known;
    }
    if (cnt > 0) {
        f[c] = (((((0.0f + fv[0]) + fv[1]) + fv[2]) + fv[3]) + fv[4] + fv[5]) / (float)cnt;
        kn[c] = (uint8_t)(sweep + 2);
    }
}

struct ExtrapArgs {
    Grid g;
    float* u;
    float* v;
    float* w;
    uint8_t* ku;
    uint8_t* kv;
    uint8_t* kw;
    int sweep;              // 0..3
    const uint32_t* brick;  // per brick of nodes: the last extrapolation that reached it
    uint32_t nbricks;
    uint32_t epoch;         // this extrapolation's number
};

// The faces of one brick's nodes, a node per thread.
__device__ __forceinline__ void extrap_brick(const ExtrapArgs& a, const BrickPos& b, int tid) {
    const Grid& g = a.g;
    const int i = b.i0 + tid % kBrick, j = b.j0 + tid / kBrick % kBrick, k = b.k0 + tid / (kBrick * kBrick);
    const bool hu = j < g.ny && k < g.nz && i <= g.nx, hv = i < g.nx && k < g.nz && j <= g.ny, hw = i < g.nx && j < g.ny && k <= g.nz;
    const size_t cu = ((size_t)k * g.ny + j) * (g.nx + 1) + i, cv = ((size_t)k * (g.ny + 1) + j) * g.nx + i,
                 cw = ((size_t)k * g.ny + j) * g.nx + i;
    const bool du = hu && !a.ku[cu], dv = hv && !a.kv[cv], dw = hw && !a.kw[cw];  // not known yet
    if (du) extrap_one(a.u, a.ku, a.sweep, g.nx + 1, g.ny, g.nz, i, j, k);
    if (dv) extrap_one(a.v, a.kv, a.sweep, g.nx, g.ny + 1, g.nz, i, j, k);
    if (dw) extrap_one(a.w, a.kw, a.sweep, g.nx, g.ny, g.nz + 1, i, j, k);
}

// A block takes every vb_.nb-th brick; those out of the liquid's reach have nothing
// to extrapolate (in a 0.2 mm pool two thirds of the nodes, before the jet has
// filled a cavity nearly all). Small scenes wait for round trips: with the gradient,
// at 2 mm 65 -> 34 us against a test of the 27 bricks around, two nodes a thread
// and conditional loads one after another. In the pool 522 -> 294 us: there the
// blocks of empty bricks and every warp's atomics for the maxima cost the time.
__device__ __forceinline__ void k_extrap_body(VB vb_, ExtrapArgs a) {
    const Grid& g = a.g;
    const int tid = (int)threadIdx.x;
    __shared__ uint32_t s_list[kBrickBS], s_n;
    // the block's bricks, kBrickBS at a time, a thread each: those within reach
    for (uint32_t base = vb_.bid; base < a.nbricks; base += vb_.nb * kBrickBS) {
        const uint32_t mine = base + (uint32_t)tid * vb_.nb;
        const bool in = mine < a.nbricks && a.brick[mine] == a.epoch;
        if (!__syncthreads_or(in)) continue;
        if (tid == 0) s_n = 0u;
        __syncthreads();
        if (in) s_list[atomicAdd(&s_n, 1u)] = mine;
        __syncthreads();
        const uint32_t n = s_n;
        for (uint32_t q = 0; q < n; ++q) extrap_brick(a, brick_of(g, s_list[q]), tid);
    }
}
__global__ void __launch_bounds__(kBrickBS) k_extrap(ExtrapArgs a) { pdl_begin(); k_extrap_body(VB{blockIdx.x, gridDim.x}, a); }

// The faces' maxima |u|, |v|, |w|, a third of the grid's blocks (at least one)
// each. Non-negative floats order like their bit patterns (a NaN counts as 0):
// an exact maximum per warp, block and grid, with an atomic for a larger value only.
constexpr int kFaceMaxBS = 256;
__device__ __forceinline__ void k_face_max_body(VB vb_, Faces f, size_t nu, size_t nv, size_t nw, unsigned int* __restrict__ out) {
    __shared__ uint32_t s_max[kFaceMaxBS / 32];
    const int c = (int)(vb_.bid % 3), tid = (int)threadIdx.x;
    const float* const p = c == 0 ? f.u : c == 1 ? f.v : f.w;
    const size_t n = c == 0 ? nu : c == 1 ? nv : nw;
    const size_t step = (size_t)(vb_.nb / 3) * kFaceMaxBS;
    const float4* const p4 = reinterpret_cast<const float4*>(p);
    float m = 0.f;
#pragma unroll 4
    for (size_t q = (size_t)(vb_.bid / 3) * kFaceMaxBS + tid; q < n / 4; q += step) {
        const float4 x = p4[q];
        m = fmaxf(fmaxf(fmaxf(fmaxf(m, fabsf(x.x)), fabsf(x.y)), fabsf(x.z)), fabsf(x.w));
    }
    if (vb_.bid < 3 && tid < (int)(n % 4)) m = fmaxf(m, fabsf(p[n / 4 * 4 + tid]));
    uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((tid & 31) == 0) s_max[tid / 32] = w;
    __syncthreads();
    if (tid >= 32) return;
    w = __reduce_max_sync(0xffffffffu, s_max[tid % (kFaceMaxBS / 32)]);
    if (tid == 0 && w > __ldcg(out + c)) atomicMax(out + c, w);
}
__global__ void __launch_bounds__(kFaceMaxBS) k_face_max(Faces f, size_t nu, size_t nv, size_t nw, unsigned int* __restrict__ out) { pdl_begin(); k_face_max_body(VB{blockIdx.x, gridDim.x}, f, nu, nv, nw, out); }

}  // namespace sdr
