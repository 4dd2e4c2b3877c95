// SDF builders on the device.
//  * k_sdf_mesh: Sdf::from_mesh_in_bounds (sdf.rs:53-86) — per node, min
//    closest-point distance (Ericson, sdf.rs:209-254) and the summed van
//    Oosterom–Strackee solid angle (sdf.rs:259-272) over all triangles, sign
//    from winding > 1/2 (sdf.rs:187-205). Triangles stream through shared
//    memory in tiles moved by the bulk-copy engine (cp.async.bulk, one
//    transaction per tile into the CTA's own shared memory, no multicast),
//    double-buffered behind an mbarrier with a bounded wait.
//  * k_sdf_scan .. k_sdf_sign: the same values for closed meshes without the
//    pass over all node-triangle pairs (further down).
//  * k_sdf_sinus: Sdf::from_fn(SinusParams::implicit) (sinus.rs:89-119).
// All arithmetic is f64 without contraction, in the reference's order.
#pragma once
#include "common.cuh"

namespace sdr {

struct D3 {
    double x, y, z;
};
__device__ __forceinline__ D3 d3(double x, double y, double z) { return D3{x, y, z}; }
__device__ __forceinline__ D3 sub3(D3 a, D3 b) { return d3(dsub(a.x, b.x), dsub(a.y, b.y), dsub(a.z, b.z)); }
__device__ __forceinline__ D3 add3(D3 a, D3 b) { return d3(dadd(a.x, b.x), dadd(a.y, b.y), dadd(a.z, b.z)); }
__device__ __forceinline__ D3 mul3(D3 a, double s) { return d3(dmul(a.x, s), dmul(a.y, s), dmul(a.z, s)); }
__device__ __forceinline__ double dot3(D3 a, D3 b) { return dadd(dadd(dmul(a.x, b.x), dmul(a.y, b.y)), dmul(a.z, b.z)); }
__device__ __forceinline__ D3 cross3(D3 a, D3 b) {
    return d3(dsub(dmul(a.y, b.z), dmul(a.z, b.y)), dsub(dmul(a.z, b.x), dmul(a.x, b.z)),
              dsub(dmul(a.x, b.y), dmul(a.y, b.x)));
}

__device__ __forceinline__ double tri_dist_sq(D3 p, D3 a, D3 b, D3 c) {  // sdf.rs:209-254
    D3 ab = sub3(b, a), ac = sub3(c, a), ap = sub3(p, a);
    double d1 = dot3(ab, ap), d2 = dot3(ac, ap);
    if (d1 <= 0.0 && d2 <= 0.0) return dot3(ap, ap);
    D3 bp = sub3(p, b);
    double d3_ = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3_ >= 0.0 && d4 <= d3_) return dot3(bp, bp);
    double vc = dsub(dmul(d1, d4), dmul(d3_, d2));
    if (vc <= 0.0 && d1 >= 0.0 && d3_ <= 0.0) {
        double v = ddiv(d1, dsub(d1, d3_));
        D3 e = sub3(p, add3(a, mul3(ab, v)));
        return dot3(e, e);
    }
    D3 cp = sub3(p, c);
    double d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    if (d6 >= 0.0 && d5 <= d6) return dot3(cp, cp);
    double vb = dsub(dmul(d5, d2), dmul(d1, d6));
    if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) {
        double w = ddiv(d2, dsub(d2, d6));
        D3 e = sub3(p, add3(a, mul3(ac, w)));
        return dot3(e, e);
    }
    double va = dsub(dmul(d3_, d6), dmul(d5, d4));
    if (va <= 0.0 && dsub(d4, d3_) >= 0.0 && dsub(d5, d6) >= 0.0) {
        double w = ddiv(dsub(d4, d3_), dadd(dsub(d4, d3_), dsub(d5, d6)));
        D3 e = sub3(p, add3(b, mul3(sub3(c, b), w)));
        return dot3(e, e);
    }
    double denom = ddiv(1.0, dadd(dadd(va, vb), vc));
    double v = dmul(vb, denom), w = dmul(vc, denom);
    D3 e = sub3(p, add3(add3(a, mul3(ab, v)), mul3(ac, w)));
    return dot3(e, e);
}

__device__ __forceinline__ double solid_angle(D3 p, D3 a, D3 b, D3 c) {  // sdf.rs:259-272
    D3 av = sub3(a, p), bv = sub3(b, p), cv = sub3(c, p);
    double la = __dsqrt_rn(dot3(av, av)), lb = __dsqrt_rn(dot3(bv, bv)), lc = __dsqrt_rn(dot3(cv, cv));
    if (la < 1e-12 || lb < 1e-12 || lc < 1e-12) return 0.0;
    double num = dot3(av, cross3(bv, cv));
    double den = dadd(dadd(dadd(dmul(dmul(la, lb), lc), dmul(dot3(av, bv), lc)), dmul(dot3(bv, cv), la)),
                      dmul(dot3(cv, av), lb));
    return dmul(2.0, atan2(num, den));
}

constexpr int kSdfBS = 128;
constexpr int kSdfTile = 128;  // triangles per stage (9216 bytes)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Bounded wait on an mbarrier phase: gives up after about one second of SM
// clock (2^31 cycles, 1.1 s at 1965 MHz) and returns false.
constexpr long long kWaitCycles = 1ll << 31;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > kWaitCycles) return false;
    }
}

// k_sdf_mesh's test hook: the tile whose bulk copy is not issued (so its
// staging wait runs out); kNoSkip in normal use.
constexpr uint32_t kNoSkip = 0xFFFFFFFFu;

// tris: padded to a whole number of tiles (9 f64 per triangle, 16-byte aligned).
__global__ void __launch_bounds__(kSdfBS) k_sdf_mesh(const double* __restrict__ tris, uint32_t ntri,
                                                     uint32_t ntiles, double ox, double oy, double oz,
                                                     double dx, int nx, int ny, int nz,
                                                     double* __restrict__ out, uint32_t* __restrict__ err,
                                                     uint32_t skip_tile = kNoSkip,
                                                     const uint32_t* __restrict__ gate = nullptr) {
    if (gate && *gate == 0u) return;  // the field is already there
    __shared__ __align__(128) double st[2][kSdfTile * 9];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int fail;
    size_t node = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t nn = (size_t)nx * ny * nz;
    int i = node % nx, j = (node / nx) % ny, k = node / ((size_t)nx * ny);
    D3 p = d3(dadd(ox, dmul((double)i, dx)), dadd(oy, dmul((double)j, dx)), dadd(oz, dmul((double)k, dx)));
    if (threadIdx.x == 0) {
        fail = 0;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t bytes = kSdfTile * 9 * sizeof(double);
    uint32_t issued = 0;  // thread 0 only
    if (threadIdx.x == 0 && ntiles > 0) {
        if (skip_tile != 0) bulk_load(st[0], tris, bytes, &bar[0]);
        issued = 1;
    }
    double min_d2 = INFINITY, wind = 0.0;
    uint32_t t = 0;
    for (; t < ntiles; ++t) {
        int b = t & 1;
        if (threadIdx.x == 0 && t + 1 < ntiles) {
            if (skip_tile != t + 1) bulk_load(st[b ^ 1], tris + (size_t)(t + 1) * kSdfTile * 9, bytes, &bar[b ^ 1]);
            issued = t + 2;
        }
        if (!mbar_wait(&bar[b], (t >> 1) & 1)) fail = 1;
        __syncthreads();
        if (fail) break;
        uint32_t cnt = min((uint32_t)kSdfTile, ntri - t * kSdfTile);
        const double* s = st[b];
        for (uint32_t q = 0; q < cnt; ++q) {
            D3 a = d3(s[9 * q], s[9 * q + 1], s[9 * q + 2]);
            D3 bb = d3(s[9 * q + 3], s[9 * q + 4], s[9 * q + 5]);
            D3 c = d3(s[9 * q + 6], s[9 * q + 7], s[9 * q + 8]);
            double d2 = tri_dist_sq(p, a, bb, c);
            if (d2 < min_d2) min_d2 = d2;
            wind = dadd(wind, solid_angle(p, a, bb, c));
        }
        __syncthreads();  // everyone is done with st[b] before it is refilled
    }
    if (fail) {
        // A bounded wait gave up: drain the copies still in flight (again
        // bounded) before the block's shared memory goes away, then report.
        if (threadIdx.x == 0) {
            for (uint32_t q = t; q < issued; ++q)
                if (q != skip_tile) mbar_wait(&bar[q & 1], (q >> 1) & 1);
            atomicOr(err, 1u);
        }
        return;
    }
    if (node >= nn) return;
    wind = ddiv(wind, dmul(4.0, 3.141592653589793));
    double dist = __dsqrt_rn(min_d2);
    out[node] = wind > 0.5 ? -dist : dist;
}

// ---------------------------------------------------------------------------
// The same field for closed meshes, without the pass over all node-triangle
// pairs (k_sdf_mesh is bound by the FP64 pipe: 25 ms for 65k nodes and 20k
// triangles). Two facts:
//  * The distance is a minimum, so a triangle that is certainly farther than
//    the nearest one found may be left out: the minimum over the others has the
//    same bits. Bounding spheres (f32, rounded outwards), per 32 triangles and
//    per triangle, rule triangles out per brick of 4 x 4 x 4 nodes, then per
//    node, an f32 distance with its error bound most of the rest; the few left
//    are evaluated as k_sdf_mesh does.
//  * Where every directed edge of the mesh is matched by its reverse, the
//    winding number is a whole number that changes only across the surface.
//    Two nodes closer to each other than their distances to the surface add up
//    to lie on the same side (each one's ball holds no surface and the balls
//    meet). So every node follows such nodes of growing distance, and only the
//    few where that ends sum the solid angles.
// A mesh with an unmatched edge, a triangle so thin that its computed distance
// may be off (k_sdf_balls), a node within 1e-10 of the extent of the surface,
// where the sign hangs on the rounding of the sum in its order, or a sum that
// is not near a whole number opens the gate of k_sdf_mesh, which then writes
// the whole field.
struct SdfFast {
    const double* tris;     // 9 f64 per triangle
    uint32_t ntri;
    double ox, oy, oz, dx;  // node grid
    int nx, ny, nz;
    double cx, cy, cz;      // centre of the node box: f32 positions are relative to it
    unsigned long long* acc;  // [0..1] edge sums, [2] bits of the largest f32 distance of a vertex or node corner
    uint32_t* gate;         // 1: k_sdf_mesh writes the field
    float4* ball;           // per triangle: bounding sphere (padded to whole groups of 32)
    float4* group;          // per 32 triangles: their bounding sphere
    float4* norm;           // per triangle: unit normal
    float4* vert;           // per triangle: three vertices; vert[3 t].w: the f32 distance holds up to this distance squared (-1: nowhere)
    double* dist;           // per node
    uint32_t* up;           // per node: the neighbour it follows, or itself (a root)
    uint32_t* roots;        // [0] their number, then the nodes
    uint8_t* inside;        // per node that is a root
    double* out;
};

__device__ __forceinline__ unsigned long long sdf_mix(unsigned long long z) {  // splitmix64 finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ unsigned long long sdf_vertex_key(const double* v, unsigned long long seed) {
    unsigned long long h = seed;
    for (int c = 0; c < 3; ++c) h = sdf_mix(h * 0x9E3779B97F4A7C15ull + (unsigned long long)__double_as_longlong(v[c]));
    return h;
}

// Per triangle: the sum over its directed edges of key(a, b) - key(b, a), under
// two seeds: zero over the mesh if and only if (up to a 2^-128 coincidence)
// every directed edge is matched by its reverse. And the mesh's extent.
__global__ void __launch_bounds__(256) k_sdf_scan(SdfFast a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long e0 = 0, e1 = 0;
    float far = 0.0f;
    if (t < a.ntri) {
        const double* v = a.tris + (size_t)t * 9;
        for (int s = 0; s < 2; ++s) {
            unsigned long long k[3], e = 0;
            for (int c = 0; c < 3; ++c) k[c] = sdf_vertex_key(v + 3 * c, s ? 0xD1B54A32D192ED03ull : 0x8CB92BA72F3D8DD7ull);
            for (int c = 0; c < 3; ++c) {
                const unsigned long long p = k[c], q = k[(c + 1) % 3];
                e += sdf_mix(p * 0x9E3779B97F4A7C15ull + q) - sdf_mix(q * 0x9E3779B97F4A7C15ull + p);
            }
            if (s) e1 = e;
            else e0 = e;
        }
        for (int c = 0; c < 3; ++c) {
            const double x = v[3 * c] - a.cx, y = v[3 * c + 1] - a.cy, z = v[3 * c + 2] - a.cz;
            const float r = __double2float_ru(sqrt(x * x + y * y + z * z));
            if (!(r < 1e12f)) *a.gate = 1u;  // not finite, or beyond the f32 bounds used here
            else far = fmaxf(far, r);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        e0 += __shfl_xor_sync(0xffffffffu, e0, o);
        e1 += __shfl_xor_sync(0xffffffffu, e1, o);
        far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(a.acc, e0);
        atomicAdd(a.acc + 1, e1);
        atomicMax(a.acc + 2, (unsigned long long)__float_as_uint(far));
    }
}

__device__ __forceinline__ float sdf_extent(const SdfFast& a) {
    const float hx = 0.5f * (float)(a.nx - 1), hy = 0.5f * (float)(a.ny - 1), hz = 0.5f * (float)(a.nz - 1);
    const float box = (float)a.dx * sqrtf(hx * hx + hy * hy + hz * hz);
    return 1.0001f * fmaxf(box, __uint_as_float((unsigned)a.acc[2]));
}

// Bounding spheres, widened by what the f32 positions of the triangles and the
// nodes may be off, and the vertices for the f32 distances. The barycentric
// coordinates of the point nearest to p are off by about 64 eps D^2 l^2 / |n|^2
// (differences of products of dot products of size l D, over the squared
// normal): a triangle is too thin if that is over a thousandth in f64 two
// extents away, and its f32 distance holds while it is under a fiftieth. That
// distance forms products of four lengths (up to 1e4 l^4 within its reach) and
// divides by |n|^2: only where both are normal numbers of f32 with room to spare.
// Other triangles are told apart by their spheres alone (squares of lengths, which
// f32 holds over all extents that pass here).
__global__ void __launch_bounds__(256) k_sdf_balls(SdfFast a) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const float ext = sdf_extent(a);
    if (t == 0 && (a.acc[0] != 0ull || a.acc[1] != 0ull || !(ext > 1e-12f && ext < 1e12f))) *a.gate = 1u;
    float4 ball = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    if (t < a.ntri) {
        const double* v = a.tris + (size_t)t * 9;
        double g[3], e1[3], e2[3], e3[3];
        for (int c = 0; c < 3; ++c) {
            g[c] = (v[c] + v[3 + c] + v[6 + c]) / 3.0;
            e1[c] = v[3 + c] - v[c];
            e2[c] = v[6 + c] - v[c];
            e3[c] = v[6 + c] - v[3 + c];
        }
        double r2 = 0.0;
        for (int q = 0; q < 3; ++q) {
            const double x = v[3 * q] - g[0], y = v[3 * q + 1] - g[1], z = v[3 * q + 2] - g[2];
            r2 = fmax(r2, x * x + y * y + z * z);
        }
        const double n0 = e1[1] * e2[2] - e1[2] * e2[1], n1 = e1[2] * e2[0] - e1[0] * e2[2],
                     n2 = e1[0] * e2[1] - e1[1] * e2[0];
        const double nn = n0 * n0 + n1 * n1 + n2 * n2;
        const double l2 =
            fmax(fmax(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2], e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2]),
                 e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2]);
        if (!(nn > 1e-10 * (double)ext * (double)ext * l2)) *a.gate = 1u;
        ball = make_float4((float)(g[0] - a.cx), (float)(g[1] - a.cy), (float)(g[2] - a.cz),
                           __double2float_ru(sqrt(r2)) * 1.000001f + 2e-6f * ext);
        const double rn = 1.0 / sqrt(nn);
        const float holds = nn > 1e-30 && l2 < 1e16 ? (float)(0.02 / (64.0 * 6e-8) * nn / l2) : -1.0f;
        a.norm[t] = make_float4((float)(n0 * rn), (float)(n1 * rn), (float)(n2 * rn), 0.0f);
        for (int q = 0; q < 3; ++q)
            a.vert[3 * (size_t)t + q] = make_float4((float)(v[3 * q] - a.cx), (float)(v[3 * q + 1] - a.cy),
                                                    (float)(v[3 * q + 2] - a.cz), holds);
    }
    a.ball[t] = ball;
    // the group's sphere, around the mean of its centres
    const bool live = t < a.ntri;
    float sx = live ? ball.x : 0.0f, sy = live ? ball.y : 0.0f, sz = live ? ball.z : 0.0f, sn = live ? 1.0f : 0.0f;
    for (int o = 16; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
        sn += __shfl_xor_sync(0xffffffffu, sn, o);
    }
    sn = fmaxf(sn, 1.0f);
    sx /= sn;
    sy /= sn;
    sz /= sn;
    const float x = ball.x - sx, y = ball.y - sy, z = ball.z - sz;
    float r = live ? sqrtf(x * x + y * y + z * z) * 1.000001f + ball.w + 1e-6f * ext : 0.0f;
    for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
    if ((threadIdx.x & 31) == 0) a.group[t / 32] = make_float4(sx, sy, sz, r);
}

// Squared distance of a point to a triangle in f32 (the cases of tri_dist_sq).
__device__ __forceinline__ float sdf_dist_f(float px, float py, float pz, float4 A, float4 B, float4 C) {
    const float abx = B.x - A.x, aby = B.y - A.y, abz = B.z - A.z, acx = C.x - A.x, acy = C.y - A.y, acz = C.z - A.z;
    const float apx = px - A.x, apy = py - A.y, apz = pz - A.z;
    auto sq = [](float x, float y, float z) { return x * x + y * y + z * z; };
    const float d1 = abx * apx + aby * apy + abz * apz, d2 = acx * apx + acy * apy + acz * apz;
    if (d1 <= 0.0f && d2 <= 0.0f) return sq(apx, apy, apz);
    const float bpx = px - B.x, bpy = py - B.y, bpz = pz - B.z;
    const float d3 = abx * bpx + aby * bpy + abz * bpz, d4 = acx * bpx + acy * bpy + acz * bpz;
    if (d3 >= 0.0f && d4 <= d3) return sq(bpx, bpy, bpz);
    const float cpx = px - C.x, cpy = py - C.y, cpz = pz - C.z;
    const float d5 = abx * cpx + aby * cpy + abz * cpz, d6 = acx * cpx + acy * cpy + acz * cpz;
    if (d6 >= 0.0f && d5 <= d6) return sq(cpx, cpy, cpz);
    const float va = d3 * d6 - d5 * d4, vb = d5 * d2 - d1 * d6, vc = d1 * d4 - d3 * d2;
    float v, w;
    if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
        v = __fdividef(d1, d1 - d3);
        w = 0.0f;
    } else if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
        v = 0.0f;
        w = __fdividef(d2, d2 - d6);
    } else if (va <= 0.0f && d4 - d3 >= 0.0f && d5 - d6 >= 0.0f) {
        w = __fdividef(d4 - d3, (d4 - d3) + (d5 - d6));
        v = 1.0f - w;
    } else {
        const float den = __fdividef(1.0f, va + vb + vc);
        v = vb * den;
        w = vc * den;
    }
    return sq(apx - (v * abx + w * acx), apy - (v * aby + w * acy), apz - (v * abz + w * acz));
}

// Is a triangle further than `near` from a point at (x, y, z) from its sphere's
// centre c? Its points are c + s with s in its plane and |s| <= w, so their
// distance squared is at least f^2 - 2 t w for a point f from c whose offset has
// the length t along the plane: tight where the triangle faces the point, as the
// candidates for its nearest one mostly do (the sphere alone leaves a shell of
// its radius). f and the height over the plane are off by less than `slack`.
__device__ __forceinline__ bool sdf_beyond(float x, float y, float z, float w, float4 nrm, float near, float slack) {
    const float f = sqrtf(x * x + y * y + z * z), h = fmaxf(fabsf(x * nrm.x + y * nrm.y + z * nrm.z) - slack, 0.0f);
    const float hi = f + slack, lo = f - slack;
    const float t = sqrtf(fmaxf(hi * hi - h * h, 0.0f) + 1e-6f * hi * hi);
    return lo * lo * 0.99999f - 2.002f * t * w > near * near;
}

constexpr int kSdfB = 4;                               // nodes of a brick along each axis
constexpr int kSdfNodes = kSdfB * kSdfB * kSdfB;       // 64
constexpr int kSdfSplit = 4;                           // threads per node
constexpr int kSdfDistBS = kSdfNodes * kSdfSplit;      // 256
constexpr int kSdfList = 512;                          // triangles a brick considers at a time
constexpr int kSdfWarpList = 256;                      // and a warp's eight nodes
static_assert(kSdfWarpList / kSdfSplit <= 64, "a bit per entry of a lane");
static_assert(kSdfB == 4 && kSdfSplit == 4 && kSdfDistBS == 256, "eight warps of 2 x 2 x 2 nodes");

// Distance of every node to the mesh, a block per brick. From the spheres: an
// upper bound u of the distance of the brick's centre, then the triangles whose
// spheres reach within u + 2 radii of it (no other can be nearest to a node of
// the brick), then the same again per warp for its eight nodes. Then per node,
// four lanes sharing the list: the f32 distances give an upper bound of the
// node's own, and the triangles that may be nearer than it within the error
// bounds are evaluated in f64. Deep inside a smooth cavity the spheres leave
// hundreds of triangles a node: the bound by the normal (sdf_beyond) and the
// distance of a vertex as upper bound leave a few (20,480 triangles, 0.8 M nodes:
// 4.6 -> 3.0 ms a field). Three blocks an SM take 3.0 ms (with a little spilling,
// 80 B of stores), two 3.5, four 3.0 to 3.8 (with more). The margins (1e-3 and 2e-6 of the extent) cover the rounding of
// the f32 and f64 distances (k_sdf_balls), so no triangle that could give the
// minimum is left out.
__global__ void __launch_bounds__(kSdfDistBS, 3) k_sdf_dist(SdfFast a, int bx, int by) {
    __shared__ float4 s_ball[kSdfList];
    __shared__ float4 s_vert[kSdfList * 3];
    __shared__ float4 s_norm[kSdfList];
    __shared__ uint32_t s_tri[kSdfList];
    __shared__ uint32_t s_n, s_ng;
    __shared__ uint32_t s_group[kSdfDistBS];  // of the groups looked at together: those within reach
    __shared__ float s_u[kSdfDistBS / 32];
    __shared__ uint16_t s_w[kSdfDistBS / 32][kSdfWarpList];
    // Other blocks of this launch may open the gate meanwhile, so a block leaves
    // as one: warps that went on alone would take unset list lengths.
    if (__syncthreads_or(*a.gate != 0u)) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int kWarps = kSdfDistBS / 32;
    const int b = blockIdx.x, sub = tid % kSdfSplit;
    const int i0 = b % bx * kSdfB, j0 = b / bx % by * kSdfB, k0 = b / (bx * by) * kSdfB;
    // a warp takes 2 x 2 x 2 nodes of the brick, four lanes each
    const int wi = (wid & 1) * 2, wj = (wid >> 1 & 1) * 2, wk = (wid >> 2 & 1) * 2;
    const int i = i0 + wi + (lane >> 2 & 1), j = j0 + wj + (lane >> 3 & 1), k = k0 + wk + (lane >> 4 & 1);
    const bool live = i < a.nx && j < a.ny && k < a.nz;
    const float ext = sdf_extent(a), slack = 2e-6f * ext;
    // the brick's centre and half diagonal (of all its places, also those beyond the grid)
    constexpr double kHalf = 0.5 * (kSdfB - 1);
    const float bcx = (float)(a.ox - a.cx + (i0 + kHalf) * a.dx), bcy = (float)(a.oy - a.cy + (j0 + kHalf) * a.dx),
                bcz = (float)(a.oz - a.cz + (k0 + kHalf) * a.dx);
    const float rad = 1.0001f * (float)(kHalf * a.dx) * 1.7320509f + slack;
    const uint32_t ngroup = (a.ntri + 31) / 32;
    auto far_of = [&](float4 q) {
        const float x = q.x - bcx, y = q.y - bcy, z = q.z - bcz;
        return sqrtf(x * x + y * y + z * z);
    };
    auto block_min = [&](float u) {
        for (int o = 16; o > 0; o >>= 1) u = fminf(u, __shfl_xor_sync(0xffffffffu, u, o));
        __syncthreads();
        if (lane == 0) s_u[wid] = u;
        __syncthreads();
        u = s_u[0];
        for (int w = 1; w < kWarps; ++w) u = fminf(u, s_u[w]);
        return u;
    };
    float u = 3e38f;
    for (uint32_t g = tid; g < ngroup; g += kSdfDistBS) {
        const float4 q = a.group[g];
        u = fminf(u, far_of(q) + q.w);
    }
    u = block_min(u) * 1.0001f;
    // the groups from g0 on, one per thread, within r of the brick's centre
    auto groups_within = [&](uint32_t g0, float r) {
        const uint32_t g = g0 + tid;
        bool in = false;
        if (g < ngroup) {
            const float4 q = a.group[g];
            in = far_of(q) * 0.9999f <= r + q.w;
        }
        __syncthreads();  // the list before has been used
        if (tid == 0) s_ng = 0u;
        __syncthreads();
        const unsigned m = __ballot_sync(0xffffffffu, in);
        uint32_t at = 0;
        if (lane == 0 && m) at = atomicAdd(&s_ng, (uint32_t)__popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (in) s_group[at] = g;
        __syncthreads();
        return s_ng;
    };
    float u2 = u;  // the same from the triangles of the groups that can hold the nearest one
    for (uint32_t g0 = 0; g0 < ngroup; g0 += kSdfDistBS) {
        const uint32_t ng = groups_within(g0, u);
        for (uint32_t e = wid; e < ng; e += kWarps) {
            const float4 t = a.ball[(size_t)s_group[e] * 32 + lane];
            if (t.w >= 0.0f) u2 = fminf(u2, far_of(t) + t.w);
        }
    }
    u = block_min(u2) * 1.0001f;
    const float reach = u * 1.001f + 2.0f * rad;  // a triangle of the brick: centre within reach + its radius
    const D3 p = d3(dadd(a.ox, dmul((double)i, a.dx)), dadd(a.oy, dmul((double)j, a.dx)), dadd(a.oz, dmul((double)k, a.dx)));
    const float px = (float)(p.x - a.cx), py = (float)(p.y - a.cy), pz = (float)(p.z - a.cz);
    float ub = (u + rad) * 1.0001f;  // upper bound of this node's distance
    // the warp's nodes: their centre, half diagonal and an upper bound of the centre's distance
    const float wx = (float)(a.ox - a.cx + (i0 + wi + 0.5) * a.dx), wy = (float)(a.oy - a.cy + (j0 + wj + 0.5) * a.dx),
                wz = (float)(a.oz - a.cz + (k0 + wk + 0.5) * a.dx);
    const float wrad = 1.0001f * (float)(0.5 * a.dx) * 1.7320509f + slack;
    float uw = (u + rad) * 1.0001f;
    double min_d2 = INFINITY;
    if (tid == 0) s_n = 0u;
    __syncthreads();
    for (uint32_t g0 = 0, e0 = 0, ng = 0;; e0 += kWarps) {
        if (e0 >= ng) {  // the next groups
            ng = groups_within(g0, reach);
            g0 += kSdfDistBS;
            e0 = 0;
        }
        const uint32_t e1 = e0 + wid;
        if (e1 < ng) {
            const uint32_t tri = s_group[e1] * 32 + lane;
            const float4 t = a.ball[tri];
            const bool in = t.w >= 0.0f && far_of(t) * 0.9999f <= reach + t.w;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            uint32_t at = 0;
            if (lane == 0 && m) at = atomicAdd(&s_n, (uint32_t)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (in) {
                const float4* v = a.vert + 3 * (size_t)tri;
                s_ball[at] = t;
                s_norm[at] = a.norm[tri];
                for (int c = 0; c < 3; ++c) s_vert[3 * at + c] = v[c];
                s_tri[at] = tri;
            }
        }
        // a round adds at most kWarps * 32 triangles
        const bool last = g0 >= ngroup && e0 + kWarps >= ng;
        __syncthreads();
        const uint32_t n = s_n;
        __syncthreads();
        if (!last && n + kWarps * 32 <= kSdfList) continue;  // room for another
        for (uint32_t c = lane; c < n; c += 32) {
            const float4 q = s_vert[3 * c];  // any point of the triangle bounds its distance
            const float x = q.x - wx, y = q.y - wy, z = q.z - wz;
            uw = fminf(uw, sqrtf(x * x + y * y + z * z) * 1.0001f + slack);
        }
        for (int o = 16; o > 0; o >>= 1) uw = fminf(uw, __shfl_xor_sync(0xffffffffu, uw, o));
        ub = fminf(ub, (uw + wrad) * 1.0001f);
        const float wreach = uw * 1.001f + 2.0f * wrad;
        uint32_t cnt = 0;  // entries of this warp's list
        for (uint32_t c0 = 0; c0 < n; c0 += 32) {
            const uint32_t c = c0 + lane;
            bool in = false;
            if (c < n) {
                const float4 q = s_ball[c];
                const float x = q.x - wx, y = q.y - wy, z = q.z - wz;
                in = !sdf_beyond(x, y, z, q.w, s_norm[c], wreach, slack);
            }
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) s_w[wid][cnt + __popc(m & ((1u << lane) - 1u))] = (uint16_t)c;
            cnt += __popc(m);
            if (cnt + 32 <= kSdfWarpList && c0 + 32 < n) continue;  // room for another 32
            __syncwarp();
            // f32 distances bound this node's; bit e / 4 of `may`: it may be the nearest
            unsigned long long may = 0ull;
            for (uint32_t e = sub; e < cnt; e += kSdfSplit) {
                const uint32_t at = s_w[wid][e];
                const float4 q = s_ball[at];
                const float x = q.x - px, y = q.y - py, z = q.z - pz, r = ub * 1.001f + q.w, f2 = x * x + y * y + z * z;
                if (f2 > r * r * 1.0002f || sdf_beyond(x, y, z, q.w, s_norm[at], ub * 1.001f, slack)) continue;
                const float4 A = s_vert[3 * at];
                float least = 0.0f;
                if (f2 > A.w) {
                    ub = fminf(ub, (sqrtf(f2) + q.w) * 1.0001f);
                } else {
                    const float d = sqrtf(sdf_dist_f(px, py, pz, A, s_vert[3 * at + 1], s_vert[3 * at + 2]));
                    least = d * 0.999f - slack;
                    ub = fminf(ub, d * 1.001f + slack);
                }
                if (least <= ub * 1.001f) may |= 1ull << (e / kSdfSplit);
            }
            for (int o = 1; o < kSdfSplit; o <<= 1) ub = fminf(ub, __shfl_xor_sync(0xffffffffu, ub, o));
            if (!live) may = 0ull;
            for (; may; may &= may - 1ull) {
                const uint32_t at = s_w[wid][(uint32_t)(__ffsll((long long)may) - 1) * kSdfSplit + sub];
                const float4 q = s_ball[at], A = s_vert[3 * at];
                const float x = q.x - px, y = q.y - py, z = q.z - pz, near = ub * 1.001f, r = near + q.w,
                            f2 = x * x + y * y + z * z;
                if (f2 > r * r * 1.0002f) continue;
                if (f2 <= A.w && sqrtf(sdf_dist_f(px, py, pz, A, s_vert[3 * at + 1], s_vert[3 * at + 2])) * 0.999f - slack > near)
                    continue;
                const double* v = a.tris + (size_t)s_tri[at] * 9;
                const double d2 = tri_dist_sq(p, d3(v[0], v[1], v[2]), d3(v[3], v[4], v[5]), d3(v[6], v[7], v[8]));
                if (d2 < min_d2) {
                    min_d2 = d2;
                    ub = fminf(ub, __double2float_ru(sqrt(d2)) * 1.0001f);
                }
            }
            cnt = 0;
            __syncwarp();
        }
        __syncthreads();
        if (last) break;
        if (tid == 0) s_n = 0u;
        // A long list (the brick at the centre of a ball: all of its triangles) is
        // left when another block has opened the gate: alone on its SM it took 7 ms
        // beside the full pass's 27 (20,480 triangles).
        if (__syncthreads_or(tid == 0 && *(volatile uint32_t*)a.gate != 0u)) return;
    }
    for (int o = 1; o < kSdfSplit; o <<= 1) min_d2 = fmin(min_d2, __shfl_xor_sync(0xffffffffu, min_d2, o));
    if (!live || sub != 0) return;
    const size_t node = ((size_t)k * a.ny + j) * a.nx + i;
    const double dist = __dsqrt_rn(min_d2);
    a.dist[node] = dist;
    if (!(dist > 1e-10 * (double)ext)) *a.gate = 1u;
}

// The neighbour of largest distance whose ball meets this node's (so both lie on
// the same side); from a local maximum the nodes 2 to 32 steps away; none: a
// root. The far looks take the real cavity's roots from 900 to a few dozen.
__global__ void __launch_bounds__(256) k_sdf_up(SdfFast a) {
    const size_t nn = (size_t)a.nx * a.ny * a.nz, n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn || *a.gate) return;
    const int i = (int)(n % a.nx), j = (int)(n / a.nx % a.ny), k = (int)(n / ((size_t)a.nx * a.ny));
    const double own = a.dist[n];
    double best = own;
    size_t to = n;
    for (int step = 1; step <= 32 && to == n; step += max(step / 2, 1))
        for (int q = 0; q < 27; ++q) {
            const int di = q % 3 - 1, dj = q / 3 % 3 - 1, dk = q / 9 - 1;
            const int x = i + di * step, y = j + dj * step, z = k + dk * step;
            if (x < 0 || y < 0 || z < 0 || x >= a.nx || y >= a.ny || z >= a.nz) continue;
            const size_t m = ((size_t)z * a.ny + y) * a.nx + x;
            const double d = a.dist[m];
            if (d > best && own + d > sqrt((double)(di * di + dj * dj + dk * dk)) * step * a.dx * 1.000001) {
                best = d;
                to = m;
            }
        }
    a.up[n] = (uint32_t)to;
    if (to == n) a.roots[1 + atomicAdd(a.roots, 1u)] = (uint32_t)n;
}

// The winding number of the roots (sdf.rs:187-205), a block each: a whole
// number up to rounding, whatever the order of the sum.
__global__ void __launch_bounds__(512) k_sdf_roots(SdfFast a) {
    __shared__ double sh[33];
    if (__syncthreads_or(*a.gate != 0u)) return;  // as one block: others may open it meanwhile
    const uint32_t nr = a.roots[0];
    for (uint32_t q = blockIdx.x; q < nr; q += gridDim.x) {
        const uint32_t n = a.roots[1 + q];
        const int i = (int)(n % a.nx), j = (int)(n / a.nx % a.ny), k = (int)(n / ((uint32_t)a.nx * a.ny));
        const D3 p = d3(dadd(a.ox, dmul((double)i, a.dx)), dadd(a.oy, dmul((double)j, a.dx)), dadd(a.oz, dmul((double)k, a.dx)));
        double w = 0.0;
        for (uint32_t t = threadIdx.x; t < a.ntri; t += blockDim.x) {
            const double* v = a.tris + (size_t)t * 9;
            w = dadd(w, solid_angle(p, d3(v[0], v[1], v[2]), d3(v[3], v[4], v[5]), d3(v[6], v[7], v[8])));
        }
        w = ddiv(block_sum<512>(w, sh), dmul(4.0, 3.141592653589793));
        if (threadIdx.x == 0) {
            a.inside[n] = w > 0.5;
            if (!(fabs(w - rint(w)) < 0.01)) *a.gate = 1u;
        }
    }
}

__global__ void __launch_bounds__(256) k_sdf_sign(SdfFast a) {
    const size_t nn = (size_t)a.nx * a.ny * a.nz, n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn || *a.gate) return;
    uint32_t r = (uint32_t)n, q;
    while ((q = a.up[r]) != r) r = q;  // distances grow strictly along the way
    a.out[n] = a.inside[r] ? -a.dist[n] : a.dist[n];
}

struct SinusD {
    double ax, ay, az, cx, cy, cz, taper, bump, sx, sz, sr, sd;
};

__device__ __forceinline__ double clampd(double x, double lo, double hi) {
    return x < lo ? lo : (x > hi ? hi : x);
}

__device__ __forceinline__ double sinus_implicit(const SinusD& s, double px, double py, double pz) {
    double qx = dsub(px, s.cx), qy = dsub(py, s.cy), qz = dsub(pz, s.cz);
    double h = dmul(dadd(ddiv(qy, s.ay), 1.0), 0.5);
    double scale = dadd(s.taper, dmul(dsub(1.0, s.taper), clampd(h, 0.0, 1.5)));
    double bump = dmul(s.bump, dadd(dmul(dmul(0.6, sin(ddiv(dmul(4.0, qx), s.ax))), cos(ddiv(dmul(3.0, qz), s.az))),
                                    dmul(0.4, sin(dadd(ddiv(dmul(5.0, qy), s.ay), 1.3)))));
    double tx = ddiv(qx, dmul(s.ax, scale)), ty = ddiv(qy, s.ay), tz = ddiv(qz, dmul(s.az, scale));
    double body = dsub(__dsqrt_rn(dadd(dadd(dmul(tx, tx), dmul(ty, ty)), dmul(tz, tz))), dadd(1.0, bump));
    body = dmul(body, fmin(fmin(s.ax, s.ay), s.az));
    double rx = dsub(px, s.sx), rz = dsub(pz, s.sz);
    double radial = dsub(__dsqrt_rn(dadd(dmul(rx, rx), dmul(rz, rz))), s.sr);
    double ytop = dsub(s.cy, dmul(0.5, s.ay));
    double ybot = dsub(dsub(s.cy, s.ay), s.sd);
    double axial = fmax(dsub(py, ytop), dsub(ybot, py));
    double socket = fmax(radial, axial);
    const double kk = 0.0015;
    double hh = clampd(dadd(0.5, ddiv(dmul(0.5, dsub(socket, body)), kk)), 0.0, 1.0);
    return dsub(dadd(dmul(socket, dsub(1.0, hh)), dmul(body, hh)), dmul(dmul(kk, hh), dsub(1.0, hh)));
}

__global__ void k_sdf_sinus(SinusD s, double ox, double oy, double oz, double dx, int nx, int ny, int nz,
                            double* __restrict__ out) {
    size_t node = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= (size_t)nx * ny * nz) return;
    int i = node % nx, j = (node / nx) % ny, k = node / ((size_t)nx * ny);
    out[node] = sinus_implicit(s, dadd(ox, dmul((double)i, dx)), dadd(oy, dmul((double)j, dx)),
                               dadd(oz, dmul((double)k, dx)));
}

}  // namespace sdr
