// Triangle-mesh voxelisation (Solver/Kernel/OpenCL/voxelise_mesh.cl): each interior cell centre
// casts one ray along a fixed oblique direction and counts Moller-Trumbore hits; an odd count marks
// the cell solid. The ray-triangle arithmetic is the reference's, term for term, so occupancy is
// bit-exact against the CPU restatement.
//
// Bound by instruction issue (ray-triangle tests), so what counts is how few (cell, triangle) pairs are
// tested. A block owns a brick of 16x8x8 cells and each of its warps two sub-bricks of 4x4x2; a triangle
// is tested by a warp only where it can be hit by one of the sub-brick's rays. Two culls, both provably
// without effect on the result:
//
//   Behind: a hit point is h = o + t*d with t > 0 and every component of d positive, so h >= o
//   componentwise, and o >= o_min, the brick's first cell centre (float rounding of the centre
//   formula is monotone in the cell index). A triangle whose largest vertex coordinate on some axis
//   is below o_min on that axis minus a margin lies behind every ray of the brick: its exact ray
//   parameter is below -margin, and the computed parameter of the exact test differs from it by
//   orders of magnitude less than that (margin = 8 cell widths + 1e-4 |o_min| + 1e-6), so the exact
//   test rejects it too.
//
//   Across: all rays are parallel, so under the shear (y, z) -> (y - x d1/d0, z - x d2/d0) a ray is one
//   point and a triangle a plane triangle. The exact test accepts only when its computed barycentric
//   coordinates lie in the triangle. With S1, S2, T the largest components of the edges and of (origin -
//   first vertex), every sum of the test's numerators and determinant is off by at most 48 eps S T
//   (resp. 48 eps S1 S2), so the true coordinates are within
//       du = 100 eps S2 (T + S1) / |det|,  dv = 100 eps S1 (T + S2) / |det|
//   of the computed ones as long as 48 eps S1 S2 <= |det| / 2 (otherwise the triangle is kept), and the
//   true hit point within du S1' + dv S2' (S' = 1.4 S: the shear adds at most 0.38 of another component)
//   of the triangle's sheared bounding box. A brick whose sheared ray origins all lie outside that box,
//   grown by this margin and the rounding of the comparison itself, cannot be hit.
//
// Measured (B200, icosphere of 5120 triangles at 128^3, radius 0.10-0.18): 0.11 ms a call, against
// 3.4-5.7 ms with the behind cull alone on bricks of 4x4x16 (0.18 ms with 8x8x8 bricks and a division per
// listed triangle). Much of it is the set-up: every block forms the edges, determinant and box of every triangle that is
// not behind it, and its warps then wait for the fullest (48 % of the issue slots, profiles/kernels_listed_cases.md).
#pragma once
#include "common.cuh"

namespace clb {

constexpr int VOX_BI = 4, VOX_BJ = 4, VOX_BK = 16;
constexpr int VOX_THREADS = VOX_BI * VOX_BJ * VOX_BK;
constexpr int VOX_CHUNK = 512;

// voxelise_mesh.cl:5-22 ray_hit
__device__ __forceinline__ int ray_hit(float o0, float o1, float o2, float d0, float d1, float d2,
                                       const float* __restrict__ t9) {
    const float a0 = t9[0], a1 = t9[1], a2 = t9[2];
    const float e10 = t9[3] - a0, e11 = t9[4] - a1, e12 = t9[5] - a2;
    const float e20 = t9[6] - a0, e21 = t9[7] - a1, e22 = t9[8] - a2;
    const float p0 = d1 * e22 - d2 * e21, p1 = d2 * e20 - d0 * e22, p2 = d0 * e21 - d1 * e20;
    const float det = e10 * p0 + e11 * p1 + e12 * p2;
    if (fabsf(det) < 1.0e-7f) return 0;
    const float inv = 1.0f / det;
    const float t0 = o0 - a0, t1 = o1 - a1, t2 = o2 - a2;
    const float uu = (t0 * p0 + t1 * p1 + t2 * p2) * inv;
    if (uu < 0.0f || uu > 1.0f) return 0;
    const float q0 = t1 * e12 - t2 * e11, q1 = t2 * e10 - t0 * e12, q2 = t0 * e11 - t1 * e10;
    const float vv = (d0 * q0 + d1 * q1 + d2 * q2) * inv;
    if (vv < 0.0f || uu + vv > 1.0f) return 0;
    return (e20 * q0 + e21 * q1 + e22 * q2) * inv > 1.0e-6f;
}

// Every triangle against every cell (the form the culled kernel is checked against).
__global__ void __launch_bounds__(VOX_THREADS) k_voxelise_all(const float* __restrict__ tris, uint8_t* __restrict__ mask,
                                                               int T, int nx, int ny, int nz, float delta, float ox,
                                                               float oy, float oz, float d0, float d1, float d2) {
    __shared__ float s_tri[VOX_CHUNK * 9];
    const int tk = threadIdx.x % VOX_BK, tj = (threadIdx.x / VOX_BK) % VOX_BJ, ti = threadIdx.x / (VOX_BK * VOX_BJ);
    const int k = blockIdx.x * VOX_BK + tk, j = blockIdx.y * VOX_BJ + tj, i = blockIdx.z * VOX_BI + ti;
    const bool active = i >= 1 && j >= 1 && k >= 1 && i < nx - 1 && j < ny - 1 && k < nz - 1;
    const float o0 = ox + ((float)i + 0.5f) * delta, o1 = oy + ((float)j + 0.5f) * delta,
                o2 = oz + ((float)k + 0.5f) * delta;
    int hits = 0;
    for (int base = 0; base < T; base += VOX_CHUNK) {
        const int n = min(VOX_CHUNK, T - base);
        for (int t = threadIdx.x; t < n * 9; t += VOX_THREADS) s_tri[t] = __ldg(tris + 9 * (i64)base + t);
        __syncthreads();
        if (active)
            for (int t = 0; t < n; ++t) hits += ray_hit(o0, o1, o2, d0, d1, d2, s_tri + 9 * t);
        __syncthreads();
    }
    if (active && (hits & 1)) mask[gidx(i, j, k, ny, nz)] = 1;
}

// The culled form. Per chunk of triangles: one thread a triangle computes its edges, determinant and grown
// sheared box and lists it when the block's brick can be hit (the ray-independent part of ray_hit, with
// the same operations, is kept: 13 floats); then each warp tests 32 listed triangles at a time against
// its sub-brick, a lane each, and runs the exact test of its 32 cells for those that remain.
// The listing visits every triangle for every block, so a block's brick is long (16) along x, the rays'
// main direction, where length costs the least sheared area; each warp has two sub-bricks.
constexpr int VC_BI = 16, VC_BJ = 8, VC_BK = 8, VC_THREADS = 512, VC_CHUNK = 512;
constexpr int VC_SUBS = VC_BI * VC_BJ * VC_BK / VC_THREADS;
static_assert(VC_SUBS == 2, "two sub-bricks of 32 cells a warp");

struct VoxTri {            // 64 bytes, read as four float4 broadcasts
    float a0, a1, a2, inv;
    float e10, e11, e12, p0;
    float e20, e21, e22, p1;
    float p2, m0, m1, m2;  // m: the triangle's largest coordinates
};

__global__ void __launch_bounds__(VC_THREADS) k_voxelise_culled(const float* __restrict__ tris,
                                                                 uint8_t* __restrict__ mask, int T, int nx, int ny,
                                                                 int nz, float delta, float ox, float oy, float oz,
                                                                 float d0, float d1, float d2) {
    __shared__ __align__(16) VoxTri s_tri[VC_CHUNK];
    __shared__ float4 s_box[VC_CHUNK];  // sheared box, grown by its margin: y lo, y hi, z lo, z hi
    __shared__ int s_count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bi = blockIdx.z * VC_BI, bj = blockIdx.y * VC_BJ, bk = blockIdx.x * VC_BK;
    const int wi = bi + 4 * (warp >> 3), wj = bj + 4 * ((warp >> 2) & 1), wk = bk + 2 * (warp & 3);  // sub-brick 0
    const int i = wi + (lane >> 3), j = wj + ((lane >> 1) & 3), k = wk + (lane & 1);  // sub-brick h: i + 8 h
    auto centre = [&](float o, int c) { return o + ((float)c + 0.5f) * delta; };
    const float o1 = centre(oy, j), o2 = centre(oz, k);
    const float r1 = d1 / d0, r2 = d2 / d0;
    // sheared ray origins of a brick of cells [i, i + ni) x ...: bounds of y - x r1 and z - x r2, and the
    // smallest origins for the behind test
    struct Brick {
        float ylo, yhi, zlo, zhi, g0, g1, g2;
    };
    auto brick = [&](int i0, int ni, int j0, int nj, int k0, int nk) {
        const float x0 = centre(ox, i0), x1 = centre(ox, i0 + ni - 1), y0 = centre(oy, j0), y1 = centre(oy, j0 + nj - 1),
                    z0 = centre(oz, k0), z1 = centre(oz, k0 + nk - 1);
        // rounding of the shear here and of a triangle's vertices (bounded by the brick's side of the
        // comparison; the vertices' own share is in their box): a few eps of the largest term
        const float r = 1.0e-6f * (fmaxf(fabsf(x0), fabsf(x1)) + fmaxf(fmaxf(fabsf(y0), fabsf(y1)), fmaxf(fabsf(z0), fabsf(z1))));
        Brick b;
        b.ylo = y0 - x1 * r1 - r;
        b.yhi = y1 - x0 * r1 + r;
        b.zlo = z0 - x1 * r2 - r;
        b.zhi = z1 - x0 * r2 + r;
        b.g0 = x0 - (8.0f * delta + 1.0e-4f * fabsf(x0) + 1.0e-6f);
        b.g1 = y0 - (8.0f * delta + 1.0e-4f * fabsf(y0) + 1.0e-6f);
        b.g2 = z0 - (8.0f * delta + 1.0e-4f * fabsf(z0) + 1.0e-6f);
        return b;
    };
    const Brick whole = brick(bi, VC_BI, bj, VC_BJ, bk, VC_BK);
    const Brick sub[VC_SUBS] = {brick(wi, 4, wj, 4, wk, 2), brick(wi + 8, 4, wj, 4, wk, 2)};
    const float x_first = centre(ox, bi), x_last = centre(ox, bi + VC_BI - 1), y_first = centre(oy, bj),
                y_last = centre(oy, bj + VC_BJ - 1), z_first = centre(oz, bk), z_last = centre(oz, bk + VC_BK - 1);
    // comparisons are written so that a NaN keeps the triangle
    auto behind = [](const Brick& b, float m0, float m1, float m2) { return m0 < b.g0 || m1 < b.g1 || m2 < b.g2; };
    auto outside = [](const Brick& b, float4 box) {
        return box.x > b.yhi || box.y < b.ylo || box.z > b.zhi || box.w < b.zlo;
    };
    int hits[VC_SUBS] = {0, 0};
    for (int base = 0; base < T; base += VC_CHUNK) {
        if (threadIdx.x == 0) s_count = 0;
        __syncthreads();
        const int t = base + threadIdx.x;
        if (t < T) {
            const float* src = tris + 9 * (i64)t;
            VoxTri v;
            v.a0 = __ldg(src);
            v.a1 = __ldg(src + 1);
            v.a2 = __ldg(src + 2);
            const float b0 = __ldg(src + 3), b1 = __ldg(src + 4), b2 = __ldg(src + 5);
            const float c0 = __ldg(src + 6), c1 = __ldg(src + 7), c2 = __ldg(src + 8);
            v.m0 = fmaxf(fmaxf(v.a0, b0), c0);
            v.m1 = fmaxf(fmaxf(v.a1, b1), c1);
            v.m2 = fmaxf(fmaxf(v.a2, b2), c2);
            if (!behind(whole, v.m0, v.m1, v.m2)) {
                v.e10 = b0 - v.a0;
                v.e11 = b1 - v.a1;
                v.e12 = b2 - v.a2;
                v.e20 = c0 - v.a0;
                v.e21 = c1 - v.a1;
                v.e22 = c2 - v.a2;
                v.p0 = d1 * v.e22 - d2 * v.e21;
                v.p1 = d2 * v.e20 - d0 * v.e22;
                v.p2 = d0 * v.e21 - d1 * v.e20;
                const float det = v.e10 * v.p0 + v.e11 * v.p1 + v.e12 * v.p2;
                const float S1 = fmaxf(fmaxf(fabsf(v.e10), fabsf(v.e11)), fabsf(v.e12));
                const float S2 = fmaxf(fmaxf(fabsf(v.e20), fabsf(v.e21)), fabsf(v.e22));
                const float tx = fmaxf(fabsf(x_first - v.a0), fabsf(x_last - v.a0));
                const float ty = fmaxf(fabsf(y_first - v.a1), fabsf(y_last - v.a1));
                const float tz = fmaxf(fabsf(z_first - v.a2), fabsf(z_last - v.a2));
                const float Tm = fmaxf(fmaxf(tx, ty), tz);
                const float eps = 6.0e-8f;
                // du S1' + dv S2' is reach / |det|; big bounds the vertices' coordinates
                const float reach = 1.6f * 100.0f * eps * S1 * S2 * (2.0f * Tm + S1 + S2);
                const float big = fmaxf(fmaxf(fabsf(v.a0), fabsf(v.a1)), fabsf(v.a2)) + S1 + S2;
                const float ay = v.a1 - v.a0 * r1, by = b1 - b0 * r1, cy = c1 - c0 * r1;
                const float az = v.a2 - v.a0 * r2, bz = b2 - b0 * r2, cz = c2 - c0 * r2;
                float4 box = make_float4(fminf(fminf(ay, by), cy), fmaxf(fmaxf(ay, by), cy), fminf(fminf(az, bz), cz),
                                         fmaxf(fmaxf(az, bz), cz));
                const bool bounded = 96.0f * eps * S1 * S2 <= fabsf(det) && reach < 1.0e30f && big < 1.0e30f;
                // the gap between the plain box and the brick against the margin, without the division
                const float gap = fmaxf(fmaxf(box.x - whole.yhi, whole.ylo - box.y), fmaxf(box.z - whole.zhi, whole.zlo - box.w));
                const bool misses = bounded && (gap - 1.0e-6f * big) * fabsf(det) > reach;
                if (!(fabsf(det) < 1.0e-7f) && !misses) {
                    v.inv = 1.0f / det;
                    const float grow = reach * fabsf(v.inv) + 1.0e-6f * big;
                    // no bound on the coordinates (or a non-finite triangle): never outside
                    box = bounded && grow < 1.0e30f ? make_float4(box.x - grow, box.y + grow, box.z - grow, box.w + grow)
                                                    : make_float4(-INFINITY, INFINITY, -INFINITY, INFINITY);
                    const int slot = atomicAdd(&s_count, 1);
                    s_tri[slot] = v;
                    s_box[slot] = box;
                }
            }
        }
        __syncthreads();
        // the kept triangles arrive in any order; the hit count (an integer) does not depend on it
        const int m = s_count;
#pragma unroll
        for (int h = 0; h < VC_SUBS; ++h) {
            const float o0 = centre(ox, i + 8 * h);
            for (int q0 = 0; q0 < m; q0 += 32) {
                const int q = q0 + lane;
                bool keep = false;
                if (q < m)
                    keep = !outside(sub[h], s_box[q]) && !behind(sub[h], s_tri[q].m0, s_tri[q].m1, s_tri[q].m2);
                unsigned todo = __ballot_sync(0xffffffffu, keep);
                while (todo) {
                    const int c = q0 + __ffs(todo) - 1;
                    todo &= todo - 1;
                    const float4* rec = reinterpret_cast<const float4*>(s_tri + c);
                    const float4 A = rec[0], E1 = rec[1], E2 = rec[2];
                    const float p2 = s_tri[c].p2;
                    // ray_hit from here on (a, inv | e1, p0 | e2, p1)
                    const float t0 = o0 - A.x, t1 = o1 - A.y, t2 = o2 - A.z;
                    const float uu = (t0 * E1.w + t1 * E2.w + t2 * p2) * A.w;
                    if (uu < 0.0f || uu > 1.0f) continue;
                    const float w0 = t1 * E1.z - t2 * E1.y, w1 = t2 * E1.x - t0 * E1.z, w2 = t0 * E1.y - t1 * E1.x;
                    const float vv = (d0 * w0 + d1 * w1 + d2 * w2) * A.w;
                    if (vv < 0.0f || uu + vv > 1.0f) continue;
                    hits[h] += (E2.x * w0 + E2.y * w1 + E2.z * w2) * A.w > 1.0e-6f;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int h = 0; h < VC_SUBS; ++h) {
        const int c = i + 8 * h;
        if (c >= 1 && j >= 1 && k >= 1 && c < nx - 1 && j < ny - 1 && k < nz - 1 && (hits[h] & 1))
            mask[gidx(c, j, k, ny, nz)] = 1;
    }
}

// voxelise_mesh.cl:24 normalize((1, 0.3713907, 0.2178311)), restated as v / sqrt(dot(v, v)) in
// correctly rounded float arithmetic; evaluated on the host so every launch uses the same three
// floats.
static inline void voxelise_direction(float out[3]) {
    volatile float x = 1.0f, y = 0.3713907f, z = 0.2178311f;
    volatile float xx = x * x, yy = y * y, zz = z * z;
    volatile float s = xx + yy;
    s = s + zz;
    const float len = sqrtf(s);
    out[0] = x / len;
    out[1] = y / len;
    out[2] = z / len;
}

}  // namespace clb
