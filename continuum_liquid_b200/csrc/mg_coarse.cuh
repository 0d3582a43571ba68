// Coarsest-level solves of levels too large for the one-launch bottom visits (mg_bottom.cuh): a grid with one short
// side stops coarsening while the others are still long (155 x 27 x 129 ends at 41 x 9 x 34, 4368 interior cells of
// a colour).
//
// A solve is 2 (pre + coarse) dependent red-black phases (multigrid.cl:232-264), 132 with the reference's counts, so
// it is bound by what one phase takes: the loads and the arithmetic of the cells a thread owns, and a barrier. A
// thread owns one cell of each colour, with its neighbour weights, the reciprocal of the diagonal and delta^2 b in
// registers; p lies in shared memory split by colour. A level of more cells than one block's threads is cut into slabs
// of planes along the longer of i and j, one per CTA of a cluster: a cell in a slab's first or last plane is also
// stored into the neighbour's ghost plane, and the cluster barrier (0.25 us) ends the phase.
//
// Time of an iteration (two phases), B200, us, a full level (in brackets one with half its cells fluid), against
// k_coarse_solve, which finds its cells again in every phase: 8 x 8 x 46 0.25 (0.17) against 1.6 (1.5); clusters:
// 10 x 23 x 18 0.35 (0.34) against 2.3 (2.2), 41 x 9 x 34 0.42 (0.34) against 10.6 (6.6), 46 x 46 x 8 0.50 (0.41)
// against 17.9 (10.6).
//
// The update is that of k_coarse_solve (the sums in the same order, divide_by for the division), the cells of a colour
// are independent, and an FP16 level's p is rounded when the solve ends, as there: the same values.
// Nothing waits on a flag: the only waits are barriers that every remaining warp passes the same number of times.
#pragma once
#include "mg_cluster.cuh"

namespace clb {

constexpr int COARSE_SLAB_THREADS = 1024;  // per CTA: one slot (colour_slots) of each colour per thread

// Interior planes [lo, hi) of slab s of cs, n0 planes with the ghost layer.
__host__ __device__ __forceinline__ void coarse_slab(int s, int cs, int n0, int* lo, int* hi) {
    *lo = 1 + (int)((long long)s * (n0 - 2) / cs);
    *hi = 1 + (int)((long long)(s + 1) * (n0 - 2) / cs);
}
__host__ __device__ __forceinline__ int coarse_slab_planes(int cs, int n0) { return (n0 - 2 + cs - 1) / cs; }
// Shared memory: p of both colours (owned planes and two ghost planes), the fluid cells of each colour, two counts.
__host__ __device__ __forceinline__ size_t coarse_slab_smem(int cs, int n0, int n1, int nz) {
    return ((size_t)2 * (coarse_slab_planes(cs, n0) + 2) * n1 * ((nz + 1) / 2) + 2 * COARSE_SLAB_THREADS + 2) * 4;
}

// along_j: slabs of planes along j instead of i. n0: planes (nx, or ny), n1: rows of a plane (ny, or nx).
template <bool H>
__global__ void __launch_bounds__(COARSE_SLAB_THREADS, 1)
    k_coarse_slabs(float* p, const float* __restrict__ b, const float4* __restrict__ opc,
                   const uint8_t* __restrict__ mask, float delta, int iterations, int n0, int n1, int nz,
                   bool along_j, const float* __restrict__ scale, int cs) {
    namespace cgx = cooperative_groups;
    constexpr int THREADS = COARSE_SLAB_THREADS;
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_begin();
    const int s = blockIdx.x;
    int lo, hi;
    coarse_slab(s, cs, n0, &lo, &hi);
    const int own = hi - lo, hz = (nz + 1) / 2, row_plane = n1 * hz;
    const int colour_words = (coarse_slab_planes(cs, n0) + 2) * row_plane;  // the same in every slab
    // strides along i and j in memory, of planes and rows there, and along i and j in shared memory
    const int gx = along_j ? n0 * nz : n1 * nz, gy = nz;
    const int g0 = along_j ? gy : gx, g1 = along_j ? gx : gy;
    const int sx = along_j ? hz : row_plane, sy = along_j ? row_plane : hz;
    float* sp = reinterpret_cast<float*>(smem);
    int* list = reinterpret_cast<int*>(sp + 2 * colour_words);  // [colour][THREADS]
    int* count = list + 2 * THREADS;
    const float d2 = H ? scale[2] : delta * delta;
    auto op = [&](int g) -> float4 {
        if constexpr (H) return ld_h4(reinterpret_cast<const Half4*>(opc), g);
        else return __ldg(opc + g);
    };
    auto ld = [&](const float* a, int g) -> float {
        if constexpr (H) return ldh(reinterpret_cast<const __half*>(a), g);
        else return a[g];
    };
    if (threadIdx.x < 2) count[threadIdx.x] = 0;
    __syncthreads();

    // q: il * n1 * nz + j * nz + k with il the plane in the slab (0: its lower ghost plane); index(q): in memory
    auto index = [&](int q) {
        const int row = q / nz, il = row / n1;
        return (il + lo - 1) * g0 + (row - il * n1) * g1 + (q - row * nz);
    };
#pragma unroll 4
    for (int q = threadIdx.x; q < (own + 2) * n1 * nz; q += THREADS) {
        const int row = q / nz, k = q - row * nz;
        const int il = row / n1, j = row - il * n1;
        sp[((il + lo - 1 + j + k) & 1) * colour_words + row * hz + (k >> 1)] = ld(p, index(q));
    }
    // the slab's cells to update, by colour (any order: cells of a colour are independent)
    const int half = (nz - 1) / 2, my = n1 - 2, slots = own * my * half;
#pragma unroll
    for (int colour = 0; colour < 2; ++colour) {
        const int r = threadIdx.x;
        int q = -1;
        if (r < slots) {
            const int row = r / half, t = r - row * half;
            const int il = 1 + row / my, j = 1 + row % my;
            const int k = 1 + 2 * t + ((il + lo - 1 + j + 1 + colour) & 1);
            if (k <= nz - 2) {
                q = (il * n1 + j) * nz + k;
                const int g = index(q);
                if (!mask[g] || !(op(g).x > 0.0f)) q = -1;
            }
        }
        const unsigned in = __ballot_sync(0xffffffffu, q >= 0);
        int base = 0;
        if ((threadIdx.x & 31) == 0 && in) base = atomicAdd(count + colour, __popc(in));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (q >= 0) list[colour * THREADS + base + __popc(in & ((1u << (threadIdx.x & 31)) - 1u))] = q;
    }
    __syncthreads();

    struct Cell {
        int c, n, up;  // words of the cell, of its slot in the other colour, of its neighbour at k + 1
        float d2b, d, r, wxp, wxm, wyp, wym, wzp, wzm;
        bool first, last;  // in the slab's first / last plane, with a neighbour there
    } cell[2];
    const int counts[2] = {count[0], count[1]};
#pragma unroll
    for (int colour = 0; colour < 2; ++colour) {
        Cell& o = cell[colour];
        // a thread without a cell takes part in the barriers only
        o.c = o.n = row_plane + hz;
        o.up = o.n + 1;
        o.d2b = o.wxp = o.wxm = o.wyp = o.wym = o.wzp = o.wzm = 0.0f;
        o.d = o.r = 1.0f;
        o.first = o.last = false;
        if (threadIdx.x < counts[colour]) {
            const int q = list[colour * THREADS + threadIdx.x], g = index(q);
            const int row = q / nz, k = q - row * nz;
            const int word = row * hz + (k >> 1);
            o.c = colour * colour_words + word;
            o.n = (colour ^ 1) * colour_words + word;
            o.up = o.n + (k & 1);
            const float4 self = op(g);
            o.d = self.x;
            o.r = 1.0f / o.d;
            o.d2b = d2 * ld(b, g);
            o.wxp = self.y;
            o.wyp = self.z;
            o.wzp = self.w;
            o.wxm = op(g - gx).y;
            o.wym = op(g - gy).z;
            o.wzm = op(g - 1).w;
            const int il = row / n1;
            o.first = il == 1 && s > 0;
            o.last = il == own && s + 1 < cs;
        }
    }

    float *left = nullptr, *right = nullptr;  // where a cell's word goes in the neighbours' ghost planes
    if (cs > 1) {
        cgx::cluster_group cluster = cgx::this_cluster();
        if (s > 0) {
            int llo, lhi;
            coarse_slab(s - 1, cs, n0, &llo, &lhi);
            left = cluster.map_shared_rank(sp, (unsigned)(s - 1)) + (lhi - llo) * row_plane;
        }
        if (s + 1 < cs) right = cluster.map_shared_rank(sp, (unsigned)(s + 1)) - own * row_plane;
        cluster_barrier();  // every slab is staged before a neighbour writes to it
    }
    // warps without a cell take no further part; the first stays, the neighbours write into this CTA's memory
    const int most = counts[0] > counts[1] ? counts[0] : counts[1];
    const int warps = most > 32 ? (most + 31) / 32 : 1;
    if ((int)(threadIdx.x >> 5) >= warps) return;
    for (int it = 0; it < iterations; ++it)
#pragma unroll
        for (int colour = 0; colour < 2; ++colour) {
            const Cell& o = cell[colour];
            if (threadIdx.x < counts[colour]) {
                const float ws = o.wxp * sp[o.n + sx] + o.wxm * sp[o.n - sx] + o.wyp * sp[o.n + sy] +
                                 o.wym * sp[o.n - sy] + o.wzp * sp[o.up] + o.wzm * sp[o.up - 1];
                const float v = divide_by(ws - o.d2b, o.d, o.r);
                sp[o.c] = v;
                if (o.first) left[o.c] = v;
                if (o.last) right[o.c] = v;
            }
            __syncwarp();  // the barriers are taken by whole warps
            if (cs > 1) cluster_barrier();
            else bar_b(warps);
        }
#pragma unroll
    for (int colour = 0; colour < 2; ++colour)
        if (threadIdx.x < counts[colour]) {
            const int g = index(list[colour * THREADS + threadIdx.x]);
            const float v = sp[cell[colour].c];
            if constexpr (H) reinterpret_cast<__half*>(p)[g] = __float2half_rn(v);
            else p[g] = v;
        }
}

}  // namespace clb
