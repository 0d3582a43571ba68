// P2G as a tiled, deterministic scatter (the tolerance-mode path on large grids; p2g_ordered.cuh keeps the reference's
// order and is the faster one below P2GT_MIN_CELLS). Same results as particles.cl:135-227 up to the order and
// rounding with which each cell's weighted sums are added: every weight is computed as the reference computes it,
// the fluid fraction (an integer count) is identical, and a face that no particle weighs is 0 in both.
//
// Each particle is visited once. A particle in bin b (b = floor(s - 0.5) per axis, s = p / dx) has nonzero weights only
// on the faces of cells b-1..b+1 along the face's own axis and b..b+1 along the other two: 12 u faces, 12 v
// faces, 12 w faces, and it is counted in one of the 8 cells b..b+1. All particles of one bin share these
// candidates, so a lane sums its bin's particles into 72 register accumulators (velocity and weight sums, in
// pairs, one fused operation a term) and adds them to the tile's shared-memory sums once per bin; the counts go to
// shared memory as they are found.
//
// Layout: a block owns a tile of TI x TJ x TK cells (10 x 10 x 30) and sums into shared memory the
// contributions of the bins of the tile and its one-bin halo: (TI+2) x (TJ+2) rows of TK+2 = 32 bins
// along k, one warp per row, one lane per bin. Rows run in 9 phases by (row i mod 3, row j mod 3):
// rows of one phase are at least 3 apart in i or j, so their candidate cells are disjoint and no two
// warps add to the same cell at the same time. Inside a row the lanes add one candidate offset at a
// time (distinct cells of each array per step, __syncwarp between steps). Every cell therefore receives its terms
// in a fixed order: no floating-point atomics (the counts use integer shared-memory atomics, which
// commute), and the same result on every run.
//
// A row's particles are one contiguous range: the warp copies it to its own buffer in shared memory (a longer row as the
// ordered walk does, in parts or equal shares of its bins: 4^3 cells of 500 particles 1310 us, in parts 4920) with consecutive
// 16-byte loads, the next phase's row before the barrier, and the lanes read their bins there (lanes that read
// their own bins from global memory touch 32 lines a load). The 16 warps of a block take one row each in
// every phase. Bound by the barriers between the phases and the FP32 pipe (46 % of the issue slots: a phase lasts as
// long as its longest row). Measured (B200, us; in brackets lanes reading global memory, two blocks of 8 warps): 160^3
// with 5.5M particles 266 (302), 200^3 523, 256^3 1044 (1126); the ordered walk takes 297, 577 and 1114, and 240
// against 274 at 144^3.
#pragma once
#include "p2g_ordered.cuh"

namespace clb {

// The number of particles is not known to the host here, so the line is drawn by cells. Ordered / tiled, us: full blocks
// of 2.8M cells 461 / 518, of 160^3 297 / 266; other fillings at 160^3, 192^3 and 256^3 (uniformly random): a layer of 8 cells
// along j 216 / 196, 303 / 284, 587 / 441, along i 163 / 131, 244 / 186, 509 / 349, along k 307 / 294, 455 / 438, 828 / 741, of 30 along
// j 389 / 410, 542 / 554, 977 / 907; half a grid of 2 a cell 452 / 416, 742 / 661, 1634 / 1473; one clump of 32^3 cells 127 /
// 152, 187 / 161, 334 / 206. Only very dense clumps stay with the walk (16^3 cells of 64 particles 412 / 490, 428 / 498, 504 / 506).
constexpr i64 P2GT_MIN_CELLS = 3500000;
constexpr int P2GT_TI = 10, P2GT_TJ = 10, P2GT_TK = 30;
constexpr int P2GT_ROWS_I = P2GT_TI + 2, P2GT_ROWS_J = P2GT_TJ + 2;
constexpr int P2GT_CELLS = P2GT_TI * P2GT_TJ * P2GT_TK;
constexpr int P2GT_WARPS = 16;
constexpr int P2GT_THREADS = 32 * P2GT_WARPS;
// shared memory: velocity sums u, v, w; weight sums u, v, w; counts
constexpr int P2GT_SHARE_COST = 16;               // as P2GO_SHARE_COST (a particle takes longer here)
constexpr int P2GT_ROW = 304;                     // particles of a row staged at a time
constexpr int P2GT_BUFFER = 6 * P2GT_ROW + 8;     // positions, velocities: each from a 16-byte boundary on
constexpr int P2GT_PAD = P2GT_CELLS + 4;           // a spare cell after each array, for what falls outside the tile
constexpr int P2GT_SMEM = (7 * P2GT_PAD + P2GT_WARPS * P2GT_BUFFER) * 4;
static_assert((3 * P2GT_ROW + 4) % 4 == 0 && (7 * P2GT_PAD) % 4 == 0, "16-byte buffers");
static_assert((P2GT_ROWS_I / 3) * (P2GT_ROWS_J / 3) == P2GT_WARPS, "one row per warp and phase");
static_assert(P2GT_TK + 2 == 32, "a row of bins is one warp");
static_assert(P2GT_ROWS_I % 3 == 0 && P2GT_ROWS_J % 3 == 0, "phases split the rows evenly");

__device__ __forceinline__ float p2gt_tent(float s, float f) { return fmaxf(0.0f, 1.0f - fabsf(s - f)); }

// One block's tile (the body of k_p2g_tiled; also run per scene by the batched P2G). The particle
// indices in offsets are indices into pos and vel.
__device__ __forceinline__ void p2g_tile(int tile, const float* __restrict__ pos, const float* __restrict__ vel,
                                         const int* __restrict__ offsets, const int* __restrict__ counts,
                                         float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                                         float* __restrict__ ff, float inv_dx, float inv_ppc, int nx, int ny, int nz,
                                         int tiles_j, int tiles_k) {
    extern __shared__ __align__(16) float p2gt_smem[];
    float* s_vel = p2gt_smem;                 // [3][PAD]
    float* s_wgt = p2gt_smem + 3 * P2GT_PAD;  // [3][PAD]
    int* s_cnt = reinterpret_cast<int*>(p2gt_smem + 6 * P2GT_PAD);
    const int tk = tile % tiles_k, tj = (tile / tiles_k) % tiles_j, ti = tile / (tiles_k * tiles_j);
    const int i0 = ti * P2GT_TI, j0 = tj * P2GT_TJ, k0 = tk * P2GT_TK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // rows holding particles: bins (i0-1+ri, j0-1+rj, k0-1 .. k0+30) inside the bin range [0, n-2]
    const int bz_lo = max(k0 - 1, 0), bz_hi = min(k0 + P2GT_TK, nz - 2);
    int any = 0;
    for (int r = threadIdx.x; r < P2GT_ROWS_I * P2GT_ROWS_J; r += P2GT_THREADS) {
        const int bx = i0 - 1 + r / P2GT_ROWS_J, by = j0 - 1 + r % P2GT_ROWS_J;
        if (bx < 0 || bx > nx - 2 || by < 0 || by > ny - 2 || bz_lo > bz_hi) continue;
        const i64 first = gidx(bx, by, bz_lo, ny, nz), last = gidx(bx, by, bz_hi, ny, nz);
        any |= (__ldg(offsets + last) + __ldg(counts + last) - __ldg(offsets + first)) > 0;
    }
    any = __syncthreads_or(any);
    if (any) {
        for (int c = threadIdx.x; c < 7 * P2GT_PAD / 4; c += P2GT_THREADS)
            reinterpret_cast<float4*>(p2gt_smem)[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float* bp = p2gt_smem + 7 * P2GT_PAD + warp * P2GT_BUFFER;
        float* bv = bp + 3 * P2GT_ROW + 4;
        const uint32_t bp32 = (uint32_t)__cvta_generic_to_shared(bp), bv32 = (uint32_t)__cvta_generic_to_shared(bv);
        const bool aligned = ((((uintptr_t)pos) | ((uintptr_t)vel)) & 15) == 0;
        const int bz = k0 - 1 + lane;
        // the warp's row in a phase: row (pi + 3 a, pj + 3 b), a = warp / 4, b = warp % 4
        const int ra = 3 * (warp / (P2GT_ROWS_J / 3)), rb = 3 * (warp % (P2GT_ROWS_J / 3));
        int begin = 0, n = 0, first = 0, last = 0, shift = 0;
        auto look_up = [&](int phase, int& b, int& c) {
            const int bx = i0 - 1 + ra + phase / 3, by = j0 - 1 + rb + phase % 3;
            b = c = 0;
            if (phase < 9 && bx >= 0 && bx <= nx - 2 && by >= 0 && by <= ny - 2 && bz >= 0 && bz <= nz - 2) {
                const i64 bin = gidx(bx, by, bz, ny, nz);
                b = __ldg(offsets + bin);
                c = __ldg(counts + bin);
            }
        };
        // from the 16-byte boundary at or before the first record (when the arrays start on one) to the last float
        auto stage = [&](int base, int m) -> int {
            int skip = 0;
            if (aligned) {
                skip = (int)((3u * (uint32_t)base) & 3u);
                const i64 at = 3 * (i64)base - skip;
                const int floats = 3 * m + skip;
                for (int t = 4 * lane; t < floats; t += 128) {
                    const int bytes = 4 * min(4, floats - t);
                    p2g_cp16(bp32 + 4 * t, pos + at + t, bytes);
                    p2g_cp16(bv32 + 4 * t, vel + at + t, bytes);
                }
            } else {
                for (int t = lane; t < 3 * m; t += 32) {
                    p2g_cp4(bp32 + 4 * t, pos + 3 * (i64)base + t);
                    p2g_cp4(bv32 + 4 * t, vel + 3 * (i64)base + t);
                }
            }
            return skip;
        };
        // A row of more particles than the buffer goes part after part of its range, which takes as long as each part's fullest
        // bin, or in rounds of shares, which cost P2GT_SHARE_COST particles each besides the fullest bin's.
        auto shares_pay = [&]() {
            const int fullest = __reduce_max_sync(0xffffffffu, n), share = P2GT_ROW / __popc(__ballot_sync(0xffffffffu, n > 0));
            return (last - first - 1) / P2GT_ROW * fullest > P2GT_SHARE_COST * ((fullest + share - 1) / share);
        };
        // A round: the next ones of every bin, in equal shares of the buffer (one range of the
        // row would be a few bins' and leave the other lanes without work). This lane's are q0 .. q1 - 1 in the buffer.
        auto stage_shares = [&](int& q0, int& q1) {
            const unsigned active = __ballot_sync(0xffffffffu, n > 0);
            const int share = P2GT_ROW / __popc(active);
            q0 = __popc(active & ((1u << lane) - 1u)) * share;
            q1 = q0 + min(n, share);
            for (unsigned left = active; left; left &= left - 1) {
                const int l = __ffs(left) - 1;
                const i64 from = 3 * (i64)__shfl_sync(0xffffffffu, begin, l);
                const int m = __shfl_sync(0xffffffffu, q1 - q0, l), to = 3 * __shfl_sync(0xffffffffu, q0, l);
                for (int t = lane; t < 3 * m; t += 32) {
                    p2g_cp4(bp32 + 4 * (to + t), pos + from + t);
                    p2g_cp4(bv32 + 4 * (to + t), vel + from + t);
                }
            }
            begin += q1 - q0;
            n -= q1 - q0;
        };
        auto take = [&](int b, int c) {
            begin = b;
            n = c;
            first = last = 0;
            const unsigned some = __ballot_sync(0xffffffffu, n > 0);
            if (some) {
                first = __shfl_sync(0xffffffffu, begin, __ffs(some) - 1);
                last = __shfl_sync(0xffffffffu, begin + n, 31 - __clz(some));
                if (last - first <= P2GT_ROW) shift = stage(first, last - first);
            }
        };
        {
            int b, c;
            look_up(0, b, c);
            take(b, c);
        }
        __syncthreads();
        for (int phase = 0; phase < 9; ++phase) {
            int next_begin, next_n;
            look_up(phase + 1, next_begin, next_n);
            if (first < last) {  // a row without particles adds nothing (warp-uniform)
                const int bx = i0 - 1 + ra + phase / 3, by = j0 - 1 + rb + phase % 3;
                // velocity and weight sums of the 12 faces of each component, as six pairs: u faces (a, b, c) and v
                // faces (b, a, c) by c, w faces (b, c, a) by c
                f32x2 vu[6], wu[6], vv[6], wv[6], vw[6], ww[6];
#pragma unroll
                for (int a = 0; a < 6; ++a) vu[a] = wu[a] = vv[a] = wv[a] = vw[a] = ww[a] = 0ull;
                const float fbx = (float)bx, fby = (float)by, fbz = (float)bz;
                const int li = bx - i0, lj = by - j0, lk = bz - k0;
                auto sum = [&](const float* bq, const float* bw, int q0, int q1) {
                    for (int q = q0; q < q1; ++q) {
                        const float sx = bq[3 * q] * inv_dx, sy = bq[3 * q + 1] * inv_dx, sz = bq[3 * q + 2] * inv_dx;
                        // the reference's face positions: cell c's u face at c + 1 on x, its v and w faces
                        // at c + 0.5; here c = b - 1, b, b + 1 (full) and b, b + 1 (half)
                        const float fx[3] = {p2gt_tent(sx, fbx), p2gt_tent(sx, fbx + 1.0f), p2gt_tent(sx, fbx + 2.0f)};
                        const float fy[3] = {p2gt_tent(sy, fby), p2gt_tent(sy, fby + 1.0f), p2gt_tent(sy, fby + 2.0f)};
                        const float fz[3] = {p2gt_tent(sz, fbz), p2gt_tent(sz, fbz + 1.0f), p2gt_tent(sz, fbz + 2.0f)};
                        const float hx[2] = {p2gt_tent(sx, fbx + 0.5f), p2gt_tent(sx, fbx + 1.5f)};
                        const float hy[2] = {p2gt_tent(sy, fby + 0.5f), p2gt_tent(sy, fby + 1.5f)};
                        const float hz[2] = {p2gt_tent(sz, fbz + 0.5f), p2gt_tent(sz, fbz + 1.5f)};
                        // weights multiplied x * y * z left to right; each sum is one fused operation per term (this
                        // kernel is the tolerance mode's: its sums already differ from the reference's order)
                        const f32x2 hz2 = pack2(hz[0], hz[1]), hy2 = pack2(hy[0], hy[1]);
                        const float v0 = bw[3 * q], v1 = bw[3 * q + 1], v2 = bw[3 * q + 2];
                        const f32x2 v02 = pack2(v0, v0), v12 = pack2(v1, v1), v22 = pack2(v2, v2);
#pragma unroll
                        for (int a = 0; a < 3; ++a)
#pragma unroll
                            for (int b = 0; b < 2; ++b) {
                                const int t = a * 2 + b;
                                const float xy = fx[a] * hy[b], xv = hx[b] * fy[a];
                                const f32x2 gu = mul2(pack2(xy, xy), hz2);
                                const f32x2 gv = mul2(pack2(xv, xv), hz2);
                                const f32x2 gw = mul2(mul2(pack2(hx[b], hx[b]), hy2), pack2(fz[a], fz[a]));
                                vu[t] = fma2(gu, v02, vu[t]);
                                wu[t] = add2(wu[t], gu);
                                vv[t] = fma2(gv, v12, vv[t]);
                                wv[t] = add2(wv[t], gv);
                                vw[t] = fma2(gw, v22, vw[t]);
                                ww[t] = add2(ww[t], gw);
                            }
                        // the particle's cell for the fluid fraction (b or b + 1 on each axis): integer adds
                        // commute, so a shared-memory atomic keeps the count exact and deterministic
                        const int ci = clampi((int)sx, 1, nx - 2) - i0, cj = clampi((int)sy, 1, ny - 2) - j0,
                                  ck = clampi((int)sz, 1, nz - 2) - k0;
                        if (ci >= 0 && ci < P2GT_TI && cj >= 0 && cj < P2GT_TJ && ck >= 0 && ck < P2GT_TK)
                            atomicAdd(s_cnt + (ci * P2GT_TJ + cj) * P2GT_TK + ck, 1);
                    }
                };
                if (last - first > P2GT_ROW && shares_pay()) {
                    do {
                        int q0, q1;
                        stage_shares(q0, q1);
                        p2g_cp_wait();
                        __syncwarp();
                        sum(bp, bv, q0, q1);
                        __syncwarp();
                    } while (__any_sync(0xffffffffu, n > 0));
                } else {
                    // (without this loop, nearly always passed once, lanes without particles went on to what follows ahead of
                    // the others, and all of it was issued twice: 2 particles a bin at 160^3 495 us, with it 410)
                    for (int base = first; base < last; base += P2GT_ROW) {
                        const int m = min(P2GT_ROW, last - base);
                        if (last - first > P2GT_ROW) {  // not staged ahead
                            __syncwarp();
                            shift = stage(base, m);
                        }
                        p2g_cp_wait();
                        __syncwarp();
                        sum(bp + shift, bv + shift, max(begin, base) - base, min(begin + n, base + m) - base);
                    }
                }
                __syncwarp();
                // add the bin's sums to the tile's cells, one candidate offset at a time: within a step the
                // lanes write distinct cells of each array (u, v and w sums are separate arrays), and a
                // __syncwarp orders the steps, which can reach the same cell from neighbouring lanes
                // (lanes whose cell the tile does not have add to the spare cell: no branch on a lane's own state)
                auto add = [&](int component, int di, int dj, int dk, float val, float wgt) {
                    const int ci = li + di, cj = lj + dj;
                    if (ci < 0 || ci >= P2GT_TI || cj < 0 || cj >= P2GT_TJ) return;  // warp-uniform
                    const int c = component * P2GT_PAD + ((unsigned)(lk + dk) < (unsigned)P2GT_TK
                                                              ? (ci * P2GT_TJ + cj) * P2GT_TK + lk + dk
                                                              : P2GT_CELLS);
                    s_vel[c] += val;
                    s_wgt[c] += wgt;
                };
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const int t = a * 2 + b;
                            auto half = [&](f32x2 v) { return c ? hi2(v) : lo2(v); };
                            add(0, a - 1, b, c, half(vu[t]), half(wu[t]));
                            add(1, b, a - 1, c, half(vv[t]), half(wv[t]));
                            add(2, b, c, a - 1, half(vw[t]), half(ww[t]));
                            __syncwarp();
                        }
            }
            take(next_begin, next_n);
            __syncthreads();
        }
        p2g_cp_wait();
    }
    // the tile's cells: the reference's normalisation (particles.cl:216-226)
    for (int c = threadIdx.x; c < P2GT_CELLS; c += P2GT_THREADS) {
        const int ci = i0 + c / (P2GT_TJ * P2GT_TK), cj = j0 + (c / P2GT_TK) % P2GT_TJ, ck = k0 + c % P2GT_TK;
        if (ci >= nx || cj >= ny || ck >= nz) continue;
        const i64 index = gidx(ci, cj, ck, ny, nz);
        if (!any) {
            u[index] = v[index] = w[index] = ff[index] = 0.0f;
            continue;
        }
        const float su = s_wgt[c], sv = s_wgt[P2GT_PAD + c], sw = s_wgt[2 * P2GT_PAD + c];
        u[index] = su > 0.0f ? s_vel[c] / su : 0.0f;
        v[index] = sv > 0.0f ? s_vel[P2GT_PAD + c] / sv : 0.0f;
        w[index] = sw > 0.0f ? s_vel[2 * P2GT_PAD + c] / sw : 0.0f;
        ff[index] = (float)s_cnt[c] * inv_ppc;
    }
}

__global__ void __launch_bounds__(P2GT_THREADS, 1)
    k_p2g_tiled(const float* __restrict__ pos, const float* __restrict__ vel, const int* __restrict__ offsets,
                const int* __restrict__ counts, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                float* __restrict__ ff, float inv_dx, float inv_ppc, int nx, int ny, int nz, int tiles_j,
                int tiles_k) {
    p2g_tile(blockIdx.x, pos, vel, offsets, counts, u, v, w, ff, inv_dx, inv_ppc, nx, ny, nz, tiles_j, tiles_k);
}

__host__ __device__ __forceinline__ int p2g_tiled_tiles(int nx, int ny, int nz, int* tiles_j, int* tiles_k) {
    const int ti = (nx + P2GT_TI - 1) / P2GT_TI;
    *tiles_j = (ny + P2GT_TJ - 1) / P2GT_TJ;
    *tiles_k = (nz + P2GT_TK - 1) / P2GT_TK;
    return ti * *tiles_j * *tiles_k;
}

}  // namespace clb
