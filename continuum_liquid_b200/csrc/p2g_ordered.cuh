// P2G in the reference's summation order, each particle visited once per face component.
//
// The reference (particles.cl:135-227) adds a cell's particles in eight partial sums: lane l visits the neighbour
// bins l, l + 8, l + 16 of the 27 in that order, and the eight sums are added as
// ((l0 + l4) + (l2 + l6)) + ((l1 + l5) + (l3 + l7)). Of the 27 bins, 12 hold particles with a nonzero weight for a
// given face component: a particle in bin b has s = p / dx in [b + 0.5, b + 1.5) on each axis (for clamped bins,
// farther away), so for the u face of cell c (at c + (1, 0.5, 0.5)) the y and z weights vanish when the bin is one
// above the cell on those axes, likewise for v and w; such a bin adds exact zeros. No lane visits more than two of
// the 12, and the second lies in a later i plane of bins than the first. So a partial sum is the ordered sum
// over one bin, or over a first bin and then a second one in a later plane, and it can be formed from the bins'
// side: a block walks the planes of bins of its tile along i; every bin adds its particles, in order, to the
// partial sums of the 12 cells it reaches, from 0 where it comes first in the cell's lane and from the stored sum
// where it comes second. In one plane no two bins reach the same partial sum, so the sums lie in shared memory
// without atomics, and one barrier a plane orders them. A cell plane is finished one or two planes later: its lanes
// are added as above and its ring slot is cleared. The same additions of the same products in the same
// order as the reference: its values bit for bit. (The fluid fraction is an integer count, by shared-memory atomics.)
//
// What bounds it: instruction issue, once the particles come from shared memory. A lane that reads its own bin's
// particles from global memory touches 32 lines with every load, and the line rate of L1 then bounds the
// kernel; so a warp takes a row of 32 bins along k, whose particles are one contiguous range, copies that range to
// its own buffer with consecutive loads, and each lane walks its bin there. A row of more particles than the buffer goes part
// by part, or, where its bins are so full that a part is a few bins' and leaves the other lanes waiting, in rounds that give
// every bin an equal share of the buffer (128^3, 4^3 cells of 500 particles each: 400 us, in parts 1030; 16^3 of 64: 410,
// 640; 40^3 of 32, still in parts: 629, in shares 640 and more). Blocks handle one component each:
// the 12 sums of a bin stay in registers at 16 warps an SM, a tile's halo is one-sided along the other axes, and
// small grids still have enough blocks.
//
// Measured (B200, us, against the gather of binning.cuh): 64^3 dam break 33 (48), 117 x 90 x 139 with 4.0M particles 199
// (539), 160^3 with 5.5M 297 (938), 256^3 with 23M 1114 (3700). 58 % of the issue slots; lanes wait for the fullest
// bin of a row (about 14 particles against 8 on average).
#pragma once
#include <type_traits>
#include <utility>

#include "binning.cuh"

namespace clb {

// Two floats in a 64-bit register, for the paired multiply and add (each half rounded as the single operation).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(f32x2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float hi2(f32x2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a + b; the assembler may join it to the paired multiplication that gave b and then rounds once.
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a + b as b * 1 + a, with the 1 from the launch's arguments: the assembler joins a paired addition (or one with a
// constant 1) to the paired multiplication before it and rounds once, where the sums here round both.
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b, f32x2 one) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(one), "l"(a));
    return r;
}

// The 12 bins with nonzero weights for the face component along axis A, in visiting order.
struct P2GRole {
    int ox, oy, oz;  // bin offset from the cell
    int lane;
    bool second;     // an earlier role has the same lane
};
struct P2GRoles {
    P2GRole r[12];
};
template <int A>
__host__ __device__ constexpr P2GRoles p2g_roles() {
    P2GRoles t{};
    int n = 0;
    for (int nb = 0; nb < 27; ++nb) {
        const int ox = nb / 9 - 1, oy = (nb / 3) % 3 - 1, oz = nb % 3 - 1;
        if ((A != 0 && ox > 0) || (A != 1 && oy > 0) || (A != 2 && oz > 0)) continue;
        bool second = false;
        for (int q = 0; q < n; ++q) second = second || t.r[q].lane == nb % 8;
        t.r[n] = P2GRole{ox, oy, oz, nb % 8, second};
        ++n;
    }
    return t;
}
// Every lane has at most two roles, and the second's bin lies in a later i plane.
template <int A>
constexpr bool p2g_roles_ok() {
    const P2GRoles t = p2g_roles<A>();
    for (int l = 0; l < 8; ++l) {
        int n = 0, plane = -2;
        for (int q = 0; q < 12; ++q)
            if (t.r[q].lane == l) {
                if (n > 0 && t.r[q].ox <= plane) return false;
                plane = t.r[q].ox;
                ++n;
            }
        if (n > 2) return false;
    }
    return true;
}
static_assert(p2g_roles_ok<0>() && p2g_roles_ok<1>() && p2g_roles_ok<2>(), "a lane's bins: one, or two in plane order");

// The roles as six pairs that share two hat functions: half 0 and 1 differ in the offset (0, -1) along k (j when the
// component's axis is k, which has three). The pair's other offsets: o1 along the first, o2 along the second of
// the remaining axes, in this order: the component's own axis offsets -1, 0, 1 (index 2, 1, 0), the other's 0, -1.
template <int A>
__host__ __device__ constexpr P2GRole p2g_pair_role(int pair, int half) {
    const int own = 1 - pair / 2, other = -(pair % 2), h = -half;
    const int ox = A == 0 ? own : other;
    const int oy = A == 1 ? own : (A == 0 ? other : h);
    const int oz = A == 2 ? own : h;
    const P2GRoles t = p2g_roles<A>();
    for (int q = 0; q < 12; ++q)
        if (t.r[q].ox == ox && t.r[q].oy == oy && t.r[q].oz == oz) return t.r[q];
    return P2GRole{9, 9, 9, -1, false};
}

template <class F, int... I>
__device__ __forceinline__ void p2g_unroll_(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void p2g_unroll(F&& f) {
    p2g_unroll_(static_cast<F&&>(f), std::make_integer_sequence<int, N>{});
}

__device__ __forceinline__ void p2g_cp4(uint32_t dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void p2g_cp16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void p2g_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A component's tile: TJ x TK cells of TI (an argument) planes. A row of bins is the 32 lanes of a warp and a plane
// has 8 rows, one per warp: one bin below the tile along j and k, and one above along the component's axis.
constexpr int P2GO_WARPS = 8, P2GO_THREADS = 32 * P2GO_WARPS;
constexpr int P2GO_SHARE_COST = 32;  // what staging a round of shares costs, in particles of a lane
constexpr int P2GO_ROW = 320;  // particles of a row staged at a time (a full row of 32 bins holds 256)
template <int A>
struct P2GTile {
    static constexpr int TJ = P2GO_WARPS - (A == 1 ? 2 : 1), TK = 32 - (A == 2 ? 2 : 1), PLANE = TJ * TK;
};
constexpr int P2GO_PLANE = 7 * 31;  // cells of the largest plane
// four planes of eight lanes' velocity and weight sums (and two planes' space for one sum that no cell has), four
// planes of counts, the warps' buffers
constexpr int P2GO_BUFFER = P2GO_ROW * 4 + 4;  // positions from a 16-byte boundary on, then the velocity component
constexpr int P2GO_SMEM = (70 * P2GO_PLANE + P2GO_WARPS * P2GO_BUFFER + 2) * 4;
static_assert((P2GO_ROW * 3 + 4) % 4 == 0 && P2GO_BUFFER % 4 == 0 && (70 * P2GO_PLANE + 2) % 4 == 0, "16-byte buffers");

struct P2GGrid {
    int nx, ny, nz, TI;
    float inv_dx, inv_ppc;
    float one;  // 1 (see add2)
};

template <int A>
__device__ __forceinline__ void p2g_ordered_tile(float* smem, int tile, const P2GGrid& g, const float* __restrict__ pos,
                                                 const float* __restrict__ vel, const int* __restrict__ offsets,
                                                 const int* __restrict__ counts, float* __restrict__ out,
                                                 float* __restrict__ ff) {
    constexpr int TJ = P2GTile<A>::TJ, TK = P2GTile<A>::TK, PLANE = P2GTile<A>::PLANE;
    const int nx = g.nx, ny = g.ny, nz = g.nz, TI = g.TI;
    float* sums = smem;  // [ring slot][lane][velocity, weight][cell of the plane]
    int* count = reinterpret_cast<int*>(smem + 66 * P2GO_PLANE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* bp = smem + 70 * P2GO_PLANE + 2 + warp * P2GO_BUFFER;
    float* bv = bp + 3 * P2GO_ROW + 4;
    const uint32_t bp32 = (uint32_t)__cvta_generic_to_shared(bp), bv32 = (uint32_t)__cvta_generic_to_shared(bv);
    const bool aligned = (((uintptr_t)pos) & 15) == 0;
    const f32x2 one = pack2(g.one, g.one);
    const int tiles_k = (nz + TK - 1) / TK, tiles_j = (ny + TJ - 1) / TJ;
    const int tk = tile % tiles_k, tj = (tile / tiles_k) % tiles_j, ti = tile / (tiles_k * tiles_j);
    const int i0 = ti * TI, j0 = tj * TJ, k0 = tk * TK;
    const int planes = min(TI, nx - i0);                     // cell planes of the tile
    const int lj = warp - 1, by = j0 + lj;                   // this warp's row of bins in every plane
    const int lk = lane - 1, bz = k0 + lk;                   // this lane's bin
    const bool in_j = by >= 0 && by <= ny - 2, in_k = bz >= 0 && bz <= nz - 2;
    const int li_end = A == 0 ? planes : planes - 1;         // bins' planes: i0 - 1 .. i0 + li_end

    // whether the tile's rows hold particles at all
    int any = 0;
    {
        const int lo = max(k0 - 1, 0), hi = min(k0 + TK - (A == 2 ? 0 : 1), nz - 2);
        for (int r = threadIdx.x; r < (li_end + 2) * P2GO_WARPS; r += P2GO_THREADS) {
            const int x = i0 - 1 + r / P2GO_WARPS, y = j0 - 1 + r % P2GO_WARPS;
            if (x < 0 || x > nx - 2 || y < 0 || y > ny - 2 || lo > hi) continue;
            const i64 a = gidx(x, y, lo, ny, nz), b = gidx(x, y, hi, ny, nz);
            any |= (__ldg(offsets + b) + __ldg(counts + b) - __ldg(offsets + a)) > 0;
        }
    }
    any = __syncthreads_or(any);
    if (any) {
        for (int c = threadIdx.x; c < (70 * P2GO_PLANE + 2) / 4; c += P2GO_THREADS)
            reinterpret_cast<float4*>(smem)[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        __syncthreads();
    }
    // A row: this lane's bin (begin, n) and the row's range [first, last), from its first non-empty bin to its last. The
    // next plane's row is looked up while this one is added and staged before the barrier, so that neither the
    // look-up nor the copy is waited for.
    int begin = 0, n = 0, first = 0, last = 0, shift = 0;
    auto look_up = [&](int li, int& b, int& c) {
        const int bx = i0 + li;
        b = c = 0;
        if (li <= li_end && bx >= 0 && bx <= nx - 2 && in_j && in_k) {
            const i64 bin = gidx(bx, by, bz, ny, nz);
            c = __ldg(counts + bin);
            b = __ldg(offsets + bin);
        }
    };
    // positions from the 16-byte boundary at or before the first (when the array starts on one), up to the
    // last float of the range; returns where the first position lies
    auto stage = [&](int base, int m) -> int {
        const float* V = vel + 3 * (i64)base + A;
        int skip = 0;
        if (aligned) {
            skip = (int)((3u * (uint32_t)base) & 3u);
            const float* P = pos + 3 * (i64)base - skip;
            const int floats = 3 * m + skip;
            for (int t = 4 * lane; t < floats; t += 128) p2g_cp16(bp32 + 4 * t, P + t, 4 * min(4, floats - t));
        } else {
            const float* P = pos + 3 * (i64)base;
            for (int t = lane; t < 3 * m; t += 32) p2g_cp4(bp32 + 4 * t, P + t);
        }
        for (int t = lane; t < m; t += 32) p2g_cp4(bv32 + 4 * t, V + 3 * t);
        return skip;
    };
    // A row of more particles than the buffer goes part after part of its range, which takes as long as each part's fullest
    // bin, or in rounds of shares, which cost P2GO_SHARE_COST particles each besides the fullest bin's.
    auto shares_pay = [&]() {
        const int fullest = __reduce_max_sync(0xffffffffu, n), share = P2GO_ROW / __popc(__ballot_sync(0xffffffffu, n > 0));
        return (last - first - 1) / P2GO_ROW * fullest > P2GO_SHARE_COST * ((fullest + share - 1) / share);
    };
    // A round: the next ones of every bin, in equal shares of the buffer (one range of the
    // row would be a few bins' and leave the other lanes without work). This lane's are q0 .. q1 - 1 in the buffer.
    auto stage_shares = [&](int& q0, int& q1) {
        const unsigned active = __ballot_sync(0xffffffffu, n > 0);
        const int share = P2GO_ROW / __popc(active);
        q0 = __popc(active & ((1u << lane) - 1u)) * share;
        q1 = q0 + min(n, share);
        for (unsigned left = active; left; left &= left - 1) {
            const int l = __ffs(left) - 1;
            const int from = __shfl_sync(0xffffffffu, begin, l), m = __shfl_sync(0xffffffffu, q1 - q0, l),
                      to = __shfl_sync(0xffffffffu, q0, l);
            const float *P = pos + 3 * (i64)from, *V = vel + 3 * (i64)from + A;
            for (int t = lane; t < 3 * m; t += 32) p2g_cp4(bp32 + 4 * (3 * to + t), P + t);
            for (int t = lane; t < m; t += 32) p2g_cp4(bv32 + 4 * (to + t), V + 3 * t);
        }
        begin += q1 - q0;
        n -= q1 - q0;
    };
    auto take = [&](int b, int c) {  // the row becomes the one at hand, its first particles staged
        begin = b;
        n = c;
        first = last = 0;
        const unsigned some = __ballot_sync(0xffffffffu, n > 0);
        if (some) {
            first = __shfl_sync(0xffffffffu, begin, __ffs(some) - 1);
            last = __shfl_sync(0xffffffffu, begin + n, 31 - __clz(some));
            shift = stage(first, min(P2GO_ROW, last - first));
        }
    };
    if (any) {
        int b, c;
        look_up(-1, b, c);
        take(b, c);
    }
    for (int li = -1; li <= li_end; ++li) {
        const int bx = i0 + li;
        if (any) {
            int next_begin, next_n;
            look_up(li + 1, next_begin, next_n);
            if (first < last) {  // warp-uniform
                const float fbx = (float)bx, fby = (float)by, fbz = (float)bz;
                // The place of a role's sums: its lane's of cell b - o, or the spare one when the tile does not have that
                // cell. A lane without particles puts back what it took (0 where it comes first), so nothing here
                // branches on a lane's own state.
                constexpr int NONE = 64 * P2GO_PLANE;
                const int here = lj * TK + lk;
                auto place = [&](const P2GRole& r) -> int {
                    const int ci = li - r.ox, cj = lj - r.oy;
                    const bool in_tile = ci >= 0 && ci < planes && cj >= 0 && cj < TJ;  // warp-uniform
                    const int c = ((ci & 3) * 16 + 2 * r.lane) * P2GO_PLANE + here - r.oy * TK - r.oz;
                    return in_tile && (unsigned)(lk - r.oz) < (unsigned)TK ? c : NONE;
                };
                f32x2 sv[6], sw[6];
                p2g_unroll<6>([&](auto index) {
                    constexpr int I = decltype(index)::value;
                    float v[2] = {0.0f, 0.0f}, w[2] = {0.0f, 0.0f};
                    p2g_unroll<2>([&](auto half) {
                        constexpr int H = decltype(half)::value;
                        constexpr P2GRole r = p2g_pair_role<A>(I, H);
                        static_assert(r.lane >= 0, "every pair is two roles");
                        if constexpr (r.second) {
                            const int c = place(r);
                            v[H] = sums[c];
                            w[H] = sums[c + P2GO_PLANE];
                        }
                    });
                    sv[I] = pack2(v[0], v[1]);
                    sw[I] = pack2(w[0], w[1]);
                });
                auto sum = [&](const float* bq, int q0, int q1) {
#pragma unroll 2
                    for (int q = q0; q < q1; ++q) {
                        const float sx = bq[3 * q] * g.inv_dx, sy = bq[3 * q + 1] * g.inv_dx, sz = bq[3 * q + 2] * g.inv_dx;
                        const float v = bv[q];
                        // hat functions at the candidate faces: along the component's own axis those of cells
                        // b - 1, b, b + 1 (at c + 1), along the others those of cells b, b + 1 (at c + 0.5)
                        float x[3], y[3], z[3];
                        if constexpr (A == 0) {
                            x[0] = tent(sx, fbx);
                            x[1] = tent(sx, fbx + 1.0f);
                            x[2] = tent(sx, fbx + 2.0f);
                        } else {
                            x[1] = tent(sx, fbx + 0.5f);
                            x[2] = tent(sx, fbx + 1.5f);
                        }
                        if constexpr (A == 1) {
                            y[0] = tent(sy, fby);
                            y[1] = tent(sy, fby + 1.0f);
                            y[2] = tent(sy, fby + 2.0f);
                        } else {
                            y[1] = tent(sy, fby + 0.5f);
                            y[2] = tent(sy, fby + 1.5f);
                        }
                        if constexpr (A == 2) {
                            z[0] = tent(sz, fbz);
                            z[1] = tent(sz, fbz + 1.0f);
                            z[2] = tent(sz, fbz + 2.0f);
                        } else {
                            z[1] = tent(sz, fbz + 0.5f);
                            z[2] = tent(sz, fbz + 1.5f);
                        }
                        // weights x * y * z, left to right; cell b - o has index 1 - o (1 is b, 2 is b + 1, 0 is b - 1)
                        const f32x2 vv = pack2(v, v);
                        // pairs along k (j when the component's axis is k)
                        const f32x2 zz = pack2(z[1], z[2]), yy = pack2(y[1], y[2]);
                        p2g_unroll<6>([&](auto index) {
                            constexpr int I = decltype(index)::value;
                            constexpr P2GRole r = p2g_pair_role<A>(I, 0);
                            f32x2 wgt;
                            if constexpr (A != 2) {
                                const float xy = x[1 - r.ox] * y[1 - r.oy];
                                wgt = mul2(pack2(xy, xy), zz);
                            } else {
                                wgt = mul2(mul2(pack2(x[1 - r.ox], x[1 - r.ox]), yy), pack2(z[1 - r.oz], z[1 - r.oz]));
                            }
                            sv[I] = add2(sv[I], mul2(wgt, vv), one);
                            sw[I] = add2(sw[I], wgt, one);
                        });
                        if constexpr (A == 0) {  // the particle's cell, for the fluid fraction: b or b + 1 on each axis
                            const int ci = clampi((int)sx, 1, nx - 2) - i0, cj = clampi((int)sy, 1, ny - 2) - j0,
                                      ck = clampi((int)sz, 1, nz - 2) - k0;
                            if (ci >= 0 && ci < planes && cj >= 0 && cj < TJ && ck >= 0 && ck < TK)
                                atomicAdd(count + (ci & 3) * P2GO_PLANE + cj * TK + ck, 1);
                        }
                    }
                };
                if (last - first > P2GO_ROW && shares_pay()) {
                    p2g_cp_wait();  // the part staged ahead
                    __syncwarp();
                    do {
                        int q0, q1;
                        stage_shares(q0, q1);
                        p2g_cp_wait();
                        __syncwarp();
                        sum(bp, q0, q1);
                        __syncwarp();
                    } while (__any_sync(0xffffffffu, n > 0));
                } else {
                    for (int base = first; base < last; base += P2GO_ROW) {
                        const int m = min(P2GO_ROW, last - base);
                        if (base > first) {
                            __syncwarp();
                            shift = stage(base, m);
                        }
                        p2g_cp_wait();
                        __syncwarp();
                        sum(bp + shift, max(begin, base) - base, min(begin + n, base + m) - base);
                    }
                }
                p2g_unroll<6>([&](auto index) {
                    constexpr int I = decltype(index)::value;
                    p2g_unroll<2>([&](auto half) {
                        constexpr int H = decltype(half)::value;
                        constexpr P2GRole r = p2g_pair_role<A>(I, H);
                        const int c = place(r);
                        sums[c] = H ? hi2(sv[I]) : lo2(sv[I]);
                        sums[c + P2GO_PLANE] = H ? hi2(sw[I]) : lo2(sw[I]);
                    });
                });
                __syncwarp();  // the buffer is free again
            }
            take(next_begin, next_n);
        }
        const int done = A == 0 ? li - 1 : li;  // the cell plane no later bins reach
        if (any) __syncthreads();
        if (done < 0) continue;
        // the ring's four slots: the next plane of bins reaches the three cell planes after this one
        for (int c = threadIdx.x; c < PLANE; c += P2GO_THREADS) {
            const int cj = j0 + c / TK, ck = k0 + c % TK;
            float value = 0.0f;
            int inside = 0;
            if (any) {
                float* l = sums + (done & 3) * 16 * P2GO_PLANE + c;
                auto tree = [&](const float* t) {  // lane q at t[2 q PLANE]
                    constexpr int L = 2 * P2GO_PLANE;
                    return ((t[0] + t[4 * L]) + (t[2 * L] + t[6 * L])) + ((t[1 * L] + t[5 * L]) + (t[3 * L] + t[7 * L]));
                };
                const float weight = tree(l + P2GO_PLANE);
                value = weight > 0.0f ? tree(l) / weight : 0.0f;
#pragma unroll
                for (int q = 0; q < 16; ++q) l[q * P2GO_PLANE] = 0.0f;
                if constexpr (A == 0) {
                    int* k = count + (done & 3) * P2GO_PLANE + c;
                    inside = *k;
                    *k = 0;
                }
            }
            if (cj < ny && ck < nz) {
                const i64 index = gidx(i0 + done, cj, ck, ny, nz);
                out[index] = value;
                if constexpr (A == 0) ff[index] = (float)inside * g.inv_ppc;
            }
        }
    }
}

// Tiles of component A; the blocks of a launch are those of u, then v, then w.
template <int A>
__host__ __device__ __forceinline__ i64 p2g_ordered_tiles(int nx, int ny, int nz, int TI) {
    return (i64)((nx + TI - 1) / TI) * ((ny + P2GTile<A>::TJ - 1) / P2GTile<A>::TJ) *
           ((nz + P2GTile<A>::TK - 1) / P2GTile<A>::TK);
}

__device__ __forceinline__ void p2g_ordered_block(float* smem, i64 block, const P2GGrid& g, const float* __restrict__ pos,
                                                  const float* __restrict__ vel, const int* __restrict__ offsets,
                                                  const int* __restrict__ counts, float* __restrict__ u,
                                                  float* __restrict__ v, float* __restrict__ w, float* __restrict__ ff) {
    const i64 nu = p2g_ordered_tiles<0>(g.nx, g.ny, g.nz, g.TI), nv = p2g_ordered_tiles<1>(g.nx, g.ny, g.nz, g.TI);
    if (block < nu) p2g_ordered_tile<0>(smem, (int)block, g, pos, vel, offsets, counts, u, ff);
    else if (block < nu + nv) p2g_ordered_tile<1>(smem, (int)(block - nu), g, pos, vel, offsets, counts, v, ff);
    else p2g_ordered_tile<2>(smem, (int)(block - nu - nv), g, pos, vel, offsets, counts, w, ff);
}

__global__ void __launch_bounds__(P2GO_THREADS, 2)
    k_p2g_ordered(const float* __restrict__ pos, const float* __restrict__ vel, const int* __restrict__ offsets,
                  const int* __restrict__ counts, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                  float* __restrict__ ff, P2GGrid g) {
    extern __shared__ __align__(16) float p2go_smem[];
    p2g_ordered_block(p2go_smem, blockIdx.x, g, pos, vel, offsets, counts, u, v, w, ff);
}

// Planes per tile. A tile walks one or two planes of bins more than it has planes of cells, so long tiles do less in
// all, but a tile is a chain of planes and a small grid needs its blocks (us with 4 / 8 / 16 planes, before the last
// refinements: 64^3 34 / 52 / 74, 96^3 148 / 134 / 153, 117 x 90 x 139 246 / 218 / 206, 256^3 1583 / 1301 / 1185).
constexpr i64 P2GO_MIN_CELLS = 1 << 17;
__host__ __device__ __forceinline__ int p2g_ordered_planes(i64 cells) {
    return cells >= (1 << 23) ? 32 : cells >= 1200000 ? 16 : cells >= (1 << 19) ? 8 : 4;
}

}  // namespace clb
