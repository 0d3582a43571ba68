// Weight gradient of the 3x3x3 convolutions on tcgen05:
//   dW[tap][ci][co] += sum_v x[v + o(tap)][ci] * dy[v][co].
//
// A GEMM with K = voxels, so both operands are read MN-major (16-byte cells of 8 channels of one voxel; eight
// consecutive voxels of a row are one K group). What bounds it: a tcgen05.mma costs at least 46 cycles whatever its
// size, and with 16 or 32 channels on either side a tap alone fills a fraction of one; gathering the 27 shifted
// copies of x (the form this replaces) costs more still. So x and dy are staged once, as slices of 16 rows x
// 16 columns (x with its halo), and the taps come from addresses:
//   M: x's cells lie as [row][8-channel plane][column], so the planes of three successive rows are one
//      sequence of M groups at a stride of one row of cells: the three dy taps of up to 40 channels are rows of one
//      128-row operand (channels go in chunks of 32);
//   N: dy's cells lie as [row][slice][plane][column], so the planes of three successive slices are one sequence of
//      N groups: the three dz taps are columns of one operand of 3 x 16 or 3 x 32;
//   dx: three starts, three accumulators.
// Three MMAs per 16 voxels then cover all 27 taps. Their accumulators stay in tensor memory while the block walks
// its tiles (a range of slices each; x slice z meets the dy slices z - 1, z, z + 1 of the range); after at most
// `flush` slices they are added to dw with FP32 reductions and start again from zero, so that no sum is longer than
// the caller's chunks_per_block chunks of 64 voxels (four rows): the tensor core's FP32 accumulation truncates, and
// its error grows with the length of the chain. Fewer than WG_FINE chunks (small volumes) are less than two slices: there
// (FINE) a slice's sums end after `flush_rows` rows already, alternate between two sets of accumulators, and go into
// the flushing warps' registers, which are added to dw once per block. 16 -> 16 at 32^3 with one chunk: 18.5 us; 39 us
// when each short sum is added to dw itself. Relative error of dw at 3 x 10 x 19 x 10, 48 -> 16, one chunk: 1.3e-7;
// 2.3e-7 with the additions to dw, 1.9e-7 in the form that gathers every tap's operand.
// Rows of the operand beyond the three dy taps read whatever lies there and feed accumulator rows nobody reads.
//
// Where W is no multiple of 16 the last tile has `over` columns, and the others of its dy are zeros. A zero times an
// infinite x is not zero, so their x has to be finite: zeros beyond W, except in the tap that looks back along x, where
// the first of them meets column W - 1. That tap's K group of eight columns is replaced there (back): over = 8 takes
// zeros; over < 8 needs no second group at all (zeros for every tap), and so leaves room for a copy of the first eight
// columns without column W - 1; over > 8 (EDGE 2) stages a copy of the second eight in eight more cells a row. The zeros
// lie behind the slots, reached by the K groups' stride, which shrinks as the start moves on. 64 -> 64, us: 8 x 50^3
// 453 (437 without this), 4 x 60^3 (EDGE 2) 330 (285).
//
// Measured (B200, 8 x 64^3, us; the form that gathered every tap's operand per block of voxels): 8 -> 16 126 (440),
// 16 -> 16 125 (907), 32 -> 32 170 (1840), 48 -> 16 248 (2758), 32 -> 64 322 (2447), 96 -> 32 485 (6125),
// 64 -> 64 644 (4861). The MMAs' fixed 46 cycles bound it now (16 -> 16: 3 per 16 voxels and 8 / 7 of the slices
// make 65 us at one MMA per 46 cycles), then the staging of two operands per slice.
//
// Roles as in conv_march.cuh: 8 warps stage slices with cp.async, one warp issues, 8 warps flush.
// Bounded waits as there (error code 4).
#pragma once
#include "conv_march.cuh"

namespace clb {
namespace conv {

constexpr int WG_STG = 8, WG_FLUSH = 8;
constexpr int WG_THREADS = 32 * (WG_STG + WG_FLUSH + 1);
constexpr int WG_T = 16, WG_RW = WG_T + 2;  // rows and columns of a tile, with halo
constexpr int WG_WIDE = WG_RW + 8;          // cells of a staged row that also holds a copy of eight columns
constexpr int WG_MAX_STAGES = 6;
constexpr int WG_CI = 32;                   // input channels per block, at most
constexpr int WG_FINE = 8;                  // chunks of 64 voxels a sum below which FINE runs

struct WgradPlan {
    int Lz, xt, yt, zt;
    int ci_chunks, co_chunks;
    int stages, x_bytes, g_bytes;  // x slices in the ring, bytes of one; bytes of the dy buffer (2 Lz slices)
    int flush, flush_rows;         // slices between flushes; FINE: rows (WG_T: a slice)
    int fine, nc;
    int over;  // W % 16
    int vec;                       // dw is 16-byte aligned
    int smem, tmem_cols;
    i64 tiles;
    int blocks_per_job, grid;
};

// NC: output channels of the block (16 or 32). FINE: short sums, added up in registers (16 output channels: 80 a thread).
// EDGE: 0 where W is a multiple of 16, 1 where its last tile has up to 8 columns, 2 where it has more.
template <int NC, bool FINE, int EDGE>
__global__ void __launch_bounds__(WG_THREADS, 1)
    k_conv_wgrad_march(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                       float* __restrict__ dw, Vol g, int Cin, int Cout, WgradPlan pl) {
    using namespace tc;
    static_assert(!FINE || NC == 16, "the registers of a flushing thread hold 16 output channels");
    constexpr bool RAGGED = EDGE > 0;
    constexpr int rw = EDGE == 2 ? WG_WIDE : WG_RW;
    constexpr int NPG = NC / 8, N3 = 3 * NC, COLS = 3 * N3;
    constexpr int SETS = FINE ? 2 : 1;  // of accumulators: short sums are taken while the next are formed
    constexpr int ST = 32 * WG_STG, NEX = (WG_RW * rw * (WG_CI / 8) + ST - 1) / ST, NEG = WG_T * WG_T * NPG / ST;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[WG_MAX_STAGES], empty[WG_MAX_STAGES], acc_full[2], acc_free[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int jobs = pl.ci_chunks * pl.co_chunks;
    const int job = blockIdx.x % jobs, first = blockIdx.x / jobs;
    const int ci0 = (job % pl.ci_chunks) * WG_CI, co0 = (job / pl.ci_chunks) * NC;
    const int np = min(WG_CI, Cin - ci0) / 8;
    const int S = pl.stages, slots = 2 * pl.Lz;
    const uint32_t xs = smem_u32(smem) + (uint32_t)pl.g_bytes, gs = smem_u32(smem);
    const uint32_t zeros = xs + (uint32_t)(S * pl.x_bytes);  // 16 rows of rw cells
    if (EDGE == 1) {
        for (int c = threadIdx.x; c < 16 * rw; c += WG_THREADS)
            reinterpret_cast<uint4*>(smem + pl.g_bytes + S * pl.x_bytes)[c] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < WG_MAX_STAGES; ++s) {
            mbar_init(&full[s], WG_STG);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < SETS; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_free[a], WG_FLUSH);
        }
        failed = 0;
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, (uint32_t)pl.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (warp < 4) {
        for (int c = 0; c < SETS * COLS; c += 16) tmem_st16_zero(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c);
        tmem_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        for (int n = 0; n < TC_WAIT_LIMIT; ++n) {
            if (mbar_try_wait(bar, parity)) return true;
            if ((n & 255) == 255 && failed) return false;
        }
        failed = 1;
        raise_device_error(4u);
        return false;
    };
    // the block's sequence of x slices: tile, then input slice z0 - 1 + i inside the volume
    struct Cursor {
        i64 tile;
        int i, i_lo, i_hi, z0, Lzt, b, x0, y0, k;  // k: tiles entered before
        bool valid;
    };
    auto enter = [&](Cursor& c, i64 t) {
        c.tile = t;
        c.valid = t < pl.tiles;
        if (!c.valid) return;
        c.x0 = (int)(t % pl.xt) * WG_T;
        i64 r = t / pl.xt;
        c.y0 = (int)(r % pl.yt) * WG_T;
        r /= pl.yt;
        c.z0 = (int)(r % pl.zt) * pl.Lz;
        c.b = (int)(r / pl.zt);
        c.Lzt = min(pl.Lz, g.D - c.z0);
        c.i = c.i_lo = c.z0 == 0 ? 1 : 0;
        c.i_hi = c.z0 + c.Lzt == g.D ? c.Lzt : c.Lzt + 1;
    };
    auto next = [&](Cursor& c) {
        if (++c.i <= c.i_hi) return;
        ++c.k;
        enter(c, c.tile + pl.blocks_per_job);
    };
    Cursor at;
    at.k = 0;
    enter(at, first);
    int s = 0, issued = 0;
    uint32_t par = 0;
    auto advance = [&]() {
        if (++s == S) {
            s = 0;
            par ^= 1u;
        }
    };

    if (warp == WG_STG + WG_FLUSH) {
        const bool leader = elect_one();
        int since = 0, flushes = 0;
        for (; at.valid; advance()) {
            if (!wait(&full[s], par)) break;
            __syncwarp();
            tc_fence_after();
            const int g0 = max(0, 2 - at.i), g1 = min(2, at.Lzt + 1 - at.i);
            const uint32_t idesc = instr_desc(TC_M, (g1 - g0 + 1) * NC, true, true);
            const int slot0 = (at.k & 1) * pl.Lz + at.i - 2 + g0;
            uint32_t dcol = tmem + (uint32_t)((flushes % SETS) * COLS + g0 * NC);
            const uint32_t x0 = xs + (uint32_t)(s * pl.x_bytes), xrow = (uint32_t)rw * 16u;
            uint64_t bd = smem_desc(gs + (uint32_t)(slot0 * NPG) * 256u, 128u, 256u);
            const uint64_t astep = (uint64_t)(np * rw), bstep = (uint64_t)(slots * NPG * 16);
            const int rows = min(WG_T, g.H - at.y0);
            auto flush = [&]() {  // ends the sums of a set; returns once the next set's last ones are taken
                if (leader) mma_commit(&acc_full[flushes % SETS]);
                __syncwarp();
                ++flushes;
                if (flushes >= SETS && !wait(&acc_free[flushes % SETS], (uint32_t)((flushes / SETS - 1) & 1))) return false;
                tc_fence_after();
                if (FINE) dcol = tmem + (uint32_t)((flushes % SETS) * COLS + g0 * NC);
                return true;
            };
            // the slice's rows: the taps from ad, the one that looks back from `back` (LAST: the overhanging tile)
            auto slice = [&](auto last, uint64_t ad, uint64_t ad_step, uint64_t back, uint64_t back_step) {
                constexpr bool LAST = decltype(last)::value;
                auto row = [&]() {
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
                        if (leader)
                            mma_bf16(dcol + (uint32_t)(dx * N3), LAST && dx == 0 ? back : ad + (uint64_t)dx, bd, idesc, 1u);
                    ad += ad_step;
                    if (LAST) back += back_step;
                    bd += bstep;
                };
                if constexpr (FINE) {
                    for (int y = 0;;) {
#pragma unroll 4
                        for (const int end = min(rows, y + pl.flush_rows); y < end; ++y) row();
                        if (y == rows) return true;
                        if (!flush()) return false;
                    }
                } else {
#pragma unroll 4
                    for (int y = 0; y < rows; ++y) row();
                    return true;
                }
            };
            bool ok;
            const uint64_t plain = smem_desc(x0, 128u, xrow);
            if (RAGGED && at.x0 + WG_T > g.W) {
                const uint64_t to_zeros = astep - (astep << 16);  // the start moves on, start + stride stays
                if (EDGE == 1 && pl.over < 8)
                    ok = slice(std::true_type{}, smem_desc(x0, zeros - x0, xrow), to_zeros,
                               smem_desc(x0 + 160u, zeros - x0 - 160u, xrow), to_zeros);
                else if (EDGE == 1)
                    ok = slice(std::true_type{}, plain, astep, smem_desc(x0, zeros - x0, xrow), to_zeros);
                else
                    ok = slice(std::true_type{}, plain, astep, smem_desc(x0, (uint32_t)WG_RW * 16u, xrow), astep);
            } else {
                ok = slice(std::false_type{}, plain, astep, plain, astep);
            }
            if (leader) mma_commit(&empty[s]);
            __syncwarp();
            ++issued;
            if (!ok) break;
            next(at);
            if (++since == pl.flush || !at.valid) {
                since = 0;
                if (!flush()) break;
            }
        }
    } else if (warp >= WG_FLUSH) {
        const int tid = (int)threadIdx.x - 32 * WG_FLUSH;
        uint32_t xoff[NEX], xdst[NEX], goff[NEG], gdst[NEG];  // source offsets in a slice (16-byte units), cells
        uint32_t xin = 0, gin = 0;
        i64 mapped = -1;
        bool ok = true;
        const int xpieces = WG_RW * rw * np, nex = (xpieces + ST - 1) / ST;
        const i64 xslice = (i64)g.H * g.W * Cin, gslice = (i64)g.H * g.W * Cout;
        const int lag = S >= 6 ? 3 : S >= 4 ? 2 : 1;
        int announce_s = 0, ahead = 0;
        auto announce = [&](int pending) {
            cp_async_wait(pending);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[announce_s]);
            announce_s = announce_s + 1 == S ? 0 : announce_s + 1;
        };
        for (int n = 0; at.valid; ++n, advance()) {
            if (n >= S && !(ok = wait(&empty[s], par ^ 1u))) break;
            if (at.tile != mapped) {
                mapped = at.tile;
                xin = gin = 0;
#pragma unroll
                for (int e = 0; e < NEX; ++e) {
                    const int f = min(tid + e * ST, xpieces - 1);
                    const int p = f % np, pos = f / np, row = pos / rw, cell = pos - row * rw;
                    int col = cell, end = WG_RW;  // a cell's column, and the first one that it leaves out
                    if (EDGE) {
                        const bool last = at.x0 + WG_T > g.W;
                        if (EDGE == 1 && last && pl.over < 8 && cell >= 10) {  // the copy of columns 0 .. 7
                            col = cell - 10;
                            end = pl.over;
                        } else if (EDGE == 2 && cell >= WG_RW) {  // the copy of columns 8 .. 15
                            col = cell - WG_RW + 8;
                            end = last ? pl.over : 0;
                        }
                    }
                    const int gy = at.y0 + row - 1, gx = at.x0 + col - 1;
                    const bool in = gy >= 0 && gy < g.H && gx >= 0 && gx < g.W && col < end;
                    xdst[e] = (uint32_t)((row * np + p) * rw + cell) * 16u;
                    xoff[e] = in ? ((uint32_t)gy * (uint32_t)g.W + (uint32_t)gx) * (uint32_t)(Cin / 8) + (uint32_t)p : 0u;
                    xin |= in ? 1u << e : 0u;
                }
#pragma unroll
                for (int e = 0; e < NEG; ++e) {
                    const int f = tid + e * ST;
                    const int p = f % NPG, pos = f / NPG, row = pos / WG_T, col = pos - row * WG_T;
                    const int gy = at.y0 + row, gx = at.x0 + col;
                    const bool in = gy < g.H && gx < g.W;
                    gdst[e] = (uint32_t)((row * slots * NPG + p) * WG_T + col) * 16u;
                    goff[e] = in ? ((uint32_t)gy * (uint32_t)g.W + (uint32_t)gx) * (uint32_t)(Cout / 8) + (uint32_t)p : 0u;
                    gin |= in ? 1u << e : 0u;
                }
            }
            const uint32_t slot = xs + (uint32_t)(s * pl.x_bytes);
            const __nv_bfloat16* xb = x + ((i64)at.b * g.D + (at.z0 - 1 + at.i)) * xslice + ci0;
#pragma unroll
            for (int e = 0; e < NEX; ++e) {
                if (e >= nex) break;
                const bool in = (xin >> e) & 1u;
                cp_async16(slot + xdst[e], xb + (in ? 8 * (i64)xoff[e] : 0), in);
            }
            // the dy slices this x slice is the first to meet
            for (int o = at.i == at.i_lo ? 0 : at.i; o <= at.i && o < at.Lzt; ++o) {
                const uint32_t dst = gs + (uint32_t)(((at.k & 1) * pl.Lz + o) * NPG) * 256u;
                const __nv_bfloat16* gb = dy + ((i64)at.b * g.D + at.z0 + o) * gslice + co0;
#pragma unroll
                for (int e = 0; e < NEG; ++e) {
                    const bool in = (gin >> e) & 1u;
                    cp_async16(dst + gdst[e], gb + (in ? 8 * (i64)goff[e] : 0), in);
                }
            }
            cp_async_commit();
            next(at);
            if (++ahead > lag) {
                announce(lag);
                --ahead;
            }
        }
        if (ok)
            for (; ahead > 0; --ahead) announce(ahead - 1);
        cp_async_wait(0);
    } else {
        const int quarter = warp & 3, half = warp >> 2;
        const int m = quarter * 32 + lane, m8 = m >> 3;
        const int ty = m8 / np, ci = ci0 + (m8 - ty * np) * 8 + (m & 7);
        const bool used = m8 < 3 * np;
        const bool any = quarter * 4 < 3 * np;  // the quarter holds some used row
        int since = 0, flushes = 0, y = 0;
        // columns 16 c .. 16 c + 15 of the accumulators are taken by the warps with c % 2 == half
        constexpr int UNITS = (COLS / 16 + 1) / 2;
        float sum[FINE ? UNITS : 1][16];
        if (FINE)
#pragma unroll
            for (int u = 0; u < UNITS; ++u)
#pragma unroll
                for (int q = 0; q < 16; ++q) sum[u][q] = 0.0f;
        auto add_to_dw = [&](int c, const float* v) {
            const int tx = 16 * c / N3, rem = 16 * c - tx * N3, gq = rem / NC, co = co0 + rem - gq * NC;
            const int tap = (2 - gq) * 9 + ty * 3 + tx;
            float* to = dw + ((i64)tap * Cin + ci) * Cout + co;
            if (pl.vec) {
#pragma unroll
                for (int q = 0; q < 16; q += 4)
                    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to + q), "f"(v[q]), "f"(v[q + 1]),
                                 "f"(v[q + 2]), "f"(v[q + 3])
                                 : "memory");
            } else {
#pragma unroll
                for (int q = 0; q < 16; ++q) atomicAdd(to + q, v[q]);
            }
        };
        while (at.valid) {
            if (FINE) y += pl.flush_rows;
            if (!FINE || y >= min(WG_T, g.H - at.y0)) {  // the slice ends
                y = 0;
                next(at);
                if (++since != pl.flush && at.valid) continue;
                since = 0;
            }
            const int set = flushes % SETS;
            if (!wait(&acc_full[set], (uint32_t)((flushes / SETS) & 1))) break;
            ++flushes;
            __syncwarp();
            tc_fence_after();
            if (any)
#pragma unroll
                for (int u = 0; u < UNITS; ++u) {
                    const int c = half + 2 * u;
                    if (c >= COLS / 16) break;  // warp-uniform
                    const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(set * COLS + 16 * c);
                    float v[16];
                    __syncwarp();
                    tmem_ld16(ta, v);
                    tmem_st16_zero(ta);
                    if (FINE) {
#pragma unroll
                        for (int q = 0; q < 16; ++q) sum[FINE ? u : 0][q] += v[q];
                    } else if (used) {
                        add_to_dw(c, v);
                    }
                }
            __syncwarp();
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_free[set]);
        }
        if (FINE && used)
#pragma unroll
            for (int u = 0; u < UNITS; ++u)
                if (half + 2 * u < COLS / 16) add_to_dw(half + 2 * u, sum[FINE ? u : 0]);
    }
    tc_fence_before();
    __syncthreads();
    if (failed && warp == WG_STG + WG_FLUSH)  // let MMAs already issued end (bounded)
        for (int n = max(0, issued - S); n < issued; ++n) mbar_wait(&empty[n % S], (uint32_t)((n / S) & 1));
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, (uint32_t)pl.tmem_cols);
}

// Slices per tile: the one with the least estimated time (rounds of tiles times their slices, two of them halo)
// that fits shared memory with a ring of at least two x slices. The ring must not reach back into the tile
// before the last (its dy slots are reused), so it is no longer than the shortest tile.
static inline bool wgrad_plan(int B, int D, int H, int W, int Cin, int Cout, int chunks_per_block, bool aligned, int sms,
                              WgradPlan& best) {
    // 32 output channels a block halve the staging of x; short sums are kept in registers, 16 channels' (FINE)
    const bool fine = chunks_per_block < WG_FINE;
    const int NC = Cout == 16 || fine ? 16 : 32;
    const int npx = (Cin < WG_CI ? Cin : WG_CI) / 8;
    WgradPlan p{};
    p.xt = (W + WG_T - 1) / WG_T;
    p.yt = (H + WG_T - 1) / WG_T;
    p.ci_chunks = (Cin + WG_CI - 1) / WG_CI;
    p.co_chunks = Cout / NC;
    const int jobs = p.ci_chunks * p.co_chunks;
    p.over = W % WG_T;
    const int rw = p.over > 8 ? WG_WIDE : WG_RW;
    p.x_bytes = WG_RW * rw * npx * 16;
    // 4 chunks of 64 voxels: one slice of 16 x 16
    p.fine = fine ? 1 : 0;
    p.nc = NC;
    p.flush = fine ? 1 : chunks_per_block / 4;
    p.flush_rows = chunks_per_block < 4 ? 4 * chunks_per_block : WG_T;
    p.vec = aligned ? 1 : 0;
    p.tmem_cols = NC == 16 && !fine ? 256 : 512;
    const int tail = 16 * rw * 16;  // operand rows past the last slot's end are read (and dropped); EDGE 1: zeros
    const int per_job = sms / jobs > 0 ? sms / jobs : 1;
    double best_cost = -1.0;
    for (int Lz = D < 16 ? D : 16; Lz >= 1; --Lz) {
        p.Lz = Lz;
        p.zt = (D + Lz - 1) / Lz;
        if (p.zt > 1 && (D + p.zt - 1) / p.zt != Lz) continue;  // an even split
        p.g_bytes = 2 * Lz * WG_T * (NC / 8) * 256;
        const int last = D - (p.zt - 1) * Lz + (p.zt > 1 ? 1 : 0);
        int stages = WG_MAX_STAGES < last + 1 ? WG_MAX_STAGES : last + 1;
        while (stages > 2 && p.g_bytes + stages * p.x_bytes + tail > CM_SMEM_LIMIT) --stages;
        if (p.g_bytes + stages * p.x_bytes + tail > CM_SMEM_LIMIT) continue;
        p.stages = stages;
        p.smem = p.g_bytes + stages * p.x_bytes + tail;
        if (p.smem < 116 * 1024) p.smem = 116 * 1024;  // one block per SM (tensor memory)
        p.tiles = (i64)B * p.zt * p.yt * p.xt;
        p.blocks_per_job = (int)(p.tiles < per_job ? p.tiles : per_job);
        p.grid = p.blocks_per_job * jobs;
        const i64 rounds = (p.tiles + p.blocks_per_job - 1) / p.blocks_per_job;
        const double cost = (double)rounds * ((Lz + 2) * (stages < 4 ? 1.3 : 1.0) + 0.5);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = p;
        }
    }
    return best_cost >= 0.0;
}

}  // namespace conv
}  // namespace clb
