// 3x3x3 convolution (forward and data gradient) as implicit GEMM on tcgen05, marching along z with all three
// dz taps of an input slice in one MMA.
//
// What bounds it: with N = 16 or 32 output channels a tcgen05.mma of M = 128, K = 16 is limited by reading its
// A operand (4 KB from shared memory, 32 cycles), not by the tensor pipe: at one MMA per tap, 27 such reads
// per 128 voxels and 16 channels cap these layers at a quarter of the dense rate. An input slice z feeds the
// output slices z - 1, z and z + 1 with the same A operand, so the weights of the three dz taps form
// one B operand of 3 N columns, and the three output slices' accumulators lie side by side in tensor memory:
// 9 MMAs (the in-plane taps) instead of 27, each at 75-100 % of the rate for N = 16 .. 64.
//
// Block: 16 rows x (8 or 16) columns of a range of Lz output slices, every accumulator in tensor memory
// (columns (tile, output slice, channel)). An M tile is 16 rows x 8 columns: eight consecutive voxels of a row
// are one 8 x 16-byte core matrix of a staged plane (8 channels of every voxel), rows follow at a stride of one
// padded row (SBO), the other 8 channels of a K = 16 step at a stride of one plane (LBO), and an in-plane tap
// is the same operand from a start shifted by its voxel offset. No position of a halo column is computed.
// Slices run through a ring of `stages` buffers. The roles run side by side, each a chain of latencies that
// would add up in one warp: 4 warps stage slices with cp.async (zero fill outside the volume), one thread issues
// the MMAs, and 8 warps store output slices (bias + ReLU, or the ReLU mask, loaded ahead) while later slices'
// MMAs run. `full` of a slot completes when its slice is staged and the storing warps have seen the MMAs of the
// slot's last slice end (so that they never fall a whole ring behind); `empty` when its MMAs have ended.
// Blocks are persistent; weights stay in shared memory unless
// they do not fit, in which case the source channels go in passes of KC channels with double-buffered weights.
// An 8-channel source (the first layer) pairs neighbouring taps in one K = 16 step instead of padding
// with zeros: the second tap's channels are "LBO" bytes further in the same plane. The ninth tap's pair is a plane of
// zeros behind the slots (a tap again with weight 0 would turn an infinite activation into NaN).
//
// Measured (B200, 128^3, us; the same layers with one MMA per tap, N = Cout, and three slices staged per output
// slice): 8 -> 16 49 (128), 16 -> 16 64 (148), 32 -> 32 132 (548), 48 -> 16 138 (723), 96 -> 32 367 (1501),
// 32 -> 64 214 (685, now 1.08 PFLOP/s), 64 -> 64 536 (1227). What bounds it now: an MMA of M = 128, K = 16 costs
// max(46, 32 + N'/4, N'/2) cycles for N' = 3 N columns (both operands are read from shared memory at 128 bytes a
// cycle), so the 16-channel layers stay at about a third of the dense rate by their shape.
//
// The sums are FP32 accumulators as everywhere in these layers. Every mbarrier wait is
// bounded: a wait that runs out records error code 4, the other warps leave their waits, and the tensor memory is
// freed after the issued MMAs have ended.
#pragma once
#include <type_traits>

#include "conv3d.cuh"

namespace clb {
namespace conv {

constexpr int CM_EPI = 8, CM_STG = 4;               // warps storing outputs, warps staging slices
constexpr int CM_THREADS = 32 * (CM_EPI + CM_STG + 1);  // and the MMA warp (the last)
constexpr int CM_TY = 16, CM_RY = CM_TY + 2;       // output rows, staged rows
constexpr int CM_NE = 16;                          // 16-byte pieces of a slice per staging thread, at most
constexpr int CM_MAX_STAGES = 8;
constexpr int CM_SMEM_LIMIT = 226 * 1024;

struct MarchPlan {
    int nx8;               // M tiles (of 8 columns) per block
    int Lz;                // output slices per block, at most
    int KC, passes;        // source channels per pass
    int np, pieces;        // planes staged per slice, 16-byte pieces per slice
    int xt, yt, zt;        // blocks along x, y, z
    int stages, slot_bytes, w_bytes, wbufs;
    int tmem_cols, smem, grid;
    i64 tiles;
};

// The zeros an 8-channel source's ninth tap is paired with: what the 16 rows and nx8 tiles of an operand reach.
__host__ __device__ constexpr int cm_zero_bytes(int nx8) { return (15 * (8 * nx8 + 2) + 8 * nx8) * 16; }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest `pending` groups of this thread (0 .. 3)
__device__ __forceinline__ void cp_async_wait(int pending) {
    if (pending >= 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
    else if (pending == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (pending == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_st16_zero(uint32_t taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(
                     taddr),
                 "r"(0)
                 : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}\n" : "=r"(p));
    return p != 0u;
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A place in the block's sequence of slices: block tile, pass over the source channels, input slice
// z0 - 1 + i (i_lo .. i_hi: the slices inside the volume).
struct MarchCursor {
    i64 tile;
    int pass, i, i_lo, i_hi, z0, Lzt, b, x0, y0;
    bool valid;
    __device__ __forceinline__ void enter(const MarchPlan& pl, const Vol& g, i64 t) {
        tile = t;
        valid = t < pl.tiles;
        if (!valid) return;
        const int xt = (int)(t % pl.xt);
        i64 r = t / pl.xt;
        const int yt = (int)(r % pl.yt);
        r /= pl.yt;
        const int zt = (int)(r % pl.zt);
        b = (int)(r / pl.zt);
        x0 = xt * 8 * pl.nx8;
        y0 = yt * CM_TY;
        z0 = zt * pl.Lz;
        Lzt = min(pl.Lz, g.D - z0);
        i_lo = z0 == 0 ? 1 : 0;
        i_hi = z0 + Lzt == g.D ? Lzt : Lzt + 1;
        i = i_lo;
        pass = 0;
    }
    __device__ __forceinline__ void next(const MarchPlan& pl, const Vol& g) {
        if (++i <= i_hi) return;
        i = i_lo;
        if (++pass < pl.passes) return;
        enter(pl, g, tile + gridDim.x);
    }
};

// NX8: M tiles of 8 columns a block; PAIRS: an 8-channel source.
template <int N, bool DGRAD, int NX8, bool PAIRS>
__global__ void __launch_bounds__(CM_THREADS, 1)
    k_conv_march(const __nv_bfloat16* __restrict__ src, const __nv_bfloat16* __restrict__ wmat,
                 const float* __restrict__ bias, const __nv_bfloat16* __restrict__ mask_src,
                 __nv_bfloat16* __restrict__ out, Vol g, int Cs, int Kpad, int relu, MarchPlan pl) {
    static_assert(N % 16 == 0 && N >= 16 && N <= 128, "N must be a multiple of 16 in [16, 128]");
    constexpr int N3 = 3 * N;
    constexpr int RW = 8 * NX8 + 2;  // staged columns
    constexpr int P = CM_RY * RW;    // voxels of a plane
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[CM_MAX_STAGES], empty[CM_MAX_STAGES], tfree;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int failed;
    using namespace tc;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* slots = smem + pl.wbufs * pl.w_bytes;
    if (threadIdx.x == 0) {
        for (int s = 0; s < CM_MAX_STAGES; ++s) {
            mbar_init(&full[s], CM_STG + CM_EPI);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&tfree, CM_EPI);
        failed = 0;
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, (uint32_t)pl.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t zeros = smem_u32(slots) + (uint32_t)(pl.stages * pl.slot_bytes);
    if (PAIRS) {
        for (int t = threadIdx.x; t < cm_zero_bytes(NX8) / 16; t += CM_THREADS)
            reinterpret_cast<uint4*>(slots + pl.stages * pl.slot_bytes)[t] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
    }
    if (warp < 4) {  // accumulators start at zero; the epilogue leaves them at zero for the next tile
        for (int c = 0; c < pl.tmem_cols; c += 16) tmem_st16_zero(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c);
        tmem_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const int S = pl.stages;
    // a bounded wait that also gives up once another warp has failed
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        for (int n = 0; n < TC_WAIT_LIMIT; ++n) {
            if (mbar_try_wait(bar, parity)) return true;
            if ((n & 255) == 255 && failed) return false;
        }
        failed = 1;
        raise_device_error(4u);
        return false;
    };
    MarchCursor at;
    at.enter(pl, g, blockIdx.x);
    // the weights of a pass from source channel c0 on, by `threads` threads (the commit is the caller's)
    auto stage_weights = [&](int buffer, int c0, int tid, int threads) {
        const uint32_t w0 = smem_u32(smem) + (uint32_t)(buffer * pl.w_bytes);
        const int count = pl.w_bytes / 16;
        for (int t = tid; t < count; t += threads) {  // (unit, K group, output slice, n)
            const int n3 = t % N3, r = t / N3, kg = r & 1, q = r >> 1;
            const int gq = n3 / N, co = n3 - gq * N;
            const int u = PAIRS ? (q < 4 ? 2 * q + kg : 8) : q % 9;
            const int c = PAIRS ? 0 : c0 + 16 * (q / 9) + 8 * kg;
            // the unit's shift reads source voxel v + (dy, dx); slice z feeds output z - 1 + gq
            const int tap = DGRAD ? gq * 9 + (8 - u) : (2 - gq) * 9 + u;
            const bool in = PAIRS ? !(q == 4 && kg == 1) : c < Cs;
            cp_async16(w0 + (uint32_t)t * 16u, in ? wmat + (i64)co * Kpad + tap * Cs + c : wmat, in);
        }
    };
    int issued = 0;  // slices whose MMAs were issued (MMA thread)
    int s = 0;       // ring slot of the slice at hand, and the parity of its use
    uint32_t par = 0;
    auto advance = [&]() {
        if (++s == S) {
            s = 0;
            par ^= 1u;
        }
    };

    if (warp == CM_EPI + CM_STG) {
        // The whole warp runs the loop and one lane issues: descriptors are then computed in uniform registers
        // in a few cycles an MMA (46 cycles of shared-memory reads and up is all an MMA leaves).
        constexpr uint32_t SBO_B = 128, LBO_B = (uint32_t)N3 * 16u, row_bytes = (uint32_t)RW * 16u;
        constexpr int MAXG = 256 / N < 3 ? 256 / N : 3;  // output slices an instruction: at most 256 columns
        const bool leader = elect_one();
        int pass_count = -1, tile_count = 0;
        for (; at.valid; advance()) {
            if (at.i == at.i_lo) {
                ++pass_count;
                if (at.pass == 0 && tile_count++ > 0 && !wait(&tfree, (uint32_t)((tile_count - 2) & 1))) break;
            }
            if (!wait(&full[s], par)) break;
            __syncwarp();
            tc_fence_after();
            // output slices i - 2 + gq (gq = 0, 1, 2) of the tile that exist
            const int g0 = max(0, 2 - at.i), g1 = min(2, at.Lzt + 1 - at.i);
            const uint32_t slot = smem_u32(slots) + (uint32_t)(s * pl.slot_bytes);
            const uint32_t w0 = smem_u32(smem) + (uint32_t)(pl.wbufs > 1 ? (pass_count & 1) * pl.w_bytes : 0);
            const uint32_t dcol = tmem + (uint32_t)((at.i - 2 + g0) * N), tcol = (uint32_t)(pl.Lz * N);
            const int cnt = min(MAXG, g1 - g0 + 1), rest = g1 - g0 + 1 - cnt;
            const uint32_t idesc = instr_desc(TC_M, cnt * N, false, false);
            const uint64_t b0 = smem_desc(w0, LBO_B, SBO_B) + (uint64_t)(g0 * N);
            auto issue = [&](uint64_t ad, uint64_t bd) {
#pragma unroll
                for (int t = 0; t < NX8; ++t) {
                    if (leader) mma_bf16(dcol + t * tcol, ad + (uint64_t)(8 * t), bd, idesc, 1u);
                    if (MAXG < 3 && rest > 0 && leader)
                        mma_bf16(dcol + t * tcol + (uint32_t)(MAXG * N), ad + (uint64_t)(8 * t),
                                 bd + (uint64_t)(MAXG * N), instr_desc(TC_M, N, false, false), 1u);
                }
            };
            if constexpr (PAIRS) {
                // taps 2 q and 2 q + 1 of the plane, tap 8 and the zeros
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    const int u0 = 2 * q, u1 = u0 + 1;
                    const int o0 = (u0 / 3) * RW + u0 % 3, o1 = (u1 / 3) * RW + u1 % 3;
                    const uint32_t pair = q < 4 ? (uint32_t)(o1 - o0) * 16u : zeros - (slot + (uint32_t)o0 * 16u);
                    issue(smem_desc(slot, pair, row_bytes) + (uint64_t)o0, b0 + (uint64_t)(q * 2 * N3));
                }
            } else {
                uint64_t ak = smem_desc(slot, (uint32_t)P * 16u, row_bytes), bk = b0;
                for (int k = 0; k < (pl.np >> 1); ++k) {
#pragma unroll
                    for (int u = 0; u < 9; ++u)
                        issue(ak + (uint64_t)((u / 3) * RW + u % 3), bk + (uint64_t)(u * 2 * N3));
                    ak += (uint64_t)(2 * P);
                    bk += (uint64_t)(9 * 2 * N3);
                }
            }
            if (leader) mma_commit(&empty[s]);
            __syncwarp();
            ++issued;
            at.next(pl, g);
        }
    } else if (warp >= CM_EPI) {
        constexpr int ST = 32 * CM_STG;
        const int tid = (int)threadIdx.x - 32 * CM_EPI;
        uint32_t goff[CM_NE];  // the tile's pieces: source offset within a slice (16-byte units, 0 outside)
        uint32_t soff[CM_NE];  // offset in the slot (bytes)
        uint32_t inside = 0, inside_last = 0;  // bit e: piece e lies in the volume (and in the last pass's channels)
        const int ne = (pl.pieces + ST - 1) / ST;
        const int last_planes = (Cs - (pl.passes - 1) * pl.KC) / 8;
        i64 mapped = -1;
        int passes = 0;        // begun so far
        bool ok = true;
        const i64 slice_elems = (i64)g.H * g.W * Cs;
        // a slice is announced once its copies have landed, `lag` slices later; the ring is longer than that, so
        // announced slices wait for the tensor core and not the other way round
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
            if (n >= S && !(ok = wait(&empty[s], par ^ 1u))) break;  // the slot's last slice
            if (at.tile != mapped) {
                mapped = at.tile;
#pragma unroll
                for (int e = 0; e < CM_NE; ++e) {
                    const int f = min(tid + e * ST, pl.pieces - 1);  // the last round repeats a piece
                    const int p8 = f % pl.np, pos = f / pl.np;
                    const int row = pos / RW, x = pos - row * RW;
                    const int gy = at.y0 + row - 1, gx = at.x0 + x - 1;
                    const bool in = gy >= 0 && gy < g.H && gx >= 0 && gx < g.W;
                    soff[e] = (uint32_t)(p8 * P + pos) * 16u;
                    goff[e] = in ? ((uint32_t)gy * (uint32_t)g.W + (uint32_t)gx) * (uint32_t)(Cs / 8) + (uint32_t)p8 : 0u;
                    inside = (inside & ~(1u << e)) | (in ? 1u << e : 0u);
                    inside_last = (inside_last & ~(1u << e)) | (in && p8 < last_planes ? 1u << e : 0u);
                    if (e + 1 >= ne) break;
                }
            }
            const uint32_t slot = smem_u32(slots) + (uint32_t)(s * pl.slot_bytes);
            const int c0 = at.pass * pl.KC;
            const __nv_bfloat16* base = src + ((i64)at.b * g.D + (at.z0 - 1 + at.i)) * slice_elems + c0;
            const uint32_t in = at.pass == pl.passes - 1 ? inside_last : inside;
#pragma unroll
            for (int e = 0; e < CM_NE; ++e) {
                if (e >= ne) break;
                const bool ok = (in >> e) & 1u;
                cp_async16(slot + soff[e], base + (ok ? 8 * (i64)goff[e] : 0), ok);
            }
            if (at.i == at.i_lo) {  // a pass begins
                if (pl.wbufs > 1) stage_weights(passes & 1, c0, tid, ST);
                ++passes;
            }
            cp_async_commit();
            at.next(pl, g);
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
        const int row = quarter * 32 + lane, y = row >> 3, xx = row & 7;  // this thread's position in an M tile
        constexpr int CG = N / 16;
        constexpr int UNITS = (NX8 * CG + 1) / 2;  // 16-column pieces of an output slice a warp stores
        uint4 mk[UNITS][2];
        auto where = [&](const MarchCursor& c, int o, int t, bool& valid) -> i64 {
            const int gy = c.y0 + y, gx = c.x0 + 8 * t + xx;
            valid = gy < g.H && gx < g.W;
            return (((i64)c.b * g.D + c.z0 + o) * g.H + gy) * g.W + gx;
        };
        auto load_mask = [&](const MarchCursor& c, int o) {
            if (!DGRAD || !mask_src) return;
#pragma unroll
            for (int h = 0; h < UNITS; ++h) {
                const int unit = 2 * h + half, t = unit / CG, col = (unit - t * CG) * 16;
                bool valid;
                const i64 v = where(c, o, t, valid);
                if (unit < NX8 * CG && valid) {
                    const uint4* m4 = reinterpret_cast<const uint4*>(mask_src + v * N + col);
                    mk[h][0] = __ldg(m4);
                    mk[h][1] = __ldg(m4 + 1);
                }
            }
        };
        auto store_slice = [&](const MarchCursor& c, int o) {
#pragma unroll
            for (int h = 0; h < UNITS; ++h) {
                const int unit = 2 * h + half, t = unit / CG, col = (unit - t * CG) * 16;
                if (unit >= NX8 * CG) continue;  // warp-uniform
                const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((t * pl.Lz + o) * N + col);
                float acc[16];
                __syncwarp();
                tmem_ld16(ta, acc);
                tmem_st16_zero(ta);
                bool valid;
                const i64 v = where(c, o, t, valid);
                if (!valid) continue;
                if (!DGRAD) {
                    if (bias) {
                        const float4* b4 = reinterpret_cast<const float4*>(bias + col);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 bv = __ldg(b4 + e);
                            acc[4 * e] += bv.x;
                            acc[4 * e + 1] += bv.y;
                            acc[4 * e + 2] += bv.z;
                            acc[4 * e + 3] += bv.w;
                        }
                    }
                    if (relu)
#pragma unroll
                        for (int e = 0; e < 16; ++e) acc[e] = fmaxf(acc[e], 0.0f);
                } else if (mask_src) {
                    const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(mk[h]);
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (!(__bfloat162float(mb[e]) > 0.0f)) acc[e] = 0.0f;
                }
                uint4* o4 = reinterpret_cast<uint4*>(out + v * N + col);
                o4[0] = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                                   pack_bf16x2(acc[6], acc[7]));
                o4[1] = make_uint4(pack_bf16x2(acc[8], acc[9]), pack_bf16x2(acc[10], acc[11]),
                                   pack_bf16x2(acc[12], acc[13]), pack_bf16x2(acc[14], acc[15]));
            }
        };
        if (pl.wbufs == 1) {  // one pass: its weights stay for the whole block
            stage_weights(0, 0, threadIdx.x, 32 * CM_EPI);
            cp_async_commit();
            cp_async_wait(0);
            fence_proxy_async();
        }
        __syncwarp();
        if (lane == 0)
            for (int k = 0; k < S; ++k) mbar_arrive(&full[k]);  // the first use of each slot waits for no MMAs
        int stored = 0;  // output slices of the tile already stored
        for (; at.valid; advance()) {
            const bool last = at.i == at.i_hi;
            // outputs that no later slice feeds, in the last pass
            const int upto = at.pass == pl.passes - 1 ? (last ? at.Lzt : at.i - 1) : 0;
            if (stored < upto) load_mask(at, stored);
            if (!wait(&empty[s], par)) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            tc_fence_after();
            while (stored < upto) {
                store_slice(at, stored);
                if (++stored < upto) load_mask(at, stored);
            }
            if (last && at.pass == pl.passes - 1) {
                stored = 0;
                __syncwarp();
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tfree);
            }
            at.next(pl, g);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (failed && warp == CM_EPI + CM_STG)  // let MMAs already issued end (bounded)
        for (int n = max(0, issued - S); n < issued; ++n) mbar_wait(&empty[n % S], (uint32_t)((n / S) & 1));
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, (uint32_t)pl.tmem_cols);
}

// Cycles of one block tile, for comparing plans (MMA issue at the larger of the A-operand read, 32 cycles, and
// the tensor pipe's N / 2, with the staging and epilogue warps in parallel, plus the ramp of a tile).
static inline double march_tile_cycles(int N, int nx8, int Lz, int np, int passes, bool pairs) {
    const double units = pairs ? 5.0 : 9.0 * (np / 2);
    double mma = 0.0;
    for (int i = 0; i <= Lz + 1; ++i) {
        const int lo = i < 2 ? 2 - i : 0, hi = Lz + 1 - i < 2 ? Lz + 1 - i : 2;
        const int cols = (hi - lo + 1) * N;
        mma += units * nx8 * (cols / 2.0 > 32.0 ? cols / 2.0 : 32.0);
    }
    // a slice costs its staging warps a fixed chain of waits and address work, and 16 bytes a piece
    const double stage = (Lz + 2) * (600.0 + CM_RY * (8 * nx8 + 2) * np / 128.0 * 30.0);
    const double store = (Lz + 2) * 250.0 + Lz * ((nx8 * (N / 16) + 1) / 2) * 400.0 / passes;
    const double warps = stage > store ? stage : store;
    return passes * (mma > warps ? mma : warps) + 2500.0;
}

// The block shape of a layer: the (columns, output slices, channels per pass) with the least estimated time
// over the whole launch (rounds of persistent blocks times a tile's cycles) within the limits of shared memory
// (226 KB), tensor memory (512 columns) and the staging threads' registers (CM_NE pieces each). More columns share
// the halo, more slices share the two extra slices a tile stages; few tiles leave SMs idle.
static inline bool march_plan(int B, int D, int H, int W, int Cs, int N, bool pairs, int sms, MarchPlan& best) {
    double best_cost = -1.0;
    const int whole = pairs ? 8 : (Cs + 15) / 16 * 16;
    for (int nx8 : {2, 1}) {
        if (nx8 == 2 && (W <= 8 || N > 32)) continue;  // two tiles of wide layers leave too few slices
        const int most = 512 / (N * nx8);
        if (most < 1) continue;
        const int RW = 8 * nx8 + 2;
        const int xt = (W + 8 * nx8 - 1) / (8 * nx8), yt = (H + CM_TY - 1) / CM_TY;
        const int zmin = (D + most - 1) / most;
        for (int step = 0; step < 12; ++step) {
            const int zw = step < 8 ? zmin + step : (D + (16 >> (step - 7)) - 1) / (16 >> (step - 7));  // Lz 8, 4, 2, 1
            if (zw < zmin || zw > D) continue;
            const int Lz = (D + zw - 1) / zw, zt = (D + Lz - 1) / Lz;
            for (int KC = whole;; KC = KC > 48 ? 48 : KC - 16) {
                const int np = pairs ? 1 : KC / 8;
                const int passes = (whole + KC - 1) / KC;
                const int pieces = CM_RY * RW * np;
                const int w_bytes = (pairs ? 5 : 9 * (np / 2)) * 2 * 3 * N * 16;
                const int wbufs = passes > 1 ? 2 : 1;
                const int slot = (pieces * 16 + 127) / 128 * 128;
                // with passes, a weight buffer is overwritten two passes later: the ring must not reach back
                // that far (its slices in flight fit one pass)
                const int last = D - (zt - 1) * Lz + (zt > 1 ? 1 : 0);
                const int fixed = wbufs * w_bytes + (pairs ? cm_zero_bytes(nx8) : 0);
                int stages = CM_MAX_STAGES;
                if (passes > 1 && stages > last + 1) stages = last + 1;
                while (stages > 2 && fixed + stages * slot > CM_SMEM_LIMIT) --stages;
                if (pieces <= CM_NE * 32 * CM_STG && fixed + stages * slot <= CM_SMEM_LIMIT) {
                    const i64 tiles = (i64)B * zt * yt * xt;
                    const i64 rounds = (tiles + sms - 1) / sms;
                    const double cost = (double)rounds * march_tile_cycles(N, nx8, Lz, np, passes, pairs) *
                                        (stages == 2 ? 1.5 : stages < 5 ? 1.1 : 1.0);
                    if (best_cost < 0 || cost < best_cost) {
                        best_cost = cost;
                        int cols = 32;
                        while (cols < nx8 * Lz * N) cols *= 2;
                        int smem = fixed + stages * slot;
                        if (smem < 116 * 1024) smem = 116 * 1024;  // one block per SM (tensor memory)
                        best = MarchPlan{nx8, Lz, KC, passes, np, pieces, xt, yt, zt, stages, slot, w_bytes, wbufs,
                                         cols, smem, (int)(tiles < sms ? tiles : sms), tiles};
                    }
                }
                if (KC <= 16) break;
            }
        }
    }
    return best_cost >= 0.0;
}

template <int N, bool DGRAD, int NX8, bool PAIRS>
static cudaError_t conv_march_launch(const __nv_bfloat16* src, const __nv_bfloat16* wmat, const float* bias,
                                     const __nv_bfloat16* mask_src, __nv_bfloat16* out, const Vol& g, int Cs, int Kpad,
                                     int relu, const MarchPlan& pl, cudaStream_t s) {
    k_conv_march<N, DGRAD, NX8, PAIRS><<<pl.grid, CM_THREADS, pl.smem, s>>>(src, wmat, bias, mask_src, out, g, Cs, Kpad,
                                                                          relu, pl);
    return cudaPeekAtLastError();
}

// The instantiation of a plan: with `set` its shared-memory limit is raised (once, at start-up), otherwise it
// is launched.
template <int N, bool DGRAD>
static cudaError_t conv_march_run(bool set, const __nv_bfloat16* src, const __nv_bfloat16* wmat, const float* bias,
                                  const __nv_bfloat16* mask_src, __nv_bfloat16* out, const Vol& g, int Cs, int Kpad,
                                  int relu, bool pairs, const MarchPlan& pl, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    auto one = [&](auto nx8, auto pr) {
        constexpr int X = decltype(nx8)::value;
        constexpr bool PR = decltype(pr)::value;
        if (set) {
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k_conv_march<N, DGRAD, X, PR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         CM_SMEM_LIMIT);
        } else if (pl.nx8 == X && pairs == PR) {
            e = conv_march_launch<N, DGRAD, X, PR>(src, wmat, bias, mask_src, out, g, Cs, Kpad, relu, pl, s);
        }
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    one(I1{}, std::false_type{});
    if constexpr (N <= 32) one(I2{}, std::false_type{});
    if constexpr (!DGRAD) {
        one(I1{}, std::true_type{});
        if constexpr (N <= 32) one(I2{}, std::true_type{});
    }
    return e;
}

}  // namespace conv
}  // namespace clb
