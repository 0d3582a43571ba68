// Bottom of the W-cycle in one launch.
//
// With L levels the second-coarsest level A = L-2 is visited 2^(L-2) times per W-cycle, and each
// visit runs (multigrid.py:53-187) pre-smoothing of A, restriction to the coarsest level B, two
// coarse solves of B (multigrid.py:127-170, 2 + 64 red-black iterations each), prolongation and
// post-smoothing of A: about 280 dependent red-black phases on a few thousand cells. As separate
// launches these are bound by launch latency; here one block of 512 threads runs the whole visit
// with both levels in shared memory and block barriers between phases.
//
// Each thread owns a fixed set of A cells and B cells of either colour (colour slots, below); the
// cell index, diagonal and delta^2 * b of each owned cell stay in registers across all sweeps (the
// neighbour weights of A cells are read from shared memory, those of B cells are registers too). The
// update formula and every summation order are those of multigrid.cl (rbgs_step, restrict_residual,
// prolongate), so the result is identical to the launch-per-kernel W-cycle.
//
// What bounds a visit is the latency of B's dependent phases (264 a visit with the reference's counts): a barrier,
// six shared-memory loads, a chain of five additions, a division and a store. So a phase is kept short:
//   * only as many warps as hold fluid cells of B take part, one cell of a colour per thread as long as 16 warps
//     suffice (a second cell costs a thread 50-90 cycles, another warp 2-6), and one warp needs no barrier;
//   * B's p lies split by colour (split_cell): consecutive words per phase instead of every second one;
//   * the addresses of a cell's six neighbours are registers, and the division is divide_by.
// Cycles of a phase (B200, 25 / 256 / 512 cells of a colour): 151 / 186 / 240; with 8 warps throughout, up to two
// cells a thread, unsplit rows and the general division 211 / 224 / 384.
#pragma once
#include "divide.cuh"
#include "multigrid.cuh"

namespace clb {

constexpr int BOTTOM_THREADS = 512;
constexpr int BOTTOM_MAX_A = 8;  // A slots of each colour per thread
constexpr int BOTTOM_MAX_B = 4;  // B slots of each colour per 256 threads

static inline size_t bottom_smem_bytes(int ca, int cb) {
    // A: p, b, op(float4); B: p, op(float4); the fluid-cell lists of both colours of both levels and
    // their four counts; each region padded to 16 bytes
    auto pad = [](size_t x) { return (x + 15) & ~(size_t)15; };
    return pad((size_t)ca * 4) * 2 + (size_t)ca * 16 + pad((size_t)cb * 4) + (size_t)cb * 16 +
           pad((size_t)(ca + cb + 8) * 4);
}

// Cells of one colour are numbered by slots: the interior rows (i, j) in index order, ceil(mz / 2)
// slots per row, slot s of a row being its (s+1)-th cell of the colour, k = k0 + 2 s with k0 the
// row's first such k (1 or 2). With an odd interior extent along k the last slot of every other row
// is empty. A colour phase updates cells of one colour only, and those are independent of each other,
// so any assignment of cells to threads gives the same result; numbering by colour keeps every lane
// of a warp busy in every phase.
__host__ __device__ __forceinline__ int colour_slots(int nx, int ny, int nz) {
    return (nx - 2) * (ny - 2) * ((nz - 1) / 2);
}

// smem / grid index of slot r of colour `colour`, or -1 for an empty slot or r past the last slot
__device__ __forceinline__ int colour_cell(int r, int colour, int nx, int ny, int nz) {
    const int half = (nz - 1) / 2, my = ny - 2;
    const int row = r / half, s = r - row * half;
    const int i = 1 + row / my, j = 1 + row % my;
    const int k = 1 + 2 * s + ((i + j + 1 + colour) & 1);
    if (i > nx - 2 || k > nz - 2) return -1;
    return (i * ny + j) * nz + k;
}

// B's p in shared memory: cells of one colour together, rows of half = (nz - 1) / 2 slots (those of the
// interior; rows of the ghost layer exist and hold 0), colour 0 first, after one word that always holds 0
// (what neighbours in the ghost layer along k read). Never more words than the level has cells. All six
// neighbours of a cell are of the other colour: along i and j in the same slot of other rows, along k in
// slots s + t - 1 and s + t of its own row, t = (k - 1) & 1.
__device__ __forceinline__ int split_cell(int i, int j, int k, int nx, int ny, int nz) {
    const int half = (nz - 1) / 2;
    return 1 + (((i + j + k) & 1) * nx * ny + i * ny + j) * half + ((k - 1) >> 1);
}

// Constants of one owned cell of the second-coarsest level: smem index, 1 / diagonal (0: a fluid cell with diagonal 0,
// not updated; -1: not fluid, or a slot without a cell) and delta^2 * b. The diagonal comes with the weights (one
// 16-byte load). With more than four cells of a colour per thread (keep_rhs) delta^2 * b is formed again in every
// sweep instead of kept, so that fewer of the owned cells spill (15 x 20 x 19 over 9 x 12 x 11, a visit: 33 us, 39
// with both kept and every thread taking two cells of B in every phase).
struct OwnedCell {
    int c;
    float r;
    float d2b;
};
__host__ __device__ constexpr bool keep_rhs(int KA) { return KA <= 4; }

// Owned coarsest-level cell with its neighbour weights in registers (constant for the whole visit).
struct OwnedCellW {
    int c;       // split_cell of the cell
    int zp, zm;  // split cells of its neighbours along k
    float d, r, d2b;
    float wxp, wxm, wyp, wym, wzp, wzm;
};

// sx, sy: split-layout strides along i and j; other: words from a cell to its slot in the other colour.
__device__ __forceinline__ float relaxed_w(const OwnedCellW& o, const float* sp, int other, int sx, int sy) {
    const int n = o.c + other;
    const float ws = o.wxp * sp[n + sx] + o.wxm * sp[n - sx] + o.wyp * sp[n + sy] + o.wym * sp[n - sy] +
                     o.wzp * sp[o.zp] + o.wzm * sp[o.zm];
    return divide_by(ws - o.d2b, o.d, o.r);
}

// One red-black update of an owned cell (multigrid.cl:225-229), p and weights in shared memory.
template <bool KEEP>
__device__ __forceinline__ float relaxed(const OwnedCell& o, const float* sp, const float4* so, const float* sb,
                                         float d2, int sx, int sy) {
    const int c = o.c;
    const float4 self = so[c];
    const float ws = self.y * sp[c + sx] + so[c - sx].y * sp[c - sx] + self.z * sp[c + sy] + so[c - sy].z * sp[c - sy] +
                     self.w * sp[c + 1] + so[c - 1].w * sp[c - 1];
    return divide_by(ws - (KEEP ? o.d2b : d2 * sb[c]), self.x, o.r);
}

// The updates of a warp's owned slots 0 .. active - 1 of one colour (active is the same in the whole warp), two
// at a time with both cells' loads ahead of either store: the cells of a colour are independent, and a phase
// costs what its chains of loads and additions take, one after the other or side by side.
template <int K, class Value, class Put>
__device__ __forceinline__ void relax_slots(int active, Value&& value, Put&& put) {
#pragma unroll
    for (int m = 0; m < K; m += 2) {
        if (m + 1 < K && m + 1 < active) {
            const float a = value(m), b = value(m + 1);
            put(m, a);
            put(m + 1, b);
        } else if (m < active) {
            put(m, value(m));
        }
    }
}

// Slots in use by this warp when `count` cells go to `threads` threads in turn.
__device__ __forceinline__ int active_slots(int count, int threads) {
    const int first = (int)(threadIdx.x & ~31u);
    return count > first ? (count - first + threads - 1) / threads : 0;
}

// The coarsest level B: thread t owns the fluid cells t, t + 512 of either colour (bottom_lists), so the first
// warps own them all, and those synchronise with a named barrier. BOTTOM_BTHREADS is what a plan counts B's
// slots by (KB slots per 256 threads: BOTTOM_KB cells of a colour per thread here).
constexpr int BOTTOM_BTHREADS = 256;
__host__ __device__ constexpr int bottom_kb(int KB) { return (KB + 1) / 2; }

// Phases of B: warps 0 .. warps - 1 take part.
__device__ __forceinline__ void bar_b(int warps) {
    if (warps > 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * warps) : "memory");
    else __syncwarp();
}

// Shared-memory arrays of a bottom visit: A's p, b and operator (float4, diagonal -1 where not
// fluid), B's p and operator, and the fluid cells of each colour of both levels; each region padded to
// 16 bytes (bottom_smem_bytes).
struct BottomSmem {
    float* spa;
    float* sba;
    float4* soa;
    float* spb;
    float4* sob;
    int* count;   // fluid cells: A colour 0, A colour 1, B colour 0, B colour 1
    int* list_a;  // two lists of CA / 2 + 1 entries
    int* list_b;  // two lists of CB / 2 + 1 entries
};

__device__ __forceinline__ BottomSmem bottom_smem(unsigned char* base, int CA, int CB) {
    auto pad = [](int x) { return (x + 3) & ~3; };  // in floats
    BottomSmem S;
    S.spa = reinterpret_cast<float*>(base);
    S.sba = S.spa + pad(CA);
    S.soa = reinterpret_cast<float4*>(S.sba + pad(CA));
    S.spb = reinterpret_cast<float*>(S.soa + CA);
    S.sob = reinterpret_cast<float4*>(S.spb + pad(CB));
    S.count = reinterpret_cast<int*>(S.sob + CB);
    S.list_a = S.count + 4;
    S.list_b = S.list_a + 2 * (CA / 2 + 1);
    return S;
}

// Lists the fluid interior cells of each colour of both levels (after the operators are staged and
// the block has synchronised). Their order is arbitrary -- cells of one colour are independent -- and
// the threads take them in turn, so a warp's owned cells are fluid but for the last ones and the empty
// slots beyond the count are empty in whole warps: a phase costs what the fluid needs, not what the
// level's size does.
__device__ __forceinline__ void bottom_lists(const BottomSmem& S, int anx, int any, int anz, int bnx, int bny,
                                             int bnz) {
    const int CA = anx * any * anz, CB = bnx * bny * bnz;
    const int la = CA / 2 + 1, lb = CB / 2 + 1;
    if (threadIdx.x < 4) S.count[threadIdx.x] = 0;
    __syncthreads();
    const int sa = colour_slots(anx, any, anz), sb = colour_slots(bnx, bny, bnz);
    for (int colour = 0; colour < 2; ++colour) {
        for (int r = threadIdx.x; r < sa; r += BOTTOM_THREADS) {
            const int c = colour_cell(r, colour, anx, any, anz);
            if (c >= 0 && S.soa[c].x >= 0.0f) S.list_a[colour * la + atomicAdd(S.count + colour, 1)] = c;
        }
        for (int r = threadIdx.x; r < sb; r += BOTTOM_THREADS) {
            const int c = colour_cell(r, colour, bnx, bny, bnz);
            if (c >= 0 && S.sob[c].x >= 0.0f) S.list_b[colour * lb + atomicAdd(S.count + 2 + colour, 1)] = c;
        }
    }
    __syncthreads();
}

// Staging of the operators of both levels and, when pa / ba are given, of A's p and b (FP16 levels
// are converted to FP32). Four cells per thread and round, all loads issued before the stores.
template <bool H>
__device__ __forceinline__ void bottom_stage(const BottomSmem& S, const float* __restrict__ pa,
                                             const float* __restrict__ ba, const float4* __restrict__ opa,
                                             const uint8_t* __restrict__ ma, int CA, const float4* __restrict__ opb,
                                             const uint8_t* __restrict__ mb, int CB) {
    auto ld = [&](const float* a, int c) -> float {
        return H ? ldh(reinterpret_cast<const __half*>(a), c) : a[c];
    };
    auto ld4 = [&](const float4* a, int c) -> float4 {
        return H ? ld_h4(reinterpret_cast<const Half4*>(a), c) : a[c];
    };
    constexpr int U = 4;
    for (int c0 = threadIdx.x; c0 < CA; c0 += U * BOTTOM_THREADS) {
        float pv[U], bv[U];
        float4 ov[U];
        uint8_t mv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * BOTTOM_THREADS;
            if (c < CA) {
                pv[u] = pa ? ld(pa, c) : 0.0f;
                bv[u] = ba ? ld(ba, c) : 0.0f;
                ov[u] = ld4(opa, c);
                mv[u] = ma[c];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * BOTTOM_THREADS;
            if (c < CA) {
                if (pa) S.spa[c] = pv[u];
                if (ba) S.sba[c] = bv[u];
                float4 o = ov[u];
                if (!mv[u]) o.x = -1.0f;
                S.soa[c] = o;
            }
        }
    }
    for (int c0 = threadIdx.x; c0 < CB; c0 += U * BOTTOM_THREADS) {
        float4 ov[U];
        uint8_t mv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * BOTTOM_THREADS;
            if (c < CB) {
                ov[u] = ld4(opb, c);
                mv[u] = mb[c];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * BOTTOM_THREADS;
            if (c < CB) {
                float4 o = ov[u];
                if (!mv[u]) o.x = -1.0f;
                S.sob[c] = o;
            }
        }
    }
}

// The cells a thread owns in a bottom visit: A cells of each colour (index, diagonal, delta^2 * b) and
// B cells of each colour with their neighbour weights. Index, diagonal and weights depend on the
// operators only, so a launch that visits A several times sets them once (bottom_cells); A's delta^2 * b
// is set again whenever A's right-hand side changes (bottom_rhs).
template <int KA, int KB>
struct BottomCells {
    OwnedCell A[2][KA];   // [colour][m]: the thread's fluid cells (bottom_lists)
    OwnedCellW B[2][bottom_kb(KB)];  // [colour][m]
};

// After the lists are built and the block has synchronised.
template <int KA, int KB>
__device__ __forceinline__ void bottom_cells(const BottomSmem& S, BottomCells<KA, KB>& R, int anx, int any, int anz,
                                             int bnx, int bny, int bnz) {
    const int la = (anx * any * anz) / 2 + 1, lb = (bnx * bny * bnz) / 2 + 1;
    const int bsx = bny * bnz, bsy = bnz;
#pragma unroll
    for (int colour = 0; colour < 2; ++colour)
#pragma unroll
        for (int m = 0; m < KA; ++m) {
            const int r = threadIdx.x + m * BOTTOM_THREADS;
            const int c = r < S.count[colour] ? S.list_a[colour * la + r] : -1;
            OwnedCell& o = R.A[colour][m];
            o.c = c < 0 ? (any + 1) * anz + 1 : c;  // a slot without a cell loads an interior cell and stores nothing
            const float d = c < 0 ? -1.0f : S.soa[c].x;  // fluid: >= 0
            o.r = d > 0.0f ? 1.0f / d : d < 0.0f ? -1.0f : 0.0f;
            o.d2b = 0.0f;
        }
#pragma unroll
    for (int colour = 0; colour < 2; ++colour)
#pragma unroll
        for (int m = 0; m < bottom_kb(KB); ++m) {
            const int r = threadIdx.x + m * BOTTOM_THREADS;
            const int c = r < S.count[2 + colour] ? S.list_b[colour * lb + r] : -1;
            OwnedCellW& o = R.B[colour][m];
            o.d2b = 0.0f;
            o.zp = o.zm = 0;
            o.c = 1 + (colour * bnx + 1) * bny * ((bnz - 1) / 2);  // a slot without a cell loads some cells, stores nothing
            o.d = o.r = -1.0f;
            o.wxp = o.wxm = o.wyp = o.wym = o.wzp = o.wzm = 0.0f;
            if (c >= 0) {
                const float4 self = S.sob[c];
                const int i = c / bsx, j = (c / bsy) % bny, k = c % bnz;
                o.c = split_cell(i, j, k, bnx, bny, bnz);
                const int up = o.c + (colour ? -1 : 1) * bnx * bny * ((bnz - 1) / 2) + ((k - 1) & 1);
                o.zp = k + 1 <= bnz - 2 ? up : 0;
                o.zm = k > 1 ? up - 1 : 0;
                o.d = self.x;
                o.r = 1.0f / o.d;
                o.wxp = self.y;
                o.wyp = self.z;
                o.wzp = self.w;
                o.wxm = S.sob[c - bsx].y;
                o.wym = S.sob[c - bsy].z;
                o.wzm = S.sob[c - 1].w;
            }
        }
}

// A's delta^2 * b of the owned cells, after A's right-hand side is in shared memory and visible.
template <int KA, int KB>
__device__ __forceinline__ void bottom_rhs(const BottomSmem& S, BottomCells<KA, KB>& R, float d2) {
#pragma unroll
    for (int colour = 0; colour < 2; ++colour)
#pragma unroll
        for (int m = 0; m < KA; ++m) {
            OwnedCell& o = R.A[colour][m];
            if (keep_rhs(KA)) o.d2b = o.r < 0.0f ? 0.0f : d2 * S.sba[o.c];
        }
}

// One visit of A from staged shared memory with the owned cells set (bottom_cells, bottom_rhs):
// pre-smoothing of A, restriction into B (B's p zeroed, multigrid.cl:114), the two coarse solves of B,
// prolongation, post-smoothing of A. bb (nullable): B's right-hand side is stored there (FP16 when H).
// KA: A slots of each colour per thread (of BOTTOM_THREADS); KB: B slots of each colour per 256 threads.
template <int KA, int KB, bool H>
__device__ __forceinline__ void bottom_core(const BottomSmem& S, BottomCells<KA, KB>& R, int anx, int any, int anz,
                                            int bnx, int bny, int bnz, float d2, float inv_delta2, int pre, int post,
                                            int coarse_iters, float* __restrict__ bb, int b_solves = 2,
                                            float w = 1.0f) {
    float* spa = S.spa;
    const float* sba = S.sba;
    const float4* soa = S.soa;
    float* spb = S.spb;
    const int CB = bnx * bny * bnz;
    auto st = [&](float* a, int c, float v) {
        if (H) reinterpret_cast<__half*>(a)[c] = __float2half_rn(v);
        else a[c] = v;
    };
    const int asx = any * anz, asy = anz, bsx = bny * bnz, bsy = bnz;
    const int half = (bnz - 1) / 2;  // split-layout strides: bny * half along i, half along j
    const int lb = CB / 2 + 1;
    constexpr int MB = bottom_kb(KB);
    OwnedCell (&A)[2][KA] = R.A;
    OwnedCellW (&B)[2][MB] = R.B;

    const int aslots[2] = {active_slots(S.count[0], BOTTOM_THREADS), active_slots(S.count[1], BOTTOM_THREADS)};
    auto smooth_a = [&](int iterations) {
        for (int it = 0; it < iterations; ++it)
#pragma unroll
            for (int colour = 0; colour < 2; ++colour) {
                relax_slots<KA>(
                    aslots[colour], [&](int m) { return relaxed<keep_rhs(KA)>(A[colour][m], spa, soa, sba, d2, asx, asy); },
                    [&](int m, float v) {
                        if (A[colour][m].r > 0.0f) spa[A[colour][m].c] = v;
                    });
                __syncthreads();
            }
    };

    __syncthreads();  // staging and the caller's writes to shared memory are complete
    smooth_a(pre);
    // restriction of the residual (multigrid.cl:90-180, right-hand-side part) of B's fluid cells (both
    // lists), one thread per coarse cell: the residuals of the eight children l = 4 di + 2 dj + dk are
    // formed independently (interior fluid children only) and added in that order, as the reference's
    // loop over di, dj, dk adds them. The sums go to B's p (free until the coarse solves), from which B's
    // owners take them.
    {
        const int n0 = S.count[2], nb = n0 + S.count[3];
        for (int g = threadIdx.x; g < nb; g += BOTTOM_THREADS) {
            const int cb = g < n0 ? S.list_b[g] : S.list_b[lb + g - n0];
            const int I = cb / bsx, J = (cb / bsy) % bny, K = cb % bnz;
            float r[8];
            bool present[8];
#pragma unroll
            for (int l = 0; l < 8; ++l) {
                const int i = 2 * I - 1 + (l >> 2), j = 2 * J - 1 + ((l >> 1) & 1), k = 2 * K - 1 + (l & 1);
                r[l] = 0.0f;
                present[l] = false;
                if (interior(i, j, k, anx, any, anz)) {
                    const int f = (i * any + j) * anz + k;
                    const float4 o = soa[f];
                    if (o.x >= 0.0f) {
                        const float ws = o.y * spa[f + asx] + soa[f - asx].y * spa[f - asx] + o.z * spa[f + asy] +
                                         soa[f - asy].z * spa[f - asy] + o.w * spa[f + 1] + soa[f - 1].w * spa[f - 1];
                        r[l] = sba[f] - (ws - o.x * spa[f]) * inv_delta2;
                        present[l] = true;
                    }
                }
            }
            float rhs = 0.0f;
#pragma unroll
            for (int l = 0; l < 8; ++l)
                if (present[l]) rhs += r[l];
            spb[split_cell(I, J, K, bnx, bny, bnz)] = rhs;
        }
    }
    __syncthreads();
    float bvals[2][MB];
#pragma unroll
    for (int colour = 0; colour < 2; ++colour)
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            // a fluid cell (slots without a cell and air cells hold -1)
            const float rhs = B[colour][m].d >= 0.0f ? spb[B[colour][m].c] : 0.0f;
            bvals[colour][m] = rhs;
            B[colour][m].d2b = d2 * rhs;
        }
    __syncthreads();
    for (int c = threadIdx.x; c < CB; c += BOTTOM_THREADS) spb[c] = 0.0f;  // multigrid.cl:114
    __syncthreads();
    const int most = max(S.count[2], S.count[3]);
    const int bwarps = min(BOTTOM_THREADS / 32, (most + 31) / 32);
    if ((int)(threadIdx.x >> 5) < bwarps) {
        // two coarse solves of the W (multigrid.py:127-170; b_solves: one when the coarsest level is
        // visited once), pre + coarse_iters iterations each
        const int bslots[2] = {active_slots(S.count[2], BOTTOM_THREADS), active_slots(S.count[3], BOTTOM_THREADS)};
        const int iterations = b_solves * (pre + coarse_iters), sx = bny * half, sy = half, other = bnx * sx;
        for (int it = 0; it < iterations; ++it)
#pragma unroll
            for (int colour = 0; colour < 2; ++colour) {
                auto put = [&](int m, float v) {
                    if (B[colour][m].d > 0.0f) spb[B[colour][m].c] = v;
                };
                auto value = [&](int m) { return relaxed_w(B[colour][m], spb, colour ? -other : other, sx, sy); };
                if (MB == 1) put(0, value(0));
                else relax_slots<MB>(bslots[colour], value, put);
                bar_b(bwarps);
            }
    }
    __syncthreads();
    // prolongation (multigrid.cl:182-201)
#pragma unroll
    for (int colour = 0; colour < 2; ++colour)
#pragma unroll
        for (int m = 0; m < KA; ++m) {
            if (A[colour][m].r < 0.0f) continue;  // interior fluid cells only
            const int c = A[colour][m].c;
            const int i = c / asx, j = (c / asy) % any, k = c % anz;
            const int I = min((i - 1) / 2 + 1, bnx - 2), J = min((j - 1) / 2 + 1, bny - 2),
                      K = min((k - 1) / 2 + 1, bnz - 2);
            spa[c] += w * spb[split_cell(I, J, K, bnx, bny, bnz)];
        }
    __syncthreads();
    smooth_a(post);
    if (bb) {
#pragma unroll
        for (int colour = 0; colour < 2; ++colour)
#pragma unroll
            for (int m = 0; m < MB; ++m)
                if (B[colour][m].d >= 0.0f)  // fluid cells
                    st(bb, S.list_b[colour * lb + threadIdx.x + m * BOTTOM_THREADS], bvals[colour][m]);
    }
}

// H = true: both levels are stored in FP16 (p, b and operator as __half, scaled values); the visit
// computes in FP32 in shared memory with kappa = scale[2] in place of delta^2 (mg_half.cuh).
template <int KA, int KB, bool H = false>
__device__ __forceinline__ void bottom_visit_block(float* __restrict__ pa, const float* __restrict__ ba,
                                                   const float4* __restrict__ opa, const uint8_t* __restrict__ ma,
                                                   int anx, int any, int anz, float* __restrict__ pb,
                                                   float* __restrict__ bb, const float4* __restrict__ opb,
                                                   const uint8_t* __restrict__ mb, int bnx, int bny, int bnz,
                                                   float delta, int pre, int post, int coarse_iters,
                                                   const float* __restrict__ scale, int b_solves = 2,
                                                   float w = 1.0f) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int CA = anx * any * anz, CB = bnx * bny * bnz;
    const BottomSmem S = bottom_smem(smem, CA, CB);
    const float d2 = H ? scale[2] : delta * delta;
    const float inv_delta2 = H ? scale[3] : 1.0f / (delta * delta);
    auto st = [&](float* a, int c, float v) {
        if (H) reinterpret_cast<__half*>(a)[c] = __float2half_rn(v);
        else a[c] = v;
    };
    bottom_stage<H>(S, pa, ba, opa, ma, CA, opb, mb, CB);
    bottom_lists(S, anx, any, anz, bnx, bny, bnz);
    BottomCells<KA, KB> R;
    bottom_cells(S, R, anx, any, anz, bnx, bny, bnz);
    bottom_rhs(S, R, d2);
    bottom_core<KA, KB, H>(S, R, anx, any, anz, bnx, bny, bnz, d2, inv_delta2, pre, post, coarse_iters, bb, b_solves,
                           w);
    const int bsx = bny * bnz, bsy = bnz;
    for (int c = threadIdx.x; c < CA; c += BOTTOM_THREADS) st(pa, c, S.spa[c]);
    for (int c = threadIdx.x; c < CB; c += BOTTOM_THREADS) {
        const int I = c / bsx, J = (c / bsy) % bny, K = c % bnz;
        st(pb, c, interior(I, J, K, bnx, bny, bnz) ? S.spb[split_cell(I, J, K, bnx, bny, bnz)] : 0.0f);
        // multigrid.cl:115 zeroes b off the interior; cells that are not fluid restrict to 0
        if (!interior(I, J, K, bnx, bny, bnz) || S.sob[c].x < 0.0f) st(bb, c, 0.0f);
    }
}

template <int KA, int KB, bool H = false>
__global__ void __launch_bounds__(BOTTOM_THREADS, 1)
    k_bottom_visit(float* __restrict__ pa, const float* __restrict__ ba, const float4* __restrict__ opa,
                   const uint8_t* __restrict__ ma, int anx, int any, int anz, float* __restrict__ pb,
                   float* __restrict__ bb, const float4* __restrict__ opb, const uint8_t* __restrict__ mb, int bnx,
                   int bny, int bnz, float delta, int pre, int post, int coarse_iters,
                   const float* __restrict__ scale, int b_solves, float w) {
    pdl_begin();
    bottom_visit_block<KA, KB, H>(pa, ba, opa, ma, anx, any, anz, pb, bb, opb, mb, bnx, bny, bnz, delta, pre, post,
                                  coarse_iters, scale, b_solves, w);
}

}  // namespace clb
