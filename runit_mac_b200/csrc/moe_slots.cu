// Expert products of a mixture-of-experts layer in 32-bit grade for several tokens: every expert's Q4_K matrices are read
// once for up to 48 (token, expert) slots.
//
// The grouped GEMV (gemv_grouped) streams a slot's expert for that slot alone: T tokens cost T * k passes over matrices, of
// which most serve an expert that another slot has just streamed.  Here the slots are sorted by expert (slots_table_kernel),
// their activations are split into two f16 halves (split_slots_kernel), and a group of slots of one expert meets its matrices on tcgen05
// (tc_rows.cuh): up to 8 slots per group where an expert has a few, up to 48 where it has many.
// The layer of width 2048, 64 experts of 1024, top 8 (us; mma.sync with tiles of 8 columns -> now): 16 tokens 86 -> 65, 32 112 -> 76, 64 144 -> 89, 128
// 199 -> 114, 256 272 -> 139; 60 experts of 768, top 4, 256 tokens 171 -> 106; 8 of 512, top 2, 64 tokens 53 -> 37.  Error against 64 bits, of the output with a
// residual of 1: 16 tokens 5.5e-8 -> 4.1e-8, 64 of 60 experts 4.9e-8 -> 4.0e-8, 256 1.12e-7 -> 0.89e-7.  (tcgen05 cuts its sums off where mma.sync did, a little
// more: with hi and lo in turn for all of K, or side by side to its end, 5.6e-8, 5.1e-8 and 1.15e-7, 1 % faster.)
#include <cuda_fp16.h>

#include "moe_internal.h"
#include "runit_internal.h"
#include "tc_rows.cuh"

namespace runit {
namespace slots {

// COLS columns of a group at most, in tiles of kTile slots.
template <int COLS> struct Shape {
    static constexpr tcr::Kind kKind = COLS == 8 ? tcr::Q4K_8 : tcr::Q4K_48;
    using C = tcr::Cfg<kKind>;
    static constexpr uint32_t kTile = COLS == 8 ? 8 : 16, kPerGroup = COLS / kTile, kImage = kTile * C::kBRow;      // bytes of a tile's 256 activations
    static constexpr uint32_t kPanel = COLS == 8 ? 16 * 128 : kTile * 128, kPanels = kImage / kPanel;               // a tile's rows of a panel
    static constexpr size_t kTableBytes = (kTile + 3) * 4;                                                          // per tile: slots, group, place in it
};

// ───────────────────────── slots by expert ─────────────────────────
// table: [0] groups, [1] tiles; from word 16: [groups][2] = expert, first tile << 3 | tiles.  place [tiles] = first tile of its group << 3 | tiles.
// order [tiles * tile]: slot, -1 = unused.  An expert's tiles are spread evenly over its groups.
__global__ void __launch_bounds__(1024) slots_table_kernel(const int32_t* __restrict__ idx, uint32_t n_slots, uint32_t E, uint32_t tile, uint32_t per_group,
                                                           int32_t* __restrict__ table, int32_t* __restrict__ place, int32_t* __restrict__ order) {
    __shared__ uint32_t cnt[256], tiles[256], groups[256];
    const uint32_t tid = threadIdx.x;
    grid_dependency_wait();
    grid_launch_dependents();
    if (tid < 256) cnt[tid] = 0;
    __syncthreads();
    for (uint32_t s = tid; s < n_slots; s += 1024) {
        const uint32_t e = (uint32_t)idx[s];
        if (e < E) atomicAdd(&cnt[e], 1u);
    }
    __syncthreads();
    uint32_t nt = 0, ng = 0;
    if (tid < 256) {
        nt = (cnt[tid] + tile - 1) / tile;
        ng = (nt + per_group - 1) / per_group;
        tiles[tid] = nt;
        groups[tid] = ng;
        cnt[tid] = 0;                              // becomes the cursor
    }
    __syncthreads();
    for (uint32_t o = 1; o < 256; o <<= 1) {       // inclusive sums
        uint32_t a = 0, b = 0;
        if (tid < 256 && tid >= o) { a = tiles[tid - o]; b = groups[tid - o]; }
        __syncthreads();
        if (tid < 256) { tiles[tid] += a; groups[tid] += b; }
        __syncthreads();
    }
    if (tid < 256) {
        const uint32_t t0 = tiles[tid] - nt, g0 = groups[tid] - ng;
        for (uint32_t i = 0; i < ng; i++) {
            const uint32_t a = i * nt / ng, n = (i + 1) * nt / ng - a, at = ((t0 + a) << 3) | n;
            table[16 + 2 * (g0 + i)] = (int32_t)tid;
            table[17 + 2 * (g0 + i)] = (int32_t)at;
            for (uint32_t j = 0; j < n; j++) place[t0 + a + j] = (int32_t)at;
        }
        if (tid == 255) { table[0] = (int32_t)groups[255]; table[1] = (int32_t)tiles[255]; }
    }
    for (uint32_t i = tid; i < tiles[255] * tile; i += 1024) order[i] = -1;
    __syncthreads();
    // the order inside an expert is not fixed; a slot's result does not depend on its column
    for (uint32_t s = tid; s < n_slots; s += 1024) {
        const uint32_t e = (uint32_t)idx[s];
        if (e < E) order[(e ? tiles[e - 1] : 0u) * tile + atomicAdd(&cnt[e], 1u)] = (int32_t)s;
    }
}

// ───────────────────────── activations of a tile ─────────────────────────
// One CTA per (tile, unit), one warp per column.  A group's images of its units lie one behind the other, its tiles' rows interleaved by
// panel; the scales likewise.
template <int COLS>
__global__ void __launch_bounds__(32 * Shape<COLS>::kTile) split_slots_kernel(const float* __restrict__ x, uint32_t xdiv, uint32_t k, const int32_t* __restrict__ table,
                                                                              const int32_t* __restrict__ place, const int32_t* __restrict__ order,
                                                                              uint8_t* __restrict__ images, float* __restrict__ scales) {
    using S = Shape<COLS>;
    constexpr uint32_t kT = 32 * S::kTile;
    __shared__ __align__(16) uint8_t out[S::kImage];
    const uint32_t tile = blockIdx.x, u = blockIdx.y, units = gridDim.y, n = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr uint32_t kSums = (S::kPanels - 1) * S::kPanel;
    if (COLS == 8)
        for (uint32_t i = threadIdx.x; i < S::kPanel / 16; i += kT) reinterpret_cast<uint4*>(out + kSums)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    grid_dependency_wait();
    grid_launch_dependents();
    if (tile >= (uint32_t)table[1]) return;
    const int32_t slot = order[tile * S::kTile + n];
    float v[8];
    tcr::load8(x + (size_t)((uint32_t)(slot < 0 ? 0 : slot) / xdiv) * k + u * 256 + 8 * lane, slot >= 0, v);
    const float scale = tcr::split_column<S::kKind>(v, lane, out, n, out + (COLS == 8 ? 0 : 4 * S::kPanel), COLS == 8 ? 8 + n : n, S::kPanel, out + kSums, n);
    const uint32_t at = (uint32_t)place[tile], first = at >> 3, nt = at & 7, mine = tile - first;
    const size_t unit = (size_t)first * units + (size_t)u * nt;        // in tiles
    if (lane == 0) scales[unit * S::kTile + mine * S::kTile + n] = scale;
    __syncthreads();
    uint8_t* dst = images + unit * S::kImage + mine * S::kPanel;
    for (uint32_t i = threadIdx.x; i < S::kImage / 16; i += kT) {
        const uint32_t panel = i / (S::kPanel / 16), r = i % (S::kPanel / 16);
        reinterpret_cast<uint4*>(dst + (size_t)panel * nt * S::kPanel)[r] = reinterpret_cast<const uint4*>(out)[i];
    }
}

// ───────────────────────── products ─────────────────────────
struct Args {
    const int32_t *table, *order;
    const uint8_t* images;
    const float* scales;
    float* y;                    // DUAL: [slot][rows] silu(gate) * up, else [slot][rows]
    uint32_t rows, units, tiles; // rows per expert (and matrix), 256-K units, row tiles per expert (DUAL: 128 outputs, else 256 rows)
    int32_t* status;
};

template <bool DUAL, int COLS> struct Policy {
    using S = Shape<COLS>;
    static constexpr int kAcc = S::C::kAcc;
    const Args& a;
    const CUtensorMap* wa;
    const CUtensorMap* wb;

    __device__ __forceinline__ bool few() const { return false; }
    __device__ __forceinline__ uint32_t begin() const { return 0; }
    __device__ __forceinline__ uint32_t end() const {
        const uint32_t items = (uint32_t)a.table[0] * a.tiles;
        return blockIdx.x < items ? (items - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    }
    __device__ __forceinline__ uint32_t steps() const { return end() * a.units * 2; }
    __device__ __forceinline__ tcr::Run run(uint32_t i) const {
        const uint32_t it = blockIdx.x + i * gridDim.x, gi = it / a.tiles, rt = it % a.tiles;
        const uint32_t e = (uint32_t)a.table[16 + 2 * gi], at = (uint32_t)a.table[17 + 2 * gi], first = at >> 3, nt = at & 7;
        tcr::Run r;
        r.map[0] = wa;
        r.map[1] = wb;
        r.row[0] = (int32_t)(e * a.rows + rt * (DUAL ? 128 : 256));
        r.row[1] = DUAL ? r.row[0] : r.row[0] + 128;
        r.u0 = 0;
        r.u1 = a.units;
        r.n = COLS == 8 ? 8 : nt * S::kTile;
        r.b = a.images + (size_t)first * a.units * S::kImage;
        r.xs = a.scales + (size_t)first * a.units * S::kTile;
        return r;
    }
    __device__ __forceinline__ void finish(uint32_t i, float (&acc)[2][kAcc], uint32_t warp, uint32_t lane) {
        const uint32_t it = blockIdx.x + i * gridDim.x, gi = it / a.tiles, rt = it % a.tiles;
        const uint32_t at = (uint32_t)a.table[17 + 2 * gi], nt = at & 7, row = (warp & 3) * 32 + lane;
        const int32_t* order = a.order + (size_t)(at >> 3) * S::kTile;
        float* y = a.y + rt * (DUAL ? 128 : 256) + row;
#pragma unroll
        for (int j = 0; j < kAcc; j++) {
            const uint32_t col = COLS == 8 ? j : 8 * (3 * (j >> 3) + (warp >> 2)) + (j & 7);
            const int32_t slot = col < nt * S::kTile ? order[col] : -1;
            if (slot >= 0) {
                float* o = y + (size_t)slot * a.rows;
                if (DUAL) o[0] = silu(acc[0][j]) * acc[1][j];
                else { o[0] = acc[0][j]; o[128] = acc[1][j]; }
            }
            acc[0][j] = acc[1][j] = 0.f;
        }
    }
};

template <bool DUAL, int COLS>
__global__ void __launch_bounds__(Shape<COLS>::C::kThreads, 1) slots_gemm_kernel(const __grid_constant__ CUtensorMap wa,
                                                                                                      const __grid_constant__ CUtensorMap wb,
                                                                                                      const __grid_constant__ Args a) {
    using C = typename Shape<COLS>::C;
    extern __shared__ uint8_t smem_raw[];
    tcr::Block<Shape<COLS>::kKind, 2> blk(smem_raw);
    grid_dependency_wait();                        // which expert comes from the table
    Policy<DUAL, COLS> p{a, &wa, &wb};
    if (blk.warp == C::kCopyW) {
        // raw superblocks of both row tiles, and the columns' scales with the first
        uint32_t s = 0, c = 0;
        for (uint32_t i = 0; i < p.end() && blk.ok; i++) {
            const tcr::Run r = p.run(i);
            for (uint32_t u = 0; u < r.u1 && blk.ok; u++, c++)
#pragma unroll
                for (uint32_t sub = 0; sub < 2; sub++, s++) {
                    if (!blk.raw_free(s)) break;
                    if (elect_one()) {
                        mbar_expect_tx(blk.raw_bar(s), C::kWBytes + (sub == 0 ? r.n * 4 : 0));
                        tma_load_2d(blk.raw(s), r.map[sub], (int32_t)(u * 144), r.row[sub], blk.raw_bar(s));
                        if (sub == 0) bulk_load_1d(blk.scales(c), r.xs + (size_t)u * r.n, r.n * 4, blk.raw_bar(s));
                    }
                    __syncwarp();
                }
        }
        mbar_drain(blk.w_full, C::kW, s);        // whatever was requested arrives before the CTA leaves, whichever role gives up, and when
    } else if (blk.warp == C::kCopyB) {
        uint32_t c = 0;
        for (uint32_t i = 0; i < p.end() && blk.ok; i++) {
            const tcr::Run r = p.run(i);
            const uint32_t bytes = r.n * C::kBRow;
            for (uint32_t u = 0; u < r.u1; u++, c++) {
                if (!blk.image_free(c)) break;
                if (elect_one()) {
                    mbar_expect_tx(blk.image_bar(c), bytes);
                    bulk_load_1d(blk.image(c), r.b + (size_t)u * bytes, bytes, blk.image_bar(c));
                }
                __syncwarp();
            }
        }
        mbar_drain(blk.b_full, C::kB, c);
    } else {
        blk.work(p);
    }
    blk.leave(a.status);
}

}  // namespace slots

// Tiles that n_slots slots of E experts can fill: an expert of c slots takes at most (c + tile - 1) / tile.
static uint32_t slots_max_tiles(uint32_t n_slots, uint32_t E, uint32_t tile) {
    const uint64_t experts = E < n_slots ? E : n_slots, t = (n_slots + (tile - 1) * experts) / tile;
    return (uint32_t)(t < n_slots ? t : n_slots);
}

// Up to 11 slots per expert on average, groups of 8, behind that of 48 (us with 8 / 48: 64 experts of 2048 x 1024, top 8: 64 tokens 96 / 106, 96 116 / 110,
// 128 142 / 119; 60 of 768, top 4: 128 tokens 85 / 92, 192 106 / 100; 16 of 1024 x 512, top 4: 48 tokens 33 / 34, 64 38 / 36).
static bool few_slots(uint64_t n_slots, uint32_t E) { return n_slots <= 11ull * E; }

// staging: 256 bytes of counts, the tables (rounded up to 256), images, scales
template <int COLS> static size_t slots_most(size_t staging_bytes, uint32_t h, uint32_t ff, uint32_t E) {
    using S = slots::Shape<COLS>;
    const size_t per_tile = S::kTableBytes + (size_t)((h > ff ? h : ff) / 256) * (S::kImage + S::kTile * 4);
    if (staging_bytes < 512 + per_tile) return 0;
    const size_t tiles = (staging_bytes - 512) / per_tile;
    // slots_max_tiles(n, E) <= tiles: (n + (tile - 1) E) / tile at most, and never more than n
    const size_t room = tiles * S::kTile, open = (size_t)(S::kTile - 1) * E, n = room > open ? room - open : 0;
    return n > tiles ? n : tiles;
}
uint32_t moe_slots_tokens(size_t staging_bytes, uint32_t h, uint32_t ff, uint32_t E, uint32_t k) {
    // every count up to the result fits: in groups of 8 as far as those are taken, in groups of 48 behind that
    const size_t small = slots_most<8>(staging_bytes, h, ff, E), large = slots_most<48>(staging_bytes, h, ff, E), line = 11ull * E;
    const size_t slots = small < line ? small : large > line ? large : line;
    return (uint32_t)(slots / k < 65536 ? slots / k : 65536);
}

template <int COLS>
static int32_t slots_run(runit_ctx* ctx, const void* gate, const void* up, const void* down, const float* x, const int32_t* idx, float* act, float* y,
                         void* staging, uint32_t n_slots, uint32_t h, uint32_t ff, uint32_t E, uint32_t k) {
    using namespace slots;
    using S = Shape<COLS>;
    using C = typename S::C;
    CUtensorMap mg, mu, md;
    int32_t st = runit_get_tmap(ctx, gate, (uint64_t)E * ff, (uint64_t)h / 256 * 144, 128, 144, &mg);
    if (st == RUNIT_OK) st = runit_get_tmap(ctx, up, (uint64_t)E * ff, (uint64_t)h / 256 * 144, 128, 144, &mu);
    if (st == RUNIT_OK) st = runit_get_tmap(ctx, down, (uint64_t)E * h, (uint64_t)ff / 256 * 144, 128, 144, &md);
    if (st != RUNIT_OK) return st;
    static bool configured[64] = {false};
    if (ctx->device >= 64 || !configured[ctx->device]) {
        RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(slots_gemm_kernel<true, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
        RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(slots_gemm_kernel<false, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
        if (ctx->device < 64) configured[ctx->device] = true;
    }
    const uint32_t mt = slots_max_tiles(n_slots, E, S::kTile), ctas = (uint32_t)ctx->sm_count, most = (h > ff ? h : ff) / 256;
    int32_t* table = (int32_t*)staging;
    int32_t* place = table + 64 + (size_t)mt * 2;
    int32_t* order = place + mt;
    uint8_t* images = (uint8_t*)staging + 256 + ((size_t)mt * S::kTableBytes + 255) / 256 * 256;
    float* scales = (float*)(images + (size_t)mt * most * S::kImage);
    auto grid = [&](uint32_t tiles) { return dim3(mt * tiles < ctas ? mt * tiles : ctas); };
    runit_launch_chain(ctx, slots_table_kernel, dim3(1), dim3(1024), idx, n_slots, E, S::kTile, S::kPerGroup, table, place, order);
    if ((st = runit_after_launch(ctx, "moe_slots_table")) != RUNIT_OK) return st;
    Args a{table, order, images, scales, act, ff, h / 256, ff / 128, ctx->d_status};
    runit_launch_chain(ctx, split_slots_kernel<COLS>, dim3(mt, h / 256), dim3(32 * S::kTile), x, k, h, (const int32_t*)table, (const int32_t*)place,
                       (const int32_t*)order, images, scales);
    if ((st = runit_after_launch(ctx, "moe_slots_split_x")) != RUNIT_OK) return st;
    runit_launch_chain_smem(ctx, slots_gemm_kernel<true, COLS>, grid(a.tiles), dim3(C::kThreads), C::kSmem, mg, mu, a);
    if ((st = runit_after_launch(ctx, "moe_slots_gate_up")) != RUNIT_OK) return st;
    runit_launch_chain(ctx, split_slots_kernel<COLS>, dim3(mt, ff / 256), dim3(32 * S::kTile), (const float*)act, 1u, ff, (const int32_t*)table,
                       (const int32_t*)place, (const int32_t*)order, images, scales);
    if ((st = runit_after_launch(ctx, "moe_slots_split_act")) != RUNIT_OK) return st;
    a.y = y;
    a.rows = h;
    a.units = ff / 256;
    a.tiles = h / 256;
    runit_launch_chain_smem(ctx, slots_gemm_kernel<false, COLS>, grid(a.tiles), dim3(C::kThreads), C::kSmem, md, md, a);
    return runit_after_launch(ctx, "moe_slots_down");
}

int32_t moe_slots_experts(runit_ctx* ctx, const void* gate, const void* up, const void* down, const float* x, const int32_t* idx, float* act,
                          float* y, void* staging, uint32_t T, uint32_t h, uint32_t ff, uint32_t E, uint32_t k) {
    return few_slots((uint64_t)T * k, E) ? slots_run<8>(ctx, gate, up, down, x, idx, act, y, staging, T * k, h, ff, E, k)
                                         : slots_run<48>(ctx, gate, up, down, x, idx, act, y, staging, T * k, h, ff, E, k);
}

}  // namespace runit
