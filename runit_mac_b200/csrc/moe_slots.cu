// Expert products of a mixture-of-experts layer in 32-bit grade for several tokens: every expert's Q4_K matrices are read
// once for up to 32 (token, expert) slots.
//
// The grouped GEMV (gemv_grouped) streams a slot's expert for that slot alone: T tokens cost T * k passes over matrices, of
// which most serve an expert that another slot has just streamed.  Here the slots are sorted by expert (slots_table_kernel),
// cut into tiles of 8 columns and groups of up to 4 tiles of one expert, and a group's products run on the tensor cores:
//   * a weight is d * (sc * q) - dmin * m.  sc * q is an integer of at most 945, exact in f16, so one AND-OR and one f16x2
//     multiply-add turn two nibbles into the operand (1024 + q) * sc - 1024 * sc without rounding; d and dmin meet the
//     256-weight sums in f32.  The unpacked operand serves all the group's columns.
//   * an activation is x = 2^e * (hi + lo) with f16 hi and lo and one power of two per 256 elements of a slot: 22 bits, error
//     at most 2^-22 of the value or 2^-35 of the unit's largest (split_slots_kernel: the largest lies near the top of f16's range, because
//     the halves of the high nibbles' activations, which are stored as x / 16, end at its smallest step).
//   * sum_j m_j * (sum of x over block j) is one more MMA per unit with 32 * m as A and the split block sums / 32 as B.
// An Inf or a NaN among a unit's activations makes its scale, and with it the token's products, NaN (as the launches per slot do).
// Bound: at 2 slots per expert (16 tokens) the unpacking, about 470 instructions per warp for 16 x 256 weights at 8 columns; at 32
// slots (256 tokens) the MMA pipe (65 % active).  Measured for the layer of width 2048, 64 experts of 1024, top 8: 16 tokens 117 ->
// 88 to 101 us (by the number of experts hit), 256 tokens 1590 -> 275 to 300 us, error against 64 bits 4.2e-6 -> 1.2e-7 of the output.  One m16 tile per warp: with two
// (half the reads of the activations' fragments, half as many warps) 256 tokens took 302 us, and 16 tokens 107 us with 256 rows per CTA.
#include <cuda_fp16.h>

#include "gemv_common.cuh"
#include "moe_internal.h"
#include "runit_internal.h"
#include "tma.cuh"

namespace runit {
namespace slots {

constexpr int kCols = 8;
constexpr uint32_t kXBytes = 8480;                 // one unit of a tile: 16 steps x 512 bytes, 256 bytes of block sums, 8 scales
// G = tiles per group at most.  4: 256 rows, sixteen consumer warps of one m16 tile, one CTA per SM with three stages of 71 KB.
// 1 (an expert has a few slots): 128 rows, eight warps, three CTAs of two stages of 27 KB, because what is left to hide is the MMA
// latency of a single tile (hi and lo have accumulators of their own) and half as many rows leave fewer idle CTAs in the last wave.
template <int G> struct Shape {
    static constexpr uint32_t kWarps = G == 1 ? 8 : 16, kRows = 16 * kWarps, kWBytes = kRows * 144;
    static constexpr uint32_t kStage = (kWBytes + G * kXBytes + 127) / 128 * 128, kStages = G == 1 ? 2 : 3, kPerSm = G == 1 ? 3 : 1;
    static constexpr uint32_t kSmem = kStages * kStage + 128, kThreads = 32 * kWarps + 32;
    static_assert(kStage % 128 == 0 && kWBytes % 256 == 0, "a tiled load lands on a multiple of 128 bytes");
    static_assert(kPerSm * (kSmem + 1024) <= 228 * 1024, "stages exceed the shared memory of an SM");
};

// ───────────────────────── slots by expert ─────────────────────────
// table: [0] groups, [1] tiles; from word 16: [groups][2] = expert, first tile << 3 | tiles; then order [tiles * 8], -1 = unused
__global__ void __launch_bounds__(1024) slots_table_kernel(const int32_t* __restrict__ idx, uint32_t n_slots, uint32_t E, uint32_t per_group,
                                                           int32_t* __restrict__ table, int32_t* __restrict__ order) {
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
        nt = (cnt[tid] + kCols - 1) / kCols;
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
            const uint32_t left = nt - i * per_group;
            table[16 + 2 * (g0 + i)] = (int32_t)tid;
            table[17 + 2 * (g0 + i)] = (int32_t)(((t0 + i * per_group) << 3) | (left < per_group ? left : per_group));
        }
        if (tid == 255) { table[0] = (int32_t)groups[255]; table[1] = (int32_t)tiles[255]; }
    }
    for (uint32_t i = tid; i < tiles[255] * kCols; i += 1024) order[i] = -1;
    __syncthreads();
    // the order inside an expert is not fixed; a slot's result does not depend on its column
    for (uint32_t s = tid; s < n_slots; s += 1024) {
        const uint32_t e = (uint32_t)idx[s];
        if (e < E) order[(e ? tiles[e - 1] : 0u) * kCols + atomicAdd(&cnt[e], 1u)] = (int32_t)s;
    }
}

// ───────────────────────── activations of a tile ─────────────────────────
// One CTA per (tile, unit), one warp per column.  Fragments: step st = 4 * chunk + 2 * half + word (half 1 = high nibbles, whose
// operand is 16 * sc * q: their activations are stored as x / 16); 16 bytes per (step, column, t): hi of elements (0, 2), (1, 3)
// of weight word t, then lo.  Behind them the block sums, [column][t] hi pair, lo pair in the order of the scale indices, and 2^e.
__global__ void __launch_bounds__(256) split_slots_kernel(const float* __restrict__ x, uint32_t xdiv, uint32_t k, const int32_t* __restrict__ table,
                                                          const int32_t* __restrict__ order, uint8_t* __restrict__ frags) {
    __shared__ __align__(16) uint8_t out[kXBytes];
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t tile = blockIdx.x, u = blockIdx.y, n = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (tile >= (uint32_t)table[1]) return;
    const int32_t slot = order[tile * kCols + n];
    float v[8], amax = 0.f;
    bool bad = false;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        v[b] = slot >= 0 ? x[(size_t)((uint32_t)slot / xdiv) * k + u * 256 + b * 32 + lane] : 0.f;
        amax = fmaxf(amax, fabsf(v[b]));
        bad |= !(fabsf(v[b]) <= 3.4028235e38f);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    bad = __any_sync(0xffffffffu, bad);
    // 2^e such that the largest |x| / 2^e lies in [2^14, 2^15): so does a 32nd of a block's sum.  e is held above -116 so that both powers
    // are normal numbers.
    int e = (int)((__float_as_uint(amax) >> 23) & 255u) - 127 - 14;
    e = e < -116 ? -116 : e;
    const float scale = bad ? __uint_as_float(0x7FC00000u) : __uint_as_float((uint32_t)(e + 127) << 23);
    const float inv = __uint_as_float((uint32_t)(127 - e) << 23);
    const uint32_t t = (lane & 15) >> 2, i = lane & 3, word = lane >> 4;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const float w = bad ? 0.f : v[b] * inv;
        const float ws = (b & 1) ? w * 0.0625f : w;
        const __half hi = __float2half_rn(ws), lo = __float2half_rn(ws - __half2float(hi));
        const uint32_t st = 4 * (b >> 1) + 2 * (b & 1) + word;
        __half* p = reinterpret_cast<__half*>(out + ((st * 8 + n) * 4 + t) * 16) + (i & 1) * 2 + (i >> 1);
        p[0] = hi;
        p[4] = lo;
        float s = w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            s *= 0.03125f;
            const uint32_t si = (b >> 1) + 4 * (b & 1);
            const __half sh = __float2half_rn(s), sl = __float2half_rn(s - __half2float(sh));
            __half* q = reinterpret_cast<__half*>(out + 8192 + (n * 4 + (si >> 1)) * 8) + (si & 1);
            q[0] = sh;
            q[2] = sl;
        }
    }
    if (lane == 0) reinterpret_cast<float*>(out + 8448)[n] = scale;
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(frags + ((size_t)tile * gridDim.y + u) * kXBytes);
    for (uint32_t j = threadIdx.x; j < kXBytes / 16; j += 256) dst[j] = reinterpret_cast<const uint4*>(out)[j];
}

// ───────────────────────── products ─────────────────────────
struct Args {
    const int32_t *table, *order;
    const uint8_t* frags;
    float* y;                    // DUAL: [slot][rows] silu(gate) * up, else [slot][rows]
    uint32_t rows, units, tiles; // rows per expert (and matrix), 256-K units, row tiles per expert
    int32_t* status;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// two nibbles in place (mask 0x000F000F or 0x00F000F0) -> f16x2 of sc * nibble (16 * sc * nibble): exact
__device__ __forceinline__ uint32_t scaled_pair(uint32_t w, uint32_t mask, __half2 sc, __half2 bias) {
    return as_u32(__hfma2(as_half2((w & mask) | 0x64006400u), sc, bias));
}
__device__ __forceinline__ uint32_t lds32(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

// A warp's m16 tile: 16 rows of the matrix; DUAL: rows 0..7 are gate rows and rows 8..15 the up rows of the same outputs, so that
// a lane holds both factors of its products.
template <bool DUAL, int G>
__global__ void __launch_bounds__(Shape<G>::kThreads, Shape<G>::kPerSm) slots_gemm_kernel(const __grid_constant__ CUtensorMap wa,
                                                                                          const __grid_constant__ CUtensorMap wb, const Args a) {
    using S = Shape<G>;
    constexpr uint32_t kStages = S::kStages, kOut = DUAL ? S::kRows / 2 : S::kRows;      // outputs of a row tile
    constexpr int LO = G == 1 ? 1 : 0;             // one tile: the products with lo have accumulators of their own
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kStages];
    const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
    const uint8_t* base_p = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const uint32_t full = smem_u32(&bars[0]), empty = smem_u32(&bars[kStages]);
    if (tid == 0) {
        for (uint32_t s = 0; s < kStages; s++) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, S::kWarps);
        }
        fence_mbar_init();
    }
    __syncthreads();
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t items = (uint32_t)a.table[0] * a.tiles;
    bool timed_out = false;
    uint32_t c = 0;
    if (warp == S::kWarps) {
        if (lane == 0) {
            for (uint32_t it = blockIdx.x; it < items && !timed_out; it += gridDim.x) {
                const uint32_t gi = it / a.tiles, rt = it % a.tiles;
                const uint32_t e = (uint32_t)a.table[16 + 2 * gi], tt = (uint32_t)a.table[17 + 2 * gi], nt = tt & 7, t0 = tt >> 3;
                const int32_t row0 = (int32_t)(e * a.rows + rt * kOut);
                for (uint32_t u = 0; u < a.units; u++, c++) {
                    const uint32_t s = c % kStages, sb = base + s * S::kStage, bar = full + 8 * s;
                    if (c >= kStages && !mbar_wait(empty + 8 * s, ((c / kStages) - 1) & 1)) { timed_out = true; break; }
                    mbar_expect_tx(bar, S::kWBytes + nt * kXBytes);
                    tma_load_2d(sb, &wa, (int32_t)(u * 144), row0, bar);
                    if (DUAL) tma_load_2d(sb + S::kWBytes / 2, &wb, (int32_t)(u * 144), row0, bar);
                    for (uint32_t j = 0; j < nt; j++)
                        bulk_load_1d(sb + S::kWBytes + j * kXBytes, a.frags + ((size_t)(t0 + j) * a.units + u) * kXBytes, kXBytes, bar);
                }
            }
            mbar_drain(full, kStages, c);          // the last loads; a warp that gave up its wait no longer waits for them
        }
    } else {
        const uint32_t row[2] = {DUAL ? warp * 8 + g : warp * 16 + g, DUAL ? S::kRows / 2 + warp * 8 + g : warp * 16 + 8 + g};
        for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
            const uint32_t gi = it / a.tiles, rt = it % a.tiles;
            const uint32_t tt = (uint32_t)a.table[17 + 2 * gi], nt = tt & 7, t0 = tt >> 3;
            float acc[G][4];
#pragma unroll
            for (int i = 0; i < G * 4; i++) (&acc[0][0])[i] = 0.f;
            for (uint32_t u = 0; u < a.units; u++, c++) {
                const uint32_t s = c % kStages;
                if (!mbar_wait(full + 8 * s, (c / kStages) & 1)) { timed_out = true; break; }
                const uint8_t* sb = base_p + s * S::kStage;
                const uint8_t* xb = sb + S::kWBytes + (g * 4 + t) * 16;
                const uint8_t* rp[2];
                Q4KScales sc[2];
                uint32_t dd[2];
                float v[G + LO][4];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    rp[r] = sb + row[r] * 144;
                    const uint4 h = *reinterpret_cast<const uint4*>(rp[r]);
                    sc[r] = q4k_unpack_scales(h.y, h.z, h.w);
                    dd[r] = h.x;
                }
#pragma unroll
                for (int i = 0; i < (G + LO) * 4; i++) (&v[0][0])[i] = 0.f;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t w[2][2];
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        w[r][0] = lds32(rp[r] + 16 + 32 * j + 4 * t);
                        w[r][1] = lds32(rp[r] + 32 + 32 * j + 4 * t);
                    }
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        const uint32_t mask = half ? 0x00F000F0u : 0x000F000Fu;
                        __half2 s2[2], b2[2];
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const uint32_t p = __byte_perm(half ? sc[r].sh : sc[r].sl, 0x64646464u, 0x4040u + 0x0101u * j);
                            s2[r] = __hsub2(as_half2(p), as_half2(0x64006400u));
                            b2[r] = __hmul2(s2[r], as_half2(0xE400E400u));      // -1024 * sc
                        }
#pragma unroll
                        for (int word = 0; word < 2; word++) {
                            uint32_t af[4];
#pragma unroll
                            for (int r = 0; r < 2; r++) {
                                af[r] = scaled_pair(w[r][word], mask, s2[r], b2[r]);
                                af[2 + r] = scaled_pair(w[r][word] >> 8, mask, s2[r], b2[r]);
                            }
#pragma unroll
                            for (int n = 0; n < G; n++)
                                if (n < (int)nt) {
                                    const uint4 bf = *reinterpret_cast<const uint4*>(xb + n * kXBytes + (4 * j + 2 * half + word) * 512);
                                    mma_f16(v[n], af, bf.x, bf.y);
                                    mma_f16(v[n + LO], af, bf.z, bf.w);
                                }
                        }
                    }
                }
                // sum of minimum * block sum, then both factors and the column's power of two
                uint32_t am[4];
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint32_t m = t < 2 ? sc[r].ml : sc[r].mh;
                    const uint32_t p = __byte_perm(m, 0x64646464u, (t & 1) ? 0x4342u : 0x4140u);
                    am[r] = am[2 + r] = as_u32(__hfma2(as_half2(p), as_half2(0x50005000u), as_half2(0xF800F800u)));      // 32 * (p - 1024), exact
                }
#pragma unroll
                for (int n = 0; n < G; n++)
                    if (n < (int)nt) {
                        const uint8_t* tail = sb + S::kWBytes + n * kXBytes + 8192;
                        const uint2 bs = *reinterpret_cast<const uint2*>(tail + (g * 4 + t) * 8);
                        const float2 xs = *reinterpret_cast<const float2*>(tail + 256 + 8 * t);
                        float mm[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_f16(mm, am, bs.x, bs.y);
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float d = half_bits_to_float(dd[i >> 1] & 0xFFFFu), dm = half_bits_to_float(dd[i >> 1] >> 16);
                            acc[n][i] = fmaf((i & 1) ? xs.y : xs.x, fmaf(d, LO ? v[n][i] + v[n + LO][i] : v[n][i], -dm * mm[i]), acc[n][i]);
                        }
                    }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * s) : "memory");
            }
            if (timed_out) break;
#pragma unroll
            for (int n = 0; n < G; n++)
                if (n < (int)nt) {
                    const int2 sl = *reinterpret_cast<const int2*>(a.order + (t0 + n) * kCols + 2 * t);
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int32_t slot = i ? sl.y : sl.x;
                        if (slot < 0) continue;
                        float* y = a.y + (size_t)slot * a.rows + rt * kOut + (DUAL ? warp * 8 : warp * 16) + g;
                        if (DUAL) y[0] = silu(acc[n][i]) * acc[n][2 + i];
                        else { y[0] = acc[n][i]; y[8] = acc[n][2 + i]; }
                    }
                }
        }
    }
    if (timed_out && a.status) atomicExch(a.status, 1);
}

}  // namespace slots

static uint32_t slots_max_tiles(uint32_t n_slots, uint32_t E) {
    const uint32_t full = n_slots / slots::kCols, open = E < n_slots ? E : n_slots;
    const uint64_t t = (uint64_t)full + open;
    return (uint32_t)(t < n_slots ? t : n_slots);
}

// staging: 256 bytes, table and order of the tiles (rounded up to 256), their activations
uint32_t moe_slots_tokens(size_t staging_bytes, uint32_t h, uint32_t ff, uint32_t E, uint32_t k) {
    const size_t per_tile = (2 + slots::kCols) * 4 + (size_t)((h > ff ? h : ff) / 256) * slots::kXBytes;
    if (staging_bytes < 512 + per_tile) return 0;
    const size_t tiles = (staging_bytes - 512) / per_tile;
    // slots_max_tiles(n, E) <= tiles: n / 8 + E tiles at most, and never more than n
    const size_t n = tiles > E ? (tiles - E) * slots::kCols : 0, slots = n > tiles ? n : tiles;
    return (uint32_t)(slots / k < 65536 ? slots / k : 65536);
}

template <int G>
static int32_t slots_run(runit_ctx* ctx, const void* gate, const void* up, const void* down, const float* x, const int32_t* idx, float* act, float* y,
                         void* staging, uint32_t n_slots, uint32_t h, uint32_t ff, uint32_t E, uint32_t k) {
    using namespace slots;
    using S = Shape<G>;
    CUtensorMap mg, mu, md;
    int32_t st = runit_get_tmap(ctx, gate, (uint64_t)E * ff, (uint64_t)h / 256 * 144, S::kRows / 2, 144, &mg);
    if (st == RUNIT_OK) st = runit_get_tmap(ctx, up, (uint64_t)E * ff, (uint64_t)h / 256 * 144, S::kRows / 2, 144, &mu);
    if (st == RUNIT_OK) st = runit_get_tmap(ctx, down, (uint64_t)E * h, (uint64_t)ff / 256 * 144, S::kRows, 144, &md);
    if (st != RUNIT_OK) return st;
    static bool configured[64] = {false};
    if (ctx->device >= 64 || !configured[ctx->device]) {
        RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(slots_gemm_kernel<true, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem));
        RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(slots_gemm_kernel<false, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem));
        if (ctx->device < 64) configured[ctx->device] = true;
    }
    const uint32_t mt = slots_max_tiles(n_slots, E), ctas = (uint32_t)ctx->sm_count * S::kPerSm;
    int32_t* table = (int32_t*)staging;
    int32_t* order = table + 64 + (size_t)mt * 2;
    uint8_t* frags = (uint8_t*)staging + 256 + ((size_t)mt * (2 + kCols) * 4 + 255) / 256 * 256;
    auto grid = [&](uint32_t tiles) { return dim3(mt * tiles < ctas ? mt * tiles : ctas); };
    runit_launch_chain(ctx, slots_table_kernel, dim3(1), dim3(1024), idx, n_slots, E, (uint32_t)G, table, order);
    if ((st = runit_after_launch(ctx, "moe_slots_table")) != RUNIT_OK) return st;
    Args a{table, order, frags, act, ff, h / 256, ff / (S::kRows / 2), ctx->d_status};
    runit_launch_chain(ctx, split_slots_kernel, dim3(mt, h / 256), dim3(256), x, k, h, (const int32_t*)table, (const int32_t*)order, frags);
    if ((st = runit_after_launch(ctx, "moe_slots_split_x")) != RUNIT_OK) return st;
    runit_launch_chain_smem(ctx, slots_gemm_kernel<true, G>, grid(a.tiles), dim3(S::kThreads), S::kSmem, mg, mu, a);
    if ((st = runit_after_launch(ctx, "moe_slots_gate_up")) != RUNIT_OK) return st;
    runit_launch_chain(ctx, split_slots_kernel, dim3(mt, ff / 256), dim3(256), (const float*)act, 1u, ff, (const int32_t*)table, (const int32_t*)order, frags);
    if ((st = runit_after_launch(ctx, "moe_slots_split_act")) != RUNIT_OK) return st;
    a.y = y;
    a.rows = h;
    a.units = ff / 256;
    a.tiles = h / S::kRows;
    runit_launch_chain_smem(ctx, slots_gemm_kernel<false, G>, grid(a.tiles), dim3(S::kThreads), S::kSmem, md, md, a);
    return runit_after_launch(ctx, "moe_slots_down");
}

int32_t moe_slots_experts(runit_ctx* ctx, const void* gate, const void* up, const void* down, const float* x, const int32_t* idx, float* act,
                          float* y, void* staging, uint32_t T, uint32_t h, uint32_t ff, uint32_t E, uint32_t k) {
    // one tile per group up to 12 slots per expert (us with one / with four: 64 experts of 2048 x 1024: 8 slots 146 / 182, 12 177 / 190, 16
    // 209 / 201, 24 283 / 225; 128 of 2048 x 768: 8 194 / 260, 12 257 / 279, 16 323 / 300; 16 of 1024 x 512: 8 32 / 38, 24 40 / 45)
    return T * k <= 12 * E ? slots_run<1>(ctx, gate, up, down, x, idx, act, y, staging, T * k, h, ff, E, k)
                          : slots_run<4>(ctx, gate, up, down, x, idx, act, y, staging, T * k, h, ff, E, k);
}

}  // namespace runit
