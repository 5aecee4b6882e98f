// Causal attention of the prefill on the tcgen05 tensor cores: softmax(q.K^T / sqrt(hd)) . V over the f16 cache with key <=
// start + query (attention.metal:36-158), head dim 64 or 128.
//
// A CTA owns 128 queries of one head and walks the keys in blocks of 128.  Warp 8's first lane issues every copy and MMA; of warps
// 0..7 two threads share a query (tensor-memory lane): warps 0..3 have keys 0..63 of a block and the first half of the head's
// dimensions, warps 4..7 the others, and the row maximum meets in shared memory:
//   S = Q.K^T     Q rounded to f16 once (shared memory, 128-byte swizzle), K by TMA; f32, two buffers of 128 columns: the product of
//                 block i + 1 runs under the softmax of block i
//   P             row maximum, exp2 and sum from tensor memory, two passes over S; P is rounded to f16 into the columns of S that the
//                 thread has already read, which makes it the A operand of the second product
//   O += P.V      V by TMA as it lies in the cache (hd contiguous: B is MN-major), accumulated in tensor memory.  P, the sum (of the
//                 unrounded P, f32) and O are relative to the row maximum so far; O is scaled by the row's own threads when that has risen, behind
//                 P, where the product that it waits for is long over.
// One CTA per SM: 161 KB (two buffers of K and V; 116 asked for at head dim 64) and all 512 tensor-memory columns.  Query blocks go from the most keys to the fewest.
// Bound: one dependent chain per SM, about 5000 clocks per block, of which the exponentials are 1024 (16 a clock) and the products 512.
// Measured, 2048 queries x 16 heads x 128: 102 us (mma.sync, 64 queries of 4 warps, 167 TFLOP/s of useful products), 58 with one
// thread per query, one buffer of S and the block's output added in registers, 51 with two threads per query, 41 as it is (421 TFLOP/s; 30
// at head dim 64); 1024 queries 45 -> 19 us, 2000 behind 1000 cached ones 156 -> 62, 33 behind 300 17 -> 9.
// The error against 64 bits is the bf16 output's, 1.677e-3, as it was.  A reference that follows the maximum only when that has risen by
// 2^8 saves the scaling of O (40 us) but rounds the largest weights, which then are not 1: 1.678e-3, and up to twice the error before bf16.
// Rows of the tensor maps end at start + T, so that what the cache holds behind the data (NaN included) reads as zeros.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "gemv_common.cuh"
#include "runit_internal.h"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace runit {
namespace atc {

constexpr int kRows = 128, kKeys = 128;
constexpr uint32_t kCols = 512;                    // tensor memory: S | P in columns 0..127 and 128..255, O from 256
constexpr uint32_t kOnePerSm = 116 * 1024;         // shared memory that only one CTA of an SM can have

template <int HD> struct Shape {
    static constexpr uint32_t kPanel = 128 * 128;  // 64 elements of 128 rows
    static constexpr uint32_t kTile = HD / 64 * kPanel;
    // Q, two blocks of K, two of V; at head dim 64 (83 KB) more than it needs: a second CTA of an SM would only sit in its allocation
    // behind the first, bound to that SM however long the first one's row of blocks is (2048 queries x 16 heads x 64: 36.1 us with two
    // resident CTAs, 28.9 with one; 2000 behind 1000 cached ones 58.3 and 49.9; 1024 15.4 and 15.1, fewer the same)
    static constexpr uint32_t kSmem = 5 * kTile + 1024 < kOnePerSm ? kOnePerSm : 5 * kTile + 1024;
    static_assert(2 * kCols <= 512 || 2 * (kSmem + 1024) > 228 * 1024, "CTAs that share an SM share its tensor memory");
};

// kind::f16 with f16 operands (formats 0), f32 accumulator; bit 16: B is MN-major
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t m, uint32_t n, uint32_t b_mn) {
    return (1u << 4) | (b_mn << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// MN-major tile in the 128-byte swizzled layout: 64 elements (128 bytes) per row of K, groups of 8 K rows 1024 bytes apart (stride
// byte offset), the next 64 elements a panel further (leading byte offset)
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr, uint32_t panel) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(panel >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// A in tensor memory: 128 lanes, 32-bit column c = K elements 2c, 2c + 1
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(d_tmem), "r"(a_tmem), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int32_t c0, int32_t c1, int32_t c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t v[16];
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = r[16 * h + j];
        tmem_st16(taddr + 16 * h, v);
    }
}
__device__ __forceinline__ float exp2_approx(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// O += P.V * scale of one block for this thread's row and half of the dimensions, over the n keys that the row sees and no others; P of
// both halves is in tensor memory at p_cols, v is the block's V as TMA put it down.
template <int HD>
__device__ __forceinline__ void visible_products(uint32_t p_cols, uint32_t o_cols, const uint8_t* v, uint32_t half, uint32_t n, float scale, bool first) {
#pragma unroll 1
    for (uint32_t c = 0; c < HD / 64; c++) {
        const uint32_t dim = HD / 2 * half + 32 * c;
        const uint8_t* panel = v + (dim >> 6) * Shape<HD>::kPanel;
        uint32_t r[32];
        float o[32];
        tmem_ld32(o_cols + 32 * c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j++) o[j] = first ? 0.f : __uint_as_float(r[j]);
#pragma unroll 1
        for (uint32_t k = 0; k < kKeys; k += 2) {
            uint32_t two;
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(two) : "r"(p_cols + (k >> 1) + (k & 64 ? 32 : 0)) : "memory");
            tmem_ld_wait();
            const float2 w = __half22float2(*reinterpret_cast<const __half2*>(&two));
#pragma unroll
            for (uint32_t e = 0; e < 2; e++) {
                if (k + e >= n) break;
                const float we = (e ? w.y : w.x) * scale;
#pragma unroll
                for (uint32_t q = 0; q < 4; q++) {
                    const uint4 x = *reinterpret_cast<const uint4*>(panel + (k + e) * 128 + (((((dim & 63) >> 3) + q) ^ ((k + e) & 7)) << 4));
                    const __half2* h = reinterpret_cast<const __half2*>(&x);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 f = __half22float2(h[j]);
                        o[8 * q + 2 * j] = fmaf(we, f.x, o[8 * q + 2 * j]);
                        o[8 * q + 2 * j + 1] = fmaf(we, f.y, o[8 * q + 2 * j + 1]);
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < 32; j++) r[j] = __float_as_uint(o[j]);
        tmem_st32(o_cols + 32 * c, r);
        tmem_st_wait();
    }
}
// Not 0 where one of two bf16 values is an Inf or a NaN.
__device__ __forceinline__ uint32_t not_finite(uint32_t b2) { return ((b2 & 0x7FFF7FFFu) + 0x00800080u) & 0x80008000u; }

struct Args {
    const float* q;
    __nv_bfloat16* out;
    uint32_t T, heads, group, start;               // group: query heads per key head
    float scale_log2;                              // log2(e) / sqrt(hd)
    int32_t* status;
};

template <int HD>
__global__ void __launch_bounds__(288, 1) attention_tc_kernel(const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv, const Args a) {
    using S = Shape<HD>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[8];
    __shared__ uint32_t tmem_holder;
    __shared__ volatile int abort_flag;
    __shared__ float part[2][2][kRows];            // [block parity][half]: row maximum of a half; at the end the sums
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t qs = base, ks = base + S::kTile, vs = base + 3 * S::kTile;      // two buffers each
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // k_full, v_full, s_full: one per buffer; p_full, o_full: one phase per block
    const uint32_t k_full = smem_u32(&bars[0]), v_full = smem_u32(&bars[2]), s_full = smem_u32(&bars[4]), p_full = smem_u32(&bars[6]), o_full = smem_u32(&bars[7]);
    const uint32_t head = blockIdx.x, q0 = (gridDim.y - 1 - blockIdx.y) * kRows;
    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < 8; i++) mbar_init(smem_u32(&bars[i]), i == 6 ? 256 : 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_holder), kCols);
        tmem_relinquish();
    }
    grid_dependency_wait();
    // queries of this CTA as f16 into the swizzled K-major tile; rows behind the last query are zeros
    if (warp < 8) {
        constexpr uint32_t CH = HD / 8;            // 16-byte chunks of a row
        for (uint32_t i = tid; i < kRows * CH; i += 256) {
            const uint32_t r = i / CH, c = i % CH;
            float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
            if (q0 + r < a.T) {
                const float4* src = reinterpret_cast<const float4*>(a.q + ((size_t)(q0 + r) * a.heads + head) * HD + c * 8);
                x0 = src[0];
                x1 = src[1];
            }
            const __half2 h[4] = {__floats2half2_rn(x0.x, x0.y), __floats2half2_rn(x0.z, x0.w), __floats2half2_rn(x1.x, x1.y), __floats2half2_rn(x1.z, x1.w)};
            uint8_t* dst = smem_raw + (qs - smem_u32(smem_raw)) + (c >> 3) * S::kPanel + r * 128 + (((c & 7) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(h);
        }
        fence_proxy_async();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    // not before the allocation is known to be done: it waits without a limit, and a block of the next grid, which allocates before its
    // own dependency wait, must not take the columns first
    grid_launch_dependents();
    const uint32_t tmem = tmem_holder;
    const uint32_t last_q = min(a.T, q0 + kRows) - 1, n_blocks = (a.start + last_q) / kKeys + 1;
    // blocks of which some row does not see all keys: the last two at most
    const uint32_t first_masked = (a.start + q0 + 1) / kKeys;
    bool ok = true;

    // A hidden key's weight of 0 meets its V all the same, and 0 x Inf is NaN.  An output that is not finite is therefore taken again, with
    // the products of the blocks that have hidden keys by visible_products; whatever is finite has met no such V.  (Looking at V
    // first instead cost 2048 queries x 16 heads x 128 42.3 us in the softmax's warps and 42.6 in a warp of its own, against 39.8; the
    // second look costs 33 queries behind 300 keys 0.2 of 9.0 us.)
    for (bool careful = false;; careful = true) {
        bool again = false;
        if (warp == 8) {
            if (lane == 0) {
                const int32_t kvh = (int32_t)(head / a.group);
                auto load = [&](const CUtensorMap* m, uint32_t dst, uint32_t bar, uint32_t i) {
                    mbar_expect_tx(bar, S::kTile);
                    for (int p = 0; p < HD / 64; p++) tma_load_3d(dst + p * S::kPanel, m, 64 * p, (int32_t)(i * kKeys), kvh, bar);
                };
                uint32_t n_k = 0, n_v = 0, n_s = 0, n_o = 0;         // started so far
                auto load_k = [&](uint32_t i) { load(&mk, ks + (i & 1) * S::kTile, k_full + 8 * (i & 1), i); n_k++; };
                auto load_v = [&](uint32_t i) { load(&mv, vs + (i & 1) * S::kTile, v_full + 8 * (i & 1), i); n_v++; };
                auto scores = [&](uint32_t i) {        // S of block i; its K has been waited for
                    const uint32_t kb = ks + (i & 1) * S::kTile;
#pragma unroll
                    for (int s = 0; s < HD / 16; s++) {
                        const uint32_t off = (s >> 2) * S::kPanel + (s & 3) * 32;
                        umma_bf16(tmem + 128 * (i & 1), umma_desc_sw128(qs + off), umma_desc_sw128(kb + off), idesc_f16(kRows, kKeys, 0), s > 0);
                    }
                    umma_commit(s_full + 8 * (i & 1));
                    n_s++;
                };
                load_k(0);
                load_v(0);
                if (n_blocks > 1) {
                    load_k(1);
                    load_v(1);
                }
                ok = mbar_wait_timed(k_full, 0, &abort_flag);
                if (ok) {
                    tc_fence_after_sync();
                    scores(0);
                }
                for (uint32_t i = 0; i < n_blocks && ok; i++) {
                    const uint32_t ph = (i >> 1) & 1;
                    // block i + 1's columns hold P of block i - 1, whose product also frees V's buffer
                    if (i > 0) {
                        if (!(ok = mbar_wait_timed(o_full, (i - 1) & 1, &abort_flag))) break;
                        if (i + 1 < n_blocks) load_v(i + 1);
                    }
                    if (i + 1 < n_blocks) {
                        if (!(ok = mbar_wait_timed(k_full + 8 * ((i + 1) & 1), ((i + 1) >> 1) & 1, &abort_flag))) break;
                        tc_fence_after_sync();
                        scores(i + 1);
                    }
                    if (!(ok = mbar_wait_timed(s_full + 8 * (i & 1), ph, &abort_flag))) break;
                    if (i + 2 < n_blocks) load_k(i + 2);      // S of block i is there: its K buffer is free
                    if (!(ok = mbar_wait_timed(v_full + 8 * (i & 1), ph, &abort_flag))) break;
                    if (!(ok = mbar_wait_timed(p_full, i & 1, &abort_flag))) break;
                    tc_fence_after_sync();
                    const uint32_t vb = vs + (i & 1) * S::kTile, pb = tmem + 128 * (i & 1);
                    if (!careful || i < first_masked) {
#pragma unroll
                        for (int s = 0; s < kKeys / 16; s++)
                            umma_f16_ts(tmem + 256, pb + 8 * s + (s >= 4 ? 32 : 0), desc_mn_sw128(vb + s * 2048, S::kPanel), idesc_f16(kRows, HD, 1), i > 0 || s > 0);
                    }
                    umma_commit(o_full);
                    n_o++;
                }
                if (ok) ok = mbar_wait_timed(o_full, (n_blocks - 1) & 1, &abort_flag);
                if (!ok) {          // nothing is in flight when the CTA leaves, whatever it gave up on
                    mbar_drain(k_full, 2, n_k);
                    mbar_drain(v_full, 2, n_v);
                    mbar_drain(s_full, 2, n_s);
                    mbar_drain(o_full, 1, n_o);
                }
            }
        } else {
            const uint32_t half = warp >> 2, row = (warp & 3) * 32 + lane, mine = tmem + (((warp & 3) * 32) << 16), qpos = a.start + q0 + row;
            const uint32_t o_cols = mine + 256 + HD / 2 * half;
            float late = 1.f;                          // what the last block's rise scaled O by
            float ref = -INFINITY, l = 0.f;            // reference in units of the scaled score times log2(e); l: this half's sum
            // a thread whose wait gave up goes on without waiting: all 256 take the same barriers
            for (uint32_t i = 0; i < n_blocks; i++) {
                if (ok) ok = mbar_wait_timed(s_full + 8 * (i & 1), (i >> 1) & 1, &abort_flag);
                __syncwarp();
                tc_fence_after_sync();
                const uint32_t s_cols = mine + 128 * (i & 1) + 64 * half, key0 = i * kKeys + 64 * half;
                const bool masked = i >= first_masked;
                float mx = -INFINITY;
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t r[32];
                    tmem_ld32(s_cols + 32 * c, r);
                    tmem_ld_wait();
                    if (masked) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (key0 + 32 * c + j <= qpos) mx = fmaxf(mx, __uint_as_float(r[j]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++) mx = fmaxf(mx, __uint_as_float(r[j]));
                    }
                }
                part[i & 1][half][row] = mx;
                asm volatile("bar.sync 1, 256;" ::: "memory");              // two blocks' slots: nobody is a whole block ahead of another
                mx = fmaxf(mx, part[i & 1][half ^ 1][row]) * a.scale_log2;
                const bool rise = mx > ref;
                const bool any = __any_sync(0xffffffffu, rise);
                const float corr = rise ? exp2_approx(ref - mx) : 1.f;
                late = corr;
                l *= corr;
                ref = rise ? mx : ref;
                const float sub = ref == -INFINITY ? 0.f : ref;             // no finite score yet: every factor is 0
                float sum = 0.f;
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t r[32], p[16];
                    tmem_ld32(s_cols + 32 * c, r);
                    tmem_ld_wait();
                    if (masked) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (key0 + 32 * c + j > qpos) r[j] = 0xFF800000u;
                    }
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        // not one multiply-add: the maximum itself must come out as exactly 1, so that a row of one key is that key's V
                        const float p0 = exp2_approx(__fsub_rn(__fmul_rn(__uint_as_float(r[2 * j]), a.scale_log2), sub));
                        const float p1 = exp2_approx(__fsub_rn(__fmul_rn(__uint_as_float(r[2 * j + 1]), a.scale_log2), sub));
                        const __half2 h = __floats2half2_rn(p0, p1);
                        sum += p0 + p1;
                        p[j] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    tmem_st16(s_cols + 16 * c, p);     // behind what this thread has read: 16 columns for 32 keys
                }
                l += sum;
                tmem_st_wait();
                // every phase of o_full is waited for in turn, so that its parity says which
                if (i > 0) {
                    if (ok) ok = mbar_wait_timed(o_full, (i - 1) & 1, &abort_flag);
                    __syncwarp();
                    if (any) {
                        tc_fence_after_sync();
#pragma unroll
                        for (int c = 0; c < HD / 64; c++) {
                            uint32_t r[32];
                            tmem_ld32(o_cols + 32 * c, r);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * corr);
                            tmem_st32(o_cols + 32 * c, r);
                        }
                        tmem_st_wait();
                    }
                }
                tc_fence_before_sync();
                mbar_arrive(p_full);
            }
            if (ok) ok = mbar_wait_timed(o_full, (n_blocks - 1) & 1, &abort_flag);
            __syncwarp();
            tc_fence_after_sync();
            // the slots of the block after the last one: its predecessor's readers have passed that block's barrier
            part[n_blocks & 1][half][row] = l;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            l += part[n_blocks & 1][half ^ 1][row];
            if (careful) {
                // P and V of the last two blocks are still there, P of the last but one relative to the reference before the last block's rise
                tc_fence_after_sync();
                for (uint32_t i = first_masked; i < n_blocks; i++) {
                    if (ok) ok = mbar_wait_timed(v_full + 8 * (i & 1), (i >> 1) & 1, &abort_flag);
                    __syncwarp();
                    visible_products<HD>(mine + 128 * (i & 1), o_cols, smem_raw + (vs - smem_u32(smem_raw)) + (i & 1) * S::kTile, half,
                                         qpos < i * kKeys ? 0 : min((uint32_t)kKeys, qpos - i * kKeys + 1), i + 1 < n_blocks ? late : 1.f, i == 0);
                }
            }
            const float inv = l > 0.f || !(l == l) ? 1.0f / l : 0.f;
            uint4* dst = reinterpret_cast<uint4*>(a.out + ((size_t)(q0 + row) * a.heads + head) * HD + HD / 2 * half);
#pragma unroll
            for (int c = 0; c < HD / 64; c++) {
                uint32_t r[32];
                tmem_ld32(o_cols + 32 * c, r);
                tmem_ld_wait();
                if (ok && q0 + row < a.T) {
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        __nv_bfloat162 h[4];
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            h[j] = __floats2bfloat162_rn(__uint_as_float(r[8 * k + 2 * j]) * inv, __uint_as_float(r[8 * k + 2 * j + 1]) * inv);
                        const uint4 w = *reinterpret_cast<const uint4*>(h);
                        dst[4 * c + k] = w;
                        again |= ((not_finite(w.x) | not_finite(w.y)) | (not_finite(w.z) | not_finite(w.w))) != 0;
                    }
                }
            }
        }
        if (!ok) {
            abort_flag = 1;
            if (a.status) atomicExch(a.status, 1);
        }
        tc_fence_before_sync();
        if (!__syncthreads_or(again) || careful || abort_flag) break;
        if (tid == 0) {
            for (int i = 0; i < 8; i++) {
                mbar_inval(smem_u32(&bars[i]));
                mbar_init(smem_u32(&bars[i]), i == 6 ? 256 : 1);
            }
            fence_mbar_init();
        }
        __syncthreads();
        tc_fence_after_sync();
    }
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kCols);
    }
}

template <int HD>
static int32_t run(runit_ctx* ctx, const CUtensorMap& mk, const CUtensorMap& mv, const Args& a) {
    static bool configured[64] = {false};
    if (ctx->device >= 64 || !configured[ctx->device]) {
        RUNIT_CUDA_TRY(ctx, cudaFuncSetAttribute(attention_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<HD>::kSmem));
        if (ctx->device < 64) configured[ctx->device] = true;
    }
    runit_launch_chain_smem(ctx, attention_tc_kernel<HD>, dim3(a.heads, (a.T + kRows - 1) / kRows), dim3(288), Shape<HD>::kSmem, mk, mv, a);
    return runit_after_launch(ctx, "prefill_attention_tc");
}

}  // namespace atc

// Every count of queries: a 128-query tile that is mostly padding still has half as many blocks in its chain as 64-key ones (33
// queries behind 300 keys 17 -> 9 us, 64 behind 1900 72 -> 28).  Addresses are 16-byte aligned (checked at the entry point).
int32_t attention_tc(runit_ctx* ctx, const float* q, const void* kcache, const void* vcache, void* out_bf16, uint32_t T, uint32_t heads, uint32_t kv_heads,
                     uint32_t hd, uint32_t max_seq, uint32_t start_pos) {
    if (!ctx->encode_tiled) return runit_fail(ctx, RUNIT_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
    auto encode = reinterpret_cast<CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                                CUtensorMapFloatOOBfill)>(ctx->encode_tiled);
    CUtensorMap m[2];
    for (int i = 0; i < 2; i++) {
        const cuuint64_t dim[3] = {hd, start_pos + T, kv_heads}, stride[2] = {hd * 2ull, (cuuint64_t)max_seq * hd * 2};
        const cuuint32_t box[3] = {64, atc::kKeys, 1}, one[3] = {1, 1, 1};
        const CUresult r = encode(&m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(i ? vcache : kcache), dim, stride, box, one,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return runit_fail(ctx, RUNIT_ERR_LAUNCH, "cuTensorMapEncodeTiled failed with %d", (int)r);
    }
    const atc::Args a{q, (__nv_bfloat16*)out_bf16, T, heads, heads / kv_heads, start_pos, 1.4426950408889634f / sqrtf((float)hd), ctx->d_status};
    return hd == 128 ? atc::run<128>(ctx, m[0], m[1], a) : atc::run<64>(ctx, m[0], m[1], a);
}

}  // namespace runit
