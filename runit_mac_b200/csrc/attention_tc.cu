// Causal attention of the prefill on the tcgen05 tensor cores: softmax(q.K^T / sqrt(hd)) . V over the f16 cache with key <=
// start + query (attention.metal:36-158), head dim 64 or 128.
//
// A CTA owns 128 queries of one head and walks the keys in blocks of 128, as two chains: one of the even blocks and one of the odd ones, each
// with scores, maximum, sum and output of its own, which meet at the end.  Eight warps serve a chain, two threads a query (tensor-memory lane):
// the first four have keys 0..63 of a block and the first half of the head's dimensions, the others the rest, and the row maximum meets in
// shared memory.  One more warp per chain issues its copies and MMAs:
//   S = Q.K^T     Q rounded to f16 once (shared memory, 128-byte swizzle), K by TMA; f32
//   P             row maximum, exp2 and sum from tensor memory, two passes over S; P is rounded to f16 into the columns of S that the
//                 thread has already read, which makes it the A operand of the second product
//   O += P.V      V by TMA as it lies in the cache (hd contiguous: B is MN-major), accumulated in tensor memory.  P, the sum (of the
//                 unrounded P, f32) and O are relative to the chain's row maximum so far; O is scaled by the row's own threads when that has risen,
//                 ahead of P.  The next S takes P's columns: its MMAs come behind those that read them.
// The chains take their exponentials in turn, so that the products of one run under the exponentials of the other.
// One CTA per SM: 161 KB (one buffer of K and V a chain; 116 asked for at head dim 64) and all 512 tensor-memory columns.  Query blocks go from the
// most keys to the fewest.
// Bound: two dependent chains per SM: a block's maximum, scaling of O, exponentials (1024 clocks at 16 a clock), hand-over and products (1024).
// Measured, 2048 queries x 16 heads x 128: 102 us (mma.sync, 64 queries of 4 warps), 41 with one chain and two buffers of S, 37 with two chains in
// step, 34.5 with the odd one started half a period late (they drift into step again), 32.8 in turn (524 TFLOP/s of useful products; 24.6 at head dim 64, 29 with one
// chain); 1024 queries 17.8 -> 15.3 us, 2000 behind 1000 cached ones 62 -> 48, 64 behind 1900 27.6 -> 22.5, a single block 6.8 -> 6.5.  O scaled between the
// exponentials instead: slower (register spills).
// The error against 64 bits is the bf16 output's, 1.677e-3, as it was.  A reference that follows the maximum only when that has risen by
// 2^8 saves the scaling of O but rounds the largest weights, which then are not 1: 1.678e-3, and up to twice the error before bf16.
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
constexpr uint32_t kSoftWarps = 16, kThreads = 32 * (kSoftWarps + 2);
constexpr int kBars = 7;                           // of a chain: k_full, v_full, s_full, p_full, o_full, done, turn
constexpr uint32_t kCols = 512;                    // tensor memory: S | P of the chains in columns 0..127 and 128..255, their O from 256 and 384
constexpr uint32_t kOnePerSm = 116 * 1024;         // shared memory that only one CTA of an SM can have

template <int HD> struct Shape {
    static constexpr uint32_t kPanel = 128 * 128;  // 64 elements of 128 rows
    static constexpr uint32_t kTile = HD / 64 * kPanel;
    // Q, a block of K and one of V for each chain; at head dim 64 (83 KB) more than it needs: a second CTA of an SM would only sit in its allocation
    // behind the first, bound to that SM however long the first one's row of blocks is (2048 queries x 16 heads x 64: 36.1 us with two
    // resident CTAs, 28.9 with one; 2000 behind 1000 cached ones 58.3 and 49.9; 1024 15.4 and 15.1, fewer the same)
    static constexpr uint32_t kSmem = 5 * kTile + 1024 < kOnePerSm ? kOnePerSm : 5 * kTile + 1024;
    static_assert(2 * kCols <= 512 || 2 * (kSmem + 1024) > 228 * 1024, "CTAs that share an SM share its tensor memory");
};

// MN-major tile in the 128-byte swizzled layout: 64 elements (128 bytes) per row of K, groups of 8 K rows 1024 bytes apart (stride
// byte offset), the next 64 elements a panel further (leading byte offset)
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr, uint32_t panel) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(panel >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
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

// O += P.V of one block for this thread's row and half of the dimensions, over the n keys that the row sees and no others; P of
// both halves is in tensor memory at p_cols, v is the block's V as TMA put it down.
template <int HD>
__device__ __forceinline__ void visible_products(uint32_t p_cols, uint32_t o_cols, const uint8_t* v, uint32_t half, uint32_t n, bool first) {
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
                const float we = e ? w.y : w.x;
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
__device__ __forceinline__ void chain_sync(uint32_t chain) {
    if (chain) asm volatile("bar.sync 2, 256;" ::: "memory");
    else asm volatile("bar.sync 1, 256;" ::: "memory");
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
__global__ void __launch_bounds__(kThreads, 1) attention_tc_kernel(const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv, const Args a) {
    using S = Shape<HD>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kBars];
    __shared__ uint32_t tmem_holder;
    __shared__ volatile int abort_flag;
    __shared__ float part[2][2][2][kRows];         // [block parity][chain][half]: row maximum of a half
    __shared__ float end_ref[2][kRows], end_sum[2][2][kRows];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t qs = base;
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t chain = warp < kSoftWarps ? warp >> 3 : warp - kSoftWarps;
    // this chain's K, V and barriers; k_full, v_full, s_full, p_full, o_full: one phase per block of the chain; done: one
    const uint32_t kb = base + S::kTile + chain * 2 * S::kTile, vb = kb + S::kTile;
    const uint32_t bar0 = smem_u32(&bars[chain * kBars]);
    const uint32_t k_full = bar0, v_full = bar0 + 8, s_full = bar0 + 16, p_full = bar0 + 24, o_full = bar0 + 32, done = bar0 + 40, turn = bar0 + 48;
    const uint32_t other_turn = smem_u32(&bars[(chain ^ 1) * kBars + 6]);
    const uint32_t head = blockIdx.x, q0 = (gridDim.y - 1 - blockIdx.y) * kRows;
    auto init_bars = [&]() {
        for (int i = 0; i < 2 * kBars; i++) mbar_init(smem_u32(&bars[i]), i % kBars == 3 ? 256 : i % kBars == 6 ? 8 : 1);
        fence_mbar_init();
    };
    if (tid == 0) {
        abort_flag = 0;
        init_bars();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_holder), kCols);
        tmem_relinquish();
    }
    grid_dependency_wait();
    // queries of this CTA as f16 into the swizzled K-major tile; rows behind the last query are zeros
    if (warp < kSoftWarps) {
        constexpr uint32_t CH = HD / 8;            // 16-byte chunks of a row
        for (uint32_t i = tid; i < kRows * CH; i += 32 * kSoftWarps) {
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
    const uint32_t tmem = tmem_holder, s_cols = tmem + 128 * chain, o_cols = tmem + 256 + 128 * chain;
    const uint32_t last_q = min(a.T, q0 + kRows) - 1, n_blocks = (a.start + last_q) / kKeys + 1;
    const uint32_t mine = (n_blocks + 1 - chain) >> 1;              // blocks chain, chain + 2, ...
    // blocks of which some row does not see all keys: the last two at most, so the last of a chain at most
    const uint32_t first_masked = (a.start + q0 + 1) / kKeys;
    bool ok = true;

    // A hidden key's weight of 0 meets its V all the same, and 0 x Inf is NaN.  An output that is not finite is therefore taken again, with
    // the products of the blocks that have hidden keys by visible_products; whatever is finite has met no such V.
    for (bool careful = false;; careful = true) {
        bool again = false;
        if (warp >= kSoftWarps) {
            const int32_t kvh = (int32_t)(head / a.group);
            uint32_t n_k = 0, n_v = 0, n_s = 0, n_o = 0, n_d = 0;    // started so far
            auto load = [&](const CUtensorMap* m, uint32_t dst, uint32_t bar, uint32_t j) {
                if (elect_one()) {
                    mbar_expect_tx(bar, S::kTile);
                    for (int p = 0; p < HD / 64; p++) tma_load_3d(dst + p * S::kPanel, m, 64 * p, (int32_t)((2 * j + chain) * kKeys), kvh, bar);
                }
                __syncwarp();
            };
            auto load_k = [&](uint32_t j) { load(&mk, kb, k_full, j); n_k++; };
            auto load_v = [&](uint32_t j) { load(&mv, vb, v_full, j); n_v++; };
            auto scores = [&]() {                  // S of the block whose K has been waited for; behind the product that reads P from these columns
                if (elect_one()) {
#pragma unroll
                    for (int s = 0; s < HD / 16; s++) {
                        const uint32_t off = (s >> 2) * S::kPanel + (s & 3) * 32;
                        umma_bf16(s_cols, umma_desc_sw128(qs + off), umma_desc_sw128(kb + off), umma_idesc_f16(kRows, kKeys, 0), s > 0);
                    }
                    umma_commit(s_full);
                }
                __syncwarp();
                n_s++;
            };
            if (mine > 0) {
                load_k(0);
                load_v(0);
                ok = mbar_wait_timed(k_full, 0, &abort_flag);
                if (__all_sync(0xffffffffu, ok)) {
                    tc_fence_after_sync();
                    scores();
                } else ok = false;
            }
            for (uint32_t j = 0; j < mine && ok; j++) {
                const uint32_t ph = j & 1;
                const bool last = j + 1 == mine;
                ok = mbar_wait_timed(s_full, ph, &abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                if (!last) load_k(j + 1);          // S is there: its K buffer is free
                ok = mbar_wait_timed(v_full, ph, &abort_flag) && mbar_wait_timed(p_full, ph, &abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                tc_fence_after_sync();
                if (elect_one()) {
                    if (!careful || 2 * j + chain < first_masked) {
#pragma unroll
                        for (int s = 0; s < kKeys / 16; s++)
                            umma_f16_ts(o_cols, s_cols + 8 * s + (s >= 4 ? 32 : 0), desc_mn_sw128(vb + s * 2048, S::kPanel), umma_idesc_f16(kRows, HD, 1), j > 0 || s > 0);
                    }
                    umma_commit(last ? done : o_full);
                }
                __syncwarp();
                if (last) {
                    n_d++;
                    break;
                }
                n_o++;
                ok = mbar_wait_timed(k_full, ph ^ 1, &abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                tc_fence_after_sync();
                scores();
                ok = mbar_wait_timed(o_full, ph, &abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                load_v(j + 1);
            }
            if (mine > 0 && ok) ok = mbar_wait_timed(done, 0, &abort_flag);
            if (!ok) {              // nothing is in flight when the CTA leaves, whatever it gave up on
                mbar_drain(k_full, 1, n_k);
                mbar_drain(v_full, 1, n_v);
                mbar_drain(s_full, 1, n_s);
                mbar_drain(o_full, 1, n_o);
                mbar_drain(done, 1, n_d);
            }
        } else {
            const uint32_t half = (warp >> 2) & 1, row = (warp & 3) * 32 + lane, lanes = ((warp & 3) * 32) << 16, qpos = a.start + q0 + row;
            const uint32_t my_o = o_cols + lanes + HD / 2 * half, my_s = s_cols + lanes + 64 * half;
            float ref = -INFINITY, l = 0.f;            // reference: the largest score so far; l: this half's sum
            // a thread whose wait gave up goes on without waiting: all threads take the same barriers
            for (uint32_t j = 0; j < mine; j++) {
                if (ok) ok = mbar_wait_timed(s_full, j & 1, &abort_flag);
                __syncwarp();
                tc_fence_after_sync();
                const uint32_t key0 = (2 * j + chain) * kKeys + 64 * half;
                const bool masked = 2 * j + chain >= first_masked;
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t r[32];
                    tmem_ld32(my_s + 32 * c, r);
                    tmem_ld_wait();
                    if (masked) {
#pragma unroll
                        for (int e = 0; e < 32; e++)
                            if (key0 + 32 * c + e > qpos) r[e] = 0xFF800000u;
                    }
#pragma unroll
                    for (int e = 0; e < 32; e++) mx4[e & 3] = fmaxf(mx4[e & 3], __uint_as_float(r[e]));
                }
                float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                part[j & 1][chain][half][row] = mx;
                chain_sync(chain);                     // two blocks' slots: nobody is a whole block ahead of another
                mx = fmaxf(mx, part[j & 1][chain][half ^ 1][row]);
                const bool rise = mx > ref;
                const float corr = rise ? exp2_approx((ref - mx) * a.scale_log2) : 1.f;
                l *= corr;
                ref = rise ? mx : ref;
                const float sub = ref == -INFINITY ? 0.f : ref;             // no finite score yet: every factor is 0
                const uint64_t scale2 = packf(a.scale_log2), sub2 = packf(-sub);
                uint64_t both = 0;
                // S of this block comes behind the product of the last one: O is complete
                if (__any_sync(0xffffffffu, rise) && j > 0) {
#pragma unroll
                    for (int c = 0; c < HD / 32; c++) {
                        uint32_t o[16];
                        tmem_ld16(my_o + 16 * c, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
                        tmem_st16(my_o + 16 * c, o);
                    }
                }
                // The chains take their exponentials in turn (block j of the odd one behind block j of the even one, and that behind block j - 1 of the
                // odd one): the products of one run under the exponentials of the other.  Left alone they fall into step.
                if (ok && (chain == 1 || j > 0)) ok = mbar_wait_timed(turn, (chain == 1 ? j : j - 1) & 1, &abort_flag);
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t r[32], p[16];
                    tmem_ld32(my_s + 32 * c, r);
                    tmem_ld_wait();
                    if (masked) {
#pragma unroll
                        for (int e = 0; e < 32; e++)
                            if (key0 + 32 * c + e > qpos) r[e] = 0xFF800000u;
                    }
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        // the difference first: the maximum itself comes out as exactly 1, so that a row of one key is that key's V
                        const uint64_t v = fmul2(fadd2(pack2(r[2 * e], r[2 * e + 1]), sub2), scale2);
                        const float p0 = exp2_approx(__uint_as_float((uint32_t)v)), p1 = exp2_approx(__uint_as_float((uint32_t)(v >> 32)));
                        const __half2 h = __floats2half2_rn(p0, p1);
                        both = fadd2(both, pack2(__float_as_uint(p0), __float_as_uint(p1)));
                        p[e] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    tmem_st16(my_s + 16 * c, p);       // behind what this thread has read: 16 columns for 32 keys
                }
                l += sum2(both);
                __syncwarp();
                if (lane == 0) mbar_arrive(other_turn);
                tmem_st_wait();
                tc_fence_before_sync();
                mbar_arrive(p_full);
            }
            if (mine > 0) {
                if (ok) ok = mbar_wait_timed(done, 0, &abort_flag);
                __syncwarp();
                tc_fence_after_sync();
                const uint32_t i = 2 * (mine - 1) + chain;
                if (careful && i >= first_masked) {    // P and V of the chain's last block are still there
                    tc_fence_before_sync();
                    chain_sync(chain);
                    tc_fence_after_sync();
                    visible_products<HD>(s_cols + lanes, my_o, smem_raw + (vb - smem_u32(smem_raw)), half, qpos < i * kKeys ? 0 : min((uint32_t)kKeys, qpos - i * kKeys + 1), mine == 1);
                }
            }
            if (half == 0) end_ref[chain][row] = ref;
            end_sum[chain][half][row] = l;
            tc_fence_before_sync();
            asm volatile("bar.sync 3, 512;" ::: "memory");
            tc_fence_after_sync();
            // both chains' sums and outputs relative to the larger of their references; four threads share a row
            const float ref0 = end_ref[0][row], ref1 = end_ref[1][row], top = fmaxf(ref0, ref1);
            const float f0 = ref0 == -INFINITY ? 0.f : exp2_approx((ref0 - top) * a.scale_log2), f1 = ref1 == -INFINITY ? 0.f : exp2_approx((ref1 - top) * a.scale_log2);
            l = (end_sum[0][0][row] + end_sum[0][1][row]) * f0 + (end_sum[1][0][row] + end_sum[1][1][row]) * f1;
            const float inv = l > 0.f || !(l == l) ? 1.0f / l : 0.f, g0 = inv * f0, g1 = inv * f1;
            const uint32_t dim0 = HD / 2 * half + HD / 4 * chain;
            uint4* dst = reinterpret_cast<uint4*>(a.out + ((size_t)(q0 + row) * a.heads + head) * HD + dim0);
#pragma unroll
            for (int c = 0; c < HD / 64; c++) {
                uint32_t x[16], y[16];
                tmem_ld16(tmem + lanes + 256 + dim0 + 16 * c, x);
                if (n_blocks > 1) tmem_ld16(tmem + lanes + 384 + dim0 + 16 * c, y);
                tmem_ld_wait();
                if (ok && q0 + row < a.T) {
                    float o[16];
#pragma unroll
                    for (int e = 0; e < 16; e++) o[e] = n_blocks > 1 ? fmaf(__uint_as_float(x[e]), g0, __uint_as_float(y[e]) * g1) : __uint_as_float(x[e]) * g0;
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        __nv_bfloat162 h[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(o[8 * k + 2 * e], o[8 * k + 2 * e + 1]);
                        const uint4 w = *reinterpret_cast<const uint4*>(h);
                        dst[2 * c + k] = w;
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
            for (int i = 0; i < 2 * kBars; i++) mbar_inval(smem_u32(&bars[i]));
            init_bars();
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
    runit_launch_chain_smem(ctx, attention_tc_kernel<HD>, dim3(a.heads, (a.T + kRows - 1) / kRows), dim3(kThreads), Shape<HD>::kSmem, mk, mv, a);
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
