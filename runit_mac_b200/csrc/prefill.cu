// Batched prefill: the whole prompt in one pass, GEMMs instead of one GEMV per token (crates/engine/src/prefill.rs:29-255).
//
// The reference's pass runs in f16 with dequantised f16 weights: per layer RMSNorm, three projection GEMMs
// (gemm.metal:39,149: 16x16 scalar tiles), batched RoPE, a host loop that copies K and V into the cache, causal
// FlashAttention with q_len = seq (attention.metal:36-158), the output GEMM, the residual add, the second RMSNorm, and for
// a mixture-of-experts model the decode block once per token (prefill.rs:156-215).  Here:
//   * the hidden state stays f32 between operators (as in this library's decode path); GEMM operands are bf16: the
//     activations are rounded once, the weights are dequantised from Q4_K to bf16 tiles inside the tcgen05 GEMM of
//     moe_grouped.cu, used with one "expert" that owns the whole matrix and the tokens in their own order;
//   * RoPE of q and k, the f16 rounding of k and v and their scatter into the cache are one launch over all positions;
//   * causal attention over the f16 cache is the kernel of attention_tc.cu; its output is written as bf16, the operand of
//     the output GEMM;
//   * the mixture-of-experts block is runit_moe_layer_q4k_bf16 on all tokens at once;
//   * the last position's hidden state then goes through the decode path's lm_head launch (RMSNorm prologue, argmax
//     epilogue), and the decoder's state is left at position n with that token, so decoding continues from the cache.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "decode_ops.cuh"
#include "gemv_common.cuh"
#include "runit_internal.h"

namespace runit {
namespace pf {

// x[t][:] = emb[token[t]][:]
__global__ void __launch_bounds__(256) embed_rows_kernel(const float* __restrict__ emb, const int32_t* __restrict__ tokens,
                                                          float* __restrict__ x, uint32_t h) {
    const uint32_t t = blockIdx.x;
    const float4* src = reinterpret_cast<const float4*>(emb + (size_t)tokens[t] * h);
    float4* dst = reinterpret_cast<float4*>(x + (size_t)t * h);
    for (uint32_t i = threadIdx.x; i < h / 4; i += 256) dst[i] = src[i];
}

// y[t][:] = bf16(x[t][:] * rsqrt(mean(x[t]^2) + eps) * gamma)   (norm.metal:95-154, same sum order as rms_norm_kernel)
__global__ void __launch_bounds__(256) rms_norm_bf16_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
                                                             __nv_bfloat16* __restrict__ y, float eps, uint32_t h) {
    __shared__ float part[8];
    const float* row = x + (size_t)blockIdx.x * h;
    __nv_bfloat16* out = y + (size_t)blockIdx.x * h;
    float s = 0.f;
    for (uint32_t i = threadIdx.x; i < h; i += 256) {
        const float v = row[i];
        s = fmaf(v, v, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += part[i];
    const float r = rsqrtf(tot / (float)h + eps);
    for (uint32_t i = threadIdx.x; i < h; i += 256) out[i] = __float2bfloat16_rn(row[i] * r * gamma[i]);
}

// Rotary embedding of q (in place) and k for every position, then k (rotated) and v into the f16 caches: the arithmetic
// per element of rope_kv_kernel (fused_rope.metal:17-56, activation.metal:13-44).  grid (T, max(heads, kv_heads)).
// q_in / k / v: rows of `ld` floats (one matrix [T][q | k | v] when the three projections were one GEMM, ld = its width;
// or three matrices with ld = 0: rows as wide as their own heads); q_out: [T][heads * hd], may be q_in when ld = 0.
__global__ void rope_cache_rows_kernel(const float* q_in, float* q_out, const float* __restrict__ k, const float* __restrict__ v,
                                       __half* __restrict__ kc, __half* __restrict__ vc, uint32_t hd, uint32_t heads, uint32_t kv_heads,
                                       uint32_t start_pos, float theta, uint32_t max_seq, uint32_t ld) {
    const uint32_t t = blockIdx.x, hid = blockIdx.y, d = threadIdx.x, half = hd / 2;
    if (d >= half) return;
    const uint32_t pos = start_pos + t;
    const float freq = 1.0f / powf(theta, (float)(2 * d) / (float)hd);
    const float angle = (float)pos * freq;
    const float c = cosf(angle), s = sinf(angle);
    if (hid < heads) {
        const float* pi = q_in + (size_t)t * (ld ? ld : heads * hd) + (size_t)hid * hd;
        float* p = q_out + ((size_t)t * heads + hid) * hd;
        const float a = pi[d], b = pi[d + half];
        p[d] = a * c - b * s;
        p[d + half] = a * s + b * c;
    }
    if (hid < kv_heads && pos < max_seq) {
        const float* p = k + (size_t)t * (ld ? ld : kv_heads * hd) + (size_t)hid * hd;
        const float a = p[d], b = p[d + half];
        const size_t o = ((size_t)hid * max_seq + pos) * hd;
        kc[o + d] = __float2half_rn(a * c - b * s);
        kc[o + d + half] = __float2half_rn(a * s + b * c);
        const float* vp = v + (size_t)t * (ld ? ld : kv_heads * hd) + (size_t)hid * hd;
        vc[o + d] = __float2half_rn(vp[d]);
        vc[o + d + half] = __float2half_rn(vp[d + half]);
    }
}

// y[t][:] = bf16(x[t][:])
__global__ void __launch_bounds__(256) to_bf16_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, size_t n4) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    const float4 a = reinterpret_cast<const float4*>(x)[i];
    __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(y) + 2 * i;
    o[0] = __floats2bfloat162_rn(a.x, a.y);
    o[1] = __floats2bfloat162_rn(a.z, a.w);
}

// x[t][:] += y[t][:]
__global__ void __launch_bounds__(256) add_rows_kernel(float* __restrict__ x, const float* __restrict__ y, size_t n4) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    float4 a = reinterpret_cast<float4*>(x)[i];
    const float4 b = reinterpret_cast<const float4*>(y)[i];
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    reinterpret_cast<float4*>(x)[i] = a;
}

// x[t][:] += y[t][:], then out[t][:] = x[t][:] * rsqrt(mean(x[t]^2) + eps) * gamma: the residual add after the o-projection
// and the RMSNorm in front of the feed-forward block as one launch, one CTA per token; the norm's arithmetic is
// rms_norm_kernel's (thread order, shuffle tree, part[0..7] in order), so the bits are those of the two launches.
__global__ void __launch_bounds__(256) add_rms_norm_rows_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ gamma,
                                                                 float* __restrict__ out, float eps, uint32_t hidden) {
    __shared__ float part[8];
    float* row = x + (size_t)blockIdx.x * hidden;
    const float* add = y + (size_t)blockIdx.x * hidden;
    float* o = out + (size_t)blockIdx.x * hidden;
    float s = 0.f;
    for (uint32_t i = threadIdx.x; i < hidden; i += 256) {
        const float v = row[i] + add[i];
        row[i] = v;
        s = fmaf(v, v, s);
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += part[i];
    const float r = rsqrtf(tot / (float)hidden + eps);
    for (uint32_t i = threadIdx.x; i < hidden; i += 256) o[i] = row[i] * r * gamma[i];     // each thread re-reads what it stored
}

}  // namespace pf
}  // namespace runit

// ───────────────────────── launchers (used by the decoder's prefill) ─────────────────────────
namespace runit {

int32_t prefill_embed(runit_ctx* ctx, const float* emb, const int32_t* tokens, float* x, uint32_t T, uint32_t h) {
    pf::embed_rows_kernel<<<T, 256, 0, ctx->stream>>>(emb, tokens, x, h);
    return runit_after_launch(ctx, "prefill_embed");
}

int32_t prefill_norm_bf16(runit_ctx* ctx, const float* x, const float* gamma, void* y_bf16, float eps, uint32_t T, uint32_t h) {
    pf::rms_norm_bf16_kernel<<<T, 256, 0, ctx->stream>>>(x, gamma, (__nv_bfloat16*)y_bf16, eps, h);
    return runit_after_launch(ctx, "prefill_rms_norm_bf16");
}

int32_t prefill_rope_cache(runit_ctx* ctx, const float* q_in, float* q_out, const float* k, const float* v, void* kcache, void* vcache,
                           uint32_t hd, uint32_t heads, uint32_t kv_heads, uint32_t start_pos, float theta, uint32_t max_seq, uint32_t T,
                           uint32_t ld) {
    const uint32_t hmax = heads > kv_heads ? heads : kv_heads;
    pf::rope_cache_rows_kernel<<<dim3(T, hmax), hd / 2, 0, ctx->stream>>>(q_in, q_out, k, v, (__half*)kcache, (__half*)vcache, hd, heads,
                                                                           kv_heads, start_pos, theta, max_seq, ld);
    return runit_after_launch(ctx, "prefill_rope_cache");
}

int32_t prefill_attention(runit_ctx* ctx, const float* q, const void* kcache, const void* vcache, void* out_bf16, uint32_t T, uint32_t heads,
                          uint32_t kv_heads, uint32_t hd, uint32_t max_seq, uint32_t start_pos) {
    RUNIT_REQUIRE(ctx, hd == 128 || hd == 64, "prefill_attention: head_dim %u unsupported (64 or 128)", hd);
    RUNIT_REQUIRE(ctx, T > 0 && heads % kv_heads == 0 && (uint64_t)start_pos + T <= max_seq, "prefill_attention: bad shape");
    return attention_tc(ctx, q, kcache, vcache, out_bf16, T, heads, kv_heads, hd, max_seq, start_pos);
}

int32_t prefill_add_rms_norm(runit_ctx* ctx, float* x, const float* y, const float* gamma, float* out, float eps, uint32_t T, uint32_t h) {
    pf::add_rms_norm_rows_kernel<<<T, 256, 0, ctx->stream>>>(x, y, gamma, out, eps, h);
    return runit_after_launch(ctx, "prefill_add_rms_norm");
}

int32_t prefill_add_rows(runit_ctx* ctx, float* x, const float* y, size_t n) {
    const size_t n4 = n / 4;
    pf::add_rows_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, ctx->stream>>>(x, y, n4);
    return runit_after_launch(ctx, "prefill_add_rows");
}

}  // namespace runit

using namespace runit;

extern "C" {

// Dense feed-forward block of a prefill pass (prefill.rs:217-227: gate GEMM, up GEMM, silu_mul, down GEMM, residual add) on
// the tensor cores: out[t] = residual[t] + Wd . bf16(silu(Wg . xb[t]) * (Wu . xb[t])), xb = bf16(x) or, with gamma,
// bf16(RMSNorm(x) * gamma).  The two GEMM launches of moe_grouped.cu with one "expert" that owns the whole matrices.
size_t runit_ffn_q4k_bf16_scratch_bytes(uint32_t T, uint32_t h, uint32_t ff) {
    const size_t rows = ((size_t)T + 255) / 256 * 256 + 256, tiles = ((size_t)T + 255) / 256;
    auto up = [](size_t v) { return (v + 1023) & ~(size_t)1023; };
    return up(4 * (3 * tiles + 4)) + up(rows * h * 2) + up(rows * ff * 2) + up((size_t)T * h * 4);
}

int32_t runit_ffn_q4k_bf16(runit_ctx_t* ctx, const void* w_gate, const void* w_up, const void* w_down, const void* x, const void* gamma,
                           float eps, const void* residual, void* out, void* scratch, size_t scratch_bytes, uint32_t T, uint32_t h,
                           uint32_t ff) {
    if (!ctx) return RUNIT_ERR_BAD_ARG;
    RUNIT_REQUIRE(ctx, w_gate && w_up && w_down && x && out && scratch && T > 0, "ffn_q4k_bf16: null pointer or no tokens");
    RUNIT_REQUIRE(ctx, h % 256 == 0 && ff % 256 == 0 && h > 0 && ff > 0, "ffn_q4k_bf16: hidden %u and intermediate %u must be multiples of 256", h, ff);
    RUNIT_REQUIRE(ctx, runit_aligned(scratch, 1024) && runit_aligned(x, 16) && runit_aligned(out, 16) && (!residual || runit_aligned(residual, 16)) &&
                           runit_aligned(w_gate, 16) && runit_aligned(w_up, 16) && runit_aligned(w_down, 16),
                  "ffn_q4k_bf16: scratch must be 1024-byte aligned, tensors 16-byte aligned");
    if (runit_ffn_q4k_bf16_scratch_bytes(T, h, ff) > scratch_bytes)
        return runit_fail(ctx, RUNIT_ERR_BUFFER_SIZE, "ffn_q4k_bf16: scratch has %zu bytes, needs %zu", scratch_bytes,
                          runit_ffn_q4k_bf16_scratch_bytes(T, h, ff));
    const size_t rows = ((size_t)T + 255) / 256 * 256 + 256, tiles = ((size_t)T + 255) / 256;
    auto up = [](size_t v) { return (v + 1023) & ~(size_t)1023; };
    uint8_t* p = (uint8_t*)scratch;
    int32_t* tables = (int32_t*)p;              p += up(4 * (3 * tiles + 4));
    void* xb = p;                               p += up(rows * h * 2);
    void* act = p;                              p += up(rows * ff * 2);
    float* y = (float*)p;
    int32_t st;
    if ((st = dense_tiles_prepare(ctx, tables, T))) return st;
    if (gamma) {
        if ((st = prefill_norm_bf16(ctx, (const float*)x, (const float*)gamma, xb, eps, T, h))) return st;
    } else {
        const size_t n4 = (size_t)T * h / 4;
        pf::to_bf16_rows_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, ctx->stream>>>((const float*)x, (__nv_bfloat16*)xb, n4);
        if ((st = runit_after_launch(ctx, "ffn_to_bf16"))) return st;
    }
    if ((st = dense_gemm_q4k_bf16(ctx, "ffn_gate_up", w_gate, w_up, ff, h, xb, (uint32_t)rows, act, ff, T, tables))) return st;
    float* dst = residual ? y : (float*)out;
    if ((st = dense_gemm_q4k_bf16(ctx, "ffn_down", w_down, nullptr, h, ff, act, (uint32_t)rows, dst, h, T, tables))) return st;
    if (!residual) return RUNIT_OK;
    if (residual != out) RUNIT_CUDA_TRY(ctx, cudaMemcpyAsync(out, residual, (size_t)T * h * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    return prefill_add_rows(ctx, (float*)out, y, (size_t)T * h);
}

// Stand-alone entry of the attention kernel (tests, other callers): q f32 [T][heads*hd] already rotated, caches f16
// [kv_heads][max_seq][hd] holding positions 0 .. start_pos + T - 1, out bf16 [T][heads*hd].
int32_t runit_prefill_attention_f16kv(runit_ctx_t* ctx, const void* q, const void* kcache, const void* vcache, void* out_bf16, uint32_t T,
                                      uint32_t heads, uint32_t kv_heads, uint32_t head_dim, uint32_t max_seq, uint32_t start_pos) {
    if (!ctx) return RUNIT_ERR_BAD_ARG;
    RUNIT_REQUIRE(ctx, q && kcache && vcache && out_bf16 && kv_heads > 0, "prefill_attention_f16kv: null pointer");
    RUNIT_REQUIRE(ctx, runit_aligned(q, 16) && runit_aligned(kcache, 16) && runit_aligned(vcache, 16) && runit_aligned(out_bf16, 16),
                  "prefill_attention_f16kv: tensors must be 16-byte aligned");
    return prefill_attention(ctx, (const float*)q, kcache, vcache, out_bf16, T, heads, kv_heads, head_dim, max_seq, start_pos);
}

}  // extern "C"
