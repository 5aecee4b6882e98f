//! The free functions of crates/kernels/src/dispatch.rs for the quantized decode path (same names, same argument
//! order), plus the operators that have no twin there, forwarding to librunit_cuda.so.  `ctx: &MetalContext` becomes
//! `&CudaContext`, `&metal::Buffer` becomes `&DeviceBuffer`, tables of peer pointers are slices of raw device pointers.
//! Generated by gen_bindings.py from include/runit_cuda.h (which cites the dispatch.rs line of every twin); do not edit.
#![allow(clippy::too_many_arguments)]
use std::ffi::c_void;

use crate::context::{CudaContext, DeviceBuffer};
use crate::error::Result;
use crate::ffi;

type B = DeviceBuffer;

pub fn gemv_q8_0_f32in_f32out(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_f32in_f32out(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q8_0_add_f32_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_add_f32_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q8_0_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q8_0_f16(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_f16(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q8_0_add_f16(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_add_f16(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q8_0_add_f32res_f16(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_add_f32res_f16(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q8_0_f32in_f32out_mr(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_f32in_f32out_mr(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q8_0_add_f32_f32in_mr(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_add_f32_f32in_mr(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q8_0_f32in_f32out_wide(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_f32in_f32out_wide(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q8_0_add_f32_f32in_wide(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_add_f32_f32in_wide(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q8_0_f32in_wide(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q8_0_f32in_wide(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn fused_qkv_q8_0_f32(ctx: &CudaContext, w_q: &B, w_k: &B, w_v: &B, x_vec: &B, out_q: &B, out_k: &B, out_v: &B, q_dim: u32, kv_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_qkv_q8_0_f32(ctx.raw, w_q.ptr as *const c_void, w_k.ptr as *const c_void, w_v.ptr as *const c_void, x_vec.ptr as *const c_void, out_q.ptr, out_k.ptr, out_v.ptr, q_dim, kv_dim, k) })
}
pub fn fused_qkv_bias_q8_0_f32(ctx: &CudaContext, w_q: &B, w_k: &B, w_v: &B, x_vec: &B, out_q: &B, out_k: &B, out_v: &B, bias_q: &B, bias_k: &B, bias_v: &B, q_dim: u32, kv_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_qkv_bias_q8_0_f32(ctx.raw, w_q.ptr as *const c_void, w_k.ptr as *const c_void, w_v.ptr as *const c_void, x_vec.ptr as *const c_void, out_q.ptr, out_k.ptr, out_v.ptr, bias_q.ptr as *const c_void, bias_k.ptr as *const c_void, bias_v.ptr as *const c_void, q_dim, kv_dim, k) })
}
pub fn fused_ffn_q8_0_f32(ctx: &CudaContext, w_gate: &B, w_up: &B, x_vec: &B, act_out: &B, ff_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_ffn_q8_0_f32(ctx.raw, w_gate.ptr as *const c_void, w_up.ptr as *const c_void, x_vec.ptr as *const c_void, act_out.ptr, ff_dim, k) })
}
pub fn gemv_q4_0_f32in_f32out(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4_0_f32in_f32out(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q4_0_add_f32_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4_0_add_f32_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q4_0_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4_0_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q4_0_f16(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4_0_f16(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q4_0_add_f16(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4_0_add_f16(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn fused_ffn_q4_0_f32(ctx: &CudaContext, w_gate: &B, w_up: &B, x_vec: &B, act_out: &B, ff_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_ffn_q4_0_f32(ctx.raw, w_gate.ptr as *const c_void, w_up.ptr as *const c_void, x_vec.ptr as *const c_void, act_out.ptr, ff_dim, k) })
}
pub fn gemv_q4k_f32in_f32out(ctx: &CudaContext, weight_q4k: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4k_f32in_f32out(ctx.raw, weight_q4k.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q4k_add_f32_f32in(ctx: &CudaContext, weight_q4k: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4k_add_f32_f32in(ctx.raw, weight_q4k.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q4k_f16(ctx: &CudaContext, weight_q4k: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4k_f16(ctx.raw, weight_q4k.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q4k_add_f16(ctx: &CudaContext, weight_q4k: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4k_add_f16(ctx.raw, weight_q4k.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q4k_add_f32res_f16(ctx: &CudaContext, weight_q4k: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q4k_add_f32res_f16(ctx.raw, weight_q4k.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn dequant_q4k_f16(ctx: &CudaContext, input: &B, output: &B, n_blocks: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_dequant_q4k_f16(ctx.raw, input.ptr as *const c_void, output.ptr, n_blocks) })
}
pub fn gemv_q5_0_f32in_f32out(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q5_0_f32in_f32out(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q5_0_add_f32_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q5_0_add_f32_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q5k_f32in_f32out(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q5k_f32in_f32out(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q5k_add_f32_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q5k_add_f32_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_q6k_f32in_f32out(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q6k_f32in_f32out(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn gemv_q6k_add_f32_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_q6k_add_f32_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemv_f16w_f32in(ctx: &CudaContext, weight: &B, input: &B, output: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_f16w_f32in(ctx.raw, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, m, k) })
}
pub fn silu_mul_f16(ctx: &CudaContext, gate: &B, up: &B, out: &B, n: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_silu_mul_f16(ctx.raw, gate.ptr as *const c_void, up.ptr as *const c_void, out.ptr, n) })
}
pub fn silu_mul_f32(ctx: &CudaContext, gate: &B, up: &B, out: &B, n: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_silu_mul_f32(ctx.raw, gate.ptr as *const c_void, up.ptr as *const c_void, out.ptr, n) })
}
pub fn scale_accumulate_f16(ctx: &CudaContext, src: &B, acc: &B, weight: f32, n: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_scale_accumulate_f16(ctx.raw, src.ptr as *const c_void, acc.ptr, weight, n) })
}
pub fn add_f16_into_f32(ctx: &CudaContext, src: &B, acc: &B, n: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_add_f16_into_f32(ctx.raw, src.ptr as *const c_void, acc.ptr, n) })
}
pub fn fused_qkv_q4_0_f32(ctx: &CudaContext, w_q: &B, w_k: &B, w_v: &B, x_vec: &B, out_q: &B, out_k: &B, out_v: &B, q_dim: u32, kv_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_qkv_q4_0_f32(ctx.raw, w_q.ptr as *const c_void, w_k.ptr as *const c_void, w_v.ptr as *const c_void, x_vec.ptr as *const c_void, out_q.ptr, out_k.ptr, out_v.ptr, q_dim, kv_dim, k) })
}
pub fn fused_qkv_q4k_f32(ctx: &CudaContext, w_q: &B, w_k: &B, w_v: &B, x_vec: &B, out_q: &B, out_k: &B, out_v: &B, q_dim: u32, kv_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_qkv_q4k_f32(ctx.raw, w_q.ptr as *const c_void, w_k.ptr as *const c_void, w_v.ptr as *const c_void, x_vec.ptr as *const c_void, out_q.ptr, out_k.ptr, out_v.ptr, q_dim, kv_dim, k) })
}
pub fn fused_ffn_q4k_f32(ctx: &CudaContext, w_gate: &B, w_up: &B, x_vec: &B, act_out: &B, ff_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_ffn_q4k_f32(ctx.raw, w_gate.ptr as *const c_void, w_up.ptr as *const c_void, x_vec.ptr as *const c_void, act_out.ptr, ff_dim, k) })
}
pub fn gemv_batched_f32(ctx: &CudaContext, fmt: i32, weight: &B, input: &B, output: &B, residual: &B, m: u32, k: u32, batch: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_batched_f32(ctx.raw, fmt, weight.ptr as *const c_void, input.ptr as *const c_void, output.ptr, residual.ptr as *const c_void, m, k, batch) })
}
pub fn rms_norm_gemv_f32(ctx: &CudaContext, fmt: i32, weight: &B, x: &B, gamma: &B, eps: f32, output: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_rms_norm_gemv_f32(ctx.raw, fmt, weight.ptr as *const c_void, x.ptr as *const c_void, gamma.ptr as *const c_void, eps, output.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn rms_norm_fused_qkv_f32(ctx: &CudaContext, fmt: i32, w_q: &B, w_k: &B, w_v: &B, x: &B, gamma: &B, eps: f32, out_q: &B, out_k: &B, out_v: &B, q_dim: u32, kv_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_rms_norm_fused_qkv_f32(ctx.raw, fmt, w_q.ptr as *const c_void, w_k.ptr as *const c_void, w_v.ptr as *const c_void, x.ptr as *const c_void, gamma.ptr as *const c_void, eps, out_q.ptr, out_k.ptr, out_v.ptr, q_dim, kv_dim, k) })
}
pub fn gemv_argmax_f32(ctx: &CudaContext, fmt: i32, weight: &B, x: &B, gamma: &B, eps: f32, logits: &B, result: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_argmax_f32(ctx.raw, fmt, weight.ptr as *const c_void, x.ptr as *const c_void, gamma.ptr as *const c_void, eps, logits.ptr, result.ptr, m, k) })
}
pub fn gemv_argmax_allgather(ctx: &CudaContext, fmt: i32, w_local: &B, x: &B, logits_local: &B, pairs_all: &[*mut c_void], world: u32, rank: u32, rows_total: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_argmax_allgather(ctx.raw, fmt, w_local.ptr as *const c_void, x.ptr as *const c_void, logits_local.ptr, pairs_all.as_ptr(), world, rank, rows_total, k) })
}
pub fn argmax_pairs(ctx: &CudaContext, pairs: &B, n: u32, result: &B) -> Result<()> {
    ctx.check(unsafe { ffi::runit_argmax_pairs(ctx.raw, pairs.ptr as *const c_void, n, result.ptr) })
}
pub fn peer_barrier_argmax(ctx: &CudaContext, signal_pads: &[*mut c_void], world: u32, rank: u32, epoch: u32, pairs: &B, result: &B) -> Result<()> {
    ctx.check(unsafe { ffi::runit_peer_barrier_argmax(ctx.raw, signal_pads.as_ptr(), world, rank, epoch, pairs.ptr as *const c_void, result.ptr) })
}
pub fn fused_qkv_f32bias_q8_0_f32(ctx: &CudaContext, w_q: &B, w_k: &B, w_v: &B, x_vec: &B, out_q: &B, out_k: &B, out_v: &B, bias_q: &B, bias_k: &B, bias_v: &B, q_dim: u32, kv_dim: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_qkv_f32bias_q8_0_f32(ctx.raw, w_q.ptr as *const c_void, w_k.ptr as *const c_void, w_v.ptr as *const c_void, x_vec.ptr as *const c_void, out_q.ptr, out_k.ptr, out_v.ptr, bias_q.ptr as *const c_void, bias_k.ptr as *const c_void, bias_v.ptr as *const c_void, q_dim, kv_dim, k) })
}
pub fn gemv_allgather_f32(ctx: &CudaContext, fmt: i32, w_local: &B, x: &B, y_all: &[*mut c_void], world: u32, rank: u32, rows_total: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_allgather_f32(ctx.raw, fmt, w_local.ptr as *const c_void, x.ptr as *const c_void, y_all.as_ptr(), world, rank, rows_total, k) })
}
pub fn moe_layer_q4k_bf16_ep(ctx: &CudaContext, router_w: &B, gate_local: &B, up_local: &B, down_local: &B, x: &B, residual: &B, out: &B, idx_out: &B, w_out: &B, scratch: &B, scratch_bytes: usize, recv_rows_all: &[*mut c_void], recv_meta_all: &[*mut c_void], recv_counts_all: &[*mut c_void], return_rows_all: &[*mut c_void], signal_pads: &[*mut c_void], T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32, world: u32, rank: u32, epoch: u32, placement: i32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_layer_q4k_bf16_ep(ctx.raw, router_w.ptr as *const c_void, gate_local.ptr as *const c_void, up_local.ptr as *const c_void, down_local.ptr as *const c_void, x.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, idx_out.ptr, w_out.ptr, scratch.ptr, scratch_bytes, recv_rows_all.as_ptr(), recv_meta_all.as_ptr(), recv_counts_all.as_ptr(), return_rows_all.as_ptr(), signal_pads.as_ptr(), T, h, ff, E, k, renorm, world, rank, epoch, placement) })
}
pub fn peer_barrier(ctx: &CudaContext, signal_pads: &[*mut c_void], world: u32, rank: u32, epoch: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_peer_barrier(ctx.raw, signal_pads.as_ptr(), world, rank, epoch) })
}
pub fn moe_router_f32(ctx: &CudaContext, router_w: &B, x: &B, logits: &B, E: u32, h: u32, T: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_router_f32(ctx.raw, router_w.ptr as *const c_void, x.ptr as *const c_void, logits.ptr, E, h, T) })
}
pub fn moe_route_topk(ctx: &CudaContext, logits: &B, logits_f16: i32, E: u32, k: u32, renorm: i32, T: u32, out_idx: &B, out_w: &B) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_route_topk(ctx.raw, logits.ptr as *const c_void, logits_f16, E, k, renorm, T, out_idx.ptr, out_w.ptr) })
}
pub fn moe_route_scored(ctx: &CudaContext, logits: &B, ld: u32, E: u32, k: u32, score: i32, renorm: i32, T: u32, out_idx: &B, out_w: &B) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_route_scored(ctx.raw, logits.ptr as *const c_void, ld, E, k, score, renorm, T, out_idx.ptr, out_w.ptr) })
}
pub fn moe_layer_q4k(ctx: &CudaContext, router_w: &B, gate: &B, up: &B, down: &B, x: &B, residual: &B, out: &B, idx_out: &B, w_out: &B, scratch: &B, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_layer_q4k(ctx.raw, router_w.ptr as *const c_void, gate.ptr as *const c_void, up.ptr as *const c_void, down.ptr as *const c_void, x.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, idx_out.ptr, w_out.ptr, scratch.ptr, scratch_bytes, T, h, ff, E, k, renorm) })
}
pub fn moe_layer_q4k_by_slot(ctx: &CudaContext, router_w: &B, gate: &B, up: &B, down: &B, x: &B, residual: &B, out: &B, idx_out: &B, w_out: &B, scratch: &B, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_layer_q4k_by_slot(ctx.raw, router_w.ptr as *const c_void, gate.ptr as *const c_void, up.ptr as *const c_void, down.ptr as *const c_void, x.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, idx_out.ptr, w_out.ptr, scratch.ptr, scratch_bytes, T, h, ff, E, k, renorm) })
}
pub fn moe_experts_q4k(ctx: &CudaContext, gate: &B, up: &B, down: &B, x_slots: &B, slot_expert: &B, y_slots: &B, act_scratch: &B, n_slots: u32, h: u32, ff: u32, n_experts: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_experts_q4k(ctx.raw, gate.ptr as *const c_void, up.ptr as *const c_void, down.ptr as *const c_void, x_slots.ptr as *const c_void, slot_expert.ptr as *const c_void, y_slots.ptr, act_scratch.ptr, n_slots, h, ff, n_experts) })
}
pub fn moe_layer_q4k_ep(ctx: &CudaContext, router_w: &B, gate_local: &B, up_local: &B, down_local: &B, x: &B, residual: &B, out: &B, idx_out: &B, w_out: &B, scratch: &B, scratch_bytes: usize, partial_all: &[*mut c_void], signal_pads: &[*mut c_void], T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32, world: u32, rank: u32, epoch: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_layer_q4k_ep(ctx.raw, router_w.ptr as *const c_void, gate_local.ptr as *const c_void, up_local.ptr as *const c_void, down_local.ptr as *const c_void, x.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, idx_out.ptr, w_out.ptr, scratch.ptr, scratch_bytes, partial_all.as_ptr(), signal_pads.as_ptr(), T, h, ff, E, k, renorm, world, rank, epoch) })
}
pub fn moe_layer_q4k_static(ctx: &CudaContext, router_w: &B, gate: &B, up: &B, down: &B, x: &B, residual: &B, out: &B, idx_out: &B, w_out: &B, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_layer_q4k_static(ctx.raw, router_w.ptr as *const c_void, gate.ptr as *const c_void, up.ptr as *const c_void, down.ptr as *const c_void, x.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, idx_out.ptr, w_out.ptr, T, h, ff, E, k, renorm) })
}
pub fn moe_layer_q4k_bf16(ctx: &CudaContext, router_w: &B, gate: &B, up: &B, down: &B, x: &B, residual: &B, out: &B, idx_out: &B, w_out: &B, scratch: &B, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_layer_q4k_bf16(ctx.raw, router_w.ptr as *const c_void, gate.ptr as *const c_void, up.ptr as *const c_void, down.ptr as *const c_void, x.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, idx_out.ptr, w_out.ptr, scratch.ptr, scratch_bytes, T, h, ff, E, k, renorm) })
}
pub fn moe_experts_grouped_q4k_bf16(ctx: &CudaContext, gate: &B, up: &B, down: &B, x: &B, idx: &B, w: &B, residual: &B, out: &B, scratch: &B, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_moe_experts_grouped_q4k_bf16(ctx.raw, gate.ptr as *const c_void, up.ptr as *const c_void, down.ptr as *const c_void, x.ptr as *const c_void, idx.ptr as *const c_void, w.ptr as *const c_void, residual.ptr as *const c_void, out.ptr, scratch.ptr, scratch_bytes, T, h, ff, E, k) })
}
pub fn rms_norm_f32_f32(ctx: &CudaContext, x: &B, y: &B, gamma: &B, eps: f32, hidden: u32, num_rows: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_rms_norm_f32_f32(ctx.raw, x.ptr as *const c_void, y.ptr, gamma.ptr as *const c_void, eps, hidden, num_rows) })
}
pub fn rms_norm_f32_f32_f32g(ctx: &CudaContext, x: &B, y: &B, gamma: &B, eps: f32, hidden: u32, num_rows: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_rms_norm_f32_f32_f32g(ctx.raw, x.ptr as *const c_void, y.ptr, gamma.ptr as *const c_void, eps, hidden, num_rows) })
}
pub fn fused_rope_qk_f32(ctx: &CudaContext, q: &B, k: &B, head_dim: u32, q_heads: u32, kv_heads: u32, pos: u32, theta: f32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fused_rope_qk_f32(ctx.raw, q.ptr, k.ptr, head_dim, q_heads, kv_heads, pos, theta) })
}
pub fn kv_copy_to_cache_f16(ctx: &CudaContext, src: &B, dst: &B, pos: u32, max_seq: u32, head_dim: u32, num_kv_heads: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_kv_copy_to_cache_f16(ctx.raw, src.ptr as *const c_void, dst.ptr, pos, max_seq, head_dim, num_kv_heads) })
}
pub fn kv_copy_to_cache_f32(ctx: &CudaContext, src: &B, dst: &B, pos: u32, max_seq: u32, head_dim: u32, num_kv_heads: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_kv_copy_to_cache_f32(ctx.raw, src.ptr as *const c_void, dst.ptr, pos, max_seq, head_dim, num_kv_heads) })
}
pub fn kv_copy_to_cache_f32_f16(ctx: &CudaContext, src: &B, dst: &B, pos: u32, max_seq: u32, head_dim: u32, num_kv_heads: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_kv_copy_to_cache_f32_f16(ctx.raw, src.ptr as *const c_void, dst.ptr, pos, max_seq, head_dim, num_kv_heads) })
}
pub fn decode_attention_f32(ctx: &CudaContext, q: &B, k: &B, v: &B, out: &B, batch: u32, kv_len: u32, num_heads: u32, num_kv_heads: u32, head_dim: u32, kv_head_stride: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_decode_attention_f32(ctx.raw, q.ptr as *const c_void, k.ptr as *const c_void, v.ptr as *const c_void, out.ptr, batch, kv_len, num_heads, num_kv_heads, head_dim, kv_head_stride) })
}
pub fn decode_attention_f16(ctx: &CudaContext, q: &B, k: &B, v: &B, out: &B, batch: u32, kv_len: u32, num_heads: u32, num_kv_heads: u32, head_dim: u32, kv_head_stride: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_decode_attention_f16(ctx.raw, q.ptr as *const c_void, k.ptr as *const c_void, v.ptr as *const c_void, out.ptr, batch, kv_len, num_heads, num_kv_heads, head_dim, kv_head_stride) })
}
pub fn decode_attention_f32q_f16kv(ctx: &CudaContext, q: &B, k: &B, v: &B, out: &B, batch: u32, kv_len: u32, num_heads: u32, num_kv_heads: u32, head_dim: u32, kv_head_stride: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_decode_attention_f32q_f16kv(ctx.raw, q.ptr as *const c_void, k.ptr as *const c_void, v.ptr as *const c_void, out.ptr, batch, kv_len, num_heads, num_kv_heads, head_dim, kv_head_stride) })
}
pub fn argmax_f16(ctx: &CudaContext, input: &B, result: &B, n: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_argmax_f16(ctx.raw, input.ptr as *const c_void, result.ptr, n) })
}
pub fn argmax_f32(ctx: &CudaContext, input: &B, result: &B, n: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_argmax_f32(ctx.raw, input.ptr as *const c_void, result.ptr, n) })
}
pub fn prefill_attention_f16kv(ctx: &CudaContext, q: &B, kcache: &B, vcache: &B, out_bf16: &B, T: u32, heads: u32, kv_heads: u32, head_dim: u32, max_seq: u32, start_pos: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_prefill_attention_f16kv(ctx.raw, q.ptr as *const c_void, kcache.ptr as *const c_void, vcache.ptr as *const c_void, out_bf16.ptr, T, heads, kv_heads, head_dim, max_seq, start_pos) })
}
pub fn ffn_q4k_bf16(ctx: &CudaContext, w_gate: &B, w_up: &B, w_down: &B, x: &B, gamma: &B, eps: f32, residual: &B, out: &B, scratch: &B, scratch_bytes: usize, T: u32, h: u32, ff: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_ffn_q4k_bf16(ctx.raw, w_gate.ptr as *const c_void, w_up.ptr as *const c_void, w_down.ptr as *const c_void, x.ptr as *const c_void, gamma.ptr as *const c_void, eps, residual.ptr as *const c_void, out.ptr, scratch.ptr, scratch_bytes, T, h, ff) })
}
pub fn gemv_bf16_f32(ctx: &CudaContext, weight: &B, x: &B, gain: &B, eps: f32, y: &B, residual: &B, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_bf16_f32(ctx.raw, weight.ptr as *const c_void, x.ptr as *const c_void, gain.ptr as *const c_void, eps, y.ptr, residual.ptr as *const c_void, m, k) })
}
pub fn gemm_bf16_rows(ctx: &CudaContext, weight: &B, x: &B, y: &B, ldy: u32, T: u32, m: u32, k: u32, exact: i32, epi: i32, pre: &B, post: &B) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemm_bf16_rows(ctx.raw, weight.ptr as *const c_void, x.ptr as *const c_void, y.ptr, ldy, T, m, k, exact, epi, pre.ptr as *const c_void, post.ptr as *const c_void) })
}
pub fn norm_gain_rows(ctx: &CudaContext, x: &B, gain: &B, eps: f32, y: &B, y_f32: i32, T: u32, width: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_norm_gain_rows(ctx.raw, x.ptr as *const c_void, gain.ptr as *const c_void, eps, y.ptr, y_f32, T, width) })
}
pub fn gated_norm_rows(ctx: &CudaContext, f32: i32, a: &B, lda: u32, n: u32, group: u32, gate: &B, ldg: u32, before: i32, weight: &B, out_scale: f32, eps: f32, T: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gated_norm_rows(ctx.raw, f32, a.ptr, lda, n, group, gate.ptr as *const c_void, ldg, before, weight.ptr as *const c_void, out_scale, eps, T) })
}
pub fn add_norm_rows(ctx: &CudaContext, x: &B, y: &B, gain: &B, eps: f32, out_gain: &B, out: &B, out_f32: i32, T: u32, width: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_add_norm_rows(ctx.raw, x.ptr, y.ptr as *const c_void, gain.ptr as *const c_void, eps, out_gain.ptr as *const c_void, out.ptr, out_f32, T, width) })
}
pub fn gemv_bf16_residual_f32(ctx: &CudaContext, weight: &B, x: &B, y: &B, y_gain: &B, gain: &B, x_out: &B, out: &B, eps: f32, cap: f32, relu2: i32, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_bf16_residual_f32(ctx.raw, weight.ptr as *const c_void, x.ptr as *const c_void, y.ptr as *const c_void, y_gain.ptr as *const c_void, gain.ptr as *const c_void, x_out.ptr, out.ptr, eps, cap, relu2, m, k) })
}
pub fn gemv_bf16_groups_f32(ctx: &CudaContext, weight: &B, x: &B, factor: &B, squares: &B, squares_n: u32, out: &B, eps: f32, plain: u32, group: u32, m: u32, k: u32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_gemv_bf16_groups_f32(ctx.raw, weight.ptr as *const c_void, x.ptr as *const c_void, factor.ptr as *const c_void, squares.ptr as *const c_void, squares_n, out.ptr, eps, plain, group, m, k) })
}
pub fn fill_weights(ctx: &CudaContext, fmt: i32, dst: &B, n_blocks: u64, seed: u64, sigma: f32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fill_weights(ctx.raw, fmt, dst.ptr, n_blocks, seed, sigma) })
}
pub fn fill_weights_q4k_zero_mean(ctx: &CudaContext, dst: &B, n_blocks: u64, seed: u64, sigma: f32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fill_weights_q4k_zero_mean(ctx.raw, dst.ptr, n_blocks, seed, sigma) })
}
pub fn fill_normal_f32(ctx: &CudaContext, dst: &B, n: u64, seed: u64, sigma: f32) -> Result<()> {
    ctx.check(unsafe { ffi::runit_fill_normal_f32(ctx.raw, dst.ptr, n, seed, sigma) })
}

/// Launch-shape variants the engine selects by row count (`use_mr = m >= 128`, crates/engine/src/forward.rs:134,193)
/// are the same kernel here; the names exist so that WeightBuf compiles unchanged.
