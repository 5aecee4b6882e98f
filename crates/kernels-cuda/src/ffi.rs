//! `extern "C"` declarations of every function in include/runit_cuda.h and include/runit_gguf.h.
//! Generated by gen_bindings.py; do not edit.
#![allow(non_camel_case_types)]
use std::ffi::c_void;
use std::os::raw::c_char;

#[repr(C)]
pub struct runit_ctx_t {
    _private: [u8; 0],
}
#[repr(C)]
pub struct runit_graph_t {
    _private: [u8; 0],
}
#[repr(C)]
pub struct runit_model_t {
    _private: [u8; 0],
}
#[repr(C)]
pub struct runit_gguf_t {
    _private: [u8; 0],
}

/// Field for field the C structs of the headers.
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_model_cfg {
    pub n_layers: i32, pub hidden: i32, pub n_heads: i32, pub n_kv_heads: i32, pub head_dim: i32, pub vocab: i32,
    pub n_experts: i32, pub top_k: i32, pub ff: i32, pub max_seq: i32, pub renorm: i32,
    pub eps: f32, pub theta: f32,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_model_weights {
    pub tok_emb: *const c_void, pub attn_norm: *const c_void, pub ffn_norm: *const c_void, pub out_norm: *const c_void,
    pub wq: *const c_void, pub wk: *const c_void, pub wv: *const c_void, pub wo: *const c_void, pub router: *const c_void,
    pub gate: *const c_void, pub up: *const c_void, pub down: *const c_void, pub lm_head: *const c_void,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_sampler_cfg {
    pub temperature: f32, pub top_k: i32, pub top_p: f32, pub repetition_penalty: f32, pub min_tokens: i32,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_gguf_tensor_info {
    pub name: *const c_char, pub dtype: u32, pub n_dims: u32, pub ne: [u64; 4],
    pub data_offset: u64, pub num_elements: u64, pub data_size: u64,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_layer_desc {
    pub heads: i32, pub dim: i32, pub rot_dim: i32, pub vdim: i32, pub kv_rank: i32, pub kv_from: i32,
    pub scale: f32, pub rot_base: f32,
    pub ff_kind: i32, pub ff_act: i32, pub ff: i32, pub n_experts: i32, pub top_k: i32, pub score: i32, pub renorm: i32, pub shared_ff: i32,
    pub norm1: *const c_void, pub norm2: *const c_void, pub w_q: *const c_void, pub kv_norm: *const c_void,
    pub w_ukv: *const c_void, pub w_o: *const c_void, pub ff_up: *const c_void, pub ff_down: *const c_void,
    pub router: *const c_void, pub shared_up: *const c_void, pub shared_down: *const c_void,
    pub mixer: i32, pub at_heads: i32, pub at_kv_heads: i32, pub at_dim: i32, pub at_vdim: i32, pub at_window: i32, pub at_unit_qk: i32,
    pub rt_heads: i32, pub rt_dim: i32, pub rt_vdim: i32, pub rt_rot_dims: i32,
    pub ss_heads: i32, pub ss_vdim: i32, pub ss_state: i32, pub ss_groups: i32, pub ss_taps: i32, pub ss_norm_groups: i32,
    pub at_scale: f32, pub at_out_scale: f32, pub rt_rot_base: f32, pub rt_out_scale: f32,
    pub at_slopes: *const c_void, pub rt_decay: *const c_void, pub ss_conv: *const c_void, pub ss_conv_b: *const c_void,
    pub ss_dt_bias: *const c_void, pub ss_a: *const c_void, pub ss_skip: *const c_void, pub ss_norm: *const c_void,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_latent_cfg {
    pub heads: u32, pub dim: u32, pub rot_dim: u32, pub vdim: u32, pub kv_rank: u32,
    pub scale: f32, pub eps: f32,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_heads_cfg {
    pub heads: u32, pub kv_heads: u32, pub dim: u32, pub vdim: u32, pub window: u32, pub cap: u32, pub unit_qk: u32,
    pub scale: f32, pub out_scale: f32, pub eps: f32,
    pub slopes: *const c_void, pub k_cache: *mut c_void, pub v_cache: *mut c_void,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_retention_cfg {
    pub heads: u32, pub dim: u32, pub vdim: u32, pub rot_dims: u32, pub out_scale: f32,
    pub freq: *const c_void, pub decay: *const c_void, pub state: *mut c_void,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_ssm_cfg {
    pub heads: u32, pub vdim: u32, pub state_dim: u32, pub groups: u32, pub taps: u32,
    pub conv: *const c_void, pub conv_b: *const c_void, pub dt_bias: *const c_void, pub a: *const c_void, pub skip: *const c_void,
    pub state: *mut c_void, pub ring: *mut c_void,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_linear_cfg {
    pub heads: u32, pub groups: u32, pub dk: u32, pub dv: u32, pub ldq: u32, pub ldk: u32, pub ldv: u32, pub ldo: u32,
    pub q: *const c_void, pub k: *const c_void, pub v: *const c_void, pub dt: *const c_void, pub log_decay: *const c_void,
    pub decay: *const c_void, pub skip: *const c_void, pub state: *mut c_void, pub out: *mut c_void,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_layered_cfg {
    pub n_layers: i32, pub width: i32, pub vocab: i32, pub max_seq: i32, pub exact: i32, pub post_norm: i32,
    pub eps: f32, pub embed_scale: f32, pub logit_cap: f32,
}
#[repr(C)]
#[derive(Clone, Copy, Debug)]
pub struct runit_layered_weights {
    pub embed: *const c_void, pub embed_norm: *const c_void, pub final_norm: *const c_void, pub head: *const c_void,
}

pub const RUNIT_OK: i32 = 0;
pub const RUNIT_ERR_NO_DEVICE: i32 = 1;
pub const RUNIT_ERR_BAD_ARG: i32 = 2;
pub const RUNIT_ERR_BUFFER_SIZE: i32 = 3;
pub const RUNIT_ERR_LAUNCH: i32 = 4;
pub const RUNIT_ERR_NCCL: i32 = 5;
pub const RUNIT_ERR_TIMEOUT: i32 = 6;
pub const RUNIT_ERR_UNSUPPORTED: i32 = 7;
pub const RUNIT_ERR_ALLOC: i32 = 8;
pub const RUNIT_BUF_DEVICE: i32 = 0;
pub const RUNIT_BUF_HOST_VISIBLE: i32 = 1;

extern "C" {
    pub fn runit_ctx_create(device: i32, out: *mut *mut runit_ctx_t) -> i32;
    pub fn runit_ctx_create_on_stream(device: i32, cuda_stream: *mut c_void, out: *mut *mut runit_ctx_t) -> i32;
    pub fn runit_ctx_destroy(ctx: *mut runit_ctx_t) -> i32;
    pub fn runit_ctx_stream(ctx: *mut runit_ctx_t) -> *mut c_void;
    pub fn runit_flush(ctx: *mut runit_ctx_t) -> i32;
    pub fn runit_last_error_string(ctx: *mut runit_ctx_t) -> *const c_char;
    pub fn runit_status_string(status: i32) -> *const c_char;
    pub fn runit_buf_alloc(ctx: *mut runit_ctx_t, bytes: usize, flags: i32, dptr: *mut *mut c_void) -> i32;
    pub fn runit_buf_free(ctx: *mut runit_ctx_t, dptr: *mut c_void) -> i32;
    pub fn runit_memcpy_h2d(ctx: *mut runit_ctx_t, dst_dev: *mut c_void, src_host: *const c_void, bytes: usize) -> i32;
    pub fn runit_memcpy_d2h(ctx: *mut runit_ctx_t, dst_host: *mut c_void, src_dev: *const c_void, bytes: usize) -> i32;
    pub fn runit_memset(ctx: *mut runit_ctx_t, dst_dev: *mut c_void, byte: i32, bytes: usize) -> i32;
    pub fn runit_launch_count(ctx: *mut runit_ctx_t) -> u64;
    pub fn runit_set_tuning(ctx: *mut runit_ctx_t, key: *const c_char, value: i32) -> i32;
    pub fn runit_graph_begin(ctx: *mut runit_ctx_t) -> i32;
    pub fn runit_graph_end(ctx: *mut runit_ctx_t, out: *mut *mut runit_graph_t) -> i32;
    pub fn runit_graph_launch(ctx: *mut runit_ctx_t, graph: *mut runit_graph_t) -> i32;
    pub fn runit_graph_destroy(ctx: *mut runit_ctx_t, graph: *mut runit_graph_t) -> i32;
    pub fn runit_graph_fused_launches(graph: *mut runit_graph_t) -> u32;
    pub fn runit_graph_kernel_launches(graph: *mut runit_graph_t) -> u32;
    pub fn runit_gemv_q8_0_f32in_f32out(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_add_f32_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_f16(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_add_f16(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_add_f32res_f16(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_f32in_f32out_mr(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_add_f32_f32in_mr(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_f32in_f32out_wide(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_add_f32_f32in_wide(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q8_0_f32in_wide(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_fused_qkv_q8_0_f32(a0: *mut runit_ctx_t, w_q: *const c_void, w_k: *const c_void, w_v: *const c_void, x_vec: *const c_void, out_q: *mut c_void, out_k: *mut c_void, out_v: *mut c_void, q_dim: u32, kv_dim: u32, k: u32) -> i32;
    pub fn runit_fused_qkv_bias_q8_0_f32(a0: *mut runit_ctx_t, w_q: *const c_void, w_k: *const c_void, w_v: *const c_void, x_vec: *const c_void, out_q: *mut c_void, out_k: *mut c_void, out_v: *mut c_void, bias_q: *const c_void, bias_k: *const c_void, bias_v: *const c_void, q_dim: u32, kv_dim: u32, k: u32) -> i32;
    pub fn runit_fused_ffn_q8_0_f32(a0: *mut runit_ctx_t, w_gate: *const c_void, w_up: *const c_void, x_vec: *const c_void, act_out: *mut c_void, ff_dim: u32, k: u32) -> i32;
    pub fn runit_gemv_q4_0_f32in_f32out(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4_0_add_f32_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4_0_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4_0_f16(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4_0_add_f16(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_fused_ffn_q4_0_f32(a0: *mut runit_ctx_t, w_gate: *const c_void, w_up: *const c_void, x_vec: *const c_void, act_out: *mut c_void, ff_dim: u32, k: u32) -> i32;
    pub fn runit_gemv_q4k_f32in_f32out(a0: *mut runit_ctx_t, weight_q4k: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4k_add_f32_f32in(a0: *mut runit_ctx_t, weight_q4k: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4k_f16(a0: *mut runit_ctx_t, weight_q4k: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4k_add_f16(a0: *mut runit_ctx_t, weight_q4k: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q4k_add_f32res_f16(a0: *mut runit_ctx_t, weight_q4k: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_dequant_q4k_f16(a0: *mut runit_ctx_t, input: *const c_void, output: *mut c_void, n_blocks: u32) -> i32;
    pub fn runit_gemv_q5_0_f32in_f32out(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q5_0_add_f32_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q5k_f32in_f32out(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q5k_add_f32_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q6k_f32in_f32out(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_q6k_add_f32_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_f16w_f32in(a0: *mut runit_ctx_t, weight: *const c_void, input: *const c_void, output: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_silu_mul_f16(a0: *mut runit_ctx_t, gate: *const c_void, up: *const c_void, out: *mut c_void, n: u32) -> i32;
    pub fn runit_silu_mul_f32(a0: *mut runit_ctx_t, gate: *const c_void, up: *const c_void, out: *mut c_void, n: u32) -> i32;
    pub fn runit_scale_accumulate_f16(a0: *mut runit_ctx_t, src: *const c_void, acc: *mut c_void, weight: f32, n: u32) -> i32;
    pub fn runit_add_f16_into_f32(a0: *mut runit_ctx_t, src: *const c_void, acc: *mut c_void, n: u32) -> i32;
    pub fn runit_fused_qkv_q4_0_f32(a0: *mut runit_ctx_t, w_q: *const c_void, w_k: *const c_void, w_v: *const c_void, x_vec: *const c_void, out_q: *mut c_void, out_k: *mut c_void, out_v: *mut c_void, q_dim: u32, kv_dim: u32, k: u32) -> i32;
    pub fn runit_fused_qkv_q4k_f32(a0: *mut runit_ctx_t, w_q: *const c_void, w_k: *const c_void, w_v: *const c_void, x_vec: *const c_void, out_q: *mut c_void, out_k: *mut c_void, out_v: *mut c_void, q_dim: u32, kv_dim: u32, k: u32) -> i32;
    pub fn runit_fused_ffn_q4k_f32(a0: *mut runit_ctx_t, w_gate: *const c_void, w_up: *const c_void, x_vec: *const c_void, act_out: *mut c_void, ff_dim: u32, k: u32) -> i32;
    pub fn runit_gemv_batched_f32(a0: *mut runit_ctx_t, fmt: i32, weight: *const c_void, input: *const c_void, output: *mut c_void, residual: *const c_void, m: u32, k: u32, batch: u32) -> i32;
    pub fn runit_gemv_batched_multi_f32(a0: *mut runit_ctx_t, fmt: i32, n_mats: u32, weights: *const *mut c_void, input: *const c_void, outputs: *const *mut c_void, rows: *const u32, k: u32, batch: u32) -> i32;
    pub fn runit_rms_norm_gemv_f32(a0: *mut runit_ctx_t, fmt: i32, weight: *const c_void, x: *const c_void, gamma: *const c_void, eps: f32, output: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_rms_norm_fused_qkv_f32(a0: *mut runit_ctx_t, fmt: i32, w_q: *const c_void, w_k: *const c_void, w_v: *const c_void, x: *const c_void, gamma: *const c_void, eps: f32, out_q: *mut c_void, out_k: *mut c_void, out_v: *mut c_void, q_dim: u32, kv_dim: u32, k: u32) -> i32;
    pub fn runit_gemv_argmax_f32(a0: *mut runit_ctx_t, fmt: i32, weight: *const c_void, x: *const c_void, gamma: *const c_void, eps: f32, logits: *mut c_void, result: *mut c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemv_argmax_allgather(a0: *mut runit_ctx_t, fmt: i32, w_local: *const c_void, x: *const c_void, logits_local: *mut c_void, pairs_all: *const *mut c_void, world: u32, rank: u32, rows_total: u32, k: u32) -> i32;
    pub fn runit_argmax_pairs(a0: *mut runit_ctx_t, pairs: *const c_void, n: u32, result: *mut c_void) -> i32;
    pub fn runit_peer_barrier_argmax(a0: *mut runit_ctx_t, signal_pads: *const *mut c_void, world: u32, rank: u32, epoch: u32, pairs: *const c_void, result: *mut c_void) -> i32;
    pub fn runit_fused_qkv_f32bias_q8_0_f32(a0: *mut runit_ctx_t, w_q: *const c_void, w_k: *const c_void, w_v: *const c_void, x_vec: *const c_void, out_q: *mut c_void, out_k: *mut c_void, out_v: *mut c_void, bias_q: *const c_void, bias_k: *const c_void, bias_v: *const c_void, q_dim: u32, kv_dim: u32, k: u32) -> i32;
    pub fn runit_gemv_allgather_f32(a0: *mut runit_ctx_t, fmt: i32, w_local: *const c_void, x: *const c_void, y_all: *const *mut c_void, world: u32, rank: u32, rows_total: u32, k: u32) -> i32;
    pub fn runit_moe_ep_prefill_scratch_bytes(T: u32, h: u32, ff: u32, E: u32, k: u32, world: u32) -> usize;
    pub fn runit_moe_layer_q4k_bf16_ep(a0: *mut runit_ctx_t, router_w: *const c_void, gate_local: *const c_void, up_local: *const c_void, down_local: *const c_void, x: *const c_void, residual: *const c_void, out: *mut c_void, idx_out: *mut c_void, w_out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, recv_rows_all: *const *mut c_void, recv_meta_all: *const *mut c_void, recv_counts_all: *const *mut c_void, return_rows_all: *const *mut c_void, signal_pads: *const *mut c_void, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32, world: u32, rank: u32, epoch: u32, placement: i32) -> i32;
    pub fn runit_peer_barrier(a0: *mut runit_ctx_t, signal_pads: *const *mut c_void, world: u32, rank: u32, epoch: u32) -> i32;
    pub fn runit_moe_router_f32(a0: *mut runit_ctx_t, router_w: *const c_void, x: *const c_void, logits: *mut c_void, E: u32, h: u32, T: u32) -> i32;
    pub fn runit_moe_route_topk(a0: *mut runit_ctx_t, logits: *const c_void, logits_f16: i32, E: u32, k: u32, renorm: i32, T: u32, out_idx: *mut c_void, out_w: *mut c_void) -> i32;
    pub fn runit_moe_route_scored(a0: *mut runit_ctx_t, logits: *const c_void, ld: u32, E: u32, k: u32, score: i32, renorm: i32, T: u32, out_idx: *mut c_void, out_w: *mut c_void) -> i32;
    pub fn runit_moe_scratch_bytes(T: u32, h: u32, ff: u32, E: u32, k: u32) -> usize;
    pub fn runit_moe_layer_q4k(a0: *mut runit_ctx_t, router_w: *const c_void, gate: *const c_void, up: *const c_void, down: *const c_void, x: *const c_void, residual: *const c_void, out: *mut c_void, idx_out: *mut c_void, w_out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> i32;
    pub fn runit_moe_layer_q4k_by_slot(a0: *mut runit_ctx_t, router_w: *const c_void, gate: *const c_void, up: *const c_void, down: *const c_void, x: *const c_void, residual: *const c_void, out: *mut c_void, idx_out: *mut c_void, w_out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> i32;
    pub fn runit_moe_experts_q4k(a0: *mut runit_ctx_t, gate: *const c_void, up: *const c_void, down: *const c_void, x_slots: *const c_void, slot_expert: *const c_void, y_slots: *mut c_void, act_scratch: *mut c_void, n_slots: u32, h: u32, ff: u32, n_experts: u32) -> i32;
    pub fn runit_moe_layer_q4k_ep(a0: *mut runit_ctx_t, router_w: *const c_void, gate_local: *const c_void, up_local: *const c_void, down_local: *const c_void, x: *const c_void, residual: *const c_void, out: *mut c_void, idx_out: *mut c_void, w_out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, partial_all: *const *mut c_void, signal_pads: *const *mut c_void, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32, world: u32, rank: u32, epoch: u32) -> i32;
    pub fn runit_moe_static_scratch_capacity() -> usize;
    pub fn runit_moe_layer_q4k_static(a0: *mut runit_ctx_t, router_w: *const c_void, gate: *const c_void, up: *const c_void, down: *const c_void, x: *const c_void, residual: *const c_void, out: *mut c_void, idx_out: *mut c_void, w_out: *mut c_void, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> i32;
    pub fn runit_moe_grouped_scratch_bytes(T: u32, h: u32, ff: u32, E: u32, k: u32) -> usize;
    pub fn runit_moe_layer_q4k_bf16(a0: *mut runit_ctx_t, router_w: *const c_void, gate: *const c_void, up: *const c_void, down: *const c_void, x: *const c_void, residual: *const c_void, out: *mut c_void, idx_out: *mut c_void, w_out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32, renorm: i32) -> i32;
    pub fn runit_moe_experts_grouped_q4k_bf16(a0: *mut runit_ctx_t, gate: *const c_void, up: *const c_void, down: *const c_void, x: *const c_void, idx: *const c_void, w: *const c_void, residual: *const c_void, out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, T: u32, h: u32, ff: u32, E: u32, k: u32) -> i32;
    pub fn runit_rms_norm_f32_f32(a0: *mut runit_ctx_t, x: *const c_void, y: *mut c_void, gamma: *const c_void, eps: f32, hidden: u32, num_rows: u32) -> i32;
    pub fn runit_rms_norm_f32_f32_f32g(a0: *mut runit_ctx_t, x: *const c_void, y: *mut c_void, gamma: *const c_void, eps: f32, hidden: u32, num_rows: u32) -> i32;
    pub fn runit_fused_rope_qk_f32(a0: *mut runit_ctx_t, q: *mut c_void, k: *mut c_void, head_dim: u32, q_heads: u32, kv_heads: u32, pos: u32, theta: f32) -> i32;
    pub fn runit_kv_copy_to_cache_f16(a0: *mut runit_ctx_t, src: *const c_void, dst: *mut c_void, pos: u32, max_seq: u32, head_dim: u32, num_kv_heads: u32) -> i32;
    pub fn runit_kv_copy_to_cache_f32(a0: *mut runit_ctx_t, src: *const c_void, dst: *mut c_void, pos: u32, max_seq: u32, head_dim: u32, num_kv_heads: u32) -> i32;
    pub fn runit_kv_copy_to_cache_f32_f16(a0: *mut runit_ctx_t, src: *const c_void, dst: *mut c_void, pos: u32, max_seq: u32, head_dim: u32, num_kv_heads: u32) -> i32;
    pub fn runit_decode_attention_f32(a0: *mut runit_ctx_t, q: *const c_void, k: *const c_void, v: *const c_void, out: *mut c_void, batch: u32, kv_len: u32, num_heads: u32, num_kv_heads: u32, head_dim: u32, kv_head_stride: u32) -> i32;
    pub fn runit_decode_attention_f16(a0: *mut runit_ctx_t, q: *const c_void, k: *const c_void, v: *const c_void, out: *mut c_void, batch: u32, kv_len: u32, num_heads: u32, num_kv_heads: u32, head_dim: u32, kv_head_stride: u32) -> i32;
    pub fn runit_decode_attention_f32q_f16kv(a0: *mut runit_ctx_t, q: *const c_void, k: *const c_void, v: *const c_void, out: *mut c_void, batch: u32, kv_len: u32, num_heads: u32, num_kv_heads: u32, head_dim: u32, kv_head_stride: u32) -> i32;
    pub fn runit_argmax_f16(a0: *mut runit_ctx_t, input: *const c_void, result: *mut c_void, n: u32) -> i32;
    pub fn runit_argmax_f32(a0: *mut runit_ctx_t, input: *const c_void, result: *mut c_void, n: u32) -> i32;
    pub fn runit_sample_f32(a0: *mut runit_ctx_t, logits: *const c_void, scores_scratch: *mut c_void, n: u32, cfg: *const runit_sampler_cfg, context: *const c_void, ctx_range: *const c_void, ctx_begin: u32, ctx_end: u32, eos_ids: *const c_void, n_eos: u32, rng_state: *mut c_void, result: *mut c_void) -> i32;
    pub fn runit_sampler_seed_state(seed: u64) -> u64;
    pub fn runit_model_create(ctx: *mut runit_ctx_t, cfg: *const runit_model_cfg, weights: *const runit_model_weights, out: *mut *mut runit_model_t) -> i32;
    pub fn runit_model_create_ep(ctx: *mut runit_ctx_t, cfg: *const runit_model_cfg, weights: *const runit_model_weights, world: u32, rank: u32, partial_all: *const *mut c_void, signal_pads: *const *mut c_void, out: *mut *mut runit_model_t) -> i32;
    pub fn runit_model_destroy(model: *mut runit_model_t) -> i32;
    pub fn runit_model_reset(model: *mut runit_model_t, token: i32, pos: i32) -> i32;
    pub fn runit_model_forward_greedy(model: *mut runit_model_t, token_id: i32, pos: i32, next_token: *mut i32) -> i32;
    pub fn runit_model_generate_greedy(model: *mut runit_model_t, prompt: *const i32, n_prompt: u32, n_gen: u32, start_pos: i32, skip_prompt_logits: i32, out_tokens: *mut i32) -> i32;
    pub fn runit_model_generate_sampled(model: *mut runit_model_t, prompt: *const i32, n_prompt: u32, n_gen: u32, start_pos: i32, cfg: *const runit_sampler_cfg, seed: u64, eos_ids: *const i32, n_eos: u32, out_tokens: *mut i32) -> i32;
    pub fn runit_model_prefill(model: *mut runit_model_t, tokens: *const i32, n: u32, next_token: *mut i32) -> i32;
    pub fn runit_prefill_attention_f16kv(a0: *mut runit_ctx_t, q: *const c_void, kcache: *const c_void, vcache: *const c_void, out_bf16: *mut c_void, T: u32, heads: u32, kv_heads: u32, head_dim: u32, max_seq: u32, start_pos: u32) -> i32;
    pub fn runit_ffn_q4k_bf16_scratch_bytes(T: u32, h: u32, ff: u32) -> usize;
    pub fn runit_ffn_q4k_bf16(a0: *mut runit_ctx_t, w_gate: *const c_void, w_up: *const c_void, w_down: *const c_void, x: *const c_void, gamma: *const c_void, eps: f32, residual: *const c_void, out: *mut c_void, scratch: *mut c_void, scratch_bytes: usize, T: u32, h: u32, ff: u32) -> i32;
    pub fn runit_model_forward(model: *mut runit_model_t, tokens: *const i32, n: u32, start_pos: u32, want: *const u32, n_want: u32, logits: *mut f32) -> i32;
    pub fn runit_gemv_bf16_f32(a0: *mut runit_ctx_t, weight: *const c_void, x: *const c_void, gain: *const c_void, eps: f32, y: *mut c_void, residual: *const c_void, m: u32, k: u32) -> i32;
    pub fn runit_gemm_bf16_rows(a0: *mut runit_ctx_t, weight: *const c_void, x: *const c_void, y: *mut c_void, ldy: u32, T: u32, m: u32, k: u32, exact: i32, epi: i32, pre: *const c_void, post: *const c_void) -> i32;
    pub fn runit_norm_gain_rows(a0: *mut runit_ctx_t, x: *const c_void, gain: *const c_void, eps: f32, y: *mut c_void, y_f32: i32, T: u32, width: u32) -> i32;
    pub fn runit_latent_query(a0: *mut runit_ctx_t, cfg: *const runit_latent_cfg, cache_f32: i32, qkv: *const c_void, ldq: u32, w_uk: *const c_void, kv_norm: *const c_void, freq: *const c_void, cache: *mut c_void, q_eff: *mut c_void, T: u32, start: u32) -> i32;
    pub fn runit_latent_attention(a0: *mut runit_ctx_t, cfg: *const runit_latent_cfg, cache_f32: i32, q_eff: *const c_void, cache: *const c_void, part_o: *mut c_void, part_ml: *mut c_void, nsplit: u32, T: u32, start: u32) -> i32;
    pub fn runit_latent_value(a0: *mut runit_ctx_t, cfg: *const runit_latent_cfg, part_o: *const c_void, part_ml: *const c_void, nsplit: u32, w_uv: *const c_void, out: *mut c_void, T: u32) -> i32;
    pub fn runit_latent_rows(a0: *mut runit_ctx_t, cfg: *const runit_latent_cfg, cache_f32: i32, qkv: *mut c_void, ldq: u32, kv_norm: *const c_void, freq: *const c_void, cache: *mut c_void, T: u32, start: u32) -> i32;
    pub fn runit_latent_prefill_attention(a0: *mut runit_ctx_t, cfg: *const runit_latent_cfg, q: *const c_void, ldq: u32, kv: *const c_void, ldkv: u32, cache: *const c_void, out: *mut c_void, ldo: u32, T: u32, start: u32) -> i32;
    pub fn runit_heads_step(a0: *mut runit_ctx_t, attn: *const runit_heads_cfg, ret: *const runit_retention_cfg, cache_f32: i32, proj: *const c_void, ao: *mut c_void, factor: *mut c_void, squares: *mut c_void, part: *mut c_void, tickets: *mut c_void, nsplit: u32, pos: *const c_void) -> i32;
    pub fn runit_heads_rows(a0: *mut runit_ctx_t, attn: *const runit_heads_cfg, ret: *const runit_retention_cfg, cache_f32: i32, proj: *mut c_void, ld: u32, T: u32, start: u32) -> i32;
    pub fn runit_head_attention_rows(a0: *mut runit_ctx_t, attn: *const runit_heads_cfg, cache_f32: i32, proj: *const c_void, ld: u32, out: *mut c_void, ldo: u32, T: u32, start: u32, part: *mut c_void, part_floats: usize, tickets: *mut c_void) -> i32;
    pub fn runit_ssm_step(a0: *mut runit_ctx_t, cfg: *const runit_ssm_cfg, proj: *const c_void, y: *mut c_void, squares: *mut c_void, pos: *const c_void) -> i32;
    pub fn runit_ssm_conv_rows(a0: *mut runit_ctx_t, cfg: *const runit_ssm_cfg, f32: i32, proj: *const c_void, ld: u32, xbc: *mut c_void, ldx: u32, dt: *mut c_void, T: u32, start: u32) -> i32;
    pub fn runit_linear_scratch_bytes(heads: u32, dk: u32, dv: u32, T: u32) -> usize;
    pub fn runit_linear_rows(a0: *mut runit_ctx_t, cfg: *const runit_linear_cfg, f32: i32, scratch: *mut c_void, T: u32, start: u32) -> i32;
    pub fn runit_gated_norm_rows(a0: *mut runit_ctx_t, f32: i32, a: *mut c_void, lda: u32, n: u32, group: u32, gate: *const c_void, ldg: u32, before: i32, weight: *const c_void, out_scale: f32, eps: f32, T: u32) -> i32;
    pub fn runit_add_norm_rows(a0: *mut runit_ctx_t, x: *mut c_void, y: *const c_void, gain: *const c_void, eps: f32, out_gain: *const c_void, out: *mut c_void, out_f32: i32, T: u32, width: u32) -> i32;
    pub fn runit_gemv_bf16_residual_f32(a0: *mut runit_ctx_t, weight: *const c_void, x: *const c_void, y: *const c_void, y_gain: *const c_void, gain: *const c_void, x_out: *mut c_void, out: *mut c_void, eps: f32, cap: f32, relu2: i32, m: u32, k: u32) -> i32;
    pub fn runit_gemv_bf16_groups_f32(a0: *mut runit_ctx_t, weight: *const c_void, x: *const c_void, factor: *const c_void, squares: *const c_void, squares_n: u32, out: *mut c_void, eps: f32, plain: u32, group: u32, m: u32, k: u32) -> i32;
    pub fn runit_model_create_layered(ctx: *mut runit_ctx_t, cfg: *const runit_layered_cfg, layers: *const runit_layer_desc, weights: *const runit_layered_weights, out: *mut *mut runit_model_t) -> i32;
    pub fn runit_model_residual(model: *mut runit_model_t) -> *mut c_void;
    pub fn runit_model_set_depth(model: *mut runit_model_t, n_layers: i32) -> i32;
    pub fn runit_model_logits(model: *mut runit_model_t) -> *mut c_void;
    pub fn runit_model_launches_per_token(model: *mut runit_model_t) -> u64;
    pub fn runit_fill_weights(a0: *mut runit_ctx_t, fmt: i32, dst: *mut c_void, n_blocks: u64, seed: u64, sigma: f32) -> i32;
    pub fn runit_fill_weights_q4k_zero_mean(a0: *mut runit_ctx_t, dst: *mut c_void, n_blocks: u64, seed: u64, sigma: f32) -> i32;
    pub fn runit_fill_normal_f32(a0: *mut runit_ctx_t, dst: *mut c_void, n: u64, seed: u64, sigma: f32) -> i32;
    pub fn runit_gguf_open(path: *const c_char, out: *mut *mut runit_gguf_t) -> i32;
    pub fn runit_gguf_open_memory(image: *const c_void, bytes: u64, out: *mut *mut runit_gguf_t) -> i32;
    pub fn runit_gguf_close(g: *mut runit_gguf_t);
    pub fn runit_gguf_last_error() -> *const c_char;
    pub fn runit_gguf_version(g: *const runit_gguf_t) -> u32;
    pub fn runit_gguf_alignment(g: *const runit_gguf_t) -> u64;
    pub fn runit_gguf_data_offset(g: *const runit_gguf_t) -> u64;
    pub fn runit_gguf_tensor_count(g: *const runit_gguf_t) -> u64;
    pub fn runit_gguf_metadata_count(g: *const runit_gguf_t) -> u64;
    pub fn runit_gguf_tensor_at(g: *const runit_gguf_t, index: u64, out: *mut runit_gguf_tensor_info) -> i32;
    pub fn runit_gguf_tensor_find(g: *const runit_gguf_t, name: *const c_char, out: *mut runit_gguf_tensor_info) -> i32;
    pub fn runit_gguf_dtype_block_size(dtype: u32) -> u64;
    pub fn runit_gguf_dtype_type_size(dtype: u32) -> u64;
    pub fn runit_gguf_dtype_tensor_data_size(dtype: u32, num_elements: u64) -> u64;
    pub fn runit_gguf_dtype_name(dtype: u32) -> *const c_char;
    pub fn runit_gguf_meta_key_at(g: *const runit_gguf_t, index: u64, key: *const *const char) -> i32;
    pub fn runit_gguf_meta_type(g: *const runit_gguf_t, key: *const c_char, r#type: *mut u32, elem_type: *mut u32, count: *mut u64) -> i32;
    pub fn runit_gguf_meta_u64(g: *const runit_gguf_t, key: *const c_char, out: *mut u64) -> i32;
    pub fn runit_gguf_meta_i64(g: *const runit_gguf_t, key: *const c_char, out: *mut i64) -> i32;
    pub fn runit_gguf_meta_f64(g: *const runit_gguf_t, key: *const c_char, out: *mut double) -> i32;
    pub fn runit_gguf_meta_bool(g: *const runit_gguf_t, key: *const c_char, out: *mut i32) -> i32;
    pub fn runit_gguf_meta_str(g: *const runit_gguf_t, key: *const c_char, out: *const *const char, len: *mut u64) -> i32;
    pub fn runit_gguf_meta_array_u64(g: *const runit_gguf_t, key: *const c_char, index: u64, out: *mut u64) -> i32;
    pub fn runit_gguf_meta_array_i64(g: *const runit_gguf_t, key: *const c_char, index: u64, out: *mut i64) -> i32;
    pub fn runit_gguf_meta_array_f64(g: *const runit_gguf_t, key: *const c_char, index: u64, out: *mut double) -> i32;
    pub fn runit_gguf_meta_array_str(g: *const runit_gguf_t, key: *const c_char, index: u64, out: *const *const char, len: *mut u64) -> i32;
    pub fn runit_gguf_read_tensor(g: *mut runit_gguf_t, name: *const c_char, host_dst: *mut c_void, capacity: u64) -> i32;
    pub fn runit_gguf_upload_tensor(ctx: *mut runit_ctx_t, g: *mut runit_gguf_t, name: *const c_char, device_dst: *mut c_void, capacity: u64) -> i32;
}
