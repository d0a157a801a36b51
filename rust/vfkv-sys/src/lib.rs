//! Raw bindings to libvfkv.so (the C ABI of include/vfkv.h and include/vfkv_next.h):
//! VulkanForge's KV-cache hot path on NVIDIA B200 -- KV append, FP8 -> F16 cache read, split-K GQA
//! decode attention -- as a drop-in for the Vulkan dispatches of `src/backend/vulkan`.
//!
//! Generated by gen_bindings.py from the headers; one declaration per exported function, same
//! names, same argument order.  NOT COMPILED in the repository this file lives in: its build image
//! has no Rust toolchain.  A test there parses the headers and this file and fails when a function
//! is missing here or its argument count differs.
//!
//! Link with `cargo:rustc-link-lib=dylib=vfkv` (build.rs) and the directory that holds libvfkv.so.
#![allow(non_camel_case_types)]

use std::os::raw::{c_char, c_void};

/// vfkv_status
pub const VFKV_OK: i32 = 0;
pub const VFKV_ERR_INVALID: i32 = 1;
pub const VFKV_ERR_OVERFLOW: i32 = 2;
pub const VFKV_ERR_OOM: i32 = 3;
pub const VFKV_ERR_CUDA: i32 = 4;
pub const VFKV_ERR_UNSUPPORTED: i32 = 5;
pub const VFKV_ERR_TIMEOUT: i32 = 6;
pub const VFKV_ERR_PRECISION: i32 = 7;
/// vfkv_dtype: the values of `KvDtype` (src/backend/vulkan/kv_cache.rs:42-74)
pub const VFKV_F32: u32 = 0;
pub const VFKV_F16: u32 = 1;
pub const VFKV_F8: u32 = 2;
/// vfkv_scale_mode
pub const VFKV_SCALE_NONE: u32 = 0;
pub const VFKV_SCALE_PER_TOKEN_HEAD: u32 = 1;
/// vfkv_prof_label: the ShaderProfiler labels of this path
pub const VFKV_PROF_KV_STORE: u32 = 0;
pub const VFKV_PROF_FP8_TO_F16: u32 = 1;
pub const VFKV_PROF_FA_SPLIT: u32 = 2;
pub const VFKV_PROF_FA_REDUCE: u32 = 3;

#[repr(C)] pub struct vfkv_ctx { _private: [u8; 0] }
#[repr(C)] pub struct vfkv_cache { _private: [u8; 0] }
#[repr(C)] pub struct vfkv_workspace { _private: [u8; 0] }
#[repr(C)] pub struct vfkv_exchange { _private: [u8; 0] }

/// KvCacheConfig (kv_cache.rs:153-176) plus n_slots and scale_mode.
#[repr(C)]
pub struct vfkv_cache_config {
    pub n_layers: u32,
    pub n_kv_heads: u32,
    pub head_dim: u32,
    pub max_seq_len: u32,
    pub dtype: u32,
    pub per_layer_head_dim: *const u32,
    pub per_layer_n_kv_heads: *const u32,
    pub n_slots: u32,
    pub scale_mode: u32,
}

#[repr(C)]
pub struct vfkv_rope_params {
    pub n_dims: u32,
    pub freq_base: f32,
    pub freq_scale: f32,
}

extern "C" {
    pub fn vfkv_ctx_create(device_ordinal: i32, out: *mut *mut vfkv_ctx) -> i32;
    pub fn vfkv_ctx_destroy(ctx: *mut vfkv_ctx) -> i32;
    pub fn vfkv_last_error(ctx: *const vfkv_ctx) -> *const c_char;
    pub fn vfkv_status_string(status: i32) -> *const c_char;
    pub fn vfkv_abi_version() -> u32;
    pub fn vfkv_ctx_poll(ctx: *mut vfkv_ctx, stream: *mut c_void) -> i32;
    pub fn vfkv_cache_create(ctx: *mut vfkv_ctx, cfg: *const vfkv_cache_config, out: *mut *mut vfkv_cache) -> i32;
    pub fn vfkv_cache_destroy(cache: *mut vfkv_cache) -> i32;
    pub fn vfkv_cache_zero_fill(cache: *mut vfkv_cache, stream: *mut c_void) -> i32;
    pub fn vfkv_cache_zero_layer(cache: *mut vfkv_cache, layer: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_cache_reset(cache: *mut vfkv_cache, slot: u32) -> i32;
    pub fn vfkv_cache_seq_len(cache: *const vfkv_cache, slot: u32, out: *mut u32) -> i32;
    pub fn vfkv_cache_set_seq_len(cache: *mut vfkv_cache, slot: u32, seq_len: u32) -> i32;
    pub fn vfkv_cache_head_dim_for(cache: *const vfkv_cache, layer: u32) -> u32;
    pub fn vfkv_cache_kv_heads_for(cache: *const vfkv_cache, layer: u32) -> u32;
    pub fn vfkv_cache_row_bytes(cache: *const vfkv_cache, layer: u32) -> u64;
    pub fn vfkv_cache_layer_size_bytes(cache: *const vfkv_cache, layer: u32) -> u64;
    pub fn vfkv_cache_layer_offset_bytes(cache: *const vfkv_cache, layer: u32) -> u64;
    pub fn vfkv_cache_layer_offset_elems(cache: *const vfkv_cache, layer: u32) -> u64;
    pub fn vfkv_cache_pos_offset_bytes(cache: *const vfkv_cache, layer: u32, pos: u32) -> u64;
    pub fn vfkv_cache_slot_offset_bytes(cache: *const vfkv_cache, layer: u32, slot: u32) -> u64;
    pub fn vfkv_cache_bytes_per_buffer(cache: *const vfkv_cache) -> u64;
    pub fn vfkv_cache_dtype(cache: *const vfkv_cache) -> u32;
    pub fn vfkv_cache_is_fp8(cache: *const vfkv_cache) -> i32;
    pub fn vfkv_cache_is_fp16(cache: *const vfkv_cache) -> i32;
    pub fn vfkv_cache_k_ptr(cache: *const vfkv_cache) -> *mut c_void;
    pub fn vfkv_cache_v_ptr(cache: *const vfkv_cache) -> *mut c_void;
    pub fn vfkv_cache_k_scale_ptr(cache: *const vfkv_cache) -> *mut f32;
    pub fn vfkv_cache_v_scale_ptr(cache: *const vfkv_cache) -> *mut f32;
    pub fn vfkv_kv_bytes_per_token(n_layers: u32, n_kv_heads: u32, head_dim: u32, per_layer_head_dim: *const u32, per_layer_n_kv_heads: *const u32, elem_size: u64) -> u64;
    pub fn vfkv_dtype_element_size(dtype: u32) -> u64;
    pub fn vfkv_dtype_from_env() -> u32;
    pub fn vfkv_guard_kv_precision(is_gemma4_moe: i32, dtype: u32, force: i32) -> i32;
    pub fn vfkv_sliding_kv_start(position: u32, sliding_window: u32) -> u32;
    pub fn vfkv_kv_store_fp8(ctx: *mut vfkv_ctx, d_src: *const f32, d_dst: *mut c_void, n_elements: u32, dst_byte_offset: u64, stream: *mut c_void) -> i32;
    pub fn vfkv_kv_copy_fp16(ctx: *mut vfkv_ctx, d_src: *const f32, d_dst: *mut c_void, n_elements: u32, dst_byte_offset: u64, stream: *mut c_void) -> i32;
    pub fn vfkv_kv_fp8_to_f16(ctx: *mut vfkv_ctx, d_src: *const c_void, d_dst: *mut c_void, n_elements: u64, stream: *mut c_void) -> i32;
    pub fn vfkv_flash_attn_split_reduce(ctx: *mut vfkv_ctx, ws: *mut vfkv_workspace, d_q: *const f32, d_k: *const c_void, d_v: *const c_void, d_out: *mut f32, dtype: u32, n_heads: u32, n_kv_heads: u32, head_dim: u32, seq_len: u32, max_seq: u32, scale: f32, kv_start: u32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_flash_attn_split_reduce_noalloc(d_q: *const f32, d_k: *const c_void, d_v: *const c_void, d_out: *mut f32, dtype: u32, n_heads: u32, n_kv_heads: u32, head_dim: u32, seq_len: u32, max_seq: u32, scale: f32, kv_start: u32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_noalloc_last_error() -> *const c_char;
    pub fn vfkv_noalloc_scratch_bytes() -> u64;
    pub fn vfkv_workspace_create(ctx: *mut vfkv_ctx, max_seqs: u32, n_q_heads: u32, head_dim: u32, max_splits: u32, out: *mut *mut vfkv_workspace) -> i32;
    pub fn vfkv_workspace_destroy(ws: *mut vfkv_workspace) -> i32;
    pub fn vfkv_workspace_bytes(ws: *const vfkv_workspace) -> u64;
    pub fn vfkv_workspace_reset(ws: *mut vfkv_workspace, stream: *mut c_void) -> i32;
    pub fn vfkv_append(cache: *mut vfkv_cache, layer: u32, d_k: *const f32, d_v: *const f32, n_tokens: u32, slot: u32, base_pos: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_append_sharded(cache: *mut vfkv_cache, layer: u32, d_k: *const f32, d_v: *const f32, n_tokens: u32, slot: u32, base_pos: u32, world: u32, page: u32, rank: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_append_batch(cache: *mut vfkv_cache, layer: u32, d_k: *const f32, d_v: *const f32, d_slot_ids: *const u32, d_positions: *const u32, n_seqs: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_fp8_to_f16(cache: *mut vfkv_cache, slot: u32, layer: u32, n_positions: u32, d_k_out: *mut c_void, d_v_out: *mut c_void, stream: *mut c_void) -> i32;
    pub fn vfkv_attend(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, layer: u32, kv_layer: u32, d_q: *const f32, d_out: *mut f32, n_q_heads: u32, slot: u32, seq_len: u32, kv_start: u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_attend_batch(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, layer: u32, kv_layer: u32, d_q: *const f32, d_out: *mut f32, n_q_heads: u32, d_slot_ids: *const u32, d_seq_lens: *const u32, d_kv_starts: *const u32, n_seqs: u32, max_seq_len_hint: u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_decode_step(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, layer: u32, d_q: *const f32, d_k: *const f32, d_v: *const f32, d_out: *mut f32, n_q_heads: u32, d_slot_ids: *const u32, d_positions: *const u32, n_seqs: u32, max_seq_len_hint: u32, window: u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_decode_token(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, d_q: *const f32, d_k: *const f32, d_v: *const f32, d_out: *mut f32, n_q_heads: u32, d_slot_ids: *const u32, d_positions: *const u32, n_seqs: u32, max_seq_len_hint: u32, windows: *const u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_decode_token_host(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, h_q: *const f32, h_k: *const f32, h_v: *const f32, h_out: *mut f32, n_q_heads: u32, h_slot_ids: *const u32, h_positions: *const u32, n_seqs: u32, windows: *const u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_decode_token_host_submit(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, h_q: *const f32, h_k: *const f32, h_v: *const f32, h_out: *mut f32, n_q_heads: u32, h_slot_ids: *const u32, h_positions: *const u32, n_seqs: u32, windows: *const u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void, ticket: *mut u64) -> i32;
    pub fn vfkv_decode_token_host_wait(ws: *mut vfkv_workspace, ticket: u64) -> i32;
    pub fn vfkv_attend_partial(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, layer: u32, kv_layer: u32, d_q: *const f32, n_q_heads: u32, slot: u32, pos_begin: u32, pos_end: u32, scale: f32, softcap: f32, n_splits: u32, d_m: *mut f32, d_l: *mut f32, d_o: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_attend_allgather(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, nccl_comm: *mut c_void, world: u32, rank: u32, layer: u32, kv_layer: u32, d_q: *const f32, n_q_heads: u32, slot: u32, pos_begin: u32, pos_end: u32, scale: f32, softcap: f32, n_splits: u32, d_packed: *mut f32, d_out: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_merge_partials(ctx: *mut vfkv_ctx, d_m: *const f32, d_l: *const f32, d_o: *const f32, n_parts: u32, n_rows: u32, head_dim: u32, d_out: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_merge_partials_packed(ctx: *mut vfkv_ctx, d_packed: *const f32, n_parts: u32, n_rows: u32, head_dim: u32, d_out: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_shard_owner(world: u32, page: u32, pos: u64) -> u32;
    pub fn vfkv_shard_local_pos(world: u32, page: u32, pos: u64) -> u64;
    pub fn vfkv_shard_local_len(world: u32, page: u32, seq_len: u64, rank: u32) -> u64;
    pub fn vfkv_shard_local_capacity(world: u32, page: u32, max_seq_len: u64) -> u64;
    pub fn vfkv_assign_sequences(lengths: *const u32, n: u32, world: u32, owner_out: *mut u32) -> i32;
    pub fn vfkv_shard_kv_heads(world: u32, rank: u32, n_kv_heads: u32, first: *mut u32, count: *mut u32) -> i32;
    pub fn vfkv_exchange_create(ctx: *mut vfkv_ctx, world: u32, rank: u32, n_rows: u32, head_dim: u32, out: *mut *mut vfkv_exchange) -> i32;
    pub fn vfkv_exchange_destroy(ex: *mut vfkv_exchange);
    pub fn vfkv_exchange_bytes(ex: *const vfkv_exchange) -> u64;
    pub fn vfkv_exchange_local_ptr(ex: *const vfkv_exchange) -> *mut c_void;
    pub fn vfkv_exchange_export(ex: *mut vfkv_exchange, handle: *mut u8) -> i32;
    pub fn vfkv_exchange_import(ex: *mut vfkv_exchange, rank: u32, handle: *const u8) -> i32;
    pub fn vfkv_exchange_set_peer(ex: *mut vfkv_exchange, rank: u32, d_peer_buffer: *mut c_void) -> i32;
    pub fn vfkv_exchange_set_timeout_ms(ex: *mut vfkv_exchange, ms: u32) -> i32;
    pub fn vfkv_exchange_ready(ex: *const vfkv_exchange) -> u32;
    pub fn vfkv_attend_push(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, ex: *mut vfkv_exchange, layer: u32, kv_layer: u32, d_q: *const f32, d_k_new: *const f32, d_v_new: *const f32, n_q_heads: u32, slot: u32, pos_begin: u32, pos_end: u32, scale: f32, softcap: f32, n_splits: u32, stream: *mut c_void) -> i32;
    pub fn vfkv_exchange_merge(ex: *mut vfkv_exchange, d_out: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_attend_exchange(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, ex: *mut vfkv_exchange, layer: u32, kv_layer: u32, d_q: *const f32, d_k_new: *const f32, d_v_new: *const f32, n_q_heads: u32, slot: u32, pos_begin: u32, pos_end: u32, scale: f32, softcap: f32, n_splits: u32, d_out: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_malloc(ctx: *mut vfkv_ctx, bytes: u64, d_out: *mut *mut c_void) -> i32;
    pub fn vfkv_free(ctx: *mut vfkv_ctx, d_ptr: *mut c_void) -> i32;
    pub fn vfkv_malloc_host(ctx: *mut vfkv_ctx, bytes: u64, h_out: *mut *mut c_void) -> i32;
    pub fn vfkv_free_host(ctx: *mut vfkv_ctx, h_ptr: *mut c_void) -> i32;
    pub fn vfkv_memcpy_h2d(ctx: *mut vfkv_ctx, d_dst: *mut c_void, h_src: *const c_void, bytes: u64, stream: *mut c_void) -> i32;
    pub fn vfkv_memcpy_d2h(ctx: *mut vfkv_ctx, h_dst: *mut c_void, d_src: *const c_void, bytes: u64, stream: *mut c_void) -> i32;
    pub fn vfkv_memset(ctx: *mut vfkv_ctx, d_dst: *mut c_void, byte: i32, bytes: u64, stream: *mut c_void) -> i32;
    pub fn vfkv_stream_synchronize(ctx: *mut vfkv_ctx, stream: *mut c_void) -> i32;
    pub fn vfkv_ctx_set_attn_impl(ctx: *mut vfkv_ctx, impl: u32) -> i32;
    pub fn vfkv_ctx_set_attn_tuning(ctx: *mut vfkv_ctx, warps: u32, stages: u32) -> i32;
    pub fn vfkv_ctx_set_dependent_launch(ctx: *mut vfkv_ctx, mode: u32) -> i32;
    pub fn vfkv_ctx_set_cluster_merge(ctx: *mut vfkv_ctx, on: u32) -> i32;
    pub fn vfkv_ctx_set_merge_wait_ms(ctx: *mut vfkv_ctx, ms: u32) -> i32;
    pub fn vfkv_ctx_debug_fail_split(ctx: *mut vfkv_ctx, split: u32) -> i32;
    pub fn vfkv_ctx_set_trace_buffer(ctx: *mut vfkv_ctx, d_buffer: *mut c_void) -> i32;
    pub fn vfkv_ctx_set_trace_ring(ctx: *mut vfkv_ctx, n_blocks: u32) -> i32;
    pub fn vfkv_ctx_launch_count(ctx: *const vfkv_ctx) -> u64;
    pub fn vfkv_ctx_kernel_count(ctx: *const vfkv_ctx) -> u64;
    pub fn vfkv_profile_enable(ctx: *mut vfkv_ctx, on: i32) -> i32;
    pub fn vfkv_profile_collect(ctx: *mut vfkv_ctx, label: u32, count: *mut u64, total_ms: *mut f64, min_ms: *mut f64, reset: i32) -> i32;
    pub fn vfkv_flash_attn(cache: *mut vfkv_cache, layer: u32, kv_layer: u32, d_q: *const f32, d_out: *mut f32, n_q_heads: u32, slot: u32, seq_len: u32, kv_start: u32, scale: f32, softcap: f32, stream: *mut c_void) -> i32;
    pub fn vfkv_scalar_attn(cache: *mut vfkv_cache, ws: *mut vfkv_workspace, layer: u32, kv_layer: u32, d_q: *const f32, d_out: *mut f32, n_q_heads: u32, slot: u32, position: u32, kv_start: u32, scale: f32, softcap: f32, stream: *mut c_void) -> i32;
    pub fn vfkv_scalar_attn_uses_split(position: u32) -> u32;
    pub fn vfkv_attend_prefill(cache: *mut vfkv_cache, layer: u32, kv_layer: u32, d_q: *const f32, d_out: *mut f32, n_q_heads: u32, slot: u32, m: u32, q_start: u32, n_kv: u32, kv_start: u32, window: u32, scale: f32, softcap: f32, stream: *mut c_void) -> i32;
    pub fn vfkv_rope_append(cache: *mut vfkv_cache, layer: u32, d_k: *const f32, d_v: *const f32, n_tokens: u32, slot: u32, base_pos: u32, rope: *const vfkv_rope_params, d_k_rot: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_rope_append_batch(cache: *mut vfkv_cache, layer: u32, d_k: *const f32, d_v: *const f32, d_slot_ids: *const u32, d_positions: *const u32, n_seqs: u32, rope: *const vfkv_rope_params, d_k_rot: *mut f32, stream: *mut c_void) -> i32;
    pub fn vfkv_rope_neox(ctx: *mut vfkv_ctx, d_x: *const f32, d_out: *mut f32, n_rows: u32, n_heads: u32, head_dim: u32, d_positions: *const u32, base_pos: u32, rope: *const vfkv_rope_params, stream: *mut c_void) -> i32;
    pub fn vfkv_longest_common_prefix(a: *const u32, n_a: u64, b: *const u32, n_b: u64) -> u64;
    pub fn vfkv_kv_reuse_prepare(cache: *mut vfkv_cache, slot: u32, cached_tokens: *const u32, n_cached: u64, full_tokens: *const u32, n_full: u64, reuse: i32, start_pos: *mut u32) -> i32;
    pub fn vfkv_kv_invalidate(cache: *mut vfkv_cache, slot: u32) -> i32;
    pub fn vfkv_compute_auto_ctx(free_bytes: u64, weight_bytes: u64, reserve_bytes: u64, kv_bytes_per_token: u64, model_max_ctx: u32, hw_cap: u32, sane_cap: u32, ctx_out: *mut u32, bound: *mut u32, avail_for_kv: *mut u64) -> i32;
    pub fn vfkv_gemma4_kv_read_layer(kv_source: *const u32, n_layers: u32, layer: u32) -> u32;
}
