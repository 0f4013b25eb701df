//! Raw FFI of `libullis_cuda.so`: one declaration per entry point of `include/ullis_cuda.h`.
//!
//! Generated by `gen_bindings.py` from the header - edit the header, not this file.
//! This crate is the only place of the `cuda` backend that may contain `unsafe` (the role
//! `src/metal/ffi.rs` plays for the Metal backend); `src/cuda.rs` wraps every call in a safe method.
//! Uncompiled where this repository is developed (no rustc there): the CPU tests check the
//! declarations against the header name by name and type by type instead.

#![allow(unsafe_code, non_camel_case_types, clippy::missing_safety_doc, clippy::too_many_arguments)]

use core::ffi::{c_char, c_void};

/// Opaque handle; only ever used behind a pointer.
#[repr(C)]
pub struct ullis_cuda_runtime {
    _private: [u8; 0],
}

/// Opaque handle; only ever used behind a pointer.
#[repr(C)]
pub struct ullis_cuda_model {
    _private: [u8; 0],
}

/// Opaque handle; only ever used behind a pointer.
#[repr(C)]
pub struct ullis_cuda_generate_state {
    _private: [u8; 0],
}

/// Opaque handle; only ever used behind a pointer.
#[repr(C)]
pub struct ullis_cuda_rosa_pushers {
    _private: [u8; 0],
}

/// Opaque handle; only ever used behind a pointer.
#[repr(C)]
pub struct ullis_cuda_train_state {
    _private: [u8; 0],
}

#[repr(C)]
#[derive(Clone, Copy, Debug, Default)]
pub struct ullis_cuda_train_result {
    pub mean_loss: f32,
    pub n_valid: u64,
    pub flips_head: u64,
    pub flips_cmix: u64,
    pub flips_rosa_o: u64,
}

#[repr(C)]
#[derive(Clone, Copy, Debug, Default)]
pub struct ullis_cuda_head_unigram_install {
    pub applied: i32,
    pub n_targets: u64,
    pub bias_rms: f32,
    pub scale_rms: f32,
    pub shrunk_kaiming_scale: i32,
}

pub const ULLIS_CUDA_OK: i32 = 0;
pub const ULLIS_CUDA_ERR_SHAPE: i32 = 1;
pub const ULLIS_CUDA_ERR_CHECKPOINT: i32 = 2;
pub const ULLIS_CUDA_ERR_CUDA: i32 = 3;
pub const ULLIS_CUDA_ERR_DEVICE_CHECK: i32 = 4;
pub const ULLIS_CUDA_ERR_NCCL: i32 = 5;
pub const ULLIS_CUDA_ERR_TIMEOUT: i32 = 6;
pub const ULLIS_CUDA_ERR_ARG: i32 = 7;
pub const ULLIS_CUDA_ERR_TOKEN: i32 = 8;
pub const ULLIS_CUDA_ERR_NOMEM: i32 = 9;
pub const ULLIS_CUDA_MODE_FAST: i32 = 0;
pub const ULLIS_CUDA_MODE_EXACT: i32 = 1;
pub const ULLIS_CUDA_SAM_EULER: i32 = 0;
pub const ULLIS_CUDA_SAM_EAGER: i32 = 1;
pub const ULLIS_CUDA_TAP_BLOCK_IN: i32 = 0;
pub const ULLIS_CUDA_TAP_LN3_OUT: i32 = 1;
pub const ULLIS_CUDA_TAP_Q_BITS: i32 = 2;
pub const ULLIS_CUDA_TAP_K_BITS: i32 = 3;
pub const ULLIS_CUDA_TAP_V_BITS: i32 = 4;
pub const ULLIS_CUDA_TAP_IDX: i32 = 5;
pub const ULLIS_CUDA_TAP_AFTER_ROSA: i32 = 6;
pub const ULLIS_CUDA_TAP_BLOCK_OUT: i32 = 7;
pub const ULLIS_CUDA_TAP_HIDDEN: i32 = 8;
pub const ULLIS_CUDA_SAM_STATIC_BYTES: usize = 64 << 20;

unsafe extern "C" {
    pub fn ullis_cuda_runtime_create(device: i32, out: *mut *mut ullis_cuda_runtime) -> i32;
    pub fn ullis_cuda_runtime_destroy(rt: *mut ullis_cuda_runtime);
    pub fn ullis_cuda_last_error(rt: *const ullis_cuda_runtime) -> *const c_char;
    pub fn ullis_cuda_runtime_set_mode(rt: *mut ullis_cuda_runtime, mode: i32) -> i32;
    pub fn ullis_cuda_runtime_set_sam(rt: *mut ullis_cuda_runtime, sam_algo: i32) -> i32;
    pub fn ullis_cuda_runtime_synchronize(rt: *mut ullis_cuda_runtime) -> i32;
    pub fn ullis_cuda_runtime_stream(rt: *mut ullis_cuda_runtime) -> *mut c_void;
    pub fn ullis_cuda_runtime_launch_count(rt: *const ullis_cuda_runtime) -> u64;
    pub fn ullis_cuda_runtime_kernel_timing(rt: *mut ullis_cuda_runtime, enabled: i32) -> i32;
    pub fn ullis_cuda_runtime_kernel_time(
        rt: *mut ullis_cuda_runtime,
        name: *const c_char,
        total_ms: *mut f32,
        launches: *mut u32,
    ) -> i32;
    pub fn ullis_cuda_runtime_kernel_names(
        rt: *mut ullis_cuda_runtime,
        buf: *mut c_char,
        len: usize,
        needed: *mut usize,
    ) -> i32;
    pub fn ullis_cuda_runtime_sam_counts(
        rt: *mut ullis_cuda_runtime,
        total: *mut u64,
        automaton: *mut u64,
        constant_q: *mut u64,
    ) -> i32;
    pub fn ullis_cuda_host_alloc(rt: *mut ullis_cuda_runtime, bytes: usize, out: *mut *mut c_void) -> i32;
    pub fn ullis_cuda_host_free(block: *mut c_void);
    pub fn ullis_cuda_runtime_wait_selftest(rt: *mut ullis_cuda_runtime, polls: u32) -> i32;
    pub fn ullis_cuda_runtime_is_sm100(rt: *const ullis_cuda_runtime) -> i32;
    pub fn ullis_cuda_model_load_safetensors(
        rt: *mut ullis_cuda_runtime,
        bytes: *const u8,
        len: usize,
        out: *mut *mut ullis_cuda_model,
    ) -> i32;
    pub fn ullis_cuda_model_destroy(model: *mut ullis_cuda_model);
    pub fn ullis_cuda_model_dims(model: *const ullis_cuda_model, dims: *mut usize) -> i32;
    pub fn ullis_cuda_model_forward_ce(
        model: *mut ullis_cuda_model,
        tokens: *const u32,
        labels: *const u32,
        ignore_id: u32,
        batch: usize,
        time: usize,
        mean_loss: *mut f32,
        loss_sum: *mut f64,
        n_valid: *mut u64,
        row_loss: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_model_upload_tokens(
        model: *mut ullis_cuda_model,
        tokens: *const u32,
        labels: *const u32,
        batch: usize,
        time: usize,
    ) -> i32;
    pub fn ullis_cuda_model_enqueue_forward_ce(
        model: *mut ullis_cuda_model,
        ignore_id: u32,
        batch: usize,
        time: usize,
    ) -> i32;
    pub fn ullis_cuda_model_read_loss(
        model: *mut ullis_cuda_model,
        mean_loss: *mut f32,
        loss_sum: *mut f64,
        n_valid: *mut u64,
        row_loss: *mut f32,
        rows: usize,
    ) -> i32;
    pub fn ullis_cuda_model_read_loss_global(
        model: *mut ullis_cuda_model,
        mean_loss: *mut f32,
        loss_sum: *mut f64,
        n_valid: *mut u64,
    ) -> i32;
    pub fn ullis_cuda_model_logits(
        model: *mut ullis_cuda_model,
        tokens: *const u32,
        batch: usize,
        time: usize,
        logits: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_model_hidden(
        model: *mut ullis_cuda_model,
        tokens: *const u32,
        batch: usize,
        time: usize,
        hidden: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_model_set_taps(model: *mut ullis_cuda_model, enabled: i32) -> i32;
    pub fn ullis_cuda_model_tap(
        model: *mut ullis_cuda_model,
        layer: i32,
        which: i32,
        out: *mut c_void,
        bytes: usize,
    ) -> i32;
    pub fn ullis_cuda_model_set_profile(model: *mut ullis_cuda_model, enabled: i32) -> i32;
    pub fn ullis_cuda_model_phase_ms(model: *mut ullis_cuda_model, ms: *mut f32) -> i32;
    pub fn ullis_cuda_generate_state_create(
        model: *mut ullis_cuda_model,
        batch: usize,
        out: *mut *mut ullis_cuda_generate_state,
    ) -> i32;
    pub fn ullis_cuda_generate_state_destroy(state: *mut ullis_cuda_generate_state);
    pub fn ullis_cuda_generate_state_reset(state: *mut ullis_cuda_generate_state) -> i32;
    pub fn ullis_cuda_generate_state_time(state: *const ullis_cuda_generate_state) -> usize;
    pub fn ullis_cuda_generate_step(
        state: *mut ullis_cuda_generate_state,
        tokens: *const u32,
        logits: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_rosa_pushers_create(
        rt: *mut ullis_cuda_runtime,
        streams: usize,
        capacity: usize,
        out: *mut *mut ullis_cuda_rosa_pushers,
    ) -> i32;
    pub fn ullis_cuda_rosa_pushers_destroy(pushers: *mut ullis_cuda_rosa_pushers);
    pub fn ullis_cuda_rosa_pushers_reset(pushers: *mut ullis_cuda_rosa_pushers) -> i32;
    pub fn ullis_cuda_rosa_pushers_push(
        pushers: *mut ullis_cuda_rosa_pushers,
        q: *const u8,
        k: *const u8,
        v: *const u8,
        steps: usize,
        idx: *mut u8,
    ) -> i32;
    pub fn ullis_cuda_train_state_create(
        model: *mut ullis_cuda_model,
        checkpoint: *const u8,
        len: usize,
        out: *mut *mut ullis_cuda_train_state,
    ) -> i32;
    pub fn ullis_cuda_train_state_destroy(state: *mut ullis_cuda_train_state);
    pub fn ullis_cuda_model_train_step(
        state: *mut ullis_cuda_train_state,
        tokens: *const u32,
        labels: *const u32,
        ignore_id: u32,
        batch: usize,
        time: usize,
        learning_rate: f32,
        result: *mut ullis_cuda_train_result,
    ) -> i32;
    pub fn ullis_cuda_train_state_read(
        state: *mut ullis_cuda_train_state,
        name: *const c_char,
        dst: *mut c_void,
        bytes: usize,
    ) -> i32;
    pub fn ullis_cuda_train_state_install_head_unigram_prior(
        state: *mut ullis_cuda_train_state,
        labels: *const u32,
        n: usize,
        ignore_id: u32,
        result: *mut ullis_cuda_head_unigram_install,
    ) -> i32;
    pub fn ullis_cuda_layer_norm(
        rt: *mut ullis_cuda_runtime,
        x: *const f32,
        weight: *const u16,
        bias: *const u16,
        y: *mut f32,
        rows: usize,
        channels: usize,
    ) -> i32;
    pub fn ullis_cuda_time_shift_delta(
        rt: *mut ullis_cuda_runtime,
        x: *const f32,
        xx: *mut f32,
        rows: usize,
        time: usize,
        channels: usize,
    ) -> i32;
    pub fn ullis_cuda_binary_linear(
        rt: *mut ullis_cuda_runtime,
        x: *const f32,
        bits: *const u32,
        scale: *const u16,
        bias: *const u16,
        y: *mut f32,
        rows: usize,
        in_features: usize,
        out_features: usize,
    ) -> i32;
    pub fn ullis_cuda_fp16_linear(
        rt: *mut ullis_cuda_runtime,
        x: *const f32,
        weight: *const u16,
        y: *mut f32,
        rows: usize,
        in_features: usize,
        out_features: usize,
    ) -> i32;
    pub fn ullis_cuda_sign_pack_bits(rt: *mut ullis_cuda_runtime, x: *const f32, bits: *mut u32, n: usize) -> i32;
    pub fn ullis_cuda_cmix_relu2(rt: *mut ullis_cuda_runtime, x: *const f32, y: *mut f32, n: usize) -> i32;
    pub fn ullis_cuda_residual_add(
        rt: *mut ullis_cuda_runtime,
        residual: *const f32,
        update: *const f32,
        out: *mut f32,
        n: usize,
    ) -> i32;
    pub fn ullis_cuda_clipped_sgd_fp16(
        rt: *mut ullis_cuda_runtime,
        parameters: *const u16,
        residual: *const f32,
        gradient: *const f32,
        learning_rate: f32,
        n: usize,
        next_parameters: *mut u16,
        next_residual: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_binaryconnect_sgd_fp16(
        rt: *mut ullis_cuda_runtime,
        parameters: *const u16,
        residual: *const f32,
        gradient: *const f32,
        learning_rate: f32,
        n: usize,
        next_parameters: *mut u16,
        next_residual: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_apply_latent_sgd(
        rt: *mut ullis_cuda_runtime,
        latent: *const u16,
        residual: *const f32,
        gradient: *const f32,
        learning_rate: f32,
        ste_scale: f32,
        n: usize,
        next_latent: *mut u16,
        next_residual: *mut f32,
        next_bits: *mut u32,
    ) -> i32;
    pub fn ullis_cuda_rosa_qkv_1bit_bwd_e(
        rt: *mut ullis_cuda_runtime,
        output_gradient: *const f32,
        idx: *const u8,
        batch: usize,
        time: usize,
        channels: usize,
        g_e: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_cmix_relu2_backward(
        rt: *mut ullis_cuda_runtime,
        input: *const f32,
        output_gradient: *const f32,
        gx: *mut f32,
        n: usize,
    ) -> i32;
    pub fn ullis_cuda_layer_norm_backward(
        rt: *mut ullis_cuda_runtime,
        input: *const f32,
        output_gradient: *const f32,
        weight: *const u16,
        rows: usize,
        channels: usize,
        gx: *mut f32,
        gw: *mut f32,
        gb: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_rosa_qkv_1bit_fwd(
        rt: *mut ullis_cuda_runtime,
        q_bits: *const u32,
        k_bits: *const u32,
        v_bits: *const u32,
        e: *const u16,
        idx: *mut u8,
        out: *mut f32,
        batch: usize,
        time: usize,
        channels: usize,
    ) -> i32;
    pub fn ullis_cuda_rosa_block_forward(
        rt: *mut ullis_cuda_runtime,
        x: *const f32,
        mix_q: *const u16,
        mix_k: *const u16,
        mix_v: *const u16,
        q_bits: *const u32,
        q_scale: *const u16,
        q_bias: *const u16,
        k_bits: *const u32,
        k_scale: *const u16,
        k_bias: *const u16,
        v_bits: *const u32,
        v_scale: *const u16,
        v_bias: *const u16,
        e: *const u16,
        o_bits: *const u32,
        o_scale: *const u16,
        o_bias: *const u16,
        batch: usize,
        time: usize,
        channels: usize,
        q_plane: *mut u32,
        k_plane: *mut u32,
        v_plane: *mut u32,
        idx: *mut u8,
        y: *mut f32,
        out: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_cmix_block_forward(
        rt: *mut ullis_cuda_runtime,
        x: *const f32,
        mix: *const u16,
        key_bits: *const u32,
        key_scale: *const u16,
        value: *const u16,
        batch: usize,
        time: usize,
        d_model: usize,
        dim_ffn: usize,
        out: *mut f32,
    ) -> i32;
    pub fn ullis_cuda_streamed_ce(
        rt: *mut ullis_cuda_runtime,
        hidden: *const f32,
        bits: *const u32,
        scale: *const u16,
        bias: *const u16,
        labels: *const u32,
        ignore_id: u32,
        rows: usize,
        time: usize,
        channels: usize,
        vocab: usize,
        row_loss: *mut f32,
        mean_loss: *mut f32,
        n_valid: *mut u64,
    ) -> i32;
    pub fn ullis_cuda_rosa_sam_static(
        device: i32,
        cuda_stream: *mut c_void,
        q_sw: *const u32,
        k_sw: *const u32,
        v_sw: *const u32,
        idx_sw: *mut u32,
        streams: usize,
        time: usize,
    ) -> i32;
    pub fn ullis_cuda_dp_unique_id(id: *mut u8) -> i32;
    pub fn ullis_cuda_dp_rendezvous(
        dir: *const c_char,
        tag: *const c_char,
        rank: i32,
        world: i32,
        timeout_ms: u32,
    ) -> i32;
    pub fn ullis_cuda_dp_init(rt: *mut ullis_cuda_runtime, rank: i32, world: i32, id: *const u8) -> i32;
    pub fn ullis_cuda_dp_allreduce_loss(rt: *mut ullis_cuda_runtime, loss_sum: *mut f64, n_valid: *mut u64) -> i32;
    pub fn ullis_cuda_dp_finalize(rt: *mut ullis_cuda_runtime) -> i32;
}
