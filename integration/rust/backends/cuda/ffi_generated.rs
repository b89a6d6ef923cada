//! GENERATED by tools/gen_rust_ffi.py from include/uzu_b200.h -- do not edit. Complete `extern "C"` surface of libuzu_b200.so:
//! opaque handles, enum constants, `#[repr(C)]` argument structs (field for field) and every entry point. Never compiled here
//! (no rustc in the build image); the struct layouts are checked against the library by tests/test_rust_ffi_gen.py.
#![allow(non_camel_case_types, dead_code)]
use std::ffi::{c_char, c_int, c_void};

#[repr(C)] pub struct uzu_context { _p: [u8; 0] }
#[repr(C)] pub struct uzu_buffer { _p: [u8; 0] }
#[repr(C)] pub struct uzu_sparse_buffer { _p: [u8; 0] }
#[repr(C)] pub struct uzu_command_buffer { _p: [u8; 0] }
#[repr(C)] pub struct uzu_engine { _p: [u8; 0] }

pub const UZU_OK: u32 = 0;
pub const UZU_ERROR_CUDA: u32 = 1;
pub const UZU_ERROR_INVALID_ARGUMENT: u32 = 2;
pub const UZU_ERROR_UNSUPPORTED: u32 = 3;
pub const UZU_ERROR_OUT_OF_MEMORY: u32 = 4;
pub const UZU_ERROR_IO: u32 = 5;
pub const UZU_ERROR_NO_DEVICE: u32 = 6;
pub const UZU_DT_BF16: u32 = 0;
pub const UZU_DT_F32: u32 = 1;
pub const UZU_DT_F16: u32 = 2;
pub const UZU_QMODE_U4: u32 = 0;
pub const UZU_QMODE_I8: u32 = 1;
pub const UZU_QMODE_U8: u32 = 2;
pub const UZU_QMETHOD_SCALE_BIAS: u32 = 0;
pub const UZU_QMETHOD_SCALE_ZERO_POINT: u32 = 1;
pub const UZU_QMETHOD_SCALE_SYMMETRIC: u32 = 2;
pub const UZU_B_FULL_PRECISION: u32 = 0;
pub const UZU_B_SCALE_BIAS_DEQUANT: u32 = 1;
pub const UZU_B_SCALE_ZERO_POINT_DEQUANT: u32 = 2;
pub const UZU_B_SCALE_SYMMETRIC_DEQUANT: u32 = 3;
pub const UZU_D_SCALE: u32 = 1;
pub const UZU_D_ACCUMULATE: u32 = 2;
pub const UZU_D_BIAS: u32 = 4;
pub const UZU_D_RHT: u32 = 8;
pub const UZU_D_SOFT_CAP: u32 = 16;
pub const UZU_ACT_SILU: u32 = 0;
pub const UZU_ACT_GELU_APPROX: u32 = 1;
pub const UZU_ACT_GELU_EXACT: u32 = 2;
pub const UZU_ACT_IDENTITY: u32 = 3;
pub const UZU_ACT_SOFTPLUS: u32 = 4;
pub const UZU_CAP_SPARSE_BUFFERS: u32 = 1;
pub const UZU_BUFFER_MANAGED: u32 = 0;
pub const UZU_BUFFER_PINNED_HOST: u32 = 1;
pub const UZU_BUFFER_DEVICE: u32 = 2;
pub const UZU_ACTIVATION_TRANSFORM_INPUT_RHT: u32 = 0;
pub const UZU_ACTIVATION_TRANSFORM_OUTPUT_RHT: u32 = 1;
pub const UZU_ACTIVATION_TRANSFORM_QUANTIZE: u32 = 2;
pub const UZU_ACTIVATION_TRANSFORM_QUANTIZE_WITH_GROUP_SUMS: u32 = 3;
pub const UZU_SAMPLING_GREEDY: u32 = 0;
pub const UZU_SAMPLING_STOCHASTIC: u32 = 1;

/// 8 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_ring_params {
    pub ring_offset: u32,
    pub ring_length: u32,
}

/// 12 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_trie_node {
    pub trie_start: u32,
    pub trie_end: u32,
    pub height: u32,
}

/// 8 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_kv_copy {
    pub source: u32,
    pub destination: u32,
}

/// 136 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_matmul_args {
    pub a: u64,
    pub b: u64,
    pub b_scales: u64,
    pub b_zero_points: u64,
    pub b_biases: u64,
    pub d: u64,
    pub bias: u64,
    pub gather_indices: u64,
    pub rht_factors: u64,
    pub b_prologue: u32,
    pub b_mode: u32,
    pub b_group_size: u32,
    pub b_signed_codes: u32,
    pub b_leading_dimension: u32,
    pub b_transpose: u32,
    pub d_transform: u32,
    pub ab_scale: f32,
    pub soft_cap: f32,
    pub m: u32,
    pub n: u32,
    pub k: u32,
    pub weights_dt: u32,
    pub input_dt: u32,
    pub output_dt: u32,
}

/// 240 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_fused_linear_args {
    pub matmul: uzu_matmul_args,
    pub prologue: u32,
    pub norm_input: u64,
    pub norm_shortcut_in: u64,
    pub norm_scales: u64,
    pub shortcut_out: u64,
    pub norm_epsilon: f32,
    pub norm_scale_offset: f32,
    pub norm_residual_add: u32,
    pub norm_full_layer: u32,
    pub act_operand: u64,
    pub act_type: u32,
    pub sg_attn: u64,
    pub sg_gate: u64,
    pub epilogue: u32,
    pub reserved0: u32,
    pub decode_stream: u64,
}

/// 32 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_tp_all_gather_args {
    pub src: u64,
    pub dst: u64,
    pub scratch: u64,
    pub rows: u32,
    pub cols_local: u32,
}

/// 112 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_normalization_args {
    pub input: u64,
    pub scales: u64,
    pub biases: u64,
    pub output: u64,
    pub shortcut: u64,
    pub hadamard_factors: u64,
    pub batch_size: u32,
    pub element_count: u32,
    pub epsilon: f32,
    pub scale_offset: f32,
    pub post_layer_scalar: f32,
    pub in_place: u32,
    pub subtract_mean: u32,
    pub full_layer: u32,
    pub copy_to_shortcut: u32,
    pub residual_add: u32,
    pub use_hadamard: u32,
    pub scale_residual_sum: u32,
    pub scale_output: u32,
    pub has_biases: u32,
    pub has_scales: u32,
}

/// 64 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_qkv_norm_args {
    pub qkv_input: u64,
    pub scales: u64,
    pub qkv_output: u64,
    pub batch_size: u32,
    pub total_heads: u32,
    pub head_dim: u32,
    pub epsilon: f32,
    pub scale_offset: f32,
    pub head_offset: u32,
    pub head_count: u32,
    pub full_layer: u32,
    pub in_place: u32,
    pub has_scales: u32,
}

/// 88 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_attention_prepare_args {
    pub qkv: u64,
    pub queries: u64,
    pub keys: u64,
    pub values: u64,
    pub cosines: u64,
    pub sines: u64,
    pub num_q_heads: u32,
    pub num_kv_heads: u32,
    pub head_dim: u32,
    pub rope_dim: u32,
    pub kv_token_offset: u32,
    pub batch_dim: u32,
    pub has_kv: u32,
    pub has_rope: u32,
    pub dynamic_position: u64,
}

/// 32 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_qk_norm_config {
    pub scales: u64,
    pub epsilon: f32,
    pub scale_offset: f32,
    pub present: u32,
    pub full_layer: u32,
    pub has_scales: u32,
    pub reserved0: u32,
}

/// 152 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_attention_prepare_norm_args {
    pub prepare: uzu_attention_prepare_args,
    pub q_norm: uzu_qk_norm_config,
    pub k_norm: uzu_qk_norm_config,
}

/// 152 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_attention_args {
    pub queries: u64,
    pub keys: u64,
    pub values: u64,
    pub out: u64,
    pub sums: u64,
    pub maxs: u64,
    pub gqa_factor: u32,
    pub sequence_length: u32,
    pub k_head_stride: u32,
    pub k_seq_stride: u32,
    pub v_head_stride: u32,
    pub v_seq_stride: u32,
    pub ring_params: uzu_ring_params,
    pub scale: f32,
    pub trie: u64,
    pub sliding_window_size: u32,
    pub sinks: u64,
    pub num_heads: u32,
    pub suffix_length: u32,
    pub head_dim: u32,
    pub has_sinks: u32,
    pub is_kv_cache_ring: u32,
    pub is_causal: u32,
    pub is_trie: u32,
    pub is_sliding_window: u32,
    pub dynamic_position: u64,
}

/// 48 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_attention_two_pass2_args {
    pub partials: u64,
    pub sums: u64,
    pub maxs: u64,
    pub out: u64,
    pub num_heads: u32,
    pub suffix_length: u32,
    pub head_dim: u32,
}

/// 32 bytes
#[repr(C)] #[derive(Clone, Copy)]
pub struct uzu_kv_cache_update_args {
    pub in_place_keys: u64,
    pub in_place_values: u64,
    pub copies: *const uzu_kv_copy,
    pub copy_count: u32,
    pub element_dim: u32,
}

/// 80 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_activation_transform_args {
    pub input: u64,
    pub fp_out: u64,
    pub q_out: u64,
    pub scales_out: u64,
    pub group_sums_out: u64,
    pub rht_factors: u64,
    pub batch_size: u32,
    pub element_count: u32,
    pub ops: u32,
    pub in_place: u32,
    pub activation_scale_group_size: u32,
    pub sum_group_size: u32,
    pub data_type: u32,
}

/// 48 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_gated_act_mul_args {
    pub act_operand: u64,
    pub value_operand: u64,
    pub fp_out: u64,
    pub gated_dim: u32,
    pub batch_dim: u32,
    pub value_offset: u32,
    pub value_row_stride: u32,
    pub act_type: u32,
    pub interleaved: u32,
}

/// 80 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_quantized_embedding_lookup_args {
    pub token_ids: u64,
    pub weights: u64,
    pub scales: u64,
    pub zero_points: u64,
    pub biases: u64,
    pub output: u64,
    pub batch_size: u32,
    pub vocab_size: u32,
    pub model_dim: u32,
    pub input_scale: f32,
    pub group_size: u32,
    pub quantization_mode: u32,
    pub quantization_method: u32,
}

/// 80 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_unified_sampling_args {
    pub logits: u64,
    pub output: u64,
    pub seeds: u64,
    pub bitmask: u64,
    pub temperature: f32,
    pub top_k: u32,
    pub top_p: f32,
    pub min_p: f32,
    pub vocab_size: u32,
    pub batch_size: u32,
    pub is_stochastic: u32,
    pub has_bitmask: u32,
    pub has_temperature: u32,
    pub has_top_k: u32,
    pub has_top_p: u32,
    pub has_min_p: u32,
}

/// 48 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_delta_net_conv_update_args {
    pub conv_weight: u64,
    pub bias: u64,
    pub in_out: u64,
    pub state: u64,
    pub kernel_size: u32,
    pub conv_dim: u32,
    pub state_stride: u32,
    pub has_bias: u32,
}

/// 80 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_delta_net_update_args {
    pub in_proj: u64,
    pub a_log: u64,
    pub dt_bias: u64,
    pub norm_weight: u64,
    pub state: u64,
    pub out: u64,
    pub num_v_heads: u32,
    pub num_k_heads: u32,
    pub head_v_dim: u32,
    pub key_dim: u32,
    pub value_dim: u32,
    pub norm_epsilon: f32,
    pub head_k_dim: u32,
}

/// 128 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_delta_net_fused_update_args {
    pub update: uzu_delta_net_update_args,
    pub conv: uzu_delta_net_conv_update_args,
}

/// 352 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_dense_linear_args {
    pub a: u64,
    pub w: u64,
    pub d: u64,
    pub bias: u64,
    pub group_offsets: u64,
    pub rows_map: u64,
    pub a_z_stride: u64,
    pub w_z_stride: u64,
    pub d_z_stride: u64,
    pub gate: u64,
    pub workspace: u64,
    pub m: u32,
    pub n: u32,
    pub k: u32,
    pub lda: u32,
    pub ldd: u32,
    pub batch: u32,
    pub weights_dt: u32,
    pub accumulate: u32,
    pub scale: f32,
    pub a_op: u32,
    pub gate_ld: u32,
    pub pair_rows: u32,
    pub glu_limit: f32,
    pub glu_alpha: f32,
    pub glu_kind: u32,
    pub d_op: u32,
    pub gate_bias: u64,
    pub col_scale: u64,
    pub row_scale: u64,
    pub post_weight: u64,
    pub post_bias: u64,
    pub next_weight: u64,
    pub next_bias: u64,
    pub next_out: u64,
    pub post_alpha: f32,
    pub post_mult: f32,
    pub next_alpha: f32,
    pub token_gate_dt: u32,
    pub token_ids: u64,
    pub token_table: u64,
    pub token_table_stride: u32,
    pub token_column: u32,
    pub token_vocab: u32,
    pub a_bf16: u32,
    pub stream_x: u64,
    pub stream_mix: u64,
    pub stream_out: u64,
    pub stream_in: u64,
    pub stream_u: u64,
    pub a_norm_weight: u64,
    pub a_norm_epsilon: f32,
    pub streams: u32,
    pub d_bf16: u32,
    pub a_residual_mult: f32,
    pub a_residual: u64,
    pub a_residual_out: u64,
    pub glu_limit_last: f32,
    pub glu_last_group: u32,
}

/// 72 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_group_rms_norm_args {
    pub input: u64,
    pub scales: u64,
    pub output: u64,
    pub row_indices: u64,
    pub rows: u32,
    pub n: u32,
    pub groups: u32,
    pub in_stride: u32,
    pub out_stride: u32,
    pub epsilon: f32,
    pub scales2: u64,
    pub output2: u64,
}

/// 96 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_norm_add_args {
    pub input: u64,
    pub weight: u64,
    pub bias: u64,
    pub residual: u64,
    pub output: u64,
    pub next_weight: u64,
    pub next_bias: u64,
    pub rows: u32,
    pub n: u32,
    pub in_stride: u32,
    pub kind: u32,
    pub next_kind: u32,
    pub alpha: f32,
    pub epsilon: f32,
    pub mult: f32,
    pub next_alpha: f32,
    pub residual_bf16: u32,
}

/// 112 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_stream_mix_args {
    pub x: u64,
    pub y: u64,
    pub mix: u64,
    pub out: u64,
    pub read: u64,
    pub u: u64,
    pub weight: u64,
    pub output: u64,
    pub token_ids: u64,
    pub table: u64,
    pub rows: u32,
    pub n: u32,
    pub streams: u32,
    pub vocab: u32,
    pub table_dt: u32,
    pub output_bf16: u32,
    pub epsilon: f32,
    pub reserved: u32,
}

/// 56 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_token_gate_args {
    pub z: u64,
    pub token_ids: u64,
    pub table: u64,
    pub out: u64,
    pub rows: u32,
    pub n: u32,
    pub vocab: u32,
    pub table_stride: u32,
    pub column: u32,
    pub weights_dt: u32,
}

/// 72 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_embedding_f32_args {
    pub token_ids: u64,
    pub table: u64,
    pub output: u64,
    pub position_turns: u64,
    pub dynamic_position: u64,
    pub rows_bf16: u64,
    pub rows: u32,
    pub vocab: u32,
    pub n: u32,
    pub weights_dt: u32,
    pub prefix: u32,
    pub scale: f32,
}

/// 56 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_glu_args {
    pub gate_up: u64,
    pub output: u64,
    pub group_offsets: u64,
    pub rows: u32,
    pub f: u32,
    pub kind: u32,
    pub output_bf16: u32,
    pub last_group: u32,
    pub limit: f32,
    pub limit_last: f32,
    pub alpha: f32,
}

/// 56 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_table_route_args {
    pub token_ids: u64,
    pub table: u64,
    pub group_offsets: u64,
    pub rows_map: u64,
    pub pair_pos: u64,
    pub rows: u32,
    pub top: u32,
    pub experts: u32,
    pub vocab: u32,
}

/// 112 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_topk_route_args {
    pub logits: u64,
    pub bias: u64,
    pub group_offsets: u64,
    pub rows_map: u64,
    pub pair_pos: u64,
    pub pair_weight: u64,
    pub rows: u32,
    pub top: u32,
    pub experts: u32,
    pub logits_stride: u32,
    pub weight_kind: u32,
    pub always: u32,
    pub compact_weight: u64,
    pub scratch: u64,
    pub correction: u64,
    pub choice_groups: u32,
    pub choice_keep: u32,
    pub weight_scale: f32,
    pub reserved: u32,
}

/// 80 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_routed_combine_args {
    pub pairs: u64,
    pub pair_pos: u64,
    pub pair_weight: u64,
    pub gate: u64,
    pub gate_bias: u64,
    pub col_scale: u64,
    pub output: u64,
    pub rows: u32,
    pub top: u32,
    pub n: u32,
    pub gate_ld: u32,
    pub accumulate: u32,
    pub weight: f32,
}

/// 120 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_sigmoid_attention_prepare_args {
    pub q: u64,
    pub k: u64,
    pub v: u64,
    pub q_scales: u64,
    pub k_scales: u64,
    pub query: u64,
    pub keys: u64,
    pub values: u64,
    pub dynamic_position: u64,
    pub rows: u32,
    pub q_n: u32,
    pub k_n: u32,
    pub v_n: u32,
    pub q_stride: u32,
    pub k_stride: u32,
    pub v_stride: u32,
    pub prefix: u32,
    pub cache_dt: u32,
    pub temp_every: u32,
    pub epsilon: f32,
    pub temp_coef: f32,
}

/// 120 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_sigmoid_attention_args {
    pub query: u64,
    pub keys: u64,
    pub values: u64,
    pub out: u64,
    pub dynamic_position: u64,
    pub dist_r1: u64,
    pub dist_r2: u64,
    pub head_bias: u64,
    pub partials: u64,
    pub tickets: u64,
    pub rows: u32,
    pub heads: u32,
    pub kv_heads: u32,
    pub dim: u32,
    pub vdim: u32,
    pub prefix: u32,
    pub cache_dt: u32,
    pub scale: f32,
    pub splits: u32,
    pub chunk_tiles: u32,
}

/// 112 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_general_delta_args {
    pub r: u64,
    pub k: u64,
    pub v: u64,
    pub rate_logit: u64,
    pub decay_logit: u64,
    pub rate_bias: u64,
    pub decay_bias: u64,
    pub unit: u64,
    pub state: u64,
    pub out: u64,
    pub r_stride: u32,
    pub k_stride: u32,
    pub v_stride: u32,
    pub rate_stride: u32,
    pub decay_stride: u32,
    pub rows: u32,
    pub heads: u32,
    pub dim: u32,
}

/// 96 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_head_norm_gate_args {
    pub x: u64,
    pub scales: u64,
    pub gate: u64,
    pub out: u64,
    pub rows: u32,
    pub heads: u32,
    pub dim: u32,
    pub x_stride: u32,
    pub gate_stride: u32,
    pub out_stride: u32,
    pub normalize: u32,
    pub epsilon: f32,
    pub gate_op: u32,
    pub reserved: u32,
    pub denom: u64,
    pub denom_floor: u64,
    pub denom_epsilon: f32,
    pub out_scale: f32,
}

/// 144 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_latent_prepare_args {
    pub kv: u64,
    pub q: u64,
    pub query: u64,
    pub cache: u64,
    pub latent_scales: u64,
    pub cosines: u64,
    pub sines: u64,
    pub dynamic_position: u64,
    pub rows: u32,
    pub heads: u32,
    pub dim: u32,
    pub rot_dim: u32,
    pub rank: u32,
    pub rot_pairs: u32,
    pub kv_stride: u32,
    pub q_stride: u32,
    pub prefix: u32,
    pub cache_dt: u32,
    pub epsilon: f32,
    pub reserved: u32,
    pub q_latent: u64,
    pub q_latent_scales: u64,
    pub q_latent_out: u64,
    pub q_rank: u32,
    pub q_latent_stride: u32,
}

/// 96 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_latent_attention_args {
    pub query: u64,
    pub cache: u64,
    pub out: u64,
    pub dynamic_position: u64,
    pub partials: u64,
    pub rows: u32,
    pub heads: u32,
    pub rank: u32,
    pub rot_dim: u32,
    pub prefix: u32,
    pub cache_dt: u32,
    pub scale: f32,
    pub splits: u32,
    pub sinks: u64,
    pub head_gate: u64,
    pub window: u32,
    pub head_gate_stride: u32,
}

/// 64 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_min_gru_args {
    pub z_logit: u64,
    pub u: u64,
    pub gate: u64,
    pub state: u64,
    pub out: u64,
    pub rows: u32,
    pub n: u32,
    pub z_stride: u32,
    pub u_stride: u32,
    pub gate_stride: u32,
    pub out_stride: u32,
}

/// 128 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_retention_args {
    pub q: u64,
    pub k: u64,
    pub v: u64,
    pub decay: u64,
    pub state: u64,
    pub out: u64,
    pub rows: u32,
    pub heads: u32,
    pub dim: u32,
    pub vdim: u32,
    pub q_stride: u32,
    pub k_stride: u32,
    pub v_stride: u32,
    pub out_stride: u32,
    pub key_scale: f32,
    pub input_op: u32,
    pub token_decay: u64,
    pub token_gain: u64,
    pub norm_out: u64,
    pub query_scale: f32,
    pub reserved1: u32,
    pub chunk_scratch: u64,
}

/// 72 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_exp_gates_args {
    pub i_pre: u64,
    pub f_pre: u64,
    pub state: u64,
    pub token_decay: u64,
    pub token_gain: u64,
    pub floor: u64,
    pub rows: u32,
    pub heads: u32,
    pub i_stride: u32,
    pub f_stride: u32,
    pub cap: f32,
    pub reserved: u32,
}

/// 128 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_delta_prepare_args {
    pub proj: u64,
    pub conv: u64,
    pub ring: u64,
    pub a_log: u64,
    pub dt_bias: u64,
    pub dynamic_position: u64,
    pub q: u64,
    pub k: u64,
    pub v: u64,
    pub decay: u64,
    pub beta: u64,
    pub rows: u32,
    pub heads: u32,
    pub kv_heads: u32,
    pub dim: u32,
    pub vdim: u32,
    pub taps: u32,
    pub stride: u32,
    pub a_offset: u32,
    pub b_offset: u32,
    pub prefix: u32,
}

/// 144 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_gated_delta_args {
    pub prep: uzu_delta_prepare_args,
    pub state: u64,
    pub out: u64,
}

/// 160 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_gated_delta_step_args {
    pub prep: uzu_delta_prepare_args,
    pub state: u64,
    pub norm: u64,
    pub out: u64,
    pub gate_offset: u32,
    pub epsilon: f32,
}

/// 168 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_window_attention_prepare_args {
    pub q: u64,
    pub k: u64,
    pub v: u64,
    pub q_scales: u64,
    pub k_scales: u64,
    pub query: u64,
    pub keys: u64,
    pub values: u64,
    pub cosines: u64,
    pub sines: u64,
    pub v_cosines: u64,
    pub v_sines: u64,
    pub dynamic_position: u64,
    pub rows: u32,
    pub heads: u32,
    pub kv_heads: u32,
    pub dim: u32,
    pub vdim: u32,
    pub rot_pairs: u32,
    pub v_pairs: u32,
    pub q_stride: u32,
    pub k_stride: u32,
    pub v_stride: u32,
    pub prefix: u32,
    pub cache_dt: u32,
    pub epsilon: f32,
    pub rot_halves: u32,
    pub unit_rms: u32,
    pub reserved: u32,
}

/// 176 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_window_attention_args {
    pub query: u64,
    pub keys: u64,
    pub values: u64,
    pub out: u64,
    pub dynamic_position: u64,
    pub head_temp: u64,
    pub v_cosines: u64,
    pub v_sines: u64,
    pub partials: u64,
    pub tickets: u64,
    pub rows: u32,
    pub heads: u32,
    pub kv_heads: u32,
    pub dim: u32,
    pub vdim: u32,
    pub prefix: u32,
    pub cache_dt: u32,
    pub window: u32,
    pub keep_first: u32,
    pub v_pairs: u32,
    pub scale: f32,
    pub softcap: f32,
    pub splits: u32,
    pub head_gate_stride: u32,
    pub sinks: u64,
    pub head_gate: u64,
    pub chunk: u32,
    pub out_stride: u32,
    pub dist_slope: u64,
    pub out_scale: f32,
    pub reserved: u32,
}

/// 296 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_side_step_args {
    pub prep: uzu_window_attention_prepare_args,
    pub retention: uzu_retention_args,
}

/// 272 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_side_attention_args {
    pub attention: uzu_window_attention_args,
    pub norm: uzu_head_norm_gate_args,
}

/// 56 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_engine_options {
    pub max_context_length: u32,
    pub use_cuda_graph: u32,
    pub fused_decode: u32,
    pub tp_rank: u32,
    pub tp_size: u32,
    pub storage_f32: u32,
    pub reserved0: u32,
    pub reserved: [u64; 3],
}

/// 48 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_sampling_method {
    pub kind: u32,
    pub has_temperature: u32,
    pub temperature: f32,
    pub has_top_k: u32,
    pub top_k: u32,
    pub has_top_p: u32,
    pub top_p: f32,
    pub has_min_p: u32,
    pub min_p: f32,
    pub seed: u64,
}

/// 56 bytes
#[repr(C)] #[derive(Default, Clone, Copy)]
pub struct uzu_model_info {
    pub model_dim: u32,
    pub hidden_dim: u32,
    pub vocab_size: u32,
    pub num_layers: u32,
    pub num_attention_layers: u32,
    pub num_delta_net_layers: u32,
    pub weight_bytes_per_token: u64,
    pub kv_bytes_per_token_per_ctx: u64,
    pub state_bytes_per_token: u64,
    pub num_layer_runs: u32,
    pub reserved: u32,
}

/// (C name, size_of) of every argument struct: ffi::abi_self_check() compares them with uzu_abi_struct_size() of the loaded library
pub const STRUCT_SIZES: &[(&str, usize)] = &[
    ("uzu_ring_params", std::mem::size_of::<uzu_ring_params>()),
    ("uzu_trie_node", std::mem::size_of::<uzu_trie_node>()),
    ("uzu_kv_copy", std::mem::size_of::<uzu_kv_copy>()),
    ("uzu_matmul_args", std::mem::size_of::<uzu_matmul_args>()),
    ("uzu_fused_linear_args", std::mem::size_of::<uzu_fused_linear_args>()),
    ("uzu_tp_all_gather_args", std::mem::size_of::<uzu_tp_all_gather_args>()),
    ("uzu_normalization_args", std::mem::size_of::<uzu_normalization_args>()),
    ("uzu_qkv_norm_args", std::mem::size_of::<uzu_qkv_norm_args>()),
    ("uzu_attention_prepare_args", std::mem::size_of::<uzu_attention_prepare_args>()),
    ("uzu_qk_norm_config", std::mem::size_of::<uzu_qk_norm_config>()),
    ("uzu_attention_prepare_norm_args", std::mem::size_of::<uzu_attention_prepare_norm_args>()),
    ("uzu_attention_args", std::mem::size_of::<uzu_attention_args>()),
    ("uzu_attention_two_pass2_args", std::mem::size_of::<uzu_attention_two_pass2_args>()),
    ("uzu_kv_cache_update_args", std::mem::size_of::<uzu_kv_cache_update_args>()),
    ("uzu_activation_transform_args", std::mem::size_of::<uzu_activation_transform_args>()),
    ("uzu_gated_act_mul_args", std::mem::size_of::<uzu_gated_act_mul_args>()),
    ("uzu_quantized_embedding_lookup_args", std::mem::size_of::<uzu_quantized_embedding_lookup_args>()),
    ("uzu_unified_sampling_args", std::mem::size_of::<uzu_unified_sampling_args>()),
    ("uzu_delta_net_conv_update_args", std::mem::size_of::<uzu_delta_net_conv_update_args>()),
    ("uzu_delta_net_update_args", std::mem::size_of::<uzu_delta_net_update_args>()),
    ("uzu_delta_net_fused_update_args", std::mem::size_of::<uzu_delta_net_fused_update_args>()),
    ("uzu_dense_linear_args", std::mem::size_of::<uzu_dense_linear_args>()),
    ("uzu_group_rms_norm_args", std::mem::size_of::<uzu_group_rms_norm_args>()),
    ("uzu_norm_add_args", std::mem::size_of::<uzu_norm_add_args>()),
    ("uzu_stream_mix_args", std::mem::size_of::<uzu_stream_mix_args>()),
    ("uzu_token_gate_args", std::mem::size_of::<uzu_token_gate_args>()),
    ("uzu_embedding_f32_args", std::mem::size_of::<uzu_embedding_f32_args>()),
    ("uzu_glu_args", std::mem::size_of::<uzu_glu_args>()),
    ("uzu_table_route_args", std::mem::size_of::<uzu_table_route_args>()),
    ("uzu_topk_route_args", std::mem::size_of::<uzu_topk_route_args>()),
    ("uzu_routed_combine_args", std::mem::size_of::<uzu_routed_combine_args>()),
    ("uzu_sigmoid_attention_prepare_args", std::mem::size_of::<uzu_sigmoid_attention_prepare_args>()),
    ("uzu_sigmoid_attention_args", std::mem::size_of::<uzu_sigmoid_attention_args>()),
    ("uzu_general_delta_args", std::mem::size_of::<uzu_general_delta_args>()),
    ("uzu_head_norm_gate_args", std::mem::size_of::<uzu_head_norm_gate_args>()),
    ("uzu_latent_prepare_args", std::mem::size_of::<uzu_latent_prepare_args>()),
    ("uzu_latent_attention_args", std::mem::size_of::<uzu_latent_attention_args>()),
    ("uzu_min_gru_args", std::mem::size_of::<uzu_min_gru_args>()),
    ("uzu_retention_args", std::mem::size_of::<uzu_retention_args>()),
    ("uzu_exp_gates_args", std::mem::size_of::<uzu_exp_gates_args>()),
    ("uzu_delta_prepare_args", std::mem::size_of::<uzu_delta_prepare_args>()),
    ("uzu_gated_delta_args", std::mem::size_of::<uzu_gated_delta_args>()),
    ("uzu_gated_delta_step_args", std::mem::size_of::<uzu_gated_delta_step_args>()),
    ("uzu_window_attention_prepare_args", std::mem::size_of::<uzu_window_attention_prepare_args>()),
    ("uzu_window_attention_args", std::mem::size_of::<uzu_window_attention_args>()),
    ("uzu_side_step_args", std::mem::size_of::<uzu_side_step_args>()),
    ("uzu_side_attention_args", std::mem::size_of::<uzu_side_attention_args>()),
    ("uzu_engine_options", std::mem::size_of::<uzu_engine_options>()),
    ("uzu_sampling_method", std::mem::size_of::<uzu_sampling_method>()),
    ("uzu_model_info", std::mem::size_of::<uzu_model_info>()),
];

#[link(name = "uzu_b200")]
extern "C" {
    pub fn uzu_last_error() -> *const c_char;
    pub fn uzu_version() -> *const c_char;
    pub fn uzu_abi_struct_size(name: *const c_char) -> usize;
    pub fn uzu_context_create(device_ordinal: c_int, out: *mut *mut uzu_context) -> c_int;
    pub fn uzu_context_destroy(ctx: *mut uzu_context);
    pub fn uzu_context_synchronize(ctx: *mut uzu_context) -> c_int;
    pub fn uzu_context_peak_memory_usage(ctx: *mut uzu_context, out_bytes: *mut usize) -> c_int;
    pub fn uzu_context_device_capabilities(ctx: *mut uzu_context) -> u32;
    pub fn uzu_context_start_capture(ctx: *mut uzu_context, trace_path: *const c_char) -> c_int;
    pub fn uzu_context_stop_capture(ctx: *mut uzu_context) -> c_int;
    pub fn uzu_context_device(ctx: *mut uzu_context) -> c_int;
    pub fn uzu_context_sm_count(ctx: *mut uzu_context) -> c_int;
    pub fn uzu_context_stream(ctx: *mut uzu_context) -> *mut c_void;
    pub fn uzu_buffer_create(ctx: *mut uzu_context, size: usize, kind: c_int, out: *mut *mut uzu_buffer) -> c_int;
    pub fn uzu_buffer_destroy(buf: *mut uzu_buffer);
    pub fn uzu_buffer_gpu_ptr(buf: *const uzu_buffer) -> u64;
    pub fn uzu_buffer_cpu_ptr(buf: *const uzu_buffer) -> *mut c_void;
    pub fn uzu_buffer_size(buf: *const uzu_buffer) -> usize;
    pub fn uzu_buffer_make_resident(ctx: *mut uzu_context, buf: *mut uzu_buffer) -> c_int;
    pub fn uzu_sparse_buffer_create(ctx: *mut uzu_context, capacity: usize, out: *mut *mut uzu_sparse_buffer) -> c_int;
    pub fn uzu_sparse_buffer_destroy(buf: *mut uzu_sparse_buffer);
    pub fn uzu_sparse_buffer_gpu_ptr(buf: *const uzu_sparse_buffer) -> u64;
    pub fn uzu_sparse_buffer_size(buf: *const uzu_sparse_buffer) -> usize;
    pub fn uzu_sparse_buffer_page_size_bytes(buf: *const uzu_sparse_buffer) -> usize;
    pub fn uzu_sparse_buffer_map(buf: *mut uzu_sparse_buffer, pages: *const u32, page_count: usize) -> c_int;
    pub fn uzu_sparse_buffer_unmap(buf: *mut uzu_sparse_buffer, pages: *const u32, page_count: usize) -> c_int;
    pub fn uzu_command_buffer_create(ctx: *mut uzu_context, name: *const c_char, out: *mut *mut uzu_command_buffer) -> c_int;
    pub fn uzu_command_buffer_destroy(cmd: *mut uzu_command_buffer);
    pub fn uzu_command_buffer_start_encoding(cmd: *mut uzu_command_buffer) -> c_int;
    pub fn uzu_command_buffer_encode_copy(cmd: *mut uzu_command_buffer, src: u64, dst: u64, bytes: usize);
    pub fn uzu_command_buffer_encode_fill(cmd: *mut uzu_command_buffer, dst: u64, bytes: usize, value: u8);
    pub fn uzu_command_buffer_encode_barrier(cmd: *mut uzu_command_buffer, after: u32, before: u32);
    pub fn uzu_command_buffer_push_debug_group(cmd: *mut uzu_command_buffer, name: *const c_char);
    pub fn uzu_command_buffer_pop_debug_group(cmd: *mut uzu_command_buffer);
    pub fn uzu_command_buffer_end_encoding(cmd: *mut uzu_command_buffer) -> c_int;
    pub fn uzu_command_buffer_submit(cmd: *mut uzu_command_buffer) -> c_int;
    pub fn uzu_command_buffer_wait_until_completed(cmd: *mut uzu_command_buffer) -> c_int;
    pub fn uzu_command_buffer_gpu_execution_time(cmd: *mut uzu_command_buffer, out_seconds: *mut f64) -> c_int;
    pub fn uzu_command_buffer_launch_count(cmd: *const uzu_command_buffer) -> u64;
    pub fn uzu_matmul_encode(cmd: *mut uzu_command_buffer, args: *const uzu_matmul_args);
    pub fn uzu_matmul_validate(args: *const uzu_matmul_args) -> c_int;
    pub fn uzu_debug_fused_linear_encode(cmd: *mut uzu_command_buffer, args: *const uzu_fused_linear_args) -> c_int;
    pub fn uzu_debug_set_qmv_tuning(warps_per_tile: c_int, k_slices: c_int, ctas_per_sm: c_int, stages: c_int);
    pub fn uzu_debug_set_qmm_tile(rows: c_int, splits: c_int) -> c_int;
    pub fn uzu_debug_set_umma(layout: c_int, desc_hi: u32, desc_lbo: u32, k_step: u32, idesc: u32, mt: c_int);
    pub fn uzu_fused_linear_supported(ctx: *mut uzu_context, args: *const uzu_fused_linear_args) -> c_int;
    pub fn uzu_fused_linear_encode(cmd: *mut uzu_command_buffer, args: *const uzu_fused_linear_args);
    pub fn uzu_tp_get_unique_id(out128: *mut u8) -> c_int;
    pub fn uzu_context_tp_init(ctx: *mut uzu_context, rank: u32, size: u32, unique_id128: *const u8) -> c_int;
    pub fn uzu_context_tp_destroy(ctx: *mut uzu_context);
    pub fn uzu_context_tp_size(ctx: *const uzu_context) -> u32;
    pub fn uzu_context_tp_rank(ctx: *const uzu_context) -> u32;
    pub fn uzu_tp_p2p_export(ctx: *mut uzu_context, capacity_f32: u32, handle_out64: *mut u8) -> c_int;
    pub fn uzu_tp_p2p_import(ctx: *mut uzu_context, handles_size_x_64: *const u8) -> c_int;
    pub fn uzu_tp_all_reduce_encode(cmd: *mut uzu_command_buffer, partial_f32: u64, count: u32, out_bf16: u64);
    pub fn uzu_tp_all_gather_encode(cmd: *mut uzu_command_buffer, args: *const uzu_tp_all_gather_args);
    pub fn uzu_normalization_encode(cmd: *mut uzu_command_buffer, args: *const uzu_normalization_args);
    pub fn uzu_qkv_norm_encode(cmd: *mut uzu_command_buffer, args: *const uzu_qkv_norm_args);
    pub fn uzu_attention_prepare_encode(cmd: *mut uzu_command_buffer, args: *const uzu_attention_prepare_args);
    pub fn uzu_attention_prepare_norm_encode(cmd: *mut uzu_command_buffer, args: *const uzu_attention_prepare_norm_args);
    pub fn uzu_attention_single_pass_encode(cmd: *mut uzu_command_buffer, args: *const uzu_attention_args);
    pub fn uzu_attention_two_pass1_encode(cmd: *mut uzu_command_buffer, args: *const uzu_attention_args);
    pub fn uzu_debug_set_prefill_attention(mode: c_int);
    pub fn uzu_debug_decode_attention_encode(cmd: *mut uzu_command_buffer, prepare: *const uzu_attention_prepare_norm_args, attention: *const uzu_attention_args) -> c_int;
    pub fn uzu_attention_two_pass2_encode(cmd: *mut uzu_command_buffer, args: *const uzu_attention_two_pass2_args);
    pub fn uzu_kv_cache_update_encode(cmd: *mut uzu_command_buffer, args: *const uzu_kv_cache_update_args);
    pub fn uzu_activation_transform_encode(cmd: *mut uzu_command_buffer, args: *const uzu_activation_transform_args);
    pub fn uzu_activation_transform_validate(args: *const uzu_activation_transform_args) -> c_int;
    pub fn uzu_sigmoid_gate_encode(cmd: *mut uzu_command_buffer, gate: u64, output: u64, total_elements: u32);
    pub fn uzu_gated_act_mul_encode(cmd: *mut uzu_command_buffer, args: *const uzu_gated_act_mul_args);
    pub fn uzu_quantized_embedding_lookup_encode(cmd: *mut uzu_command_buffer, args: *const uzu_quantized_embedding_lookup_args);
    pub fn uzu_full_precision_embedding_lookup_encode(cmd: *mut uzu_command_buffer, token_ids: u64, weights: u64, output: u64, batch_size: u32, vocab_size: u32, model_dim: u32, input_scale: f32);
    pub fn uzu_logit_transform_encode(cmd: *mut uzu_command_buffer, logits: u64, length: u32, scale: f32, soft_cap: f32, has_soft_cap: u32);
    pub fn uzu_tensor_add_scale_encode(cmd: *mut uzu_command_buffer, input: u64, bias: u64, output: u64, num_cols: u32, length: u32, scale: f32);
    pub fn uzu_tensor_copy_encode(cmd: *mut uzu_command_buffer, src: u64, dst: u64, length: u32);
    pub fn uzu_tensor_add_bias_encode(cmd: *mut uzu_command_buffer, input: u64, bias: u64, output: u64, num_cols: u32, length: u32);
    pub fn uzu_tensor_add_swap_encode(cmd: *mut uzu_command_buffer, skip_buffer: u64, main_buffer: u64, length: u32);
    pub fn uzu_unified_sampling_encode(cmd: *mut uzu_command_buffer, args: *const uzu_unified_sampling_args);
    pub fn uzu_delta_net_conv_update_encode(cmd: *mut uzu_command_buffer, args: *const uzu_delta_net_conv_update_args);
    pub fn uzu_delta_net_update_encode(cmd: *mut uzu_command_buffer, args: *const uzu_delta_net_update_args);
    pub fn uzu_delta_net_fused_update_supported(args: *const uzu_delta_net_fused_update_args) -> c_int;
    pub fn uzu_delta_net_fused_update_encode(cmd: *mut uzu_command_buffer, args: *const uzu_delta_net_fused_update_args);
    pub fn uzu_debug_set_delta_prefill(mode: c_int);
    pub fn uzu_dense_linear_encode(cmd: *mut uzu_command_buffer, args: *const uzu_dense_linear_args);
    pub fn uzu_debug_dense_umma_error() -> u32;
    pub fn uzu_debug_set_wait_error(ctx: *mut uzu_context, code: u32);
    pub fn uzu_group_rms_norm_encode(cmd: *mut uzu_command_buffer, args: *const uzu_group_rms_norm_args);
    pub fn uzu_norm_add_encode(cmd: *mut uzu_command_buffer, args: *const uzu_norm_add_args);
    pub fn uzu_stream_mix_encode(cmd: *mut uzu_command_buffer, args: *const uzu_stream_mix_args);
    pub fn uzu_token_gate_encode(cmd: *mut uzu_command_buffer, args: *const uzu_token_gate_args);
    pub fn uzu_rows_to_bf16_encode(cmd: *mut uzu_command_buffer, src: u64, src_stride: u32, dst: u64, rows: u32, n: u32);
    pub fn uzu_embedding_f32_encode(cmd: *mut uzu_command_buffer, token_ids: u64, table: u64, weights_dt: u32, output: u64, rows: u32, vocab: u32, n: u32);
    pub fn uzu_embedding_f32_scaled_encode(cmd: *mut uzu_command_buffer, token_ids: u64, table: u64, weights_dt: u32, output: u64, rows: u32, vocab: u32, n: u32, scale: f32);
    pub fn uzu_embedding_f32_position_encode(cmd: *mut uzu_command_buffer, args: *const uzu_embedding_f32_args);
    pub fn uzu_glu_encode(cmd: *mut uzu_command_buffer, args: *const uzu_glu_args);
    pub fn uzu_clamped_glu_encode(cmd: *mut uzu_command_buffer, gate_up: u64, output: u64, rows: u32, f: u32, limit: f32, alpha: f32);
    pub fn uzu_silu_glu_encode(cmd: *mut uzu_command_buffer, gate_up: u64, output: u64, rows: u32, f: u32);
    pub fn uzu_unary_f32_encode(cmd: *mut uzu_command_buffer, input: u64, in_stride: u32, output: u64, out_stride: u32, rows: u32, n: u32, op: u32);
    pub fn uzu_residual_add_encode(cmd: *mut uzu_command_buffer, x: u64, a: u64, b: u64, length: u32);
    pub fn uzu_logit_cap_f32_encode(cmd: *mut uzu_command_buffer, logits_f32: u64, logits_bf16: u64, length: u32, cap: f32, has_cap: u32);
    pub fn uzu_table_route_encode(cmd: *mut uzu_command_buffer, args: *const uzu_table_route_args);
    pub fn uzu_routed_combine_encode(cmd: *mut uzu_command_buffer, pairs: u64, pair_pos: u64, output: u64, rows: u32, top: u32, n: u32, weight: f32, accumulate: u32);
    pub fn uzu_topk_route_encode(cmd: *mut uzu_command_buffer, args: *const uzu_topk_route_args);
    pub fn uzu_routed_combine_gated_encode(cmd: *mut uzu_command_buffer, args: *const uzu_routed_combine_args);
    pub fn uzu_sigmoid_attention_prepare_encode(cmd: *mut uzu_command_buffer, args: *const uzu_sigmoid_attention_prepare_args);
    pub fn uzu_sigmoid_attention_encode(cmd: *mut uzu_command_buffer, args: *const uzu_sigmoid_attention_args);
    pub fn uzu_general_delta_encode(cmd: *mut uzu_command_buffer, args: *const uzu_general_delta_args);
    pub fn uzu_head_norm_gate_encode(cmd: *mut uzu_command_buffer, args: *const uzu_head_norm_gate_args);
    pub fn uzu_latent_prepare_encode(cmd: *mut uzu_command_buffer, args: *const uzu_latent_prepare_args);
    pub fn uzu_latent_attention_encode(cmd: *mut uzu_command_buffer, args: *const uzu_latent_attention_args);
    pub fn uzu_min_gru_encode(cmd: *mut uzu_command_buffer, args: *const uzu_min_gru_args);
    pub fn uzu_retention_encode(cmd: *mut uzu_command_buffer, args: *const uzu_retention_args);
    pub fn uzu_exp_gates_encode(cmd: *mut uzu_command_buffer, args: *const uzu_exp_gates_args);
    pub fn uzu_delta_prepare_encode(cmd: *mut uzu_command_buffer, args: *const uzu_delta_prepare_args);
    pub fn uzu_gated_delta_encode(cmd: *mut uzu_command_buffer, args: *const uzu_gated_delta_args);
    pub fn uzu_gated_delta_step_encode(cmd: *mut uzu_command_buffer, args: *const uzu_gated_delta_step_args);
    pub fn uzu_window_attention_prepare_encode(cmd: *mut uzu_command_buffer, args: *const uzu_window_attention_prepare_args);
    pub fn uzu_window_attention_encode(cmd: *mut uzu_command_buffer, args: *const uzu_window_attention_args);
    pub fn uzu_side_step_encode(cmd: *mut uzu_command_buffer, args: *const uzu_side_step_args);
    pub fn uzu_side_attention_encode(cmd: *mut uzu_command_buffer, args: *const uzu_side_attention_args);
    pub fn uzu_engine_create(ctx: *mut uzu_context, model_dir: *const c_char, opts: *const uzu_engine_options, out: *mut *mut uzu_engine) -> c_int;
    pub fn uzu_engine_destroy(e: *mut uzu_engine);
    pub fn uzu_engine_info(e: *const uzu_engine, out: *mut uzu_model_info) -> c_int;
    pub fn uzu_engine_reset(e: *mut uzu_engine) -> c_int;
    pub fn uzu_engine_context_length(e: *const uzu_engine) -> u32;
    pub fn uzu_engine_snapshot(e: *mut uzu_engine) -> c_int;
    pub fn uzu_engine_restore(e: *mut uzu_engine) -> c_int;
    pub fn uzu_engine_prefill(e: *mut uzu_engine, tokens: *const u32, count: u32, sampling: *const uzu_sampling_method, out_token: *mut u32) -> c_int;
    pub fn uzu_engine_next(e: *mut uzu_engine, out_token: *mut u32) -> c_int;
    pub fn uzu_engine_flush(e: *mut uzu_engine, out_token: *mut u32) -> c_int;
    pub fn uzu_engine_decode_device(e: *mut uzu_engine, steps: u32, out_tokens_dev: u64) -> c_int;
    pub fn uzu_engine_forward(e: *mut uzu_engine, tokens: *const u32, count: u32, row_begin: u32, row_end: u32, out_logits: *mut u16) -> c_int;
    pub fn uzu_engine_slot_acquire(e: *mut uzu_engine, out_slot: *mut u32) -> c_int;
    pub fn uzu_engine_slot_release(e: *mut uzu_engine, slot: u32) -> c_int;
    pub fn uzu_engine_forward_rows(e: *mut uzu_engine, slot: u32, tokens: *const u32, count: u32, rows: *const u32, nrows: u32, out_logits: *mut f32) -> c_int;
    pub fn uzu_engine_debug_layer_outputs(e: *mut uzu_engine, enable: u32, out: *mut f32, capacity_floats: u32, out_count: *mut u32) -> c_int;
    pub fn uzu_engine_batch_begin(e: *mut uzu_engine, sequences: u32) -> c_int;
    pub fn uzu_engine_batch_prefill(e: *mut uzu_engine, sequence: u32, tokens: *const u32, count: u32, out_token: *mut u32) -> c_int;
    pub fn uzu_engine_batch_step(e: *mut uzu_engine, tokens_in: *const u32, tokens_out: *mut u32) -> c_int;
    pub fn uzu_engine_batch_decode_timed(e: *mut uzu_engine, first_tokens: *const u32, steps: u32, out_seconds: *mut f64) -> c_int;
    pub fn uzu_engine_batch_logits(e: *mut uzu_engine, out_logits: *mut u16) -> c_int;
    pub fn uzu_engine_batch_context_length(e: *const uzu_engine, sequence: u32) -> u32;
    pub fn uzu_engine_launch_count(e: *const uzu_engine) -> u64;
    pub fn uzu_engine_debug_step_captures(e: *const uzu_engine) -> u64;
    pub fn uzu_engine_decode_timed(e: *mut uzu_engine, steps: u32, out_seconds: *mut f64) -> c_int;
    pub fn uzu_engine_step_host(e: *mut uzu_engine, token_in: u32, token_out: *mut u32) -> c_int;
    pub fn uzu_engine_decode_mode(e: *const uzu_engine) -> c_int;
    pub fn uzu_engine_decode_mode_reason(e: *const uzu_engine) -> *const c_char;
    pub fn uzu_engine_set_decode_mode(e: *mut uzu_engine, persistent: c_int) -> c_int;
    pub fn uzu_engine_last_logits(e: *mut uzu_engine, out_logits: *mut u16) -> c_int;
    pub fn uzu_engine_speculation_supported(e: *const uzu_engine) -> c_int;
    pub fn uzu_engine_trie_pass(e: *mut uzu_engine, tokens: *const u32, nodes: *const uzu_trie_node, seeds: *const u64, count: u32, sampling: *const uzu_sampling_method, out_tokens: *mut u32, out_logits: *mut u16) -> c_int;
    pub fn uzu_engine_trie_accept(e: *mut uzu_engine, accepted_indices: *const u32, count: u32, next_token: u32) -> c_int;
    pub fn uzu_engine_debug_decode_trace(e: *mut uzu_engine, cta: u32, capacity: u32, out_kinds: *mut u32, out_cycles: *mut u64, out_nops: *mut u32) -> c_int;
    pub fn uzu_engine_time_linears(e: *mut uzu_engine, iters: u32, out_seconds: *mut f64, out_launches: *mut u64) -> c_int;
    pub fn uzu_engine_time_prefill_linears(e: *mut uzu_engine, m: u32, iters: u32, out_seconds: *mut f64, out_flops: *mut f64) -> c_int;
    pub fn uzu_engine_time_linears_select(e: *mut uzu_engine, iters: u32, select: u32, out_seconds: *mut f64, out_launches: *mut u64) -> c_int;
}
