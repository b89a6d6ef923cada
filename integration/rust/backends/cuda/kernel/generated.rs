//! GENERATED by tools/gen_rust_kernels.py from integration/rust/kernel_table.json + include/uzu_b200.h -- do not edit.
//! 72 kernel traits of backends/common/kernel (traitgen.rs:15-81): 20 implemented over libuzu_b200.so, the rest
//! NotSupported stubs. Never compiled here (no rustc in the build image); structure checked by tests/test_rust_kernels_gen.py.
#![allow(clippy::style, clippy::complexity, clippy::perf)]
use crate::{
    backends::common::{kernel::*, BufferArg, BufferArgMut, Encoder},
    data_type::DataType,
};

use super::{addr, addr_mut, dt};
use crate::backends::cuda::{ffi_generated as ffi, Cuda, CudaContext, CudaError};

/// backends/cpu/kernel/activation/activation.rs:7
pub struct CudaActivationKernel;
impl ActivationKernel for CudaActivationKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, in_place: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("Activation: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'output, 'encoder>(&self, input: Option<impl BufferArg<'input, Cuda>>, output: impl BufferArgMut<'output, Cuda>, n: u32, act_type: crate::backends::common::gpu_types::activation_type::ActivationType, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaActivationKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/activation_transform/activation_transform.rs:43
#[allow(non_snake_case, dead_code)]
pub struct CudaActivationTransformKernel { T: DataType, ops: crate::backends::common::gpu_types::ActivationTransformOp, in_place: bool, activation_scale_group_size: u32, sum_group_size: u32 }
impl ActivationTransformKernel for CudaActivationTransformKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, ops: crate::backends::common::gpu_types::ActivationTransformOp, in_place: bool, activation_scale_group_size: u32, sum_group_size: u32) -> Result<Self, CudaError> {
        if T != DataType::BF16 && T != DataType::F32 { return Err(CudaError::NotSupported("ActivationTransform: T must be bf16 or f32")); }
        Ok(Self { T, ops, in_place, activation_scale_group_size, sum_group_size })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'fp_out, 'q_out, 'scales_out, 'group_sums_out, 'rht_factors, 'encoder>(&self, input: Option<impl BufferArg<'input, Cuda>>, fp_out: Option<impl BufferArgMut<'fp_out, Cuda>>, q_out: Option<impl BufferArgMut<'q_out, Cuda>>, scales_out: Option<impl BufferArgMut<'scales_out, Cuda>>, group_sums_out: Option<impl BufferArgMut<'group_sums_out, Cuda>>, rht_factors: impl BufferArg<'rht_factors, Cuda>, batch_size: u32, element_count: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_activation_transform_args {
            input: input.map(addr).unwrap_or(0),
            fp_out: fp_out.map(addr_mut).unwrap_or(0),
            q_out: q_out.map(addr_mut).unwrap_or(0),
            scales_out: scales_out.map(addr_mut).unwrap_or(0),
            group_sums_out: group_sums_out.map(addr_mut).unwrap_or(0),
            rht_factors: addr(rht_factors),
            batch_size: batch_size,
            element_count: element_count,
            ops: self.ops as u32,
            in_place: self.in_place as u32,
            activation_scale_group_size: self.activation_scale_group_size,
            sum_group_size: self.sum_group_size,
            data_type: dt(self.T),
        };
        unsafe { ffi::uzu_activation_transform_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/attention/ancestor_attention.rs:7
pub struct CudaAncestorAttentionKernel;
impl AncestorAttentionKernel for CudaAncestorAttentionKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, HEAD_DIM: u32, num_heads: u32) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("AncestorAttention: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'prefix_kv, 'node_kv, 'current_qkv, 'cosines, 'sines, 'node_metadata, 'ancestor_indices, 'ancestor_counts, 'node_indices, 'output, 'encoder>(&self, prefix_kv: impl BufferArg<'prefix_kv, Cuda>, node_kv: impl BufferArgMut<'node_kv, Cuda>, current_qkv: impl BufferArg<'current_qkv, Cuda>, cosines: impl BufferArg<'cosines, Cuda>, sines: impl BufferArg<'sines, Cuda>, node_metadata: impl BufferArg<'node_metadata, Cuda>, ancestor_indices: impl BufferArg<'ancestor_indices, Cuda>, ancestor_counts: impl BufferArg<'ancestor_counts, Cuda>, node_indices: impl BufferArg<'node_indices, Cuda>, output: impl BufferArgMut<'output, Cuda>, rows: u32, prefix_length: u32, ancestor_stride: u32, node_capacity: u32, max_depth: u32, scale: f32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaAncestorAttentionKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/attention/attention_fallback.rs:10
pub struct CudaAttentionFallbackScatterScoresKernel;
impl AttentionFallbackScatterScoresKernel for CudaAttentionFallbackScatterScoresKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, is_kv_cache_ring: bool, is_causal: bool, is_trie: bool, is_sliding_window: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("AttentionFallbackScatterScores: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'group_scores, 'scores, 'trie, 'encoder>(&self, group_scores: impl BufferArg<'group_scores, Cuda>, scores: impl BufferArgMut<'scores, Cuda>, ring_params: Option<crate::backends::common::gpu_types::ring::RingParams>, trie: Option<impl BufferArg<'trie, Cuda>>, sliding_window_size: Option<u32>, group_index: u32, gqa_factor: u32, sequence_length: u32, suffix_length: u32, total_elements: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaAttentionFallbackScatterScoresKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/attention/attention_fallback.rs:77
pub struct CudaAttentionFallbackScatterValuesKernel;
impl AttentionFallbackScatterValuesKernel for CudaAttentionFallbackScatterValuesKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("AttentionFallbackScatterValues: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'group_output, 'out, 'encoder>(&self, group_output: impl BufferArg<'group_output, Cuda>, out: impl BufferArgMut<'out, Cuda>, group_index: u32, gqa_factor: u32, suffix_length: u32, num_heads: u32, head_dim: u32, total_elements: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaAttentionFallbackScatterValuesKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/attention/attention_prepare.rs:34
#[allow(non_snake_case, dead_code)]
pub struct CudaAttentionPrepareKernel { ElementT: DataType, RopeT: DataType, has_kv: bool, has_rope: bool }
impl AttentionPrepareKernel for CudaAttentionPrepareKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, ElementT: DataType, RopeT: DataType, has_kv: bool, has_rope: bool) -> Result<Self, CudaError> {
        if ElementT != DataType::BF16 { return Err(CudaError::NotSupported("AttentionPrepare: ElementT must be bf16")); }
        Ok(Self { ElementT, RopeT, has_kv, has_rope })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'qkv, 'queries, 'keys, 'values, 'cosines, 'sines, 'encoder>(&self, qkv: impl BufferArg<'qkv, Cuda>, queries: impl BufferArgMut<'queries, Cuda>, keys: Option<impl BufferArgMut<'keys, Cuda>>, values: Option<impl BufferArgMut<'values, Cuda>>, cosines: Option<impl BufferArg<'cosines, Cuda>>, sines: Option<impl BufferArg<'sines, Cuda>>, num_q_heads: u32, num_kv_heads: Option<u32>, head_dim: u32, rope_dim: Option<u32>, kv_token_offset: Option<u32>, batch_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_attention_prepare_args {
            qkv: addr(qkv),
            queries: addr_mut(queries),
            keys: keys.map(addr_mut).unwrap_or(0),
            values: values.map(addr_mut).unwrap_or(0),
            cosines: cosines.map(addr).unwrap_or(0),
            sines: sines.map(addr).unwrap_or(0),
            num_q_heads: num_q_heads,
            num_kv_heads: num_kv_heads.unwrap_or_default(),
            head_dim: head_dim,
            rope_dim: rope_dim.unwrap_or_default(),
            kv_token_offset: kv_token_offset.unwrap_or_default(),
            batch_dim: batch_dim,
            has_kv: self.has_kv as u32,
            has_rope: self.has_rope as u32,
            dynamic_position: 0,
        };
        unsafe { ffi::uzu_attention_prepare_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/attention/attention_single_pass.rs:10
#[allow(non_snake_case, dead_code)]
pub struct CudaAttentionSinglePassKernel { T: DataType, HEAD_DIM: u32, has_sinks: bool, is_kv_cache_ring: bool, is_causal: bool, is_trie: bool, is_sliding_window: bool }
impl AttentionSinglePassKernel for CudaAttentionSinglePassKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, HEAD_DIM: u32, has_sinks: bool, is_kv_cache_ring: bool, is_causal: bool, is_trie: bool, is_sliding_window: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("AttentionSinglePass: T must be bf16")); }
        if HEAD_DIM == 512 { return Err(CudaError::NotSupported("head_dim 512 (AttentionFallback path)")); }
        Ok(Self { T, HEAD_DIM, has_sinks, is_kv_cache_ring, is_causal, is_trie, is_sliding_window })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'queries, 'keys, 'values, 'out, 'trie, 'sinks, 'encoder>(&self, queries: impl BufferArg<'queries, Cuda>, keys: impl BufferArg<'keys, Cuda>, values: impl BufferArg<'values, Cuda>, out: impl BufferArgMut<'out, Cuda>, gqa_factor: u32, sequence_length: u32, k_head_stride: u32, k_seq_stride: u32, v_head_stride: u32, v_seq_stride: u32, ring_params: Option<crate::backends::common::gpu_types::ring::RingParams>, scale: f32, trie: Option<impl BufferArg<'trie, Cuda>>, sliding_window_size: Option<u32>, sinks: Option<impl BufferArg<'sinks, Cuda>>, num_heads: u32, suffix_length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_attention_args {
            queries: addr(queries),
            keys: addr(keys),
            values: addr(values),
            out: addr_mut(out),
            sums: 0,
            maxs: 0,
            gqa_factor: gqa_factor,
            sequence_length: sequence_length,
            k_head_stride: k_head_stride,
            k_seq_stride: k_seq_stride,
            v_head_stride: v_head_stride,
            v_seq_stride: v_seq_stride,
            ring_params: ring_params.map(|r| ffi::uzu_ring_params { ring_offset: r.ring_offset, ring_length: r.ring_length }).unwrap_or(ffi::uzu_ring_params { ring_offset: 0, ring_length: 0 }),
            scale: scale,
            trie: trie.map(addr).unwrap_or(0),
            sliding_window_size: sliding_window_size.unwrap_or_default(),
            sinks: sinks.map(addr).unwrap_or(0),
            num_heads: num_heads,
            suffix_length: suffix_length,
            head_dim: self.HEAD_DIM,
            has_sinks: self.has_sinks as u32,
            is_kv_cache_ring: self.is_kv_cache_ring as u32,
            is_causal: self.is_causal as u32,
            is_trie: self.is_trie as u32,
            is_sliding_window: self.is_sliding_window as u32,
            dynamic_position: 0,
        };
        unsafe { ffi::uzu_attention_single_pass_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/attention/attention_two_pass.rs:12
#[allow(non_snake_case, dead_code)]
pub struct CudaAttentionTwoPass1Kernel { T: DataType, HEAD_DIM: u32, has_sinks: bool, is_kv_cache_ring: bool, is_causal: bool, is_trie: bool, is_sliding_window: bool }
impl AttentionTwoPass1Kernel for CudaAttentionTwoPass1Kernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, HEAD_DIM: u32, has_sinks: bool, is_kv_cache_ring: bool, is_causal: bool, is_trie: bool, is_sliding_window: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("AttentionTwoPass1: T must be bf16")); }
        if HEAD_DIM == 512 { return Err(CudaError::NotSupported("head_dim 512 (AttentionFallback path)")); }
        Ok(Self { T, HEAD_DIM, has_sinks, is_kv_cache_ring, is_causal, is_trie, is_sliding_window })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'queries, 'keys, 'values, 'out, 'sums, 'maxs, 'trie, 'sinks, 'encoder>(&self, queries: impl BufferArg<'queries, Cuda>, keys: impl BufferArg<'keys, Cuda>, values: impl BufferArg<'values, Cuda>, out: impl BufferArgMut<'out, Cuda>, sums: impl BufferArgMut<'sums, Cuda>, maxs: impl BufferArgMut<'maxs, Cuda>, gqa_factor: u32, sequence_length: u32, k_head_stride: u32, k_seq_stride: u32, v_head_stride: u32, v_seq_stride: u32, ring_params: Option<crate::backends::common::gpu_types::ring::RingParams>, scale: f32, num_heads: u32, suffix_length: u32, trie: Option<impl BufferArg<'trie, Cuda>>, sliding_window_size: Option<u32>, sinks: Option<impl BufferArg<'sinks, Cuda>>, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_attention_args {
            queries: addr(queries),
            keys: addr(keys),
            values: addr(values),
            out: addr_mut(out),
            sums: addr_mut(sums),
            maxs: addr_mut(maxs),
            gqa_factor: gqa_factor,
            sequence_length: sequence_length,
            k_head_stride: k_head_stride,
            k_seq_stride: k_seq_stride,
            v_head_stride: v_head_stride,
            v_seq_stride: v_seq_stride,
            ring_params: ring_params.map(|r| ffi::uzu_ring_params { ring_offset: r.ring_offset, ring_length: r.ring_length }).unwrap_or(ffi::uzu_ring_params { ring_offset: 0, ring_length: 0 }),
            scale: scale,
            trie: trie.map(addr).unwrap_or(0),
            sliding_window_size: sliding_window_size.unwrap_or_default(),
            sinks: sinks.map(addr).unwrap_or(0),
            num_heads: num_heads,
            suffix_length: suffix_length,
            head_dim: self.HEAD_DIM,
            has_sinks: self.has_sinks as u32,
            is_kv_cache_ring: self.is_kv_cache_ring as u32,
            is_causal: self.is_causal as u32,
            is_trie: self.is_trie as u32,
            is_sliding_window: self.is_sliding_window as u32,
            dynamic_position: 0,
        };
        unsafe { ffi::uzu_attention_two_pass1_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/attention/attention_two_pass.rs:143
#[allow(non_snake_case, dead_code)]
pub struct CudaAttentionTwoPass2Kernel { T: DataType, HEAD_DIM: u32 }
impl AttentionTwoPass2Kernel for CudaAttentionTwoPass2Kernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, HEAD_DIM: u32) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("AttentionTwoPass2: T must be bf16")); }
        Ok(Self { T, HEAD_DIM })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'partials, 'sums, 'maxs, 'out, 'encoder>(&self, partials: impl BufferArg<'partials, Cuda>, sums: impl BufferArg<'sums, Cuda>, maxs: impl BufferArg<'maxs, Cuda>, out: impl BufferArgMut<'out, Cuda>, num_heads: u32, suffix_length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_attention_two_pass2_args {
            partials: addr(partials),
            sums: addr(sums),
            maxs: addr(maxs),
            out: addr_mut(out),
            num_heads: num_heads,
            suffix_length: suffix_length,
            head_dim: self.HEAD_DIM,
        };
        unsafe { ffi::uzu_attention_two_pass2_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/gdn/tree_verify/tree_gram.rs:9
pub struct CudaBuildTreeGramKernel;
impl BuildTreeGramKernel for CudaBuildTreeGramKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, USE_MXU: bool, use_h0: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("BuildTreeGram: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'q, 'k, 'trie, 'prefix, 'beta, 'h0, 'h0_idx, 'a_packed, 'qkd, 'a_inv, 'kh0, 'encoder>(&self, q: impl BufferArg<'q, Cuda>, k: impl BufferArg<'k, Cuda>, trie: impl BufferArg<'trie, Cuda>, prefix: impl BufferArg<'prefix, Cuda>, beta: impl BufferArg<'beta, Cuda>, h0: Option<impl BufferArg<'h0, Cuda>>, h0_idx: Option<impl BufferArg<'h0_idx, Cuda>>, a_packed: impl BufferArgMut<'a_packed, Cuda>, qkd: impl BufferArgMut<'qkd, Cuda>, a_inv: impl BufferArgMut<'a_inv, Cuda>, kh0: Option<impl BufferArgMut<'kh0, Cuda>>, scale: f32, batch_size: u32, tree_size: u32, k_heads: u32, value_heads: u32, head_k_dim: u32, head_v_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaBuildTreeGramKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/tree_verify/out.rs:7
pub struct CudaBuildTreeOutKernel;
impl BuildTreeOutKernel for CudaBuildTreeOutKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, QKT: DataType, OutputT: DataType, use_mxu: bool, transposed_h0: bool, use_h0: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("BuildTreeOut: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'q, 'prefix, 'qkd, 'u, 'h0, 'h0_indices, 'o, 'encoder>(&self, q: impl BufferArg<'q, Cuda>, prefix: impl BufferArg<'prefix, Cuda>, qkd: impl BufferArg<'qkd, Cuda>, u: impl BufferArg<'u, Cuda>, h0: Option<impl BufferArg<'h0, Cuda>>, h0_indices: Option<impl BufferArg<'h0_indices, Cuda>>, o: impl BufferArgMut<'o, Cuda>, scale: f32, batch_size: u32, tree_size: u32, qk_heads: u32, value_heads: u32, head_k_dim: u32, head_v_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaBuildTreeOutKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/tree_verify/prefix.rs:5
pub struct CudaBuildTreePrefixKernel;
impl BuildTreePrefixKernel for CudaBuildTreePrefixKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("BuildTreePrefix: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'trie, 'log_decay, 'prefix, 'encoder>(&self, trie: impl BufferArg<'trie, Cuda>, log_decay: impl BufferArg<'log_decay, Cuda>, prefix: impl BufferArgMut<'prefix, Cuda>, batch_size: u32, tree_size: u32, value_heads: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaBuildTreePrefixKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/sampling/context_ring_update.rs:5
pub struct CudaContextRingUpdateKernel;
impl ContextRingUpdateKernel for CudaContextRingUpdateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("ContextRingUpdate: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'context_ring, 'encoder>(&self, input: impl BufferArg<'input, Cuda>, context_ring: impl BufferArgMut<'context_ring, Cuda>, suffix_repetition_length: u32, input_length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaContextRingUpdateKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/conv1d.rs:41
pub struct CudaConv1dDecodeKernel;
impl Conv1dDecodeKernel for CudaConv1dDecodeKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, has_bias: bool, state_in_place: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("Conv1dDecode: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x, 'w, 'b, 'state, 'x_out, 'b_out, 'c_out, 'next_state, 'encoder>(&self, x: impl BufferArg<'x, Cuda>, w: impl BufferArg<'w, Cuda>, b: Option<impl BufferArg<'b, Cuda>>, state: Option<impl BufferArg<'state, Cuda>>, x_out: impl BufferArgMut<'x_out, Cuda>, b_out: impl BufferArgMut<'b_out, Cuda>, c_out: impl BufferArgMut<'c_out, Cuda>, next_state: impl BufferArgMut<'next_state, Cuda>, kernel_size: u32, row_stride: u32, state_stride: u32, num_channels: u32, suffix_len: u32, inner_dim: u32, proj_dim: u32, activation_type: crate::backends::common::gpu_types::activation_type::ActivationType, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaConv1dDecodeKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/conv1d.rs:7
pub struct CudaConv1dPackKernel;
impl Conv1dPackKernel for CudaConv1dPackKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, StateT: DataType, InputT: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("Conv1dPack: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'state_in, 'x, 'padded, 'encoder>(&self, state_in: impl BufferArg<'state_in, Cuda>, x: impl BufferArg<'x, Cuda>, padded: impl BufferArgMut<'padded, Cuda>, state_stride: u32, row_stride: u32, suffix_len: u32, num_channels: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaConv1dPackKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/conv1d.rs:129
pub struct CudaConv1dScanKernel;
impl Conv1dScanKernel for CudaConv1dScanKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, has_bias: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("Conv1dScan: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'padded, 'w, 'b, 'x_out, 'b_out, 'c_out, 'state_out, 'encoder>(&self, padded: impl BufferArg<'padded, Cuda>, w: impl BufferArg<'w, Cuda>, b: Option<impl BufferArg<'b, Cuda>>, x_out: impl BufferArgMut<'x_out, Cuda>, b_out: impl BufferArgMut<'b_out, Cuda>, c_out: impl BufferArgMut<'c_out, Cuda>, state_out: impl BufferArgMut<'state_out, Cuda>, suffix_len: u32, kernel_size: u32, row_stride: u32, state_stride: u32, num_channels: u32, inner_dim: u32, proj_dim: u32, activation_type: crate::backends::common::gpu_types::activation_type::ActivationType, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaConv1dScanKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/tree_verify/conv_scan.rs:7
pub struct CudaConvTreeScanKernel;
impl ConvTreeScanKernel for CudaConvTreeScanKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, kernel_size: u32, has_bias: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("ConvTreeScan: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_proj, 'conv_weight, 'bias, 'base_state, 'parents, 'out_proj, 'suffix_state, 'encoder>(&self, in_proj: impl BufferArg<'in_proj, Cuda>, conv_weight: impl BufferArg<'conv_weight, Cuda>, bias: Option<impl BufferArg<'bias, Cuda>>, base_state: impl BufferArg<'base_state, Cuda>, parents: impl BufferArg<'parents, Cuda>, out_proj: impl BufferArgMut<'out_proj, Cuda>, suffix_state: impl BufferArgMut<'suffix_state, Cuda>, suffix_len: u32, total_proj_dim: u32, conv_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaConvTreeScanKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/conv_scan.rs:16
pub struct CudaDeltaNetConvScanKernel;
impl DeltaNetConvScanKernel for CudaDeltaNetConvScanKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, has_bias: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("DeltaNetConvScan: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'conv_padded, 'conv_weight, 'bias, 'in_proj, 'state_out, 'encoder>(&self, conv_padded: impl BufferArg<'conv_padded, Cuda>, conv_weight: impl BufferArg<'conv_weight, Cuda>, bias: Option<impl BufferArg<'bias, Cuda>>, in_proj: impl BufferArgMut<'in_proj, Cuda>, state_out: impl BufferArgMut<'state_out, Cuda>, suffix_len: u32, kernel_size: u32, row_stride: u32, state_stride: u32, conv_dim: u32, out_stride: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaDeltaNetConvScanKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/conv_update.rs:8
#[allow(non_snake_case, dead_code)]
pub struct CudaDeltaNetConvUpdateKernel { T: DataType, has_bias: bool }
impl DeltaNetConvUpdateKernel for CudaDeltaNetConvUpdateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, has_bias: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("DeltaNetConvUpdate: T must be bf16")); }
        Ok(Self { T, has_bias })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'conv_weight, 'bias, 'in_out, 'state, 'encoder>(&self, conv_weight: impl BufferArg<'conv_weight, Cuda>, bias: Option<impl BufferArg<'bias, Cuda>>, in_out: impl BufferArgMut<'in_out, Cuda>, state: impl BufferArgMut<'state, Cuda>, kernel_size: u32, conv_dim: u32, state_stride: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_delta_net_conv_update_args {
            conv_weight: addr(conv_weight),
            bias: bias.map(addr).unwrap_or(0),
            in_out: addr_mut(in_out),
            state: addr_mut(state),
            kernel_size: kernel_size,
            conv_dim: conv_dim,
            state_stride: state_stride,
            has_bias: self.has_bias as u32,
        };
        unsafe { ffi::uzu_delta_net_conv_update_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/gdn/norm_gate.rs:16
pub struct CudaDeltaNetNormGateKernel;
impl DeltaNetNormGateKernel for CudaDeltaNetNormGateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("DeltaNetNormGate: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_out, 'in_proj, 'norm_weight, 'encoder>(&self, in_out: impl BufferArgMut<'in_out, Cuda>, in_proj: impl BufferArg<'in_proj, Cuda>, norm_weight: impl BufferArg<'norm_weight, Cuda>, num_v_heads: u32, head_v_dim: u32, value_dim: u32, conv_dim: u32, total_proj_dim: u32, norm_epsilon: f32, suffix_len: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaDeltaNetNormGateKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/prefill.rs:7
pub struct CudaDeltaNetPrefillKernel;
impl DeltaNetPrefillKernel for CudaDeltaNetPrefillKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, HEAD_K_DIM: u32) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("DeltaNetPrefill: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'q_norm, 'k_norm, 'beta_buf, 'decay_buf, 'in_proj, 'state, 'out, 'encoder>(&self, q_norm: impl BufferArg<'q_norm, Cuda>, k_norm: impl BufferArg<'k_norm, Cuda>, beta_buf: impl BufferArg<'beta_buf, Cuda>, decay_buf: impl BufferArg<'decay_buf, Cuda>, in_proj: impl BufferArg<'in_proj, Cuda>, state: impl BufferArgMut<'state, Cuda>, out: impl BufferArgMut<'out, Cuda>, num_v_heads: u32, num_k_heads: u32, head_v_dim: u32, key_dim: u32, value_dim: u32, suffix_len: u32, num_dv_groups: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaDeltaNetPrefillKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/prefill_prep.rs:8
pub struct CudaDeltaNetPrefillPrepKernel;
impl DeltaNetPrefillPrepKernel for CudaDeltaNetPrefillPrepKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, QKT: DataType, HEAD_K_DIM: u32, write_log_decay: bool, write_compact_v: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("DeltaNetPrefillPrep: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_proj, 'a_log, 'dt_bias, 'q_norm_out, 'k_norm_out, 'compact_v_out, 'beta_out, 'decay_out, 'encoder>(&self, in_proj: impl BufferArg<'in_proj, Cuda>, a_log: impl BufferArg<'a_log, Cuda>, dt_bias: impl BufferArg<'dt_bias, Cuda>, q_norm_out: impl BufferArgMut<'q_norm_out, Cuda>, k_norm_out: impl BufferArgMut<'k_norm_out, Cuda>, compact_v_out: Option<impl BufferArgMut<'compact_v_out, Cuda>>, beta_out: impl BufferArgMut<'beta_out, Cuda>, decay_out: impl BufferArgMut<'decay_out, Cuda>, num_v_heads: u32, num_k_heads: u32, key_dim: u32, value_dim: u32, suffix_len: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaDeltaNetPrefillPrepKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/update.rs:13
#[allow(non_snake_case, dead_code)]
pub struct CudaDeltaNetUpdateKernel { T: DataType, HEAD_K_DIM: u32 }
impl DeltaNetUpdateKernel for CudaDeltaNetUpdateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, HEAD_K_DIM: u32) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("DeltaNetUpdate: T must be bf16")); }
        Ok(Self { T, HEAD_K_DIM })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_proj, 'a_log, 'dt_bias, 'norm_weight, 'state, 'out, 'encoder>(&self, in_proj: impl BufferArg<'in_proj, Cuda>, a_log: impl BufferArg<'a_log, Cuda>, dt_bias: impl BufferArg<'dt_bias, Cuda>, norm_weight: impl BufferArg<'norm_weight, Cuda>, state: impl BufferArgMut<'state, Cuda>, out: impl BufferArgMut<'out, Cuda>, num_v_heads: u32, num_k_heads: u32, head_v_dim: u32, key_dim: u32, value_dim: u32, norm_epsilon: f32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_delta_net_update_args {
            in_proj: addr(in_proj),
            a_log: addr(a_log),
            dt_bias: addr(dt_bias),
            norm_weight: addr(norm_weight),
            state: addr_mut(state),
            out: addr_mut(out),
            num_v_heads: num_v_heads,
            num_k_heads: num_k_heads,
            head_v_dim: head_v_dim,
            key_dim: key_dim,
            value_dim: value_dim,
            norm_epsilon: norm_epsilon,
            head_k_dim: self.HEAD_K_DIM,
        };
        unsafe { ffi::uzu_delta_net_update_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/embedding/full_precision_embedding.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaFullPrecisionEmbeddingLookupKernel { T: DataType }
impl FullPrecisionEmbeddingLookupKernel for CudaFullPrecisionEmbeddingLookupKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("FullPrecisionEmbeddingLookup: T must be bf16")); }
        Ok(Self { T })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'token_ids, 'weights, 'output, 'encoder>(&self, token_ids: impl BufferArg<'token_ids, Cuda>, weights: impl BufferArg<'weights, Cuda>, output: impl BufferArgMut<'output, Cuda>, batch_size: u32, vocab_size: u32, model_dim: u32, input_scale: f32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_full_precision_embedding_lookup_encode(encoder.as_command_buffer_mut().raw(), addr(token_ids), addr(weights), addr_mut(output), batch_size, vocab_size, model_dim, input_scale) };
    }
}

/// backends/cpu/kernel/gated_act_mul/gated_act_mul.rs:13
#[allow(non_snake_case, dead_code)]
pub struct CudaGatedActMulKernel { T: DataType, ops: crate::backends::common::gpu_types::GatedActMulOp, interleaved: bool, use_hadamard: bool, activation_scale_group_size: u32, sum_group_size: u32 }
impl GatedActMulKernel for CudaGatedActMulKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, ops: crate::backends::common::gpu_types::GatedActMulOp, interleaved: bool, use_hadamard: bool, activation_scale_group_size: u32, sum_group_size: u32) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("GatedActMul: T must be bf16")); }
        if use_hadamard { return Err(CudaError::NotSupported("GatedActMul with a fused Hadamard")); }
        if ops != crate::backends::common::gpu_types::GatedActMulOp::FullPrecision { return Err(CudaError::NotSupported("GatedActMul with int8 activation outputs (A8)")); }
        Ok(Self { T, ops, interleaved, use_hadamard, activation_scale_group_size, sum_group_size })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'act_operand, 'value_operand, 'fp_out, 'q_out, 'scales_out, 'group_sums_out, 'hadamard_factors, 'encoder>(&self, act_operand: impl BufferArg<'act_operand, Cuda>, value_operand: Option<impl BufferArg<'value_operand, Cuda>>, fp_out: Option<impl BufferArgMut<'fp_out, Cuda>>, q_out: Option<impl BufferArgMut<'q_out, Cuda>>, scales_out: Option<impl BufferArgMut<'scales_out, Cuda>>, group_sums_out: Option<impl BufferArgMut<'group_sums_out, Cuda>>, hadamard_factors: Option<impl BufferArg<'hadamard_factors, Cuda>>, gated_dim: u32, batch_dim: u32, value_offset: u32, value_row_stride: u32, act_type: crate::backends::common::gpu_types::ActivationType, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_gated_act_mul_args {
            act_operand: addr(act_operand),
            value_operand: value_operand.map(addr).unwrap_or(0),
            fp_out: fp_out.map(addr_mut).unwrap_or(0),
            gated_dim: gated_dim,
            batch_dim: batch_dim,
            value_offset: value_offset,
            value_row_stride: value_row_stride,
            act_type: act_type as u32,
            interleaved: self.interleaved as u32,
        };
        unsafe { ffi::uzu_gated_act_mul_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/attention/kv_cache_update.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaKVCacheUpdateKernel { T: DataType }
impl KVCacheUpdateKernel for CudaKVCacheUpdateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("KVCacheUpdate: T must be bf16")); }
        Ok(Self { T })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_place_keys, 'in_place_values, 'encoder>(&self, in_place_keys: impl BufferArgMut<'in_place_keys, Cuda>, in_place_values: impl BufferArgMut<'in_place_values, Cuda>, copies: &[crate::backends::common::gpu_types::kv_cache_update::Copy], copy_count: u32, element_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_kv_cache_update_args {
            in_place_keys: addr_mut(in_place_keys),
            in_place_values: addr_mut(in_place_values),
            copies: copies.as_ptr() as *const ffi::uzu_kv_copy,
            copy_count: copy_count,
            element_dim: element_dim,
        };
        unsafe { ffi::uzu_kv_cache_update_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/logit_transform/logit_transform.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaLogitTransformKernel { T: DataType, has_soft_cap: bool }
impl LogitTransformKernel for CudaLogitTransformKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, has_soft_cap: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("LogitTransform: T must be bf16")); }
        Ok(Self { T, has_soft_cap })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'logits, 'encoder>(&self, logits: impl BufferArgMut<'logits, Cuda>, length: u32, scale: f32, soft_cap: f32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_logit_transform_encode(encoder.as_command_buffer_mut().raw(), addr_mut(logits), length, scale, soft_cap, self.has_soft_cap as u32) };
    }
}

/// backends/cpu/kernel/moe/scatter_buckets.rs:7
pub struct CudaMoeBlockBasesFromPartialsKernel;
impl MoeBlockBasesFromPartialsKernel for CudaMoeBlockBasesFromPartialsKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeBlockBasesFromPartials: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'partials, 'block_bases, 'block_alloc, 'encoder>(&self, partials: impl BufferArg<'partials, Cuda>, block_bases: impl BufferArgMut<'block_bases, Cuda>, block_alloc: impl BufferArgMut<'block_alloc, Cuda>, e_input: u32, num_blocks: u32, num_tiles: u32, capacity_per_expert: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeBlockBasesFromPartialsKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_map.rs:22
pub struct CudaMoeBuildTileMapKernel;
impl MoeBuildTileMapKernel for CudaMoeBuildTileMapKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeBuildTileMap: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'offsets, 'tile_row_offsets, 'tile_counts, 'tile_map, 'encoder>(&self, offsets: impl BufferArg<'offsets, Cuda>, tile_row_offsets: impl BufferArg<'tile_row_offsets, Cuda>, tile_counts: impl BufferArg<'tile_counts, Cuda>, tile_map: impl BufferArgMut<'tile_map, Cuda>, e: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeBuildTileMapKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/counts_offsets_fused.rs:3
pub struct CudaMoeCountsOffsetsFusedKernel;
impl MoeCountsOffsetsFusedKernel for CudaMoeCountsOffsetsFusedKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeCountsOffsetsFused: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'topk_ids, 'offsets, 'sum_k_out, 'partials, 'encoder>(&self, topk_ids: impl BufferArg<'topk_ids, Cuda>, offsets: impl BufferArgMut<'offsets, Cuda>, sum_k_out: impl BufferArgMut<'sum_k_out, Cuda>, partials: impl BufferArgMut<'partials, Cuda>, t_input: u32, e_input: u32, k_input: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeCountsOffsetsFusedKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/experts_two_pass_decode.rs:32
pub struct CudaMoeExpertsDecodeDownFused2DKernel;
impl MoeExpertsDecodeDownFused2DKernel for CudaMoeExpertsDecodeDownFused2DKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, AccumT: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeExpertsDecodeDownFused2D: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'hidden, 'row_expert_map, 'w2_all, 'down_biases, 'y_out, 'encoder>(&self, hidden: impl BufferArg<'hidden, Cuda>, row_expert_map: impl BufferArg<'row_expert_map, Cuda>, w2_all: impl BufferArg<'w2_all, Cuda>, down_biases: impl BufferArg<'down_biases, Cuda>, y_out: impl BufferArgMut<'y_out, Cuda>, total_rows: u32, d_model: u32, d_ff: u32, e: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeExpertsDecodeDownFused2DKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/experts_two_pass_decode.rs:7
pub struct CudaMoeExpertsDecodePassAKernel;
impl MoeExpertsDecodePassAKernel for CudaMoeExpertsDecodePassAKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, gating_sel: u32) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeExpertsDecodePassA: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x_perm, 'expert_offsets, 'w13_all, 'hidden_out, 'up_biases, 'tile_map, '__dsl_indirect_dispatch_buffer, 'encoder>(&self, x_perm: impl BufferArg<'x_perm, Cuda>, expert_offsets: impl BufferArg<'expert_offsets, Cuda>, w13_all: impl BufferArg<'w13_all, Cuda>, hidden_out: impl BufferArgMut<'hidden_out, Cuda>, up_biases: impl BufferArg<'up_biases, Cuda>, d_model: u32, d_ff: u32, e: u32, gate_clip_min: f32, gate_clip_max: f32, up_clip_min: f32, up_clip_max: f32, silu_alpha: f32, tile_map: impl BufferArg<'tile_map, Cuda>, __dsl_indirect_dispatch_buffer: impl BufferArg<'__dsl_indirect_dispatch_buffer, Cuda>, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeExpertsDecodePassAKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/experts_two_pass_prefill.rs:7
pub struct CudaMoeExpertsPrefillPassAKernel;
impl MoeExpertsPrefillPassAKernel for CudaMoeExpertsPrefillPassAKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, gating_sel: u32) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeExpertsPrefillPassA: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x_perm, 'expert_offsets, 'w13_all, 'up_biases, 'hidden_out, 'tile_map, '__dsl_indirect_dispatch_buffer, 'encoder>(&self, x_perm: impl BufferArg<'x_perm, Cuda>, expert_offsets: impl BufferArg<'expert_offsets, Cuda>, w13_all: impl BufferArg<'w13_all, Cuda>, up_biases: impl BufferArg<'up_biases, Cuda>, hidden_out: impl BufferArgMut<'hidden_out, Cuda>, d_model: u32, d_ff: u32, e: u32, gate_clip_min: f32, gate_clip_max: f32, up_clip_min: f32, up_clip_max: f32, silu_alpha: f32, tile_map: impl BufferArg<'tile_map, Cuda>, __dsl_indirect_dispatch_buffer: impl BufferArg<'__dsl_indirect_dispatch_buffer, Cuda>, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeExpertsPrefillPassAKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/experts_two_pass_prefill.rs:32
pub struct CudaMoeExpertsPrefillPassBKernel;
impl MoeExpertsPrefillPassBKernel for CudaMoeExpertsPrefillPassBKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeExpertsPrefillPassB: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'hidden, 'expert_offsets, 'w2_all, 'down_biases, 'output, 'tile_map, '__dsl_indirect_dispatch_buffer, 'encoder>(&self, hidden: impl BufferArg<'hidden, Cuda>, expert_offsets: impl BufferArg<'expert_offsets, Cuda>, w2_all: impl BufferArg<'w2_all, Cuda>, down_biases: impl BufferArg<'down_biases, Cuda>, output: impl BufferArgMut<'output, Cuda>, d_model: u32, d_ff: u32, e: u32, tile_map: impl BufferArg<'tile_map, Cuda>, __dsl_indirect_dispatch_buffer: impl BufferArg<'__dsl_indirect_dispatch_buffer, Cuda>, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeExpertsPrefillPassBKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/finalize.rs:7
pub struct CudaMoeFinalizeKernel;
impl MoeFinalizeKernel for CudaMoeFinalizeKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeFinalize: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'tok2row, 'probs, 'y_partial, 'y, 'encoder>(&self, tok2row: impl BufferArg<'tok2row, Cuda>, probs: impl BufferArg<'probs, Cuda>, y_partial: impl BufferArg<'y_partial, Cuda>, y: impl BufferArgMut<'y, Cuda>, t_count: u32, d_model: u32, k_input: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeFinalizeKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/gather.rs:57
pub struct CudaMoeGatherXPerm1DKernel;
impl MoeGatherXPerm1DKernel for CudaMoeGatherXPerm1DKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeGatherXPerm1D: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x, 'bucketed_ids, 'x_perm, 'sumk_buf, 'encoder>(&self, x: impl BufferArg<'x, Cuda>, bucketed_ids: impl BufferArg<'bucketed_ids, Cuda>, x_perm: impl BufferArgMut<'x_perm, Cuda>, sumk_buf: impl BufferArg<'sumk_buf, Cuda>, d_model: u32, t: u32, k: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeGatherXPerm1DKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/gather.rs:43
pub struct CudaMoeGatherXPerm2DKernel;
impl MoeGatherXPerm2DKernel for CudaMoeGatherXPerm2DKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeGatherXPerm2D: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x, 'bucketed_ids, 'x_perm, 'sumk_buf, 'encoder>(&self, x: impl BufferArg<'x, Cuda>, bucketed_ids: impl BufferArg<'bucketed_ids, Cuda>, x_perm: impl BufferArgMut<'x_perm, Cuda>, sumk_buf: impl BufferArg<'sumk_buf, Cuda>, d_model: u32, t: u32, k: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeGatherXPerm2DKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_pass_a.rs:23
pub struct CudaMoePassABuildRowMapKernel;
impl MoePassABuildRowMapKernel for CudaMoePassABuildRowMapKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoePassABuildRowMap: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'expert_offsets, 'row_expert_map, 'encoder>(&self, expert_offsets: impl BufferArg<'expert_offsets, Cuda>, row_expert_map: impl BufferArgMut<'row_expert_map, Cuda>, total_rows: u32, e: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoePassABuildRowMapKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_pass_a.rs:33
pub struct CudaMoePassABuildTileMapKernel;
impl MoePassABuildTileMapKernel for CudaMoePassABuildTileMapKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoePassABuildTileMap: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'expert_offsets, 'tile_offsets, 'row_expert_map, 'tile_map, 'encoder>(&self, expert_offsets: impl BufferArg<'expert_offsets, Cuda>, tile_offsets: impl BufferArg<'tile_offsets, Cuda>, row_expert_map: impl BufferArg<'row_expert_map, Cuda>, tile_map: impl BufferArgMut<'tile_map, Cuda>, total_rows: u32, h_blocks: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoePassABuildTileMapKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_pass_a.rs:3
pub struct CudaMoePassATileCountsKernel;
impl MoePassATileCountsKernel for CudaMoePassATileCountsKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoePassATileCounts: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'expert_offsets, 'tile_counts, 'encoder>(&self, expert_offsets: impl BufferArg<'expert_offsets, Cuda>, tile_counts: impl BufferArgMut<'tile_counts, Cuda>, e: u32, h_blocks: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoePassATileCountsKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_pass_a.rs:13
pub struct CudaMoePassATileScanKernel;
impl MoePassATileScanKernel for CudaMoePassATileScanKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoePassATileScan: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'tile_counts, 'tile_offsets, 'total_tiles, 'encoder>(&self, tile_counts: impl BufferArg<'tile_counts, Cuda>, tile_offsets: impl BufferArgMut<'tile_offsets, Cuda>, total_tiles: impl BufferArgMut<'total_tiles, Cuda>, e: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoePassATileScanKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_pass_a.rs:45
pub struct CudaMoePassAWriteDispatchArgsKernel;
impl MoePassAWriteDispatchArgsKernel for CudaMoePassAWriteDispatchArgsKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoePassAWriteDispatchArgs: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'total_tiles, 'dispatch_args, 'encoder>(&self, total_tiles: impl BufferArg<'total_tiles, Cuda>, dispatch_args: impl BufferArgMut<'dispatch_args, Cuda>, num_tiles_y: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoePassAWriteDispatchArgsKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/router_topk.rs:7
pub struct CudaMoeRouterTopKKernel;
impl MoeRouterTopKKernel for CudaMoeRouterTopKKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, ScalarT: DataType, has_biases: bool, has_router_scales: bool, has_per_expert_scales: bool, has_router_input_scale: bool, normalize_router_input: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeRouterTopK: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'weight, 'bias, 'router_scale, 'per_expert_scale, 'topk_ids, 'topk_probs, 'encoder>(&self, input: impl BufferArg<'input, Cuda>, weight: impl BufferArg<'weight, Cuda>, bias: Option<impl BufferArg<'bias, Cuda>>, router_scale: Option<impl BufferArg<'router_scale, Cuda>>, per_expert_scale: Option<impl BufferArg<'per_expert_scale, Cuda>>, topk_ids: impl BufferArgMut<'topk_ids, Cuda>, topk_probs: impl BufferArgMut<'topk_probs, Cuda>, t: u32, d_model: u32, e: u32, k: u32, renorm: bool, router_norm_epsilon: Option<f32>, router_input_scale: Option<f32>, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeRouterTopKKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/scatter_buckets.rs:20
pub struct CudaMoeScatterBucketsMapKernel;
impl MoeScatterBucketsMapKernel for CudaMoeScatterBucketsMapKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeScatterBucketsMap: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'topk_ids, 'topk_probs, 'offsets, 'block_bases, 'block_alloc, 'out_ids, 'out_probs, 'tok2row, 'encoder>(&self, topk_ids: impl BufferArg<'topk_ids, Cuda>, topk_probs: impl BufferArg<'topk_probs, Cuda>, offsets: impl BufferArg<'offsets, Cuda>, block_bases: impl BufferArg<'block_bases, Cuda>, block_alloc: impl BufferArg<'block_alloc, Cuda>, out_ids: impl BufferArgMut<'out_ids, Cuda>, out_probs: impl BufferArgMut<'out_probs, Cuda>, t: u32, e: u32, k: u32, num_blocks: u32, num_tiles: u32, tok2row: impl BufferArgMut<'tok2row, Cuda>, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeScatterBucketsMapKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_map.rs:3
pub struct CudaMoeTileCountsKernel;
impl MoeTileCountsKernel for CudaMoeTileCountsKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeTileCounts: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'offsets, 'tile_counts, 'encoder>(&self, offsets: impl BufferArg<'offsets, Cuda>, tile_counts: impl BufferArgMut<'tile_counts, Cuda>, e: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeTileCountsKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_map.rs:12
pub struct CudaMoeTileScanKernel;
impl MoeTileScanKernel for CudaMoeTileScanKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeTileScan: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'tile_counts, 'tile_row_offsets, 'total_tiles_buf, 'encoder>(&self, tile_counts: impl BufferArg<'tile_counts, Cuda>, tile_row_offsets: impl BufferArgMut<'tile_row_offsets, Cuda>, total_tiles_buf: impl BufferArgMut<'total_tiles_buf, Cuda>, e: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeTileScanKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/moe/tiles_map.rs:33
pub struct CudaMoeWriteDispatchArgsKernel;
impl MoeWriteDispatchArgsKernel for CudaMoeWriteDispatchArgsKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("MoeWriteDispatchArgs: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'total_tiles_buf, 'dispatch_args, 'encoder>(&self, total_tiles_buf: impl BufferArg<'total_tiles_buf, Cuda>, dispatch_args: impl BufferArgMut<'dispatch_args, Cuda>, num_tiles_n: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaMoeWriteDispatchArgsKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/normalization/normalization.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaNormalizationKernel { InputT: DataType, AffineT: DataType, OutputT: DataType, AccumT: DataType, in_place: bool, subtract_mean: bool, full_layer: bool, copy_to_shortcut: bool, residual_add: bool, use_hadamard: bool, scale_residual_sum: bool, scale_output: bool, has_biases: bool, has_scales: bool }
impl NormalizationKernel for CudaNormalizationKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, InputT: DataType, AffineT: DataType, OutputT: DataType, AccumT: DataType, in_place: bool, subtract_mean: bool, full_layer: bool, copy_to_shortcut: bool, residual_add: bool, use_hadamard: bool, scale_residual_sum: bool, scale_output: bool, has_biases: bool, has_scales: bool) -> Result<Self, CudaError> {
        if InputT != DataType::BF16 { return Err(CudaError::NotSupported("Normalization: InputT must be bf16")); }
        if OutputT != DataType::BF16 { return Err(CudaError::NotSupported("Normalization: OutputT must be bf16")); }
        if use_hadamard { return Err(CudaError::NotSupported("in-norm Hadamard (Mirai RHT)")); }
        Ok(Self { InputT, AffineT, OutputT, AccumT, in_place, subtract_mean, full_layer, copy_to_shortcut, residual_add, use_hadamard, scale_residual_sum, scale_output, has_biases, has_scales })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'scales, 'biases, 'output, 'shortcut, 'hadamard_factors, 'encoder>(&self, input: Option<impl BufferArg<'input, Cuda>>, scales: Option<impl BufferArg<'scales, Cuda>>, biases: Option<impl BufferArg<'biases, Cuda>>, output: impl BufferArgMut<'output, Cuda>, shortcut: Option<impl BufferArgMut<'shortcut, Cuda>>, hadamard_factors: Option<impl BufferArg<'hadamard_factors, Cuda>>, batch_size: u32, element_count: u32, epsilon: f32, scale_offset: f32, post_layer_scalar: f32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_normalization_args {
            input: input.map(addr).unwrap_or(0),
            scales: scales.map(addr).unwrap_or(0),
            biases: biases.map(addr).unwrap_or(0),
            output: addr_mut(output),
            shortcut: shortcut.map(addr_mut).unwrap_or(0),
            hadamard_factors: hadamard_factors.map(addr).unwrap_or(0),
            batch_size: batch_size,
            element_count: element_count,
            epsilon: epsilon,
            scale_offset: scale_offset,
            post_layer_scalar: post_layer_scalar,
            in_place: self.in_place as u32,
            subtract_mean: self.subtract_mean as u32,
            full_layer: self.full_layer as u32,
            copy_to_shortcut: self.copy_to_shortcut as u32,
            residual_add: self.residual_add as u32,
            use_hadamard: self.use_hadamard as u32,
            scale_residual_sum: self.scale_residual_sum as u32,
            scale_output: self.scale_output as u32,
            has_biases: self.has_biases as u32,
            has_scales: self.has_scales as u32,
        };
        unsafe { ffi::uzu_normalization_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/pooling/pooling.rs:7
pub struct CudaPoolingMeanKernel;
impl PoolingMeanKernel for CudaPoolingMeanKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("PoolingMean: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'output, 'encoder>(&self, input: impl BufferArg<'input, Cuda>, output: impl BufferArgMut<'output, Cuda>, seq_len: u32, hidden_dim: u32, batch_size: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaPoolingMeanKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/attention/qkv_norm.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaQKVNormKernel { InputT: DataType, ScaleT: DataType, OutputT: DataType, AccumT: DataType, in_place: bool, has_scales: bool }
impl QKVNormKernel for CudaQKVNormKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, InputT: DataType, ScaleT: DataType, OutputT: DataType, AccumT: DataType, in_place: bool, has_scales: bool) -> Result<Self, CudaError> {
        if InputT != DataType::BF16 { return Err(CudaError::NotSupported("QKVNorm: InputT must be bf16")); }
        if OutputT != DataType::BF16 { return Err(CudaError::NotSupported("QKVNorm: OutputT must be bf16")); }
        Ok(Self { InputT, ScaleT, OutputT, AccumT, in_place, has_scales })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'qkv_input, 'scales, 'qkv_output, 'encoder>(&self, qkv_input: Option<impl BufferArg<'qkv_input, Cuda>>, scales: Option<impl BufferArg<'scales, Cuda>>, qkv_output: impl BufferArgMut<'qkv_output, Cuda>, batch_size: u32, total_heads: u32, head_dim: u32, epsilon: f32, scale_offset: f32, head_offset: u32, head_count: u32, full_layer: bool, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_qkv_norm_args {
            qkv_input: qkv_input.map(addr).unwrap_or(0),
            scales: scales.map(addr).unwrap_or(0),
            qkv_output: addr_mut(qkv_output),
            batch_size: batch_size,
            total_heads: total_heads,
            head_dim: head_dim,
            epsilon: epsilon,
            scale_offset: scale_offset,
            head_offset: head_offset,
            head_count: head_count,
            full_layer: full_layer as u32,
            in_place: self.in_place as u32,
            has_scales: self.has_scales as u32,
        };
        unsafe { ffi::uzu_qkv_norm_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/embedding/quant_embedding.rs:11
#[allow(non_snake_case, dead_code)]
pub struct CudaQuantizedEmbeddingLookupKernel { T: DataType, group_size: u32, quantization_mode: crate::backends::common::gpu_types::QuantizationMode, quantization_method: crate::backends::common::gpu_types::QuantizationMethod, use_hadamard: bool }
impl QuantizedEmbeddingLookupKernel for CudaQuantizedEmbeddingLookupKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, group_size: u32, quantization_mode: crate::backends::common::gpu_types::QuantizationMode, quantization_method: crate::backends::common::gpu_types::QuantizationMethod, use_hadamard: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("QuantizedEmbeddingLookup: T must be bf16")); }
        if use_hadamard { return Err(CudaError::NotSupported("quantized embedding with an output Hadamard")); }
        Ok(Self { T, group_size, quantization_mode, quantization_method, use_hadamard })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'token_ids, 'weights, 'scales, 'zero_points, 'biases, 'output, 'output_hadamard_factors, 'encoder>(&self, token_ids: impl BufferArg<'token_ids, Cuda>, weights: impl BufferArg<'weights, Cuda>, scales: impl BufferArg<'scales, Cuda>, zero_points: Option<impl BufferArg<'zero_points, Cuda>>, biases: Option<impl BufferArg<'biases, Cuda>>, output: impl BufferArgMut<'output, Cuda>, output_hadamard_factors: Option<impl BufferArg<'output_hadamard_factors, Cuda>>, batch_size: u32, vocab_size: u32, model_dim: u32, input_scale: f32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_quantized_embedding_lookup_args {
            token_ids: addr(token_ids),
            weights: addr(weights),
            scales: addr(scales),
            zero_points: zero_points.map(addr).unwrap_or(0),
            biases: biases.map(addr).unwrap_or(0),
            output: addr_mut(output),
            batch_size: batch_size,
            vocab_size: vocab_size,
            model_dim: model_dim,
            input_scale: input_scale,
            group_size: self.group_size,
            quantization_mode: self.quantization_mode as u32,
            quantization_method: self.quantization_method as u32,
        };
        unsafe { ffi::uzu_quantized_embedding_lookup_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/sampling/repetition_penalty.rs:7
pub struct CudaRepetitionPenaltyKernel;
impl RepetitionPenaltyKernel for CudaRepetitionPenaltyKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("RepetitionPenalty: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'original_logits, 'logits_copy, 'context_ring, 'token_ids, 'encoder>(&self, original_logits: impl BufferArg<'original_logits, Cuda>, logits_copy: impl BufferArgMut<'logits_copy, Cuda>, context_ring: impl BufferArg<'context_ring, Cuda>, token_ids: impl BufferArg<'token_ids, Cuda>, repetition_penalty: f32, suffix_repetition_length: u32, vocab_size: u32, sampling_start: u32, sampling_length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaRepetitionPenaltyKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/ssd_prefill.rs:31
pub struct CudaSSDPrefillKernel;
impl SSDPrefillKernel for CudaSSDPrefillKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("SSDPrefill: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x, 'dt_raw, 'b, 'c, 'd, 'z, 'state, 'y, 'encoder>(&self, x: impl BufferArg<'x, Cuda>, dt_raw: impl BufferArg<'dt_raw, Cuda>, b: impl BufferArg<'b, Cuda>, c: impl BufferArg<'c, Cuda>, d: impl BufferArg<'d, Cuda>, z: impl BufferArg<'z, Cuda>, state: impl BufferArgMut<'state, Cuda>, y: impl BufferArgMut<'y, Cuda>, suffix_len: u32, group_size: u32, state_size: u32, x_strides: &[u32; 3], dt_strides: &[u32; 2], cb_strides: &[u32; 3], state_strides: &[u32; 3], num_heads: u32, head_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaSSDPrefillKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/ssd_prefill.rs:7
pub struct CudaSSDPrefill64Kernel;
impl SSDPrefill64Kernel for CudaSSDPrefill64Kernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("SSDPrefill64: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x, 'dt_raw, 'b, 'c, 'd, 'z, 'state, 'y, 'encoder>(&self, x: impl BufferArg<'x, Cuda>, dt_raw: impl BufferArg<'dt_raw, Cuda>, b: impl BufferArg<'b, Cuda>, c: impl BufferArg<'c, Cuda>, d: impl BufferArg<'d, Cuda>, z: impl BufferArg<'z, Cuda>, state: impl BufferArgMut<'state, Cuda>, y: impl BufferArgMut<'y, Cuda>, suffix_len: u32, group_size: u32, state_size: u32, x_strides: &[u32; 3], dt_strides: &[u32; 2], cb_strides: &[u32; 3], state_strides: &[u32; 3], num_heads: u32, head_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaSSDPrefill64Kernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/ssd_update.rs:7
pub struct CudaSSDUpdateKernel;
impl SSDUpdateKernel for CudaSSDUpdateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, state_in_place: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("SSDUpdate: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'x, 'dt_raw, 'b, 'c, 'd, 'z, 'state, 'y, 'next_state, 'encoder>(&self, x: impl BufferArg<'x, Cuda>, dt_raw: impl BufferArg<'dt_raw, Cuda>, b: impl BufferArg<'b, Cuda>, c: impl BufferArg<'c, Cuda>, d: impl BufferArg<'d, Cuda>, z: impl BufferArg<'z, Cuda>, state: Option<impl BufferArg<'state, Cuda>>, y: impl BufferArgMut<'y, Cuda>, next_state: impl BufferArgMut<'next_state, Cuda>, group_size: u32, state_size: u32, x_strides: &[u32; 3], dt_strides: &[u32; 2], cb_strides: &[u32; 3], state_strides: &[u32; 4], b_size: u32, h_size: u32, dh_size: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaSSDUpdateKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/short_conv/short_conv.rs:114
pub struct CudaShortConvDecodeKernel;
impl ShortConvDecodeKernel for CudaShortConvDecodeKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, WeightT: DataType, has_bias: bool, state_in_place: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("ShortConvDecode: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_proj, 'w, 'b, 'state, 'out, 'next_state, 'encoder>(&self, in_proj: impl BufferArg<'in_proj, Cuda>, w: impl BufferArg<'w, Cuda>, b: Option<impl BufferArg<'b, Cuda>>, state: Option<impl BufferArg<'state, Cuda>>, out: impl BufferArgMut<'out, Cuda>, next_state: impl BufferArgMut<'next_state, Cuda>, suffix_len: u32, kernel_size: u32, in_proj_stride: u32, state_stride: u32, model_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaShortConvDecodeKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/short_conv/short_conv.rs:7
pub struct CudaShortConvPackKernel;
impl ShortConvPackKernel for CudaShortConvPackKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("ShortConvPack: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'state_in, 'in_proj, 'padded, 'encoder>(&self, state_in: impl BufferArg<'state_in, Cuda>, in_proj: impl BufferArg<'in_proj, Cuda>, padded: impl BufferArgMut<'padded, Cuda>, state_stride: u32, suffix_len: u32, in_proj_stride: u32, model_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaShortConvPackKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/short_conv/short_conv.rs:44
pub struct CudaShortConvPrefillKernel;
impl ShortConvPrefillKernel for CudaShortConvPrefillKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, WeightT: DataType, has_bias: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("ShortConvPrefill: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'padded, 'in_proj, 'w, 'b, 'out, 'state_out, 'encoder>(&self, padded: impl BufferArg<'padded, Cuda>, in_proj: impl BufferArg<'in_proj, Cuda>, w: impl BufferArg<'w, Cuda>, b: Option<impl BufferArg<'b, Cuda>>, out: impl BufferArgMut<'out, Cuda>, state_out: impl BufferArgMut<'state_out, Cuda>, suffix_len: u32, kernel_size: u32, in_proj_stride: u32, state_stride: u32, model_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaShortConvPrefillKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/short_conv/short_conv.rs:185
pub struct CudaShortConvTrieKernel;
impl ShortConvTrieKernel for CudaShortConvTrieKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, WeightT: DataType, has_bias: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("ShortConvTrie: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'in_proj, 'w, 'b, 'base_state, 'parents, 'out, 'suffix_state, 'encoder>(&self, in_proj: impl BufferArg<'in_proj, Cuda>, w: impl BufferArg<'w, Cuda>, b: Option<impl BufferArg<'b, Cuda>>, base_state: impl BufferArg<'base_state, Cuda>, parents: impl BufferArg<'parents, Cuda>, out: impl BufferArgMut<'out, Cuda>, suffix_state: impl BufferArgMut<'suffix_state, Cuda>, suffix_len: u32, kernel_size: u32, in_proj_stride: u32, state_stride: u32, model_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaShortConvTrieKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/attention/sigmoid_gate.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaSigmoidGateKernel { T: DataType }
impl SigmoidGateKernel for CudaSigmoidGateKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("SigmoidGate: T must be bf16")); }
        Ok(Self { T })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'gate, 'output, 'encoder>(&self, gate: impl BufferArg<'gate, Cuda>, output: impl BufferArgMut<'output, Cuda>, total_elements: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_sigmoid_gate_encode(encoder.as_command_buffer_mut().raw(), addr(gate), addr_mut(output), total_elements) };
    }
}

/// backends/cpu/kernel/softmax/softmax.rs:7
pub struct CudaSoftmaxKernel;
impl SoftmaxKernel for CudaSoftmaxKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, has_sinks: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("Softmax: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'values, 'sinks, 'encoder>(&self, values: impl BufferArgMut<'values, Cuda>, sinks: Option<impl BufferArg<'sinks, Cuda>>, row_length: u32, outer_dim: u32, batch_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaSoftmaxKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/ssm/split_inproj.rs:7
pub struct CudaSplitInProjKernel;
impl SplitInProjKernel for CudaSplitInProjKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("SplitInProj: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'conv_out, 'z_out, 'dt_out, 'z_bias, 'encoder>(&self, input: impl BufferArg<'input, Cuda>, conv_out: impl BufferArgMut<'conv_out, Cuda>, z_out: impl BufferArgMut<'z_out, Cuda>, dt_out: impl BufferArgMut<'dt_out, Cuda>, z_bias: impl BufferArg<'z_bias, Cuda>, suffix_length: u32, total_dim: u32, conv_dim: u32, inner_dim: u32, num_heads: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaSplitInProjKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/gdn/tree_verify/state_advance.rs:7
pub struct CudaStateAdvanceKernel;
impl StateAdvanceKernel for CudaStateAdvanceKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, HEAD_K_DIM: u32, num_v_heads: u32, num_k_heads: u32) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("StateAdvance: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'k_norm, 'v, 'log_decay_buf, 'beta_buf, 'accepted_indices, 'state, 'encoder>(&self, k_norm: impl BufferArg<'k_norm, Cuda>, v: impl BufferArg<'v, Cuda>, log_decay_buf: impl BufferArg<'log_decay_buf, Cuda>, beta_buf: impl BufferArg<'beta_buf, Cuda>, accepted_indices: impl BufferArg<'accepted_indices, Cuda>, state: impl BufferArgMut<'state, Cuda>, accepted_len: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaStateAdvanceKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/tensor_add_bias/tensor_add_bias.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaTensorAddBiasKernel { T: DataType, BiasT: DataType, in_place: bool }
impl TensorAddBiasKernel for CudaTensorAddBiasKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, BiasT: DataType, in_place: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("TensorAddBias: T must be bf16")); }
        if BiasT != DataType::BF16 { return Err(CudaError::NotSupported("TensorAddBias: BiasT must be bf16")); }
        Ok(Self { T, BiasT, in_place })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'bias, 'output, 'encoder>(&self, input: Option<impl BufferArg<'input, Cuda>>, bias: impl BufferArg<'bias, Cuda>, output: impl BufferArgMut<'output, Cuda>, num_cols: u32, length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_tensor_add_bias_encode(encoder.as_command_buffer_mut().raw(), input.map(addr).unwrap_or(0), addr(bias), addr_mut(output), num_cols, length) };
    }
}

/// backends/cpu/kernel/tensor_add_scale/tensor_add_scale.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaTensorAddScaleKernel { T: DataType, in_place: bool }
impl TensorAddScaleKernel for CudaTensorAddScaleKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, in_place: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("TensorAddScale: T must be bf16")); }
        Ok(Self { T, in_place })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'input, 'bias, 'output, 'encoder>(&self, input: Option<impl BufferArg<'input, Cuda>>, bias: impl BufferArg<'bias, Cuda>, output: impl BufferArgMut<'output, Cuda>, num_cols: u32, length: u32, scale: f32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_tensor_add_scale_encode(encoder.as_command_buffer_mut().raw(), input.map(addr).unwrap_or(0), addr(bias), addr_mut(output), num_cols, length, scale) };
    }
}

/// backends/cpu/kernel/tensor_add_swap/tensor_add_swap.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaTensorAddSwapKernel { T: DataType }
impl TensorAddSwapKernel for CudaTensorAddSwapKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("TensorAddSwap: T must be bf16")); }
        Ok(Self { T })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'skip_buffer, 'main_buffer, 'encoder>(&self, skip_buffer: impl BufferArgMut<'skip_buffer, Cuda>, main_buffer: impl BufferArgMut<'main_buffer, Cuda>, length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_tensor_add_swap_encode(encoder.as_command_buffer_mut().raw(), addr_mut(skip_buffer), addr_mut(main_buffer), length) };
    }
}

/// backends/cpu/kernel/tensor_copy/tensor_copy.rs:7
#[allow(non_snake_case, dead_code)]
pub struct CudaTensorCopyKernel { T: DataType }
impl TensorCopyKernel for CudaTensorCopyKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("TensorCopy: T must be bf16")); }
        Ok(Self { T })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'src_buffer, 'dst_buffer, 'encoder>(&self, src_buffer: impl BufferArg<'src_buffer, Cuda>, dst_buffer: impl BufferArgMut<'dst_buffer, Cuda>, length: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unsafe { ffi::uzu_tensor_copy_encode(encoder.as_command_buffer_mut().raw(), addr(src_buffer), addr_mut(dst_buffer), length) };
    }
}

/// backends/cpu/kernel/gdn/tree_verify/tree_update_solve.rs:9
pub struct CudaTreeUpdateSolveKernel;
impl TreeUpdateSolveKernel for CudaTreeUpdateSolveKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, BV: u32, use_h0: bool) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("TreeUpdateSolve: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'kh0, 'v, 'prefix, 'beta, 'a_packed, 'a_inv, 'h0_idx, 'u, 'encoder>(&self, kh0: Option<impl BufferArg<'kh0, Cuda>>, v: impl BufferArg<'v, Cuda>, prefix: impl BufferArg<'prefix, Cuda>, beta: impl BufferArg<'beta, Cuda>, a_packed: impl BufferArg<'a_packed, Cuda>, a_inv: impl BufferArg<'a_inv, Cuda>, h0_idx: Option<impl BufferArg<'h0_idx, Cuda>>, u: impl BufferArgMut<'u, Cuda>, batch_size: u32, tree_size: u32, value_heads: u32, head_v_dim: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaTreeUpdateSolveKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/sampling/unified_sampling.rs:13
#[allow(non_snake_case, dead_code)]
pub struct CudaUnifiedSamplingKernel { T: DataType, is_stochastic: bool, has_bitmask: bool, has_temperature: bool, has_top_k: bool, has_top_p: bool, has_min_p: bool }
impl UnifiedSamplingKernel for CudaUnifiedSamplingKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext, T: DataType, is_stochastic: bool, has_bitmask: bool, has_temperature: bool, has_top_k: bool, has_top_p: bool, has_min_p: bool) -> Result<Self, CudaError> {
        if T != DataType::BF16 { return Err(CudaError::NotSupported("UnifiedSampling: T must be bf16")); }
        Ok(Self { T, is_stochastic, has_bitmask, has_temperature, has_top_k, has_top_p, has_min_p })
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'logits, 'output, 'seeds, 'bitmask, 'encoder>(&self, logits: impl BufferArg<'logits, Cuda>, output: impl BufferArgMut<'output, Cuda>, seeds: Option<impl BufferArg<'seeds, Cuda>>, bitmask: Option<impl BufferArg<'bitmask, Cuda>>, temperature: Option<f32>, top_k: Option<u32>, top_p: Option<f32>, min_p: Option<f32>, vocab_size: u32, batch_size: u32, encoder: &'encoder mut Encoder<Cuda>) {
        let args = ffi::uzu_unified_sampling_args {
            logits: addr(logits),
            output: addr_mut(output),
            seeds: seeds.map(addr).unwrap_or(0),
            bitmask: bitmask.map(addr).unwrap_or(0),
            temperature: temperature.unwrap_or_default(),
            top_k: top_k.unwrap_or_default(),
            top_p: top_p.unwrap_or_default(),
            min_p: min_p.unwrap_or_default(),
            vocab_size: vocab_size,
            batch_size: batch_size,
            is_stochastic: self.is_stochastic as u32,
            has_bitmask: self.has_bitmask as u32,
            has_temperature: self.has_temperature as u32,
            has_top_k: self.has_top_k as u32,
            has_top_p: self.has_top_p as u32,
            has_min_p: self.has_min_p as u32,
        };
        unsafe { ffi::uzu_unified_sampling_encode(encoder.as_command_buffer_mut().raw(), &args) };
    }
}

/// backends/cpu/kernel/weaver/weaver_frontier_insert_children.rs:16
pub struct CudaWeaverFrontierInsertChildrenKernel;
impl WeaverFrontierInsertChildrenKernel for CudaWeaverFrontierInsertChildrenKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("WeaverFrontierInsertChildren: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'packed_tree, 'node_metadata, 'node_valid, 'child_ids, 'child_logprobs, 'frontier, 'encoder>(&self, packed_tree: impl BufferArg<'packed_tree, Cuda>, node_metadata: impl BufferArg<'node_metadata, Cuda>, node_valid: impl BufferArg<'node_valid, Cuda>, child_ids: impl BufferArg<'child_ids, Cuda>, child_logprobs: impl BufferArg<'child_logprobs, Cuda>, frontier: impl BufferArgMut<'frontier, Cuda>, frontier_capacity: u32, tree_slot_count: u32, node_count: u32, expand_width: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaWeaverFrontierInsertChildrenKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/weaver/weaver_frontier_select.rs:7
pub struct CudaWeaverFrontierSelectKernel;
impl WeaverFrontierSelectKernel for CudaWeaverFrontierSelectKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("WeaverFrontierSelect: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'frontier, 'packed_tree, 'slot_ancestors, 'node_token_ids, 'node_metadata, 'node_ancestor_indices, 'node_valid, 'candidate_pool_ids, 'candidate_pool_logits, 'node_candidate_ids, 'node_candidate_logits, 'encoder>(&self, frontier: impl BufferArgMut<'frontier, Cuda>, packed_tree: impl BufferArgMut<'packed_tree, Cuda>, slot_ancestors: impl BufferArgMut<'slot_ancestors, Cuda>, node_token_ids: impl BufferArgMut<'node_token_ids, Cuda>, node_metadata: impl BufferArgMut<'node_metadata, Cuda>, node_ancestor_indices: impl BufferArgMut<'node_ancestor_indices, Cuda>, node_valid: impl BufferArgMut<'node_valid, Cuda>, candidate_pool_ids: impl BufferArg<'candidate_pool_ids, Cuda>, candidate_pool_logits: impl BufferArg<'candidate_pool_logits, Cuda>, node_candidate_ids: impl BufferArgMut<'node_candidate_ids, Cuda>, node_candidate_logits: impl BufferArgMut<'node_candidate_logits, Cuda>, frontier_capacity: u32, tree_slot_count: u32, node_count: u32, batch_start_slot: u32, ancestor_stride: u32, max_depth: u32, lookahead_count: u32, candidate_depth_count: u32, candidates_per_depth: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaWeaverFrontierSelectKernel cannot be constructed")
    }
}

/// backends/cpu/kernel/weaver/weaver_top_children.rs:9
pub struct CudaWeaverTopChildrenKernel;
impl WeaverTopChildrenKernel for CudaWeaverTopChildrenKernel {
    type Backend = Cuda;
    #[allow(non_snake_case, unused_variables, clippy::too_many_arguments)]
    fn new(context: &CudaContext) -> Result<Self, CudaError> {
        Err(CudaError::NotSupported("WeaverTopChildren: outside the CUDA decode hot path"))
    }
    #[allow(unused_variables, clippy::too_many_arguments)]
    fn encode<'residual_logits, 'candidate_logits, 'candidate_ids, 'depth_seeds, 'node_metadata, 'output_token_ids, 'output_model_logprobs, 'encoder>(&self, residual_logits: impl BufferArg<'residual_logits, Cuda>, candidate_logits: impl BufferArg<'candidate_logits, Cuda>, candidate_ids: impl BufferArg<'candidate_ids, Cuda>, depth_seeds: impl BufferArg<'depth_seeds, Cuda>, node_metadata: impl BufferArg<'node_metadata, Cuda>, output_token_ids: impl BufferArgMut<'output_token_ids, Cuda>, output_model_logprobs: impl BufferArgMut<'output_model_logprobs, Cuda>, rows: u32, candidates: u32, expand_width: u32, vocab_size: u32, encoder: &'encoder mut Encoder<Cuda>) {
        unreachable!("CudaWeaverTopChildrenKernel cannot be constructed")
    }
}

/// `autogen_kernels!()` of this backend (build/cpu/compiler.rs:632-658 emits the CPU one): every generated associated type of `Kernels`.
macro_rules! autogen_cuda_kernels {
    () => {
        type ActivationKernel = crate::backends::cuda::kernel::generated::CudaActivationKernel;
        type ActivationTransformKernel = crate::backends::cuda::kernel::generated::CudaActivationTransformKernel;
        type AncestorAttentionKernel = crate::backends::cuda::kernel::generated::CudaAncestorAttentionKernel;
        type AttentionFallbackScatterScoresKernel = crate::backends::cuda::kernel::generated::CudaAttentionFallbackScatterScoresKernel;
        type AttentionFallbackScatterValuesKernel = crate::backends::cuda::kernel::generated::CudaAttentionFallbackScatterValuesKernel;
        type AttentionPrepareKernel = crate::backends::cuda::kernel::generated::CudaAttentionPrepareKernel;
        type AttentionSinglePassKernel = crate::backends::cuda::kernel::generated::CudaAttentionSinglePassKernel;
        type AttentionTwoPass1Kernel = crate::backends::cuda::kernel::generated::CudaAttentionTwoPass1Kernel;
        type AttentionTwoPass2Kernel = crate::backends::cuda::kernel::generated::CudaAttentionTwoPass2Kernel;
        type BuildTreeGramKernel = crate::backends::cuda::kernel::generated::CudaBuildTreeGramKernel;
        type BuildTreeOutKernel = crate::backends::cuda::kernel::generated::CudaBuildTreeOutKernel;
        type BuildTreePrefixKernel = crate::backends::cuda::kernel::generated::CudaBuildTreePrefixKernel;
        type ContextRingUpdateKernel = crate::backends::cuda::kernel::generated::CudaContextRingUpdateKernel;
        type Conv1dDecodeKernel = crate::backends::cuda::kernel::generated::CudaConv1dDecodeKernel;
        type Conv1dPackKernel = crate::backends::cuda::kernel::generated::CudaConv1dPackKernel;
        type Conv1dScanKernel = crate::backends::cuda::kernel::generated::CudaConv1dScanKernel;
        type ConvTreeScanKernel = crate::backends::cuda::kernel::generated::CudaConvTreeScanKernel;
        type DeltaNetConvScanKernel = crate::backends::cuda::kernel::generated::CudaDeltaNetConvScanKernel;
        type DeltaNetConvUpdateKernel = crate::backends::cuda::kernel::generated::CudaDeltaNetConvUpdateKernel;
        type DeltaNetNormGateKernel = crate::backends::cuda::kernel::generated::CudaDeltaNetNormGateKernel;
        type DeltaNetPrefillKernel = crate::backends::cuda::kernel::generated::CudaDeltaNetPrefillKernel;
        type DeltaNetPrefillPrepKernel = crate::backends::cuda::kernel::generated::CudaDeltaNetPrefillPrepKernel;
        type DeltaNetUpdateKernel = crate::backends::cuda::kernel::generated::CudaDeltaNetUpdateKernel;
        type FullPrecisionEmbeddingLookupKernel = crate::backends::cuda::kernel::generated::CudaFullPrecisionEmbeddingLookupKernel;
        type GatedActMulKernel = crate::backends::cuda::kernel::generated::CudaGatedActMulKernel;
        type KVCacheUpdateKernel = crate::backends::cuda::kernel::generated::CudaKVCacheUpdateKernel;
        type LogitTransformKernel = crate::backends::cuda::kernel::generated::CudaLogitTransformKernel;
        type MoeBlockBasesFromPartialsKernel = crate::backends::cuda::kernel::generated::CudaMoeBlockBasesFromPartialsKernel;
        type MoeBuildTileMapKernel = crate::backends::cuda::kernel::generated::CudaMoeBuildTileMapKernel;
        type MoeCountsOffsetsFusedKernel = crate::backends::cuda::kernel::generated::CudaMoeCountsOffsetsFusedKernel;
        type MoeExpertsDecodeDownFused2DKernel = crate::backends::cuda::kernel::generated::CudaMoeExpertsDecodeDownFused2DKernel;
        type MoeExpertsDecodePassAKernel = crate::backends::cuda::kernel::generated::CudaMoeExpertsDecodePassAKernel;
        type MoeExpertsPrefillPassAKernel = crate::backends::cuda::kernel::generated::CudaMoeExpertsPrefillPassAKernel;
        type MoeExpertsPrefillPassBKernel = crate::backends::cuda::kernel::generated::CudaMoeExpertsPrefillPassBKernel;
        type MoeFinalizeKernel = crate::backends::cuda::kernel::generated::CudaMoeFinalizeKernel;
        type MoeGatherXPerm1DKernel = crate::backends::cuda::kernel::generated::CudaMoeGatherXPerm1DKernel;
        type MoeGatherXPerm2DKernel = crate::backends::cuda::kernel::generated::CudaMoeGatherXPerm2DKernel;
        type MoePassABuildRowMapKernel = crate::backends::cuda::kernel::generated::CudaMoePassABuildRowMapKernel;
        type MoePassABuildTileMapKernel = crate::backends::cuda::kernel::generated::CudaMoePassABuildTileMapKernel;
        type MoePassATileCountsKernel = crate::backends::cuda::kernel::generated::CudaMoePassATileCountsKernel;
        type MoePassATileScanKernel = crate::backends::cuda::kernel::generated::CudaMoePassATileScanKernel;
        type MoePassAWriteDispatchArgsKernel = crate::backends::cuda::kernel::generated::CudaMoePassAWriteDispatchArgsKernel;
        type MoeRouterTopKKernel = crate::backends::cuda::kernel::generated::CudaMoeRouterTopKKernel;
        type MoeScatterBucketsMapKernel = crate::backends::cuda::kernel::generated::CudaMoeScatterBucketsMapKernel;
        type MoeTileCountsKernel = crate::backends::cuda::kernel::generated::CudaMoeTileCountsKernel;
        type MoeTileScanKernel = crate::backends::cuda::kernel::generated::CudaMoeTileScanKernel;
        type MoeWriteDispatchArgsKernel = crate::backends::cuda::kernel::generated::CudaMoeWriteDispatchArgsKernel;
        type NormalizationKernel = crate::backends::cuda::kernel::generated::CudaNormalizationKernel;
        type PoolingMeanKernel = crate::backends::cuda::kernel::generated::CudaPoolingMeanKernel;
        type QKVNormKernel = crate::backends::cuda::kernel::generated::CudaQKVNormKernel;
        type QuantizedEmbeddingLookupKernel = crate::backends::cuda::kernel::generated::CudaQuantizedEmbeddingLookupKernel;
        type RepetitionPenaltyKernel = crate::backends::cuda::kernel::generated::CudaRepetitionPenaltyKernel;
        type SSDPrefillKernel = crate::backends::cuda::kernel::generated::CudaSSDPrefillKernel;
        type SSDPrefill64Kernel = crate::backends::cuda::kernel::generated::CudaSSDPrefill64Kernel;
        type SSDUpdateKernel = crate::backends::cuda::kernel::generated::CudaSSDUpdateKernel;
        type ShortConvDecodeKernel = crate::backends::cuda::kernel::generated::CudaShortConvDecodeKernel;
        type ShortConvPackKernel = crate::backends::cuda::kernel::generated::CudaShortConvPackKernel;
        type ShortConvPrefillKernel = crate::backends::cuda::kernel::generated::CudaShortConvPrefillKernel;
        type ShortConvTrieKernel = crate::backends::cuda::kernel::generated::CudaShortConvTrieKernel;
        type SigmoidGateKernel = crate::backends::cuda::kernel::generated::CudaSigmoidGateKernel;
        type SoftmaxKernel = crate::backends::cuda::kernel::generated::CudaSoftmaxKernel;
        type SplitInProjKernel = crate::backends::cuda::kernel::generated::CudaSplitInProjKernel;
        type StateAdvanceKernel = crate::backends::cuda::kernel::generated::CudaStateAdvanceKernel;
        type TensorAddBiasKernel = crate::backends::cuda::kernel::generated::CudaTensorAddBiasKernel;
        type TensorAddScaleKernel = crate::backends::cuda::kernel::generated::CudaTensorAddScaleKernel;
        type TensorAddSwapKernel = crate::backends::cuda::kernel::generated::CudaTensorAddSwapKernel;
        type TensorCopyKernel = crate::backends::cuda::kernel::generated::CudaTensorCopyKernel;
        type TreeUpdateSolveKernel = crate::backends::cuda::kernel::generated::CudaTreeUpdateSolveKernel;
        type UnifiedSamplingKernel = crate::backends::cuda::kernel::generated::CudaUnifiedSamplingKernel;
        type WeaverFrontierInsertChildrenKernel = crate::backends::cuda::kernel::generated::CudaWeaverFrontierInsertChildrenKernel;
        type WeaverFrontierSelectKernel = crate::backends::cuda::kernel::generated::CudaWeaverFrontierSelectKernel;
        type WeaverTopChildrenKernel = crate::backends::cuda::kernel::generated::CudaWeaverTopChildrenKernel;
    };
}
pub(crate) use autogen_cuda_kernels;
