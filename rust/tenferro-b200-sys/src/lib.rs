//! Raw FFI bindings to `libtenferro_b200.so` (the C ABI declared in `include/tenferro_b200.h`).
//!
//! GENERATED by `gen_sys.py` from the header - do not edit; run the script again instead.
//! Uncompiled here: the machines this library is built on carry no Rust toolchain.  The
//! test suite checks every declaration below against the header by name and arity.
#![allow(non_camel_case_types, non_upper_case_globals, non_snake_case)]

use core::ffi::{c_char, c_int, c_uint, c_ulonglong, c_void};

// ---- enums: C enums cross the boundary as ints, so each is an integer type plus constants
pub type tfb_status = c_int;
pub const TFB_OK: tfb_status = 0;
pub const TFB_ERR_SHAPE_MISMATCH: tfb_status = 1;
pub const TFB_ERR_RANK_MISMATCH: tfb_status = 2;
pub const TFB_ERR_DEVICE: tfb_status = 3;
pub const TFB_ERR_NO_COMPATIBLE_DEVICE: tfb_status = 4;
pub const TFB_ERR_CROSS_MEMORY_SPACE: tfb_status = 5;
pub const TFB_ERR_INVALID_ARGUMENT: tfb_status = 6;
pub const TFB_ERR_STRIDED: tfb_status = 7;

pub type tfb_dtype = c_int;
pub const TFB_F32: tfb_dtype = 0;
pub const TFB_F64: tfb_dtype = 1;
pub const TFB_C32: tfb_dtype = 2;
pub const TFB_C64: tfb_dtype = 3;

pub type tfb_op = c_int;
pub const TFB_OP_BATCHED_GEMM: tfb_op = 0;
pub const TFB_OP_REDUCE: tfb_op = 1;
pub const TFB_OP_TRACE: tfb_op = 2;
pub const TFB_OP_PERMUTE: tfb_op = 3;
pub const TFB_OP_ANTI_TRACE: tfb_op = 4;
pub const TFB_OP_ANTI_DIAG: tfb_op = 5;
pub const TFB_OP_CONTRACT: tfb_op = 6;
pub const TFB_OP_ELEMENTWISE_MUL: tfb_op = 7;

pub type tfb_reduce_op = c_int;
pub const TFB_REDUCE_SUM: tfb_reduce_op = 0;
pub const TFB_REDUCE_MAX: tfb_reduce_op = 1;
pub const TFB_REDUCE_MIN: tfb_reduce_op = 2;

pub type tfb_extension = c_int;
pub const TFB_EXT_CONTRACT: tfb_extension = 0;
pub const TFB_EXT_ELEMENTWISE_MUL: tfb_extension = 1;

pub type tfb_algebra = c_int;
pub const TFB_ALGEBRA_STANDARD: tfb_algebra = 0;
pub const TFB_ALGEBRA_MAX_PLUS: tfb_algebra = 1;
pub const TFB_ALGEBRA_MIN_PLUS: tfb_algebra = 2;

pub type tfb_op_kind = c_int;
pub const TFB_KIND_CONTRACT: tfb_op_kind = 0;
pub const TFB_KIND_BATCHED_GEMM: tfb_op_kind = 1;
pub const TFB_KIND_REDUCE: tfb_op_kind = 2;
pub const TFB_KIND_TRACE: tfb_op_kind = 3;
pub const TFB_KIND_PERMUTE: tfb_op_kind = 4;
pub const TFB_KIND_ELEMENTWISE_MUL: tfb_op_kind = 5;

pub type tfb_space_kind = c_int;
pub const TFB_SPACE_MAIN_MEMORY: tfb_space_kind = 0;
pub const TFB_SPACE_GPU_MEMORY: tfb_space_kind = 1;

pub type tfb_device_kind = c_int;
pub const TFB_DEVICE_CPU: tfb_device_kind = 0;
pub const TFB_DEVICE_CUDA: tfb_device_kind = 1;
pub const TFB_DEVICE_HIP: tfb_device_kind = 2;

// ---- flags
pub const TFB_VIEW_CONJ: u32 = 1;

// ---- opaque handles
#[repr(C)]
pub struct tfb_ctx {
    _private: [u8; 0],
}
#[repr(C)]
pub struct tfb_plan {
    _private: [u8; 0],
}
#[repr(C)]
pub struct tfb_event {
    _private: [u8; 0],
}
#[repr(C)]
pub struct tfb_subscripts {
    _private: [u8; 0],
}
#[repr(C)]
pub struct tfb_tree {
    _private: [u8; 0],
}
#[repr(C)]
pub struct tfb_graph {
    _private: [u8; 0],
}
#[repr(C)]
pub struct tfb_grouped_plan {
    _private: [u8; 0],
}

// ---- plain structs
#[repr(C)]
#[derive(Clone, Copy)]
pub struct tfb_compute_device {
    pub kind: i32,
    pub device_id: i32,
}

#[repr(C)]
#[derive(Clone, Copy)]
pub struct tfb_desc {
    pub op: i32,
    pub reduce_op: i32,
    pub modes_a: *const u32,
    pub n_modes_a: usize,
    pub modes_b: *const u32,
    pub n_modes_b: usize,
    pub modes_c: *const u32,
    pub n_modes_c: usize,
    pub paired: *const u32,
    pub n_pairs: usize,
    pub batch_dims: *const usize,
    pub n_batch_dims: usize,
    pub m: usize,
    pub n: usize,
    pub k: usize,
}

#[repr(C)]
#[derive(Clone, Copy)]
pub struct tfb_view {
    pub base: *mut c_void,
    pub rank: usize,
    pub dims: *const usize,
    pub strides: *const isize,
    pub offset: isize,
    pub flags: u32,
}

#[repr(C)]
#[derive(Clone, Copy)]
pub struct tfb_gemm_problem {
    pub m: i64,
    pub n: i64,
    pub k: i64,
    pub a: *const c_void,
    pub a_rs: i64,
    pub a_cs: i64,
    pub b: *const c_void,
    pub b_rs: i64,
    pub b_cs: i64,
    pub c: *mut c_void,
    pub c_rs: i64,
    pub c_cs: i64,
}

#[link(name = "tenferro_b200")]
extern "C" {
    pub fn tfb_last_error(buf: *mut c_char, cap: usize) -> usize;
    pub fn tfb_version() -> *const c_char;
    pub fn tfb_ctx_create(device_id: c_int, out: *mut *mut tfb_ctx) -> tfb_status;
    pub fn tfb_ctx_destroy(ctx: *mut tfb_ctx) -> tfb_status;
    pub fn tfb_ctx_device(ctx: *const tfb_ctx, device_id: *mut c_int) -> tfb_status;
    pub fn tfb_ctx_stream(ctx: *const tfb_ctx, stream: *mut *mut c_void) -> tfb_status;
    pub fn tfb_ctx_set_stream(ctx: *mut tfb_ctx, stream: *mut c_void) -> tfb_status;
    pub fn tfb_ctx_synchronize(ctx: *mut tfb_ctx) -> tfb_status;
    pub fn tfb_ctx_properties(ctx: *const tfb_ctx, sm_count: *mut c_int, total_mem: *mut usize, cc_major: *mut c_int, cc_minor: *mut c_int) -> tfb_status;
    pub fn tfb_alloc(ctx: *mut tfb_ctx, bytes: usize, out: *mut *mut c_void) -> tfb_status;
    pub fn tfb_free(ctx: *mut tfb_ctx, ptr: *mut c_void) -> tfb_status;
    pub fn tfb_pool_stats(ctx: *mut tfb_ctx, reserved: *mut usize, used: *mut usize) -> tfb_status;
    pub fn tfb_memcpy_h2d_async(ctx: *mut tfb_ctx, dst: *mut c_void, src: *const c_void, bytes: usize) -> tfb_status;
    pub fn tfb_memcpy_d2h_async(ctx: *mut tfb_ctx, dst: *mut c_void, src: *const c_void, bytes: usize) -> tfb_status;
    pub fn tfb_memcpy_d2d_async(ctx: *mut tfb_ctx, dst: *mut c_void, src: *const c_void, bytes: usize) -> tfb_status;
    pub fn tfb_memcpy_h2d_2d_async(ctx: *mut tfb_ctx, dst: *mut c_void, dst_pitch: usize, src: *const c_void, src_pitch: usize, width: usize, height: usize) -> tfb_status;
    pub fn tfb_memcpy_d2h_2d_async(ctx: *mut tfb_ctx, dst: *mut c_void, dst_pitch: usize, src: *const c_void, src_pitch: usize, width: usize, height: usize) -> tfb_status;
    pub fn tfb_memcpy_p2p_async(ctx: *mut tfb_ctx, dst: *mut c_void, dst_device: c_int, src: *const c_void, src_device: c_int, bytes: usize) -> tfb_status;
    pub fn tfb_memset_async(ctx: *mut tfb_ctx, dst: *mut c_void, value: c_int, bytes: usize) -> tfb_status;
    pub fn tfb_host_alloc(bytes: usize, out: *mut *mut c_void) -> tfb_status;
    pub fn tfb_host_free(ptr: *mut c_void) -> tfb_status;
    pub fn tfb_kernel_launch_count() -> c_ulonglong;
    pub fn tfb_ctx_profile_begin(ctx: *mut tfb_ctx) -> tfb_status;
    pub fn tfb_ctx_profile_read(ctx: *mut tfb_ctx, kernel: *const c_char, launches: *mut usize, total_ms: *mut f64) -> tfb_status;
    pub fn tfb_ctx_profile_end(ctx: *mut tfb_ctx) -> tfb_status;
    pub fn tfb_probe_fp64_tflops(ctx: *mut tfb_ctx, tflops: *mut f64) -> tfb_status;
    pub fn tfb_probe_hbm_gbs(ctx: *mut tfb_ctx, gbs: *mut f64) -> tfb_status;
    pub fn tfb_probe_tf32_tflops(ctx: *mut tfb_ctx, tflops: *mut f64) -> tfb_status;
    pub fn tfb_probe_tf32_tflops_sustained(ctx: *mut tfb_ctx, seconds: f64, tflops: *mut f64) -> tfb_status;
    pub fn tfb_probe_mma_issue_cycles(ctx: *mut tfb_ctx, m: c_int, n: c_int, issuers: c_int, issue_cycles: *mut f64, complete_cycles: *mut f64) -> tfb_status;
    pub fn tfb_selftest_wait_expiry(ctx: *mut tfb_ctx, polls: c_uint) -> tfb_status;
    pub fn tfb_ctx_capture_begin(ctx: *mut tfb_ctx) -> tfb_status;
    pub fn tfb_ctx_capture_end(ctx: *mut tfb_ctx, out: *mut *mut tfb_graph) -> tfb_status;
    pub fn tfb_graph_launch(graph: *mut tfb_graph) -> tfb_status;
    pub fn tfb_graph_destroy(graph: *mut tfb_graph);
    pub fn tfb_event_record(ctx: *mut tfb_ctx, out: *mut *mut tfb_event) -> tfb_status;
    pub fn tfb_event_record_completion(ctx: *mut tfb_ctx, out: *mut *mut tfb_event) -> tfb_status;
    pub fn tfb_event_wait(ctx: *mut tfb_ctx, ev: *mut tfb_event) -> tfb_status;
    pub fn tfb_event_synchronize(ev: *mut tfb_event) -> tfb_status;
    pub fn tfb_event_query(ev: *mut tfb_event, ready: *mut c_int) -> tfb_status;
    pub fn tfb_event_elapsed_ms(start: *mut tfb_event, stop: *mut tfb_event, ms: *mut f32) -> tfb_status;
    pub fn tfb_event_destroy(ev: *mut tfb_event) -> tfb_status;
    pub fn tfb_preferred_compute_devices(space_kind: i32, space_id: usize, op_kind: i32, out: *mut tfb_compute_device, cap: usize, n_out: *mut usize) -> tfb_status;
    pub fn tfb_compute_device_format(dev: tfb_compute_device, buf: *mut c_char, cap: usize) -> usize;
    pub fn tfb_has_extension(dtype: i32, ext: i32) -> c_int;
    pub fn tfb_plan_create(ctx: *mut tfb_ctx, desc: *const tfb_desc, dtype: i32, n_shapes: usize, ranks: *const usize, dims: *const *const usize, out: *mut *mut tfb_plan) -> tfb_status;
    pub fn tfb_plan_destroy(plan: *mut tfb_plan) -> tfb_status;
    pub fn tfb_plan_kernel_name(plan: *const tfb_plan) -> *const c_char;
    pub fn tfb_plan_force_kernel(plan: *mut tfb_plan, kernel: c_int) -> tfb_status;
    pub fn tfb_plan_set_algebra(plan: *mut tfb_plan, algebra: i32) -> tfb_status;
    pub fn tfb_has_extension_for_algebra(algebra: i32, dtype: i32, ext: i32) -> c_int;
    pub fn tfb_execute(plan: *mut tfb_plan, alpha: *const c_void, n_inputs: usize, inputs: *const tfb_view, beta: *const c_void, output: *const tfb_view) -> tfb_status;
    pub fn tfb_reduce_static(ctx: *mut tfb_ctx, dtype: i32, reduce_op: i32, modes_a: *const u32, n_modes_a: usize, a: *const tfb_view, modes_c: *const u32, n_modes_c: usize, c: *const tfb_view, alpha: *const c_void, beta: *const c_void) -> tfb_status;
    pub fn tfb_grouped_gemm(ctx: *mut tfb_ctx, dtype: i32, n_problems: usize, problems: *const tfb_gemm_problem, alpha: *const c_void, beta: *const c_void) -> tfb_status;
    pub fn tfb_grouped_plan_create(ctx: *mut tfb_ctx, dtype: i32, n_problems: usize, problems: *const tfb_gemm_problem, out: *mut *mut tfb_grouped_plan) -> tfb_status;
    pub fn tfb_grouped_plan_execute(plan: *mut tfb_grouped_plan, alpha: *const c_void, beta: *const c_void) -> tfb_status;
    pub fn tfb_grouped_plan_destroy(plan: *mut tfb_grouped_plan);
    pub fn tfb_subscripts_new(n_inputs: usize, input_ranks: *const usize, inputs: *const *const u32, output_rank: usize, output: *const u32, out: *mut *mut tfb_subscripts) -> tfb_status;
    pub fn tfb_subscripts_parse(notation: *const c_char, out: *mut *mut tfb_subscripts) -> tfb_status;
    pub fn tfb_subscripts_destroy(subs: *mut tfb_subscripts) -> tfb_status;
    pub fn tfb_subscripts_n_inputs(subs: *const tfb_subscripts) -> usize;
    pub fn tfb_subscripts_input(subs: *const tfb_subscripts, i: usize, labels: *mut u32, cap: usize) -> usize;
    pub fn tfb_subscripts_output(subs: *const tfb_subscripts, labels: *mut u32, cap: usize) -> usize;
    pub fn tfb_subscripts_has_order(subs: *const tfb_subscripts) -> c_int;
    pub fn tfb_tree_optimize(subs: *const tfb_subscripts, ranks: *const usize, dims: *const *const usize, out: *mut *mut tfb_tree) -> tfb_status;
    pub fn tfb_tree_from_pairs(subs: *const tfb_subscripts, ranks: *const usize, dims: *const *const usize, n_pairs: usize, pairs: *const usize, out: *mut *mut tfb_tree) -> tfb_status;
    pub fn tfb_tree_destroy(tree: *mut tfb_tree) -> tfb_status;
    pub fn tfb_tree_n_steps(tree: *const tfb_tree) -> usize;
    pub fn tfb_tree_pairs(tree: *const tfb_tree, pairs: *mut usize, cap: usize) -> usize;
    pub fn tfb_tree_macs(tree: *const tfb_tree) -> f64;
    pub fn tfb_tree_output_dims(tree: *const tfb_tree, dims: *mut usize, cap: usize) -> usize;
    pub fn tfb_einsum_with_plan_into(ctx: *mut tfb_ctx, tree: *const tfb_tree, dtype: i32, n_operands: usize, operands: *const tfb_view, alpha: *const c_void, beta: *const c_void, output: *const tfb_view) -> tfb_status;
}
