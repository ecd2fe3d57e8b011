/* Test-only exports of libmaidenx_cuda.so: host-side views of the launch planners and hooks that let a test
 * reach a state it must not produce on a GPU.  Not part of the op layer's public interface (maidenx_cuda.h);
 * no counterpart in the reference. */
#ifndef MAIDENX_CUDA_TESTING_H
#define MAIDENX_CUDA_TESTING_H
#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Host-only views of the launch planners, for tests that run without a GPU: which kernel class a call with this
 * HOST metadata and these base addresses would take.  Elementwise: 0 empty, 1 flat, 2 row, 3 tile, 4 generic,
 * 5 serial (an in-place lhs that overlaps itself), 6 error, 7 flat with shifted loads (operands not 16-byte aligned).  Reduction: 0 empty, 1 rows, 2 columns, 3 generic
 * scatter, 4 error, 5 first and last dim folded around a kept one, with the recognised [outer, reduced, inner] extents. */
int mx_debug_elementwise_plan(size_t num_els, size_t num_dims, const size_t* host_metadata, int num_inputs, int inplace, size_t elem_size,
                              size_t out_elem_size, const void* out, const void* a, const void* b, int* merged_rank, int* vector_ok,
                              int* transposed_mask);
/* Would cuda_matmul_<bf16|f16> with this HOST metadata run on the tcgen05 kernel (its batches) or on the CUDA-core kernels (0)?
 * Also returns the operand layouts (0 = K-major, 1 = MN-major) and the extents of the launch. */
int mx_debug_matmul_forward_path(size_t num_els, const size_t* host_metadata, const void* a, const void* b, const void* out, int* a_mn_major,
                                 int* b_mn_major, size_t* m, size_t* n, size_t* k);
/* The decision of every cuda_matmul / cuda_matmul_backward call (elem_size 2: bf16 / f16, 4: f32; which: 0 forward with x = a, y = b,
 * 1 grad_a with x = g, y = b, 2 grad_b with x = g, y = a): 0 = CUDA-core kernels, else the number of batches of the tensor-core launch.
 * *prepared: 1 the first operand of the product is copied to padded rows, 2 the second, 4 or 8 the output is written without tensor
 * stores, element-wise or in pairs.  The two calls above and below are this one for the forward product. */
int mx_debug_matmul_plan(size_t elem_size, int which, size_t num_els, size_t nea, size_t neb, const size_t* host_metadata, const void* x, const void* y,
                         const void* out, int* a_mn_major, int* b_mn_major, size_t* m, size_t* n, size_t* k, int* prepared);
int mx_debug_reduce_plan(size_t num_els, size_t num_dims, size_t num_red_dims, const size_t* host_metadata, int sum_to_shape, size_t* outer,
                         size_t* reduced, size_t* inner);

/* Would cuda_matmul_f32 with this HOST metadata run on the tcgen05 split-tf32 kernel (its batches) or on the CUDA-core kernels (0)? */
int mx_debug_matmul_forward_path_f32(size_t num_els, const size_t* host_metadata, const void* a, const void* b, const void* out, int* a_mn_major,
                                     int* b_mn_major, size_t* m, size_t* n, size_t* k);
/* Tuning aid: row-tiles per column sweep in the one-CTA tensor-core kernel's tile order (default 16). */
void mx_debug_set_gemm_group_m(int rows);
/* Pairs of CTAs of the two-CTA tensor-core kernel that can be resident at once on the current device (-1: query failed). */
int mx_debug_gemm_max_resident_pairs(void);
/* The 16-bit Conv2d layer's input gradient (direct form, strides of 1) as one product without a column matrix: 1 = by the rule (default), 0 = never, 2 = wherever
 * possible. */
void mx_debug_set_conv_implicit(int mode);
/* f32 products as pairs of f16 values: 1 = by the rule on their cost (default), 0 = never, 2 = wherever possible, 3 = the same, emptying the accumulator after
 * every 32 values of K.  The query: the calling thread's last f32 product ran as pairs in this many slices (0: not as pairs). */
void mx_debug_set_gemm_f32_pairs(int mode);
int mx_debug_gemm_f32_last_pairs(void);
/* 16-bit operands whose rows are 16-byte multiples but no whole 128-byte lines are copied in lines where that pays: 1 = by the rule (default), 0 = never, 2 =
 * always.  The query: the operands that the calling thread's last product on the tensor cores copied first, for this or because it had to (1 A, 2 B). */
void mx_debug_set_gemm_realign(int mode);
int mx_debug_gemm_last_copies(void);
/* Short reductions (K <= 256, one batch, many row tiles) keep the B panel of a column tile in shared memory and stream
 * only A.  set: 1 = on (default), 0 = always the general schedule.  The query returns the CTAs per column tile a launch
 * with these tile counts takes (0 = general schedule). */
void mx_debug_set_gemm_keep_b(int on);
int mx_debug_gemm_keep_b_ctas(int tiles_m, int tiles_n, int num_kb, int batch, int ctas);
/* The schedule of the calling thread's last launch of the one-CTA tensor-core kernel: 0 = general, 1 = the B panel of a column tile kept, 2 = the same for a
 * batch that shares A. */
int mx_debug_gemm_last_schedule(void);
/* How many K slices the tensor-core path cuts a product with `tiles` output tiles and reduction length `k` into
 * (1 = no split) on `sms` SMs; block_k = 64 for bf16 / f16, 32 for f32. */
int mx_debug_splitk_slices(size_t tiles, size_t k, int block_k, int sms);
/* f32 tensor-core products whose reduction is cut into the CTAs of a cluster: 1 = where that is the cheapest form (default), 0 =
 * nowhere, 2 = wherever one fits. */
void mx_debug_set_gemm_f32_cluster(int on);
/* 1 (default): long f32 reductions multiply the large part of A by both parts of B in one instruction; 0: never. */
void mx_debug_set_gemm_f32_wide(int on);
/* What the calling thread's last f32 product on the tensor cores was: form[0] K slices, form[1] CTAs of a cluster of slices (0: none), form[2]
 * 1 = both parts of B in one instruction, form[3] columns of a tile. */
void mx_debug_gemm_f32_last_form(int form[4]);
/* Writes `value` (0 clears) into the calling thread's tensor-core error word the way a kernel of an earlier launch
 * whose bounded wait ran out would have left it.  Returns 0, or -1 without a usable device. */
int mx_debug_tc_gemm_poke_status(int value);

#ifdef __cplusplus
}
#endif
#endif /* MAIDENX_CUDA_TESTING_H */
