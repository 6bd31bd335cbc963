// Host interface of the backward kernels (backward.cu, tc_wgrad_f32.cu) and of the kernels that copy or
// convert whole tensors (transpose.cu, quantize.cu).
#pragma once

#include "common.cuh"

namespace ksmm {

// One operand of a weight gradient: the factor's input or the gradient of its output.  `ld` is the
// row stride in elements of a batch-last operand (the batch, or more where rows are padded).
struct WgradOperand {
  const void* ptr;
  int last;    // 1: (features, batch), 0: (batch, features)
  int64_t ld;
  int regrouped = 0;  // batch-first rows in block order (i, l, k) instead of (i, k, l)
};

// block transposes of kernel-format weights: (nblk, c, b) -> (nblk, b, c)
int launch_transpose_blocks(const void* in, void* out, int64_t nblk, int c, int b, int es, cudaStream_t stream);

// dW of the factor of `p` (pattern, batch, type; p.out = dW in kernel format).  The workspace holds
// copies of operands that cannot be addressed as they stand, and the partial sums.
size_t wgrad_workspace_bytes(const Problem& p, const WgradOperand& x, const WgradOperand& g);
int wgrad_launch(const Problem& p, WgradOperand x, WgradOperand g, void* workspace, size_t workspace_bytes,
                 cudaStream_t stream);
// Gradient of a bias: the sum over the batch of a gradient of `feats` features, in fp32, stored as `dtype`.
// The workspace holds bias_grad_workspace_bytes(feats) for a batch-first gradient.
size_t bias_grad_workspace_bytes(int64_t feats);
int launch_bias_grad(const void* g, int last, int64_t ld, void* out, void* workspace, int64_t batch, int64_t feats,
                     int dtype, cudaStream_t stream);
// the same from fp32 partial sums (slices, feats)
int launch_bias_sum(const float* part, int slices, void* out, int64_t feats, int dtype, cudaStream_t stream);
// the weight gradient of such a factor runs on the tensor cores for every pair of operand layouts
bool wgrad_any_layout(const Problem& p);
// the fp32 tensor-core kernel: partial tiles (splits, a*d, c, b) into `part`; nt = 64 or 128 columns
int wgrad_f32_launch(const Problem& p, const WgradOperand& x, const WgradOperand& g, float* part, int nt, int splits,
                     cudaStream_t stream);

// in: rows x cols with row stride in_ld (0 = cols), out: cols x rows with row stride out_ld (0 = rows)
int launch_transpose(const void* in, void* out, int64_t rows, int64_t cols, int es, cudaStream_t stream,
                     int64_t out_ld = 0, int64_t in_ld = 0, float* sums = nullptr, int sum_dtype = 0);
// with `sums` (elements of sum_dtype): sums[t][col] over the rows of row tile t, fp32
int transpose_row_tiles(int64_t rows, int es);
// rows x cols from row stride in_ld to row stride out_ld (elements of es bytes); rows of the destination
// are aligned to 16 bytes
int launch_copy_rows(const void* in, int64_t in_ld, void* out, int64_t out_ld, int64_t rows, int64_t cols, int es,
                     cudaStream_t stream);

// Per-tensor e4m3 quantisation of (rows, cols) with row stride in_ld: out has the same order (row stride
// out_ld) or, with transpose (in_ld = cols), is (cols, rows).  `parts` holds quantize_parts_bytes().
size_t quantize_parts_bytes();
int launch_quantize(const void* in, int dtype, int64_t in_ld, void* out, int64_t out_ld, int64_t rows, int64_t cols,
                    bool transpose, void* parts, float* scale, cudaStream_t stream);

}  // namespace ksmm
