// Ends of a layer fused into one launch (layer_tail.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

constexpr int kTailMaxWidth = 8192;

// Per row of D features, in fp32 and rounded once:
//   v = x + routed + shared * sigmoid(h . gate_w)          x_out = bf16(v)
//   h_out = x_out rsqrt(mean(x_out^2) + eps) (1 + norm_w)   (norm_w instead of 1 + norm_w without `one_plus`)
// routed is fp32; any of x, routed, shared may be nullptr (nothing added); without gate_w shared counts as it is; without norm_w
// there is no h_out. D a multiple of 8, at most kTailMaxWidth; all rows contiguous on 16-byte boundaries; x_out may be x.
struct LayerTailArgs {
  const __nv_bfloat16* x;
  const float* routed;
  const __nv_bfloat16* shared;
  const __nv_bfloat16* h;
  const __nv_bfloat16* gate_w;
  const __nv_bfloat16* norm_w;
  __nv_bfloat16* x_out;
  __nv_bfloat16* h_out;
  int rows, D, one_plus;
  float eps;
};
cudaError_t launch_layer_tail(const LayerTailArgs& a, cudaStream_t stream);

// counts[e] = pairs of expert e, pos[p] = rank of pair p among its expert's, out[0 .. n_out) = 0, in one launch. At most
// kPrepareMaxPairs pairs and kPrepareMaxExperts experts; n_out a multiple of 4 on a 16-byte boundary.
// With `order`: the pairs sorted by expert, and `flags` [n_flags] cleared (what the expert kernel of one rank starts from).
constexpr int kPrepareMaxPairs = 8192, kPrepareMaxExperts = 512;
cudaError_t launch_moe_prepare_zero(const int* idx, int n_pairs, int n_experts, int* counts, int* pos, float* out, int64_t n_out,
                                    int* order, int* flags, int n_flags, cudaStream_t stream);

// out = silu(g) * u, rounded once; rows of I features (a multiple of 8), g and u with row strides (multiples of 8), out contiguous; all
// on 16-byte boundaries.
cudaError_t launch_silu_mul(const __nv_bfloat16* g, int64_t ldg, const __nv_bfloat16* u, int64_t ldu, __nv_bfloat16* out, int64_t rows,
                            int I, cudaStream_t stream);

// ids[r] = place of the largest of row r (bf16, N values), the first of equal ones; a NaN is the largest, as in torch.
cudaError_t launch_argmax_rows(const __nv_bfloat16* x, int64_t ldx, int rows, int N, int64_t* ids, cudaStream_t stream);

}  // namespace b200
