// The embedding side of a call (sm_100a): phase table, clamped phase bias and the clamp's gradient, one launch each.
//
// PoPE.forward / AxialPoPE.forward (PoPE_pytorch/pope.py:125-147, pope_nd.py:66-106) are a chain of small elementwise
// PyTorch kernels -- 4 for a sequence, about 25 for a grid -- whose results are a few hundred KB: the launches and the host
// work between them are the whole cost (a training step at (2, 8, 2048, 96) spent 0.25 of its 0.53 ms there).  One kernel
// writes everything: positions, freqs[p][c] = positions[p][axis(c)] * inv_freqs[c] (one fp32 multiply, as the module does
// it), the flat inverse frequencies and axis numbers that the factored form needs, and the clamped bias.
#include "kernels.h"
#include "tc_common.cuh"

namespace pope {

// One thread per (position, feature); the threads behind the table take the bias and the small vectors.
__global__ void __launch_bounds__(256) pope_table_kernel(PopeTableArgs p, int n, int r) {
  pdl_wait();
  const int64_t total = (int64_t)n * r, bias_n = p.bias ? (int64_t)p.H * r : 0;
  int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (idx < total) {
    const int pos = (int)(idx / r), c = (int)(idx - (int64_t)pos * r);
    int axis = 0, first = 0;
    while (axis + 1 < p.axes && c >= first + p.width[axis]) first += p.width[axis++];
    // column a of the positions is grid dimension axes - 1 - a: column 0 varies fastest
    int rest = pos;
    for (int a = 0; a < axis; ++a) rest /= p.dims[p.axes - 1 - a];
    const float x = (float)(axis + 1 < p.axes ? rest % p.dims[p.axes - 1 - axis] : rest) + p.offset;
    const float inv = p.inv_freqs[axis][c - first];
    p.freqs[idx] = __fmul_rn(x, inv);
    if (c == first) p.positions[(int64_t)pos * p.axes + axis] = x;
    if (pos == 0 && p.inv_flat) p.inv_flat[c] = inv, p.axis_of[c] = axis;
    return;
  }
  idx -= total;
  if (idx < bias_n) {
    const float b = p.bias[idx];
    p.bias_out[idx] = b < POPE_BIAS_MIN ? POPE_BIAS_MIN : b > 0.f ? 0.f : b;   // NaN stays NaN
  }
}

cudaError_t pope_table(const PopeTableArgs& p, cudaStream_t st) {
  int64_t n = 1;
  int r = 0;
  for (int a = 0; a < p.axes; ++a) n *= p.dims[a], r += p.width[a];
  const int64_t work = n * r + (p.bias ? (int64_t)p.H * r : 0);
  if (work == 0) return cudaSuccess;
  return launch_dependent(pope_table_kernel, dim3((unsigned)((work + 255) / 256)), dim3(256), 0, st, p, (int)n, r);
}

__global__ void __launch_bounds__(256) pope_clamp_bwd_kernel(const float* bias, const float* grad, float* out, int64_t n) {
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i < n) out[i] = (bias[i] >= POPE_BIAS_MIN && bias[i] <= 0.f) ? grad[i] : 0.f;
}

cudaError_t pope_clamp_bwd(const PopeClampBwdArgs& p, cudaStream_t st) {
  if (p.n == 0) return cudaSuccess;
  return launch_dependent(pope_clamp_bwd_kernel, dim3((unsigned)((p.n + 255) / 256)), dim3(256), 0, st, p.bias, p.grad, p.grad_bias, p.n);
}

}  // namespace pope
