// Stand-alone PoPE transform (sm_100a): q, k -> q', k' of width 2r + (d - r) in the reference's interleaved layout
// [a0 cos, a0 sin, a1 cos, a1 sin, ..., pass-through features], fp32, for callers that feed their own attention.
// Replaces the chain of elementwise PyTorch kernels of PoPE_pytorch/pope.py:37-86 (softplus, add, cos, sin, two
// products, stack, reshape, cat: about ten passes over the data) by ONE pass: bytes = inputs + outputs.
// Phases as the reference computes them: query row i uses freqs[Nk - Nq + i] (:64), key row j uses fl(freqs[j] + bias[h])
// (:56); accurate sincosf, expf and a log1p good to 1.1 ulp, since the result IS the user-visible value here (no 16-bit rounding
// follows).  The backward is the chain rule of the same map:
//   dx = (g_c cos + g_s sin) sigmoid(x),  dphase = a (g_s cos - g_c sin)  -> dfreqs (query and key rows), dbias (key rows).
#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "tc_common.cuh"

namespace pope {

struct ApplySide {
  const void* x;      // (units, rows, d) input
  Strides sx;
  float* y;           // (units, rows, d + r) output / its gradient
  Strides sy;
  void* dx;           // backward only
  Strides sdx;
  int heads, rows, pos0;
  const float* bias;  // key side: per-head phase; query side: null
  int64_t bias_sh;
  float* dbias;       // backward, key side only (may be null)
  int64_t dbias_sh;
};

struct ApplyP {
  ApplySide side[2];  // 0 = queries, 1 = keys
  int B, d, r;
  const float* freqs;
  Strides sf;
  float* dfreqs;      // backward (may be null)
  Strides sdf;
};

constexpr int AP_THREADS = 256;
constexpr int AP_ITEMS = 2;    // rotated items per thread and unit
constexpr int AP_ROWS = 64;    // most rows per block

// N consecutive elements as fp32
template <int N, typename T> __device__ __forceinline__ void ap_load(const T* src, float (&x)[N]) {
  if constexpr (N == 1) {
    x[0] = to_f32<T>(src[0]);
  } else {
    struct alignas(N * sizeof(T)) Pack { T v[N]; };
    const Pack w = *reinterpret_cast<const Pack*>(src);
#pragma unroll
    for (int e = 0; e < N; ++e) x[e] = to_f32<T>(w.v[e]);
  }
}
template <int N, typename T> __device__ __forceinline__ void ap_store(T* dst, const float (&x)[N]) {
  if constexpr (N == 1) {
    dst[0] = from_f32<T>(x[0]);
  } else {
    struct alignas(N * sizeof(T)) Pack { T v[N]; } w;
#pragma unroll
    for (int e = 0; e < N; ++e) w.v[e] = from_f32<T>(x[e]);
    *reinterpret_cast<Pack*>(dst) = w;
  }
}

// log(1 + t) / t for t in [0, 1]: the polynomial through the Chebyshev points of degree 9 (relative error 5e-9; in fp32, times t,
// 1.1 ulp at most, as log1pf, at half of its instructions and without a branch)
__device__ __forceinline__ float log1p_over(float t) {
  float q = -3.176057010e-03f;
  q = fmaf(q, t, 1.954252722e-02f);
  q = fmaf(q, t, -5.637361275e-02f);
  q = fmaf(q, t, 1.054362379e-01f);
  q = fmaf(q, t, -1.526966707e-01f);
  q = fmaf(q, t, 1.966327426e-01f);
  q = fmaf(q, t, -2.495161626e-01f);
  q = fmaf(q, t, 3.332971050e-01f);
  q = fmaf(q, t, -4.999989265e-01f);
  q = fmaf(q, t, 9.999999947e-01f);
  return q;
}
// 1 / w for w in [1, 2], one Newton step behind the approximate reciprocal: within 1 ulp
__device__ __forceinline__ float rcp_near1(float w) {
  const float q = __fdividef(1.f, w);
  return fmaf(q, fmaf(-w, q, 1.f), q);
}

// grid (row blocks, unit groups, 2 sides).  A block takes `rows_pb` rows of `group` units (u = head x B + batch entry, so that
// the entries of a head are neighbours).  An item is RW rotated features of a row, or PW plain ones; rotated and plain items
// are dealt out separately, so that no warp holds both, and a thread keeps its AP_ITEMS rotated items for all units of the
// group: their cosines and sines (accurate sincosf) are taken once per phase, not once per unit.
// VEC: pairs of rotated features and quads of plain ones, every access of a warp in whole 16- to 4-byte pieces.
//
// Bytes = inputs + outputs: (4, 16, 2048, 64), r = 32, bf16 moves 134 MB forward and 168 MB backward, 21 and 26 us at the
// copy rate; the kernels take 33 and 57.  Bound by instruction issue (0.68 per clock and scheduler with log1pf, two
// exponentials and 64-bit offsets, when they took 39 and 64).  One thread per feature and row, half of every warp rotated and a
// sincosf per unit, the training step took 228 us; now 115.  More warps (40 registers) spill and are slower (54 + 73 before the
// last change), four items per thread too (57 + 104).
template <typename T, bool BACKWARD, bool VEC>
__global__ void __launch_bounds__(AP_THREADS, 4) apply_qk_kernel(ApplyP p, int rows_pb, int group) {
  constexpr int RW = VEC ? 2 : 1, PW = VEC ? 4 : 1;
  __shared__ float red[BACKWARD ? AP_THREADS * AP_ITEMS * RW : 1];
  pdl_wait();
  const ApplySide& s = p.side[blockIdx.z];
  const int units = p.B * s.heads, u0 = blockIdx.y * group, u1 = min(u0 + group, units);
  const int row0 = blockIdx.x * rows_pb, nrow = min(rows_pb, s.rows - row0);
  if (u0 >= units || nrow <= 0) return;
  const int RP = p.r / RW, PP = (p.d - p.r) / PW;   // rotated and plain items of a row
  using Off = std::conditional_t<VEC, int, int64_t>;   // offsets inside a block's rows (VEC: known to fit)
  const Off sxn = (Off)s.sx.n, syn = (Off)s.sy.n, sdxn = (Off)s.sdx.n;
  int row[AP_ITEMS], c[AP_ITEMS];
  Off xo[AP_ITEMS], yo[AP_ITEMS], dxo[AP_ITEMS];
  bool act[AP_ITEMS];
  float cs[AP_ITEMS][RW], sn[AP_ITEMS][RW], df[AP_ITEMS][RW], db[AP_ITEMS][RW];
#pragma unroll
  for (int k = 0; k < AP_ITEMS; ++k) {
    const int item = threadIdx.x + AP_THREADS * k;
    row[k] = RP > 0 ? item / RP : nrow, c[k] = (item - row[k] * RP) * RW, act[k] = row[k] < nrow;
    xo[k] = row[k] * sxn + c[k], yo[k] = row[k] * syn + 2 * c[k], dxo[k] = row[k] * sdxn + c[k];
#pragma unroll
    for (int e = 0; e < RW; ++e) cs[k][e] = sn[k][e] = df[k][e] = db[k][e] = 0.f;
  }
  // plain items: one column of them per thread, every prpp-th row
  const int prpp = PP > 0 ? AP_THREADS / PP : 1, prow = PP > 0 ? threadIdx.x / PP : 0;
  const int pc = p.r + (PP > 0 ? (threadIdx.x - prow * PP) * PW : 0), pend = PP > 0 && prow < prpp ? nrow : 0;
  int h = u0 / p.B, b = u0 - h * p.B;
  auto flush_freqs = [&]() {   // the gradient of the phases of (b, h), summed over the units that shared them
    if (!BACKWARD || !p.dfreqs) return;
#pragma unroll
    for (int k = 0; k < AP_ITEMS; ++k)
#pragma unroll
      for (int e = 0; e < RW; ++e) {
        if (act[k]) atomicAdd(p.dfreqs + b * p.sdf.b + h * p.sdf.h + (int64_t)(s.pos0 + row0 + row[k]) * p.sdf.n + c[k] + e, df[k][e]);
        df[k][e] = 0.f;
      }
  };
  auto flush_bias = [&]() {    // one atomic per (block, head, feature); block-uniform
    if (!BACKWARD || !s.dbias) return;
#pragma unroll
    for (int k = 0; k < AP_ITEMS; ++k)
#pragma unroll
      for (int e = 0; e < RW; ++e) red[(threadIdx.x + AP_THREADS * k) * RW + e] = db[k][e], db[k][e] = 0.f;
    __syncthreads();
    for (int f = threadIdx.x; f < p.r; f += AP_THREADS) {
      float sum = 0.f;
      for (int i = 0; i < nrow; ++i) sum += red[i * p.r + f];
      atomicAdd(s.dbias + h * s.dbias_sh + f, sum);
    }
    __syncthreads();
  };
  bool fresh = true;
  for (int u = u0; u < u1; ++u) {
    const T* x = static_cast<const T*>(s.x) + b * s.sx.b + h * s.sx.h + (int64_t)row0 * s.sx.n;
    float* y = s.y + b * s.sy.b + h * s.sy.h + (int64_t)row0 * s.sy.n;
    T* dx = BACKWARD ? static_cast<T*>(s.dx) + b * s.sdx.b + h * s.sdx.h + (int64_t)row0 * s.sdx.n : nullptr;
    float xv[AP_ITEMS][RW], g[AP_ITEMS][2 * RW];
#pragma unroll
    for (int k = 0; k < AP_ITEMS; ++k) {
      if (!act[k]) continue;
      ap_load<RW>(x + xo[k], xv[k]);
      if (BACKWARD) ap_load<2 * RW>(y + yo[k], g[k]);
    }
    for (int rr = prow; rr < pend; rr += prpp) {
      float v[PW];
      if (!BACKWARD) {
        ap_load<PW>(x + (rr * sxn + pc), v);
        ap_store<PW>(y + (rr * syn + p.r + pc), v);
      } else {
        ap_load<PW>(y + (rr * syn + p.r + pc), v);
        ap_store<PW>(dx + (rr * sdxn + pc), v);
      }
    }
#pragma unroll
    for (int k = 0; k < AP_ITEMS; ++k) {
      if (!act[k]) continue;
      if (fresh) {
        const float* f = p.freqs + b * p.sf.b + h * p.sf.h + (int64_t)(s.pos0 + row0 + row[k]) * p.sf.n + c[k];
#pragma unroll
        for (int e = 0; e < RW; ++e) sincosf(s.bias ? f[e] + s.bias[h * s.bias_sh + c[k] + e] : f[e], &sn[k][e], &cs[k][e]);
      }
      float out[BACKWARD ? RW : 2 * RW];
#pragma unroll
      for (int e = 0; e < RW; ++e) {
        const float xe = xv[k][e], t = expf(-fabsf(xe));
        const float a = fmaf(t, log1p_over(t), fmaxf(xe, 0.f));
        if constexpr (BACKWARD) {
          const float gc = g[k][2 * e], gs = g[k][2 * e + 1];
          out[e] = (gc * cs[k][e] + gs * sn[k][e]) * ((xe >= 0.f ? 1.f : t) * rcp_near1(1.f + t));
          const float dphase = a * (gs * cs[k][e] - gc * sn[k][e]);
          df[k][e] += dphase, db[k][e] += dphase;
        } else {
          out[2 * e] = a * cs[k][e], out[2 * e + 1] = a * sn[k][e];
        }
      }
      if constexpr (BACKWARD) ap_store<RW>(dx + dxo[k], out);
      else ap_store<2 * RW>(y + yo[k], out);
    }
    const int h2 = b + 1 == p.B ? h + 1 : h, b2 = b + 1 == p.B ? 0 : b + 1;
    fresh = (h2 != h && (s.bias || p.sf.h != 0)) || (b2 != b && p.sf.b != 0);
    // (a table that is broadcast by a stride of 0 has a gradient with a slice for every unit: its own strides decide)
    if (BACKWARD && ((h2 != h && p.sdf.h != 0) || (b2 != b && p.sdf.b != 0) || u + 1 == u1)) flush_freqs();
    if (BACKWARD && (h2 != h || u + 1 == u1)) flush_bias();
    h = h2, b = b2;
  }
}

// Whether every row of both sides can be read and written in pieces of 2 and 4 elements.
template <typename T>
static bool apply_vectors(const ApplyP& p) {
  if (p.d % 4 != 0 || p.r % 4 != 0) return false;
  auto ok = [](const void* ptr, const Strides& st, size_t esz) {
    return reinterpret_cast<uintptr_t>(ptr) % (4 * esz) == 0 && st.b % 4 == 0 && st.h % 4 == 0 && st.n % 4 == 0;
  };
  for (const ApplySide& s : p.side) {
    if (s.sx.n >= (1 << 24) || s.sy.n >= (1 << 24) || s.sdx.n >= (1 << 24) || std::min({s.sx.n, s.sy.n, s.sdx.n}) < 0) return false;   // 32-bit offsets
    if (!ok(s.x, s.sx, sizeof(T)) || !ok(s.y, s.sy, 4) || (s.dx && !ok(s.dx, s.sdx, sizeof(T)))) return false;
  }
  return true;
}

template <typename T, bool BACKWARD, bool VEC>
static cudaError_t launch_apply_v(const ApplyP& p, int units_max, int rows_max, cudaStream_t st) {
  if (p.d > AP_THREADS) return cudaErrorInvalidValue;
  const int items = p.r / (VEC ? 2 : 1);
  const int rows_pb = items > 0 ? std::min(AP_ROWS, AP_ITEMS * AP_THREADS / items) : AP_ROWS;
  const int blocks = (rows_max + rows_pb - 1) / rows_pb;
  // Units per block: up to 8, whole heads where possible, while six blocks per SM (one and a half times what is resident)
  // are left.  At (4, 16, 2048, 64), r = 32: 1 unit 55 + 81 us (forward + backward), 2 units 44 + 68, 4 units 40 + 64,
  // 8 units 39 + 64, 16 units 43 + 68 (before the arithmetic was cut).
  int group = (int)std::min<int64_t>(8, std::max<int64_t>(1, (int64_t)blocks * units_max * 2 / (148 * 6)));
  if (group > p.B) group -= group % p.B;
  const dim3 grid((unsigned)blocks, (unsigned)((units_max + group - 1) / group), 2);
  return launch_dependent(apply_qk_kernel<T, BACKWARD, VEC>, grid, dim3(AP_THREADS), 0, st, p, rows_pb, group);
}

template <typename T, bool BACKWARD>
static cudaError_t launch_apply(const ApplyP& p, int units_max, int rows_max, cudaStream_t st) {
  return apply_vectors<T>(p) ? launch_apply_v<T, BACKWARD, true>(p, units_max, rows_max, st)
                             : launch_apply_v<T, BACKWARD, false>(p, units_max, rows_max, st);
}

static ApplyP apply_params(const PopeShape& s, const PopeEmbed& e) {
  ApplyP p = {};
  p.B = s.B, p.d = s.d, p.r = s.r;
  p.freqs = e.freqs, p.sf = Strides(e.sf);
  p.side[0].heads = s.H, p.side[0].rows = s.Nq, p.side[0].pos0 = s.Nk - s.Nq;
  p.side[1].heads = s.Hk, p.side[1].rows = s.Nk, p.side[1].pos0 = 0;
  p.side[1].bias = s.r > 0 ? e.bias : nullptr, p.side[1].bias_sh = e.bias_stride_h;
  return p;
}

cudaError_t apply_qk_fwd(const PopeApplyArgs& a, cudaStream_t st) {
  const PopeShape& s = a.shape;
  ApplyP p = apply_params(s, a.embed);
  p.side[0].x = a.q, p.side[0].sx = Strides(a.sq), p.side[0].y = a.q_out, p.side[0].sy = Strides(a.sqo);
  p.side[1].x = a.k, p.side[1].sx = Strides(a.sk), p.side[1].y = a.k_out, p.side[1].sy = Strides(a.sko);
  const int units = s.B * (s.H > s.Hk ? s.H : s.Hk);
  switch (s.dtype) {
    case POPE_F32: return launch_apply<float, false>(p, units, s.Nk, st);
    case POPE_BF16: return launch_apply<__nv_bfloat16, false>(p, units, s.Nk, st);
    default: return launch_apply<__half, false>(p, units, s.Nk, st);
  }
}

cudaError_t apply_qk_bwd(const PopeApplyBwdArgs& a, cudaStream_t st) {
  const PopeShape& s = a.shape;
  ApplyP p = apply_params(s, a.embed);
  p.side[0].x = a.q, p.side[0].sx = Strides(a.sq), p.side[0].y = const_cast<float*>(a.dq_out), p.side[0].sy = Strides(a.sdqo);
  p.side[0].dx = a.dq, p.side[0].sdx = Strides(a.sdq);
  p.side[1].x = a.k, p.side[1].sx = Strides(a.sk), p.side[1].y = const_cast<float*>(a.dk_out), p.side[1].sy = Strides(a.sdko);
  p.side[1].dx = a.dk, p.side[1].sdx = Strides(a.sdk);
  p.side[1].dbias = s.r > 0 ? a.dbias : nullptr, p.side[1].dbias_sh = a.dbias_stride_h;
  p.dfreqs = s.r > 0 ? a.dfreqs : nullptr, p.sdf = Strides(a.sdf);
  const int units = s.B * (s.H > s.Hk ? s.H : s.Hk);
  switch (s.dtype) {
    case POPE_F32: return launch_apply<float, true>(p, units, s.Nk, st);
    case POPE_BF16: return launch_apply<__nv_bfloat16, true>(p, units, s.Nk, st);
    default: return launch_apply<__half, true>(p, units, s.Nk, st);
  }
}

}  // namespace pope
