// Exact-arithmetic (fp32 FMA) PoPE attention in 64 x 64 tiles: forward and backward for every dtype, any head dim and rotate
// dim with d + r <= 256, any stride, grouped heads, 2- to 4-D phase tables, key-padding and causal masks.
//
// What bounds it is the fp32 FMA rate (128 per clock and SM), so everything else is kept off the inner loops:
//   * a pre-pass transforms every operand once per call (accurate sincosf / log1pf / expf) into fp32 tile images in the
//     caller's workspace.  The kernels of simt_attn.cu transform the keys again in every CTA; at (1, 8, 1024, 64), r = 64 that
//     was half of their instructions.
//   * an image tile is feature-major, [feature][64 rows], one contiguous bulk copy, its 16-byte groups of four rows
//     permuted by  group ^ (feature / 4 mod 16).  That one layout feeds both kinds of product without bank conflicts: with the
//     features as the contraction index (scores: four rows of both operands per feature) and with the rows as the contraction
//     index (gradients and P V: four keys of a feature at a time).
//   * a thread owns a 4 x 4 piece of the score tile and 4 rows x (columns / 16) of the accumulators: two 16-byte shared loads
//     per 16 FMAs, a quarter of what one row x one key per lane needed.
// Measured at (1, 8, 1024, 64), r = 64, causal, fp32: see the table at the launch functions.
//
// Semantics: PoPE_pytorch/triton_pope_flash_attn.py:23-218 (top-left causal mask, bottom-right positions, mask True = keep,
// zero output and -inf LSE for empty rows).
#include <math_constants.h>

#include <algorithm>

#include "kernels.h"
#include "tc_common.cuh"

namespace pope {

constexpr int ST_ROWS = 64;        // rows of a tile
constexpr int ST_THREADS = 256;    // 16 x 16 threads, 4 x 4 scores each

struct TiledP {
  int H, Hk, Nq, Nk, d, r, KD;     // KD = d + r rounded up to 8: features of a Q' / K' tile
  int qt, kt, causal, dtype;       // tiles per unit
  float scale, scale_log2;
  const float *qimg, *kimg, *vimg, *gimg;   // [unit][tile][KD | DP][64]: Q', K', V, dO
  int DP;                          // features of a V / dO tile: d rounded up to 8
  const uint8_t* mask;
  int64_t msb, msn;
  void* o;
  Strides so;
  float* lse;
  const float *lse_in, *delta;
  void *dq, *dk, *dv;
  Strides sdq, sdk, sdv, sdf;
  float *dfreqs, *dbias;
  int64_t dbias_sh;
  unsigned int* status;
};

__device__ __forceinline__ void put(void* base, int64_t i, float v, int dtype) {
  if (dtype == POPE_F32) static_cast<float*>(base)[i] = v;
  else if (dtype == POPE_BF16) static_cast<__nv_bfloat16*>(base)[i] = __float2bfloat16_rn(v);
  else static_cast<__half*>(base)[i] = __float2half_rn(v);
}

// ---- pre-pass --------------------------------------------------------------------------------------------------------
// One operand: rows of `units` (batch, head) slices of x.  r > 0: the first r features become a cos / a sin of table row
// pos0 + row (+ the head's bias); r = 0: a plain transpose.
struct TileJob {
  const void* x;
  Strides sx;
  int units, heads, rows, r, pos0, feats;   // feats = features of an image tile (KD or DP)
  const float* bias;
  int64_t bias_sh;
  float* img;
};
struct TileJobs { TileJob job[4]; };

// grid (tiles, units, jobs).  Lanes take consecutive rows of one feature: the stores of a warp are whole lines, and the
// loads, a line per lane, come back from L1 for the next 31 features.
template <typename T>
__global__ void __launch_bounds__(256) tile_image_kernel(TileJobs jobs, int d, const float* __restrict__ freqs, Strides sf) {
  pdl_wait();
  pdl_trigger();
  const TileJob& jb = jobs.job[blockIdx.z];
  const int tile = blockIdx.x, u = blockIdx.y;
  if (u >= jb.units || tile * ST_ROWS >= jb.rows) return;
  const int b = u / jb.heads, h = u % jb.heads;
  const int row = threadIdx.x & 63, j = tile * ST_ROWS + row;
  const bool ok = j < jb.rows;
  const T* x = static_cast<const T*>(jb.x) + b * jb.sx.b + h * jb.sx.h + (int64_t)j * jb.sx.n;
  const float* f = freqs + b * sf.b + h * sf.h + (int64_t)(jb.pos0 + j) * sf.n;
  const float* bias = jb.bias ? jb.bias + h * jb.bias_sh : nullptr;
  float* img = jb.img + ((int64_t)u * ((jb.rows + ST_ROWS - 1) / ST_ROWS) + tile) * jb.feats * ST_ROWS;
  auto at = [&](int c) { return img + c * ST_ROWS + ((((row >> 2) ^ (c >> 2)) & 15) << 2) + (row & 3); };
  for (int c = threadIdx.x >> 6; c < d; c += 4) {
    float v = ok ? to_f32<T>(x[c]) : 0.f;
    if (c < jb.r) {
      float cs = 0.f, sn = 0.f;
      if (ok) {
        sincosf(bias ? f[c] + bias[c] : f[c], &sn, &cs);
        const float a = softplus_f(v);
        cs *= a, sn *= a;
      }
      *at(c) = cs, *at(d + c) = sn;
    } else {
      *at(c) = v;
    }
  }
  for (int c = d + jb.r + (threadIdx.x >> 6); c < jb.feats; c += 4) *at(c) = 0.f;
}

static cudaError_t launch_tile_images(const TileJobs& jobs, int njobs, const PopeShape& s, const PopeEmbed& e, cudaStream_t st) {
  int tiles = 0, units = 0;
  for (int i = 0; i < njobs; ++i) {
    tiles = max(tiles, (jobs.job[i].rows + ST_ROWS - 1) / ST_ROWS), units = max(units, jobs.job[i].units);
  }
  const dim3 grid((unsigned)tiles, (unsigned)units, (unsigned)njobs), block(256);
  switch (s.dtype) {
    case POPE_F32: return launch_dependent(tile_image_kernel<float>, grid, block, 0, st, jobs, s.d, e.freqs, Strides(e.sf));
    case POPE_BF16: return launch_dependent(tile_image_kernel<__nv_bfloat16>, grid, block, 0, st, jobs, s.d, e.freqs, Strides(e.sf));
    default: return launch_dependent(tile_image_kernel<__half>, grid, block, 0, st, jobs, s.d, e.freqs, Strides(e.sf));
  }
}

// ---- tile products ---------------------------------------------------------------------------------------------------
// c[i][j] += sum over features k < n of A[k][4 ty + i] B[k][4 tx + j], both feature-major tiles
__device__ __forceinline__ void mm_features(float (&c)[4][4], const float* A, const float* B, int n, int ty, int tx) {
#pragma unroll 2
  for (int k4 = 0; k4 < n; k4 += 4) {
    const int sw = (k4 >> 2) & 15;
    const float* a = A + k4 * ST_ROWS + ((ty ^ sw) << 2);
    const float* b = B + k4 * ST_ROWS + ((tx ^ sw) << 2);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 av = *reinterpret_cast<const float4*>(a + k * ST_ROWS), bv = *reinterpret_cast<const float4*>(b + k * ST_ROWS);
      const float x[4] = {av.x, av.y, av.z, av.w}, y[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = fmaf(x[i], y[j], c[i][j]);
    }
  }
}

// c[i][m] += sum over the 64 tile rows t of S[4 ty + i][t] B[feature(m)][t]: S is a row-major score tile (put_scores), B a
// feature-major tile; feature(m) = 4 tx + m % 4 + 64 (m / 4)
template <int NC>
__device__ __forceinline__ void mm_rows(float (&c)[4][NC], const float* S, const float* B, int ty, int tx) {
  const float* s = S + ty * 4 * ST_ROWS;
  const float* b = B + tx * 4 * ST_ROWS;
#pragma unroll 2
  for (int g = 0; g < 16; ++g) {
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(s + i * ST_ROWS + ((g ^ ty) << 2));
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const float4 y = *reinterpret_cast<const float4*>(b + ((m >> 2) * 64 + (m & 3)) * ST_ROWS + ((g ^ tx) << 2));
#pragma unroll
      for (int i = 0; i < 4; ++i) c[i][m] = fmaf(x[i].w, y.w, fmaf(x[i].z, y.z, fmaf(x[i].y, y.y, fmaf(x[i].x, y.x, c[i][m]))));
    }
  }
}

__device__ __forceinline__ void put_scores(float* S, const float (&v)[4][4], int ty, int tx) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(S + (ty * 4 + i) * ST_ROWS + ((tx ^ ty) << 2)) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
}

template <int N> __device__ __forceinline__ void zero(float (&c)[4][N]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) c[i][j] = 0.f;
}

// one image tile by bulk copy; a thread of the CTA calls it after every thread is done with the buffer
__device__ __forceinline__ void fetch(float* dst, const float* img, int feats, uint64_t* bar) {
  mbar_expect_tx(bar, feats * ST_ROWS * 4);
  bulk_load(dst, img, feats * ST_ROWS * 4, bar);
}

// ---- forward ---------------------------------------------------------------------------------------------------------
// Shared memory: Q' tile, K' tile, V tile, P.  The K' buffer is free once the scores are in registers and refilled behind
// the softmax and P V, the V buffer is refilled behind the next scores; where two CTAs fit an SM they cover the rest.
template <int ND>
__global__ void __launch_bounds__(ST_THREADS, ND == 4 ? 2 : 1) attn_fwd_tiled_kernel(TiledP p) {
  extern __shared__ __align__(128) float st_smem[];
  const int QF = p.KD * ST_ROWS, VF = ND * 16 * ST_ROWS;
  float *Qs = st_smem, *Ks = Qs + QF, *Vs = Ks + QF, *Ps = Vs + VF;
  uint64_t* bars = reinterpret_cast<uint64_t*>(Ps + ST_ROWS * ST_ROWS);   // Q', K', V landed
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int u = blockIdx.y, b = u / p.H, h = u % p.H, hk = h % p.Hk, uk = b * p.Hk + hk;
  const int qtile = gridDim.x - 1 - blockIdx.x, i0 = qtile * ST_ROWS;   // heavy (late) row blocks first
  int n_end = p.Nk;
  if (p.causal) n_end = min(n_end, min(i0 + ST_ROWS, p.Nq));
  const int T = (n_end + ST_ROWS - 1) / ST_ROWS;
  const float* kimg = p.kimg + (int64_t)uk * p.kt * QF;
  const float* vimg = p.vimg + (int64_t)uk * p.kt * p.DP * ST_ROWS;
  const uint8_t* mask = p.mask ? p.mask + b * p.msb : nullptr;
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
    mbar_init_fence();
    pdl_wait();
    fetch(Qs, p.qimg + ((int64_t)u * p.qt + qtile) * QF, p.KD, &bars[0]);
    fetch(Ks, kimg, p.KD, &bars[1]);
    fetch(Vs, vimg, p.DP, &bars[2]);
  }
  __syncthreads();
  bool failed = !mbar_wait(&bars[0], 0, WAIT_LIMIT);
  float m[4], l[4], o[4][ND];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = -CUDART_INF_F, l[i] = 0.f;
  zero(o);
  for (int t = 0; t < T; ++t) {
    const int n0 = t * ST_ROWS;
    float s[4][4];
    zero(s);
    if (!failed) failed = !mbar_wait(&bars[1], t & 1, WAIT_LIMIT);
    mm_features(s, Qs, Ks, p.KD, ty, tx);
    const int j0 = n0 + tx * 4;
    bool ok[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) ok[j] = j0 + j < p.Nk && (!mask || mask[(int64_t)(j0 + j) * p.msn] != 0);
    __syncthreads();   // the K' tile and (from the last round) P have been read
    if (tid == 0 && t + 1 < T) fetch(Ks, kimg + (int64_t)(t + 1) * QF, p.KD, &bars[1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gi = i0 + ty * 4 + i;
      float mx = -CUDART_INF_F;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = ok[j] && (!p.causal || j0 + j <= gi) ? s[i][j] * p.scale_log2 : -CUDART_INF_F;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int off = 8; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m[i], mx), m_use = m_new == -CUDART_INF_F ? 0.f : m_new;
      const float alpha = exp2f(m[i] - m_use);   // 0 on the first visible tile
      m[i] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = exp2f(s[i][j] - m_use), sum += s[i][j];
      l[i] = l[i] * alpha + sum;                 // this lane's columns; the lanes of a row are summed at the end
#pragma unroll
      for (int c = 0; c < ND; ++c) o[i][c] *= alpha;
    }
    put_scores(Ps, s, ty, tx);
    __syncthreads();
    if (!failed) failed = !mbar_wait(&bars[2], t & 1, WAIT_LIMIT);
    mm_rows<ND>(o, Ps, Vs, ty, tx);
    if (t + 1 < T) {
      __syncthreads();   // the V tile has been read
      if (tid == 0) fetch(Vs, vimg + (int64_t)(t + 1) * p.DP * ST_ROWS, p.DP, &bars[2]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gi = i0 + ty * 4 + i;
#pragma unroll
    for (int off = 8; off >= 1; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
    if (gi >= p.Nq) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    const int64_t base = b * p.so.b + h * p.so.h + (int64_t)gi * p.so.n;
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      const int col = tx * 4 + (c & 3) + 64 * (c >> 2);
      if (col < p.d) put(p.o, base + col, o[i][c] * inv, p.dtype);
    }
    if (tx == 0) p.lse[(int64_t)u * p.Nq + gi] = l[i] > 0.f ? m[i] * LN2 + logf(l[i]) : -CUDART_INF_F;
  }
  if (failed) atomicOr(p.status, 1u);
}

// ---- backward ----------------------------------------------------------------------------------------------------------
// Epilogue: X' gradients of 64 rows in `acc` [64][ASTR] -> dx, dphase.  Everything the chain rule needs is in the resident
// image tile: with xc = a cos, xs = a sin,  a = sqrt(xc^2 + xs^2),  sigmoid(x) = 1 - exp(-a),
//   dx = (gc xc + gs xs) / a * sigmoid(x),  dphase = gs xc - gc xs.
__device__ __forceinline__ void chain_rule(const TiledP& p, const float* acc, int astr, const float* X, int row0, int rows, void* dx, int64_t base,
                                           int64_t sn, float* df, int64_t sfn, int pos0, float* dbias) {
  for (int c = threadIdx.x & 63; c < p.d; c += 64) {
    float sum = 0.f;
    for (int row = threadIdx.x >> 6; row < ST_ROWS && row0 + row < rows; row += 4) {
      float g = acc[row * astr + c];
      if (c < p.r) {
        const int grp = row >> 2, e = row & 3;
        const float gs = acc[row * astr + p.d + c];
        const float xc = X[c * ST_ROWS + (((grp ^ (c >> 2)) & 15) << 2) + e];
        const float xs = X[(p.d + c) * ST_ROWS + (((grp ^ ((p.d + c) >> 2)) & 15) << 2) + e];
        const float a = sqrtf(xc * xc + xs * xs), dph = gs * xc - g * xs;
        g = a > 0.f ? (g * xc + gs * xs) / a * -expm1f(-a) : 0.f;
        sum += dph;
        if (df) atomicAdd(df + (int64_t)(pos0 + row0 + row) * sfn + c, dph);
      }
      put(dx, base + (int64_t)(row0 + row) * sn + c, g, p.dtype);
    }
    if (dbias && c < p.r) atomicAdd(dbias + c, sum);
  }
}

// accumulator columns -> row-major staging tile
template <int N> __device__ __forceinline__ void stage_acc(float* dst, int stride, const float (&c)[4][N], int width, int ty, int tx) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int m = 0; m < N; ++m) {
      const int col = tx * 4 + (m & 3) + 64 * (m >> 2);
      if (col < width) dst[(ty * 4 + i) * stride + col] = c[i][m];
    }
}

// dq: 64 query rows resident (Q', dO); streams K' and V tiles:  S, dP -> dS -> dQ' += dS K'
template <int ND, int NK>
__device__ __forceinline__ void bwd_dq_tiled(const TiledP& p, float* smem, uint64_t* bars, int qtile, int u) {
  const int QF = p.KD * ST_ROWS, QA = NK * 16 * ST_ROWS, VF = p.DP * ST_ROWS;
  float *Qs = smem, *Gs = Qs + QF, *Ks = Gs + VF, *Vs = Ks + QA, *Ss = Vs + VF;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int b = u / p.H, h = u % p.H, hk = h % p.Hk, uk = b * p.Hk + hk, i0 = qtile * ST_ROWS;
  int n_end = p.Nk;
  if (p.causal) n_end = min(n_end, min(i0 + ST_ROWS, p.Nq));
  const int T = (n_end + ST_ROWS - 1) / ST_ROWS;
  const float* kimg = p.kimg + (int64_t)uk * p.kt * QF;
  const float* vimg = p.vimg + (int64_t)uk * p.kt * VF;
  const uint8_t* mask = p.mask ? p.mask + b * p.msb : nullptr;
  if (tid == 0) {
    mbar_expect_tx(&bars[0], (QF + VF) * 4);
    bulk_load(Qs, p.qimg + ((int64_t)u * p.qt + qtile) * QF, QF * 4, &bars[0]);
    bulk_load(Gs, p.gimg + ((int64_t)u * p.qt + qtile) * VF, VF * 4, &bars[0]);
    fetch(Ks, kimg, p.KD, &bars[1]);
    fetch(Vs, vimg, p.DP, &bars[2]);
  }
  float lse2[4], dl[4], acc[4][NK];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gi = i0 + ty * 4 + i;
    const float l = gi < p.Nq ? p.lse_in[(int64_t)u * p.Nq + gi] : -CUDART_INF_F;
    lse2[i] = l == -CUDART_INF_F ? CUDART_INF_F : l * LOG2E;   // +inf: probabilities are exactly 0
    dl[i] = gi < p.Nq ? p.delta[(int64_t)u * p.Nq + gi] : 0.f;
  }
  zero(acc);
  bool failed = !mbar_wait(&bars[0], 0, WAIT_LIMIT);
  for (int t = 0; t < T; ++t) {
    const int j0 = t * ST_ROWS + tx * 4;
    float s[4][4], dp[4][4];
    zero(s), zero(dp);
    if (!failed) failed = !mbar_wait(&bars[2], t & 1, WAIT_LIMIT);
    mm_features(dp, Gs, Vs, p.DP, ty, tx);
    bool ok[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) ok[j] = j0 + j < p.Nk && (!mask || mask[(int64_t)(j0 + j) * p.msn] != 0);
    if (!failed) failed = !mbar_wait(&bars[1], t & 1, WAIT_LIMIT);
    mm_features(s, Qs, Ks, p.KD, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool vis = ok[j] && (!p.causal || j0 + j <= i0 + ty * 4 + i);
        s[i][j] = vis ? exp2f(s[i][j] * p.scale_log2 - lse2[i]) * (dp[i][j] - dl[i]) * p.scale : 0.f;
      }
    put_scores(Ss, s, ty, tx);
    __syncthreads();   // dS is written, the V tile has been read
    if (tid == 0 && t + 1 < T) fetch(Vs, vimg + (int64_t)(t + 1) * VF, p.DP, &bars[2]);
    mm_rows<NK>(acc, Ss, Ks, ty, tx);
    __syncthreads();   // the K' tile and dS have been read
    if (tid == 0 && t + 1 < T) fetch(Ks, kimg + (int64_t)(t + 1) * QF, p.KD, &bars[1]);
  }
  const int astr = p.d + p.r + 1;
  stage_acc<NK>(Gs, astr, acc, p.d + p.r, ty, tx);   // dO, K', V and dS are dead: [64][d + r + 1] fits them
  __syncthreads();
  float* df = p.dfreqs ? p.dfreqs + b * p.sdf.b + h * p.sdf.h : nullptr;
  chain_rule(p, Gs, astr, Qs, i0, p.Nq, p.dq, b * p.sdq.b + h * p.sdq.h, p.sdq.n, df, p.sdf.n, p.Nk - p.Nq, nullptr);
  if (failed) atomicOr(p.status, 1u);
}

// dk / dv: 64 key rows resident (K', V); streams the Q' and dO tiles of every grouped query head:
// S^T, dP^T -> P^T -> dV += P^T dO, dS^T -> dK' += dS^T Q'
template <int ND, int NK>
__device__ __forceinline__ void bwd_dkdv_tiled(const TiledP& p, float* smem, uint64_t* bars, int ktile, int uk) {
  const int QF = p.KD * ST_ROWS, QA = NK * 16 * ST_ROWS, VF = p.DP * ST_ROWS, VA = ND * 16 * ST_ROWS;
  float *Ks = smem, *Vs = Ks + QF, *Qs = Vs + VF, *Gs = Qs + QA, *Ss = Gs + VA;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int b = uk / p.Hk, hk = uk % p.Hk, j0 = ktile * ST_ROWS, groups = p.H / p.Hk;
  const int t_first = p.causal ? ktile : 0;   // under the causal mask queries before this tile see none of its keys
  const int per = p.qt > t_first ? p.qt - t_first : 0, T = per * groups;
  const uint8_t* mask = p.mask ? p.mask + b * p.msb : nullptr;
  auto unit = [&](int t) { return b * p.H + (t / per) * p.Hk + hk; };
  auto qtile = [&](int t) { return t_first + t % per; };
  auto fetch_q = [&](int t) { fetch(Qs, p.qimg + ((int64_t)unit(t) * p.qt + qtile(t)) * QF, p.KD, &bars[1]); };
  auto fetch_g = [&](int t) { fetch(Gs, p.gimg + ((int64_t)unit(t) * p.qt + qtile(t)) * VF, p.DP, &bars[2]); };
  if (tid == 0 && T > 0) {
    mbar_expect_tx(&bars[0], (QF + VF) * 4);
    bulk_load(Ks, p.kimg + ((int64_t)uk * p.kt + ktile) * QF, QF * 4, &bars[0]);
    bulk_load(Vs, p.vimg + ((int64_t)uk * p.kt + ktile) * VF, VF * 4, &bars[0]);
    fetch_q(0), fetch_g(0);
  }
  float ak[4][NK], av[4][ND];
  zero(ak), zero(av);
  bool ok[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gj = j0 + ty * 4 + i;
    ok[i] = gj < p.Nk && (!mask || mask[(int64_t)gj * p.msn] != 0);
  }
  bool failed = T > 0 && !mbar_wait(&bars[0], 0, WAIT_LIMIT);
  for (int t = 0; t < T; ++t) {
    const int q0 = qtile(t) * ST_ROWS + tx * 4;
    const float *lse = p.lse_in + (int64_t)unit(t) * p.Nq, *delta = p.delta + (int64_t)unit(t) * p.Nq;
    float lse2[4], dl[4], s[4][4], dp[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float l = q0 + j < p.Nq ? __ldg(lse + q0 + j) : -CUDART_INF_F;
      lse2[j] = l == -CUDART_INF_F ? CUDART_INF_F : l * LOG2E;
      dl[j] = q0 + j < p.Nq ? __ldg(delta + q0 + j) : 0.f;
    }
    zero(s), zero(dp);
    if (!failed) failed = !mbar_wait(&bars[1], t & 1, WAIT_LIMIT);
    mm_features(s, Ks, Qs, p.KD, ty, tx);
    if (!failed) failed = !mbar_wait(&bars[2], t & 1, WAIT_LIMIT);
    mm_features(dp, Vs, Gs, p.DP, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool vis = ok[i] && (!p.causal || j0 + ty * 4 + i <= q0 + j);
        s[i][j] = vis ? exp2f(s[i][j] * p.scale_log2 - lse2[j]) : 0.f;
        dp[i][j] = s[i][j] * (dp[i][j] - dl[j]) * p.scale;
      }
    put_scores(Ss, s, ty, tx);
    __syncthreads();
    mm_rows<ND>(av, Ss, Gs, ty, tx);
    __syncthreads();   // P^T and the dO tile have been read
    if (tid == 0 && t + 1 < T) fetch_g(t + 1);
    put_scores(Ss, dp, ty, tx);
    __syncthreads();
    mm_rows<NK>(ak, Ss, Qs, ty, tx);
    __syncthreads();   // dS^T and the Q' tile have been read
    if (tid == 0 && t + 1 < T) fetch_q(t + 1);
  }
  const int astr = p.d + p.r + 1;
  stage_acc<NK>(Qs, astr, ak, p.d + p.r, ty, tx);   // Q', dO and the scores are dead: [64][d + r + 1] fits them
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gj = j0 + ty * 4 + i;
    if (gj >= p.Nk) continue;
    const int64_t base = b * p.sdv.b + hk * p.sdv.h + (int64_t)gj * p.sdv.n;
#pragma unroll
    for (int m = 0; m < ND; ++m) {
      const int col = tx * 4 + (m & 3) + 64 * (m >> 2);
      if (col < p.d) put(p.dv, base + col, av[i][m], p.dtype);
    }
  }
  __syncthreads();
  float* df = p.dfreqs ? p.dfreqs + b * p.sdf.b + hk * p.sdf.h : nullptr;
  // (a tile that no query sees has zero gradients; its K' tile was never fetched, so zeros stand in for it)
  if (T == 0) {
    for (int i = tid; i < QF; i += ST_THREADS) Ks[i] = 0.f;
    __syncthreads();
  }
  chain_rule(p, Qs, astr, Ks, j0, p.Nk, p.dk, b * p.sdk.b + hk * p.sdk.h, p.sdk.n, df, p.sdf.n, 0, p.dbias ? p.dbias + hk * p.dbias_sh : nullptr);
  if (failed) atomicOr(p.status, 1u);
}

// Both sides in one launch: the CTAs of one side fill what the other leaves idle.  Blocks come heaviest first (under the
// causal mask: late query tiles, early key tiles).
template <int ND, int NK>
__global__ void __launch_bounds__(ST_THREADS, (ND == 4 && NK <= 8) ? 2 : 1) attn_bwd_tiled_kernel(TiledP p, int nq_units, int nk_units) {
  extern __shared__ __align__(128) float st_smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(st_smem);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
    mbar_init_fence();
  }
  __syncthreads();
  pdl_wait();
  const int level = blockIdx.x / (nq_units + nk_units), w = blockIdx.x % (nq_units + nk_units);
  if (w < nk_units) {
    if (level < p.kt) bwd_dkdv_tiled<ND, NK>(p, st_smem + 32, bars, level, w);
  } else if (level < p.qt) {
    bwd_dq_tiled<ND, NK>(p, st_smem + 32, bars, p.qt - 1 - level, w - nk_units);
  }
}

// ---- host side ---------------------------------------------------------------------------------------------------------
static int up(int x, int m) { return (x + m - 1) / m * m; }
static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }
static size_t img_bytes(int units, int rows, int feats) { return up256((size_t)units * ((rows + ST_ROWS - 1) / ST_ROWS) * ST_ROWS * feats * 4); }

static size_t fwd_smem(int KD, int ND) { return (size_t)(2 * KD + ND * 16 + ST_ROWS) * ST_ROWS * 4 + 64; }
// dk / dv side: K', V resident, Q', dO streamed, one score tile (the dq side needs no more); the staged gradients,
// 64 x (d + r + 1), fit the streamed buffers of either side
static size_t bwd_smem(int KD, int DP, int ND, int NK) { return (size_t)(KD + DP + NK * 16 + ND * 16 + ST_ROWS) * ST_ROWS * 4 + 128; }

// Tiles of 64 query rows: fewer than 32 leave most of a tile empty, and the key-split kernels of simt_attn.cu serve those.
// Wider operands than these do not fit shared memory in tiles of 64 rows.
bool attn_fwd_tiled_supported(const PopeShape& s) { return s.Nq >= 32 && s.d + s.r <= 256; }
bool attn_bwd_tiled_supported(const PopeShape& s) { return s.Nq >= 32 && s.d <= 128 && s.d + s.r <= 256; }

size_t attn_fwd_tiled_workspace(const PopeShape& s) {
  const int KD = up(s.d + s.r, 8), DP = up(s.d, 8);
  return img_bytes(s.B * s.H, s.Nq, KD) + img_bytes(s.B * s.Hk, s.Nk, KD) + img_bytes(s.B * s.Hk, s.Nk, DP);
}
size_t attn_bwd_tiled_workspace(const PopeShape& s) {
  return attn_fwd_tiled_workspace(s) + img_bytes(s.B * s.H, s.Nq, up(s.d, 8)) + up256((size_t)s.B * s.H * s.Nq * 4);
}

static TiledP tiled_params(const PopeShape& s, int causal, float scale, const uint8_t* mask, int64_t msb, int64_t msn, float* ws) {
  TiledP p = {};
  p.H = s.H, p.Hk = s.Hk, p.Nq = s.Nq, p.Nk = s.Nk, p.d = s.d, p.r = s.r, p.KD = up(s.d + s.r, 8), p.DP = up(s.d, 8);
  p.qt = (s.Nq + ST_ROWS - 1) / ST_ROWS, p.kt = (s.Nk + ST_ROWS - 1) / ST_ROWS, p.causal = causal, p.dtype = s.dtype;
  p.scale = scale, p.scale_log2 = scale * LOG2E;
  p.mask = mask, p.msb = msb, p.msn = msn;
  p.qimg = ws;
  p.kimg = p.qimg + img_bytes(s.B * s.H, s.Nq, p.KD) / 4;
  p.vimg = p.kimg + img_bytes(s.B * s.Hk, s.Nk, p.KD) / 4;
  p.gimg = p.vimg + img_bytes(s.B * s.Hk, s.Nk, p.DP) / 4;
  p.status = tc_status_ptr();
  return p;
}

static TileJob tile_job(const void* x, const PopeStride3& sx, int batch, int heads, int rows, int r, int pos0, int feats, const float* img) {
  TileJob j = {};
  j.x = x, j.sx = Strides(sx), j.units = batch * heads, j.heads = heads, j.rows = rows, j.r = r, j.pos0 = pos0, j.feats = feats;
  j.img = const_cast<float*>(img);
  return j;
}

template <int ND>
static cudaError_t launch_fwd_tiled(const TiledP& p, const PopeShape& s, cudaStream_t st) {
  const size_t smem = fwd_smem(p.KD, ND);
  cudaError_t e = ensure_max_smem<attn_fwd_tiled_kernel<ND>>();
  if (e != cudaSuccess) return e;
  return launch_dependent(attn_fwd_tiled_kernel<ND>, dim3(p.qt, s.B * s.H), dim3(ST_THREADS), smem, st, p);
}

cudaError_t attn_fwd_tiled(const PopeAttnArgs& a, cudaStream_t st) {
  const PopeShape& s = a.shape;
  TiledP p = tiled_params(s, a.causal, a.softmax_scale, a.mask, a.mask_stride_b, a.mask_stride_n, static_cast<float*>(a.workspace));
  if (!p.status) return cudaErrorInvalidSymbol;
  p.o = a.out, p.so = Strides(a.so), p.lse = a.lse;
  TileJobs jobs = {};
  jobs.job[0] = tile_job(a.q, a.sq, s.B, s.H, s.Nq, s.r, s.Nk - s.Nq, p.KD, p.qimg);
  jobs.job[1] = tile_job(a.k, a.sk, s.B, s.Hk, s.Nk, s.r, 0, p.KD, p.kimg);
  jobs.job[1].bias = s.r > 0 ? a.embed.bias : nullptr, jobs.job[1].bias_sh = a.embed.bias_stride_h;
  jobs.job[2] = tile_job(a.v, a.sv, s.B, s.Hk, s.Nk, 0, 0, p.DP, p.vimg);
  const cudaError_t e = launch_tile_images(jobs, 3, s, a.embed, st);
  if (e != cudaSuccess) return e;
  return s.d <= 64 ? launch_fwd_tiled<4>(p, s, st) : s.d <= 128 ? launch_fwd_tiled<8>(p, s, st) : launch_fwd_tiled<16>(p, s, st);
}

template <int ND, int NK>
static cudaError_t launch_bwd_tiled(const TiledP& p, const PopeShape& s, cudaStream_t st) {
  const size_t smem = bwd_smem(p.KD, p.DP, ND, NK);
  cudaError_t e = ensure_max_smem<attn_bwd_tiled_kernel<ND, NK>>();
  if (e != cudaSuccess) return e;
  const int nq = s.B * s.H, nk = s.B * s.Hk;
  return launch_dependent(attn_bwd_tiled_kernel<ND, NK>, dim3((unsigned)((nq + nk) * std::max(p.qt, p.kt))), dim3(ST_THREADS), smem, st, p, nq, nk);
}

cudaError_t attn_bwd_tiled(const PopeAttnBwdArgs& a, cudaStream_t st) {
  const PopeShape& s = a.shape;
  float* ws = static_cast<float*>(a.workspace);
  float* delta = ws;
  TiledP p = tiled_params(s, a.causal, a.softmax_scale, a.mask, a.mask_stride_b, a.mask_stride_n, ws + up256((size_t)s.B * s.H * s.Nq * 4) / 4);
  if (!p.status) return cudaErrorInvalidSymbol;
  p.lse_in = a.lse, p.delta = delta;
  p.dq = a.dq, p.dk = a.dk, p.dv = a.dv, p.sdq = Strides(a.sdq), p.sdk = Strides(a.sdk), p.sdv = Strides(a.sdv), p.sdf = Strides(a.sdf);
  p.dfreqs = s.r > 0 ? a.dfreqs : nullptr, p.dbias = s.r > 0 ? a.dbias : nullptr, p.dbias_sh = a.dbias_stride_h;
  cudaError_t e = attn_bwd_delta(a, delta, st);
  if (e != cudaSuccess) return e;
  TileJobs jobs = {};
  jobs.job[0] = tile_job(a.q, a.sq, s.B, s.H, s.Nq, s.r, s.Nk - s.Nq, p.KD, p.qimg);
  jobs.job[1] = tile_job(a.k, a.sk, s.B, s.Hk, s.Nk, s.r, 0, p.KD, p.kimg);
  jobs.job[1].bias = s.r > 0 ? a.embed.bias : nullptr, jobs.job[1].bias_sh = a.embed.bias_stride_h;
  jobs.job[2] = tile_job(a.v, a.sv, s.B, s.Hk, s.Nk, 0, 0, p.DP, p.vimg);
  jobs.job[3] = tile_job(a.dout, a.sdo, s.B, s.H, s.Nq, 0, 0, p.DP, p.gimg);
  if ((e = launch_tile_images(jobs, 4, s, a.embed, st)) != cudaSuccess) return e;
  const int kd = s.d + s.r;
  if (s.d <= 64) return kd <= 64 ? launch_bwd_tiled<4, 4>(p, s, st) : launch_bwd_tiled<4, 8>(p, s, st);
  return kd <= 128 ? launch_bwd_tiled<8, 8>(p, s, st) : kd <= 192 ? launch_bwd_tiled<8, 12>(p, s, st) : launch_bwd_tiled<8, 16>(p, s, st);
}

}  // namespace pope
