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
//   * a thread owns 4 rows x 8 columns of the score tile (4 x 4 where the accumulators are wide) and a warp 16 rows x 64
//     columns, 4 x 8 lanes: of the three 16-byte loads per 32 FMAs the lanes of a half-warp share addresses, six
//     wavefronts in eight clocks of the FMA pipe.  (4 x 4 per thread and 2 x 16 lanes: six wavefronts in four clocks, and
//     shared memory set the pace.)
//   * small grids are cut along the streamed operand: a cluster of 2 or 4 CTAs shares a tile, each takes a part of the
//     stream, and the partial accumulators meet in distributed shared memory.
// Measured at (1, 8, 1024, 64), r = 64, causal, fp32, a whole training step: 1131 us with the kernels of simt_attn.cu, 609 in tiles
// with 4 x 4 scores per thread, 341 with 4 x 8 and clusters, 337 with the images of a tile dealt over several CTAs (80 us at the
// nominal fp32 rate).
//
// Semantics: PoPE_pytorch/triton_pope_flash_attn.py:23-218 (top-left causal mask, bottom-right positions, mask True = keep,
// zero output and -inf LSE for empty rows).
#include <math_constants.h>

#include <algorithm>

#include "kernels.h"
#include "tc_common.cuh"

namespace pope {

constexpr int ST_ROWS = 64;        // rows of a tile

// Thread layout: TX = 8: 128 threads, 4 x 8 scores each; TX = 16: 256 threads, 4 x 4.  Rows 4 ty + i; column (or feature) j of
// a thread is 4 tx + j % 4 + 4 TX (j / 4).
template <int TX> struct Lay {
  static constexpr int THREADS = 16 * TX, CS = 64 / TX;
  int tx, ty;
  __device__ __forceinline__ Lay() {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    tx = (lane & 7) + (TX == 16 ? (w & 1) * 8 : 0), ty = (TX == 16 ? w >> 1 : w) * 4 + (lane >> 3);
  }
  __device__ __forceinline__ int col(int j) const { return tx * 4 + (j & 3) + 4 * TX * (j >> 2); }
};

struct TiledP {
  int H, Hk, Nq, Nk, d, r, KD;     // KD = d + r rounded up to 8: features of a Q' / K' tile
  int qt, kt, causal, dtype;       // tiles per unit
  int split;                       // CTAs of a cluster that share a tile
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

// grid (tiles x slices, units, jobs).  Lanes take consecutive rows of one feature: the stores of a warp are whole lines, and the
// loads, a line per lane, come back from L1 for the next 31 features.  A thread takes every 4 slices-th feature, four at a time
// with their loads up front.
template <typename T>
__global__ void __launch_bounds__(256) tile_image_kernel(TileJobs jobs, int d, int slices, const float* freqs, Strides sf) {
  pdl_wait();
  pdl_trigger();
  const TileJob& jb = jobs.job[blockIdx.z];
  const int tile = blockIdx.x / slices, u = blockIdx.y;
  if (u >= jb.units || tile * ST_ROWS >= jb.rows) return;
  const int c0 = (blockIdx.x % slices) * 4 + (threadIdx.x >> 6), step = 4 * slices;
  const int b = u / jb.heads, h = u % jb.heads;
  const int row = threadIdx.x & 63, j = tile * ST_ROWS + row;
  const bool ok = j < jb.rows;
  const T* x = static_cast<const T*>(jb.x) + b * jb.sx.b + h * jb.sx.h + (int64_t)j * jb.sx.n;
  const float* f = freqs + b * sf.b + h * sf.h + (int64_t)(jb.pos0 + j) * sf.n;
  const float* bias = jb.bias ? jb.bias + h * jb.bias_sh : nullptr;
  float* img = jb.img + ((int64_t)u * ((jb.rows + ST_ROWS - 1) / ST_ROWS) + tile) * jb.feats * ST_ROWS;
  auto at = [&](int c) { return img + c * ST_ROWS + ((((row >> 2) ^ (c >> 2)) & 15) << 2) + (row & 3); };
  constexpr int CU = 4;
  for (int first = c0; first < d; first += CU * step) {
    float v[CU], ph[CU];
#pragma unroll
    for (int i = 0; i < CU; ++i) {
      const int c = first + i * step;
      v[i] = ok && c < d ? to_f32<T>(x[c]) : 0.f;
      ph[i] = ok && c < jb.r ? (bias ? f[c] + bias[c] : f[c]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < CU; ++i) {
      const int c = first + i * step;
      if (c >= d) break;
      if (c < jb.r) {
        float cs = 0.f, sn = 0.f;
        if (ok) {
          sincosf(ph[i], &sn, &cs);
          const float a = softplus_f(v[i]);
          cs *= a, sn *= a;
        }
        *at(c) = cs, *at(d + c) = sn;
      } else {
        *at(c) = v[i];
      }
    }
  }
  for (int c = d + jb.r + c0; c < jb.feats; c += step) *at(c) = 0.f;
}

static cudaError_t launch_tile_images(const TileJobs& jobs, int njobs, const PopeShape& s, const PopeEmbed& e, cudaStream_t st) {
  int tiles = 0, units = 0;
  for (int i = 0; i < njobs; ++i) {
    tiles = max(tiles, (jobs.job[i].rows + ST_ROWS - 1) / ST_ROWS), units = max(units, jobs.job[i].units);
  }
  // feature slices: until every SM has eight CTAs, at most four.  At (1, 8, 1024, 64), r = 64, four operands of the backward:
  // 1 slice 19.4 us, 2 slices 16.5, 4 slices 15.5
  int slices = 1;
  while (slices < 4 && (int64_t)tiles * units * njobs * slices * 2 <= 148 * 16) slices *= 2;
  const dim3 grid((unsigned)(tiles * slices), (unsigned)units, (unsigned)njobs), block(256);
  switch (s.dtype) {
    case POPE_F32: return launch_dependent(tile_image_kernel<float>, grid, block, 0, st, jobs, s.d, slices, e.freqs, Strides(e.sf));
    case POPE_BF16: return launch_dependent(tile_image_kernel<__nv_bfloat16>, grid, block, 0, st, jobs, s.d, slices, e.freqs, Strides(e.sf));
    default: return launch_dependent(tile_image_kernel<__half>, grid, block, 0, st, jobs, s.d, slices, e.freqs, Strides(e.sf));
  }
}

// ---- tile products ---------------------------------------------------------------------------------------------------
// c[i][j] += sum over features k < n of A[k][row(i)] B[k][col(j)], both feature-major tiles
template <int TX>
__device__ __forceinline__ void mm_features(float (&c)[4][64 / TX], const float* A, const float* B, int n, Lay<TX> L) {
  constexpr int CS = 64 / TX;
#pragma unroll 2
  for (int k4 = 0; k4 < n; k4 += 4) {
    const int sw = (k4 >> 2) & 15;
    const float* a = A + k4 * ST_ROWS + ((L.ty ^ sw) << 2);
    const float* b[CS / 4];
#pragma unroll
    for (int q = 0; q < CS / 4; ++q) b[q] = B + k4 * ST_ROWS + (((L.tx + TX * q) ^ sw) << 2);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 av = *reinterpret_cast<const float4*>(a + k * ST_ROWS);
      const float x[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int q = 0; q < CS / 4; ++q) {
        const float4 bv = *reinterpret_cast<const float4*>(b[q] + k * ST_ROWS);
        const float y[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) c[i][q * 4 + j] = fmaf(x[i], y[j], c[i][q * 4 + j]);
      }
    }
  }
}

// c[i][m] += sum over the 64 tile rows t of S[row(i)][t] B[col(m)][t]: S is a row-major score tile (put_scores), B a
// feature-major tile
template <int TX, int NC>
__device__ __forceinline__ void mm_rows(float (&c)[4][NC], const float* S, const float* B, Lay<TX> L) {
  const float* s = S + L.ty * 4 * ST_ROWS;
  const float* b = B + L.tx * 4 * ST_ROWS;
#pragma unroll 2
  for (int g = 0; g < 16; ++g) {
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(s + i * ST_ROWS + ((g ^ L.ty) << 2));
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const float4 y = *reinterpret_cast<const float4*>(b + ((m >> 2) * 4 * TX + (m & 3)) * ST_ROWS + ((g ^ ((L.tx + TX * (m >> 2)) & 15)) << 2));
#pragma unroll
      for (int i = 0; i < 4; ++i) c[i][m] = fmaf(x[i].w, y.w, fmaf(x[i].z, y.z, fmaf(x[i].y, y.y, fmaf(x[i].x, y.x, c[i][m]))));
    }
  }
}

template <int TX>
__device__ __forceinline__ void put_scores(float* S, const float (&v)[4][64 / TX], Lay<TX> L) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 64 / TX / 4; ++q)
      *reinterpret_cast<float4*>(S + (L.ty * 4 + i) * ST_ROWS + (((L.tx + TX * q) ^ L.ty) << 2)) =
          make_float4(v[i][q * 4], v[i][q * 4 + 1], v[i][q * 4 + 2], v[i][q * 4 + 3]);
}

template <int N> __device__ __forceinline__ void zero(float (&c)[4][N]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) c[i][j] = 0.f;
}

// the sum of *p over the CTAs that share a tile
__device__ __forceinline__ float over_split(const float* p, int split) {
  if (split == 1) return *p;
  float v = 0.f;
  for (int r = 0; r < split; ++r) v += dsmem_ld(p, r);
  return v;
}
__device__ __forceinline__ void split_sync(int split) {
  if (split == 1) __syncthreads();
  else __syncwarp(), cluster_sync();
}

// every thread is done with a buffer that a copy is about to refill
__device__ __forceinline__ void release_sync() { fence_async_smem(), __syncthreads(); }

// one image tile by bulk copy; a thread of the CTA calls it behind release_sync()
__device__ __forceinline__ void fetch(float* dst, const float* img, int feats, uint64_t* bar) {
  mbar_expect_tx(bar, feats * ST_ROWS * 4);
  bulk_load(dst, img, feats * ST_ROWS * 4, bar);
}

// ---- forward ---------------------------------------------------------------------------------------------------------
// Shared memory: Q' tile, K' tile, V tile, P.  The K' buffer is free once the scores are in registers and refilled behind
// the softmax and P V, the V buffer is refilled behind the next scores; where two CTAs fit an SM they cover the rest.
// ND: output features per thread.
template <int ND>
__global__ void __launch_bounds__(128, ND == 8 ? 2 : 1) attn_fwd_tiled_kernel(TiledP p) {
  constexpr int TX = 8, CS = 8;
  extern __shared__ __align__(128) float st_smem[];
  const int QF = p.KD * ST_ROWS, VF = ND * TX * ST_ROWS;
  float *Qs = st_smem, *Ks = Qs + QF, *Vs = Ks + QF, *Ps = Vs + VF, *ml = Ps + ST_ROWS * ST_ROWS;   // ml: [64] maxima, [64] sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(ml + 2 * ST_ROWS);   // Q', K', V landed
  const int tid = threadIdx.x;
  const Lay<TX> L;
  const int u = blockIdx.y, b = u / p.H, h = u % p.H, hk = h % p.Hk, uk = b * p.Hk + hk;
  const int rank = blockIdx.x % p.split, qtile = p.qt - 1 - blockIdx.x / p.split, i0 = qtile * ST_ROWS;   // heavy (late) row blocks first
  int n_end = p.Nk;
  if (p.causal) n_end = min(n_end, min(i0 + ST_ROWS, p.Nq));
  const int tiles = (n_end + ST_ROWS - 1) / ST_ROWS, t0 = tiles * rank / p.split, T = tiles * (rank + 1) / p.split - t0;
  const float* kimg = p.kimg + ((int64_t)uk * p.kt + t0) * QF;
  const float* vimg = p.vimg + ((int64_t)uk * p.kt + t0) * p.DP * ST_ROWS;
  const uint8_t* mask = p.mask ? p.mask + b * p.msb : nullptr;
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
    mbar_init_fence();
  }
  pdl_wait();
  if (tid == 0 && T > 0) {
    fetch(Qs, p.qimg + ((int64_t)u * p.qt + qtile) * QF, p.KD, &bars[0]);
    fetch(Ks, kimg, p.KD, &bars[1]);
    fetch(Vs, vimg, p.DP, &bars[2]);
  }
  __syncthreads();
  bool failed = T > 0 && !mbar_wait(&bars[0], 0, WAIT_LIMIT);
  float m[4], l[4], o[4][ND];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i] = -CUDART_INF_F, l[i] = 0.f;
  zero(o);
  for (int t = 0; t < T; ++t) {
    const int n0 = (t0 + t) * ST_ROWS;
    float s[4][CS];
    zero(s);
    uint32_t ok = 0;
#pragma unroll
    for (int j = 0; j < CS; ++j) {
      const int key = n0 + L.col(j);
      ok |= (uint32_t)(key < p.Nk && (!mask || mask[(int64_t)key * p.msn] != 0)) << j;
    }
    if (!failed) failed = !mbar_wait(&bars[1], t & 1, WAIT_LIMIT);
    mm_features<TX>(s, Qs, Ks, p.KD, L);
    release_sync();   // the K' tile and (from the last round) P have been read
    if (tid == 0 && t + 1 < T) fetch(Ks, kimg + (int64_t)(t + 1) * QF, p.KD, &bars[1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gi = i0 + L.ty * 4 + i;
      float mx = -CUDART_INF_F;
#pragma unroll
      for (int j = 0; j < CS; ++j) {
        s[i][j] = ((ok >> j) & 1u) && (!p.causal || n0 + L.col(j) <= gi) ? s[i][j] * p.scale_log2 : -CUDART_INF_F;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int off = 4; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m[i], mx), m_use = m_new == -CUDART_INF_F ? 0.f : m_new;
      const float alpha = exp2f(m[i] - m_use);   // 0 on the first visible tile
      m[i] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < CS; ++j) s[i][j] = exp2f(s[i][j] - m_use), sum += s[i][j];
      l[i] = l[i] * alpha + sum;                 // this lane's columns; the lanes of a row are summed at the end
#pragma unroll
      for (int c = 0; c < ND; ++c) o[i][c] *= alpha;
    }
    put_scores<TX>(Ps, s, L);
    __syncthreads();
    if (!failed) failed = !mbar_wait(&bars[2], t & 1, WAIT_LIMIT);
    mm_rows<TX, ND>(o, Ps, Vs, L);
    if (t + 1 < T) {
      release_sync();   // the V tile has been read
      if (tid == 0) fetch(Vs, vimg + (int64_t)(t + 1) * p.DP * ST_ROWS, p.DP, &bars[2]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], off);
  if (p.split == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int gi = i0 + L.ty * 4 + i;
      if (gi >= p.Nq) continue;
      const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
      const int64_t base = b * p.so.b + h * p.so.h + (int64_t)gi * p.so.n;
#pragma unroll
      for (int c = 0; c < ND; ++c)
        if (L.col(c) < p.d) put(p.o, base + L.col(c), o[i][c] * inv, p.dtype);
      if (L.tx == 0) p.lse[(int64_t)u * p.Nq + gi] = l[i] > 0.f ? m[i] * LN2 + logf(l[i]) : -CUDART_INF_F;
    }
  } else {
    // the parts of the key range meet: (max, sum, output) of every CTA in its own shared memory, each CTA finishes its
    // share of the rows
    float* os = Vs;   // [64][ND * TX]; V and P are dead
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = L.ty * 4 + i;
#pragma unroll
      for (int c = 0; c < ND; ++c) os[row * (ND * TX) + L.col(c)] = o[i][c];
      if (L.tx == 0) ml[row] = m[i], ml[ST_ROWS + row] = l[i];
    }
    split_sync(p.split);
    const int r0 = ST_ROWS * rank / p.split, r1 = ST_ROWS * (rank + 1) / p.split;
    for (int row = r0 + (tid >> 5); row < r1 && i0 + row < p.Nq; row += 4) {
      float M = -CUDART_INF_F, sum = 0.f, w[4];
      for (int r = 0; r < p.split; ++r) M = fmaxf(M, dsmem_ld(ml + row, r));
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        w[r] = r < p.split && M != -CUDART_INF_F ? exp2f(dsmem_ld(ml + row, r) - M) : 0.f;
        if (r < p.split) sum += w[r] * dsmem_ld(ml + ST_ROWS + row, r);
      }
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
      const int64_t base = b * p.so.b + h * p.so.h + (int64_t)(i0 + row) * p.so.n;
      for (int c = tid & 31; c < p.d; c += 32) {
        float v = 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r < p.split) v = fmaf(w[r], dsmem_ld(os + row * (ND * TX) + c, r), v);
        put(p.o, base + c, v * inv, p.dtype);
      }
      if ((tid & 31) == 0) p.lse[(int64_t)u * p.Nq + i0 + row] = sum > 0.f ? M * LN2 + logf(sum) : -CUDART_INF_F;
    }
    split_sync(p.split);   // nobody leaves while its shared memory is read
  }
  if (failed) atomicOr(p.status, 1u);
}

// ---- backward ----------------------------------------------------------------------------------------------------------
// Epilogue: X' gradients of rows [r0, r1) of a tile, staged as [64][astr] by every CTA that shares it -> dx, dphase.  Everything the chain rule needs is in the resident
// image tile: with xc = a cos, xs = a sin,  a = hypot(xc, xs),  sigmoid(x) = 1 - exp(-a),
//   dx = (gc xc + gs xs) / a * sigmoid(x),  dphase = gs xc - gc xs.
__device__ __forceinline__ void chain_rule(const TiledP& p, const float* acc, int astr, const float* X, int row0, int rows, void* dx, int64_t base,
                                           int64_t sn, float* df, int64_t sfn, int pos0, float* dbias, int rank) {
  const int r0 = ST_ROWS * rank / p.split, r1 = ST_ROWS * (rank + 1) / p.split;
  for (int c = threadIdx.x & 63; c < p.d; c += 64) {
    float sum = 0.f;
    for (int row = r0 + (threadIdx.x >> 6); row < r1 && row0 + row < rows; row += blockDim.x >> 6) {
      float g = over_split(acc + row * astr + c, p.split);
      if (c < p.r) {
        const int grp = row >> 2, e = row & 3;
        const float gs = over_split(acc + row * astr + p.d + c, p.split);
        const float xc = X[c * ST_ROWS + (((grp ^ (c >> 2)) & 15) << 2) + e];
        const float xs = X[(p.d + c) * ST_ROWS + (((grp ^ ((p.d + c) >> 2)) & 15) << 2) + e];
        const float a = hypotf(xc, xs), dph = gs * xc - g * xs;   // (the squares leave the range of fp32 below x = -44 and above 1e19)
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
template <int TX, int N> __device__ __forceinline__ void stage_acc(float* dst, int stride, const float (&c)[4][N], int width, Lay<TX> L) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int m = 0; m < N; ++m)
      if (L.col(m) < width) dst[(L.ty * 4 + i) * stride + L.col(m)] = c[i][m];
}

// dq: 64 query rows resident (Q', dO); streams K' and V tiles:  S, dP -> dS -> dQ' += dS K'
template <int TX, int ND, int NK>
__device__ __forceinline__ void bwd_dq_tiled(const TiledP& p, float* smem, uint64_t* bars, int qtile, int u, int rank) {
  constexpr int CS = 64 / TX;
  const int QF = p.KD * ST_ROWS, QA = NK * TX * ST_ROWS, VF = p.DP * ST_ROWS;
  float *Qs = smem, *Gs = Qs + QF, *Ks = Gs + VF, *Vs = Ks + QA, *Ss = Vs + VF;
  const int tid = threadIdx.x;
  const Lay<TX> L;
  const int b = u / p.H, h = u % p.H, hk = h % p.Hk, uk = b * p.Hk + hk, i0 = qtile * ST_ROWS;
  int n_end = p.Nk;
  if (p.causal) n_end = min(n_end, min(i0 + ST_ROWS, p.Nq));
  const int tiles = (n_end + ST_ROWS - 1) / ST_ROWS, t0 = tiles * rank / p.split, T = tiles * (rank + 1) / p.split - t0;
  const float* kimg = p.kimg + ((int64_t)uk * p.kt + t0) * QF;
  const float* vimg = p.vimg + ((int64_t)uk * p.kt + t0) * VF;
  const uint8_t* mask = p.mask ? p.mask + b * p.msb : nullptr;
  if (tid == 0) {
    mbar_expect_tx(&bars[0], (QF + VF) * 4);
    bulk_load(Qs, p.qimg + ((int64_t)u * p.qt + qtile) * QF, QF * 4, &bars[0]);
    bulk_load(Gs, p.gimg + ((int64_t)u * p.qt + qtile) * VF, VF * 4, &bars[0]);
    if (T > 0) fetch(Ks, kimg, p.KD, &bars[1]), fetch(Vs, vimg, p.DP, &bars[2]);
  }
  float lse2[4], dl[4], acc[4][NK];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gi = i0 + L.ty * 4 + i;
    const float l = gi < p.Nq ? p.lse_in[(int64_t)u * p.Nq + gi] : -CUDART_INF_F;
    lse2[i] = l == -CUDART_INF_F ? CUDART_INF_F : l * LOG2E;   // +inf: probabilities are exactly 0
    dl[i] = gi < p.Nq ? p.delta[(int64_t)u * p.Nq + gi] : 0.f;
  }
  zero(acc);
  bool failed = !mbar_wait(&bars[0], 0, WAIT_LIMIT);
  for (int t = 0; t < T; ++t) {
    const int n0 = (t0 + t) * ST_ROWS;
    float s[4][CS], dp[4][CS];
    zero(s), zero(dp);
    uint32_t ok = 0;
#pragma unroll
    for (int j = 0; j < CS; ++j) {
      const int key = n0 + L.col(j);
      ok |= (uint32_t)(key < p.Nk && (!mask || mask[(int64_t)key * p.msn] != 0)) << j;
    }
    if (!failed) failed = !mbar_wait(&bars[2], t & 1, WAIT_LIMIT);
    mm_features<TX>(dp, Gs, Vs, p.DP, L);
    if (!failed) failed = !mbar_wait(&bars[1], t & 1, WAIT_LIMIT);
    mm_features<TX>(s, Qs, Ks, p.KD, L);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < CS; ++j) {
        const bool vis = ((ok >> j) & 1u) && (!p.causal || n0 + L.col(j) <= i0 + L.ty * 4 + i);
        s[i][j] = vis ? exp2f(s[i][j] * p.scale_log2 - lse2[i]) * (dp[i][j] - dl[i]) * p.scale : 0.f;
      }
    put_scores<TX>(Ss, s, L);
    release_sync();   // dS is written, the V tile has been read
    if (tid == 0 && t + 1 < T) fetch(Vs, vimg + (int64_t)(t + 1) * VF, p.DP, &bars[2]);
    mm_rows<TX, NK>(acc, Ss, Ks, L);
    release_sync();   // the K' tile and dS have been read
    if (tid == 0 && t + 1 < T) fetch(Ks, kimg + (int64_t)(t + 1) * QF, p.KD, &bars[1]);
  }
  const int astr = p.d + p.r + 1;
  stage_acc<TX, NK>(Gs, astr, acc, p.d + p.r, L);   // dO, K', V and dS are dead: [64][d + r + 1] fits them
  split_sync(p.split);
  float* df = p.dfreqs ? p.dfreqs + b * p.sdf.b + h * p.sdf.h : nullptr;
  chain_rule(p, Gs, astr, Qs, i0, p.Nq, p.dq, b * p.sdq.b + h * p.sdq.h, p.sdq.n, df, p.sdf.n, p.Nk - p.Nq, nullptr, rank);
  if (p.split > 1) split_sync(p.split);   // nobody leaves while its shared memory is read
  if (failed) atomicOr(p.status, 1u);
}

// dk / dv: 64 key rows resident (K', V); streams the Q' and dO tiles of every grouped query head:
// S^T, dP^T -> P^T -> dV += P^T dO, dS^T -> dK' += dS^T Q'
template <int TX, int ND, int NK>
__device__ __forceinline__ void bwd_dkdv_tiled(const TiledP& p, float* smem, uint64_t* bars, int ktile, int uk, int rank) {
  constexpr int CS = 64 / TX;
  const int QF = p.KD * ST_ROWS, QA = NK * TX * ST_ROWS, VF = p.DP * ST_ROWS, VA = ND * TX * ST_ROWS;
  float *Ks = smem, *Vs = Ks + QF, *Qs = Vs + VF, *Gs = Qs + QA, *Ss = Gs + VA;
  const int tid = threadIdx.x;
  const Lay<TX> L;
  const int b = uk / p.Hk, hk = uk % p.Hk, j0 = ktile * ST_ROWS, groups = p.H / p.Hk;
  const int t_first = p.causal ? ktile : 0;   // under the causal mask queries before this tile see none of its keys
  const int per = p.qt > t_first ? p.qt - t_first : 0, total = per * groups;
  const int s0 = total * rank / p.split, T = total * (rank + 1) / p.split - s0;   // this CTA's part of the stream
  const uint8_t* mask = p.mask ? p.mask + b * p.msb : nullptr;
  auto unit = [&](int t) { return b * p.H + ((s0 + t) / per) * p.Hk + hk; };
  auto qtile = [&](int t) { return t_first + (s0 + t) % per; };
  auto fetch_q = [&](int t) { fetch(Qs, p.qimg + ((int64_t)unit(t) * p.qt + qtile(t)) * QF, p.KD, &bars[1]); };
  auto fetch_g = [&](int t) { fetch(Gs, p.gimg + ((int64_t)unit(t) * p.qt + qtile(t)) * VF, p.DP, &bars[2]); };
  if (tid == 0) {
    mbar_expect_tx(&bars[0], (QF + VF) * 4);
    bulk_load(Ks, p.kimg + ((int64_t)uk * p.kt + ktile) * QF, QF * 4, &bars[0]);
    bulk_load(Vs, p.vimg + ((int64_t)uk * p.kt + ktile) * VF, VF * 4, &bars[0]);
    if (T > 0) fetch_q(0), fetch_g(0);
  }
  float ak[4][NK], av[4][ND];
  zero(ak), zero(av);
  bool ok[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gj = j0 + L.ty * 4 + i;
    ok[i] = gj < p.Nk && (!mask || mask[(int64_t)gj * p.msn] != 0);
  }
  bool failed = !mbar_wait(&bars[0], 0, WAIT_LIMIT);
  for (int t = 0; t < T; ++t) {
    const int q0 = qtile(t) * ST_ROWS;
    const float *lse = p.lse_in + (int64_t)unit(t) * p.Nq, *delta = p.delta + (int64_t)unit(t) * p.Nq;
    float lse2[CS], dl[CS], s[4][CS], dp[4][CS];
#pragma unroll
    for (int j = 0; j < CS; ++j) {
      const int i = q0 + L.col(j);
      const float l = i < p.Nq ? lse[i] : -CUDART_INF_F;
      lse2[j] = l == -CUDART_INF_F ? CUDART_INF_F : l * LOG2E;
      dl[j] = i < p.Nq ? delta[i] : 0.f;
    }
    zero(s), zero(dp);
    if (!failed) failed = !mbar_wait(&bars[1], t & 1, WAIT_LIMIT);
    mm_features<TX>(s, Ks, Qs, p.KD, L);
    if (!failed) failed = !mbar_wait(&bars[2], t & 1, WAIT_LIMIT);
    mm_features<TX>(dp, Vs, Gs, p.DP, L);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < CS; ++j) {
        const bool vis = ok[i] && (!p.causal || j0 + L.ty * 4 + i <= q0 + L.col(j));
        s[i][j] = vis ? exp2f(s[i][j] * p.scale_log2 - lse2[j]) : 0.f;
        dp[i][j] = s[i][j] * (dp[i][j] - dl[j]) * p.scale;
      }
    put_scores<TX>(Ss, s, L);
    __syncthreads();
    mm_rows<TX, ND>(av, Ss, Gs, L);
    release_sync();   // P^T and the dO tile have been read
    if (tid == 0 && t + 1 < T) fetch_g(t + 1);
    put_scores<TX>(Ss, dp, L);
    __syncthreads();
    mm_rows<TX, NK>(ak, Ss, Qs, L);
    release_sync();   // dS^T and the Q' tile have been read
    if (tid == 0 && t + 1 < T) fetch_q(t + 1);
  }
  const int astr = p.d + p.r + 1;
  stage_acc<TX, NK>(Qs, astr, ak, p.d + p.r, L);   // Q', dO and the scores are dead: [64][d + r + 1] fits them
  // dV: with one CTA per tile straight from the registers, else through the (dead) buffers behind the staged dK'
  float* vs = Qs + ST_ROWS * astr;   // [64][d + 1]
  if (p.split > 1) stage_acc<TX, ND>(vs, p.d + 1, av, p.d, L);
  split_sync(p.split);
  const int64_t vbase = b * p.sdv.b + hk * p.sdv.h + (int64_t)j0 * p.sdv.n;
  if (p.split > 1) {
    for (int idx = tid; idx < (ST_ROWS / p.split) * p.d; idx += Lay<TX>::THREADS) {
      const int row = ST_ROWS / p.split * rank + idx / p.d, c = idx % p.d;
      if (j0 + row < p.Nk) put(p.dv, vbase + row * p.sdv.n + c, over_split(vs + row * (p.d + 1) + c, p.split), p.dtype);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < ND; ++m)
        if (L.col(m) < p.d && j0 + L.ty * 4 + i < p.Nk) put(p.dv, vbase + (L.ty * 4 + i) * p.sdv.n + L.col(m), av[i][m], p.dtype);
  }
  float* df = p.dfreqs ? p.dfreqs + b * p.sdf.b + hk * p.sdf.h : nullptr;
  chain_rule(p, Qs, astr, Ks, j0, p.Nk, p.dk, b * p.sdk.b + hk * p.sdk.h, p.sdk.n, df, p.sdf.n, 0, p.dbias ? p.dbias + hk * p.dbias_sh : nullptr, rank);
  if (p.split > 1) split_sync(p.split);   // nobody leaves while its shared memory is read
  if (failed) atomicOr(p.status, 1u);
}

// Both sides in one launch: the CTAs of one side fill what the other leaves idle.  Blocks come heaviest first (under the
// causal mask: late query tiles, early key tiles).
template <int TX, int ND, int NK>
__global__ void __launch_bounds__(16 * TX, NK * TX <= 128 ? 2 : 1) attn_bwd_tiled_kernel(TiledP p, int nq_units, int nk_units) {
  extern __shared__ __align__(128) float st_smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(st_smem);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
    mbar_init_fence();
  }
  __syncthreads();
  pdl_wait();
  const int rank = blockIdx.x % p.split, id = blockIdx.x / p.split, level = id / (nq_units + nk_units), w = id % (nq_units + nk_units);
  if (w < nk_units) {
    if (level < p.kt) bwd_dkdv_tiled<TX, ND, NK>(p, st_smem + 32, bars, level, w, rank);
  } else if (level < p.qt) {
    bwd_dq_tiled<TX, ND, NK>(p, st_smem + 32, bars, p.qt - 1 - level, w - nk_units, rank);
  }
}

// ---- host side ---------------------------------------------------------------------------------------------------------
static int up(int x, int m) { return (x + m - 1) / m * m; }
static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }
static size_t img_bytes(int units, int rows, int feats) { return up256((size_t)units * ((rows + ST_ROWS - 1) / ST_ROWS) * ST_ROWS * feats * 4); }

static size_t fwd_smem(int KD, int d_wide) { return (size_t)(2 * KD + d_wide + ST_ROWS + 2) * ST_ROWS * 4 + 64; }
// dk / dv side: K', V resident, Q', dO streamed, one score tile (the dq side needs no more); the staged gradients,
// 64 x (2 d + r + 2), fit the streamed buffers and the score tile of either side
static size_t bwd_smem(int KD, int DP, int d_wide, int k_wide) { return (size_t)(KD + DP + k_wide + d_wide + ST_ROWS) * ST_ROWS * 4 + 128; }

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

// CTAs per tile: until two per SM are there, as long as each keeps at least two streamed tiles
static int tiled_split(int64_t ctas, int stream) {
  int n = 1;
  while (n < 4 && ctas * n < 2 * 148 && stream >= 4 * n) n *= 2;
  return n;
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
  const size_t smem = fwd_smem(p.KD, ND * 8);
  cudaError_t e = ensure_max_smem<attn_fwd_tiled_kernel<ND>>();
  if (e != cudaSuccess) return e;
  return launch_clusters(attn_fwd_tiled_kernel<ND>, p.split, dim3(p.qt * p.split, s.B * s.H), dim3(128), smem, st, true, p);
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
  p.split = tiled_split((int64_t)p.qt * s.B * s.H, p.kt);
  return s.d <= 64 ? launch_fwd_tiled<8>(p, s, st) : s.d <= 128 ? launch_fwd_tiled<16>(p, s, st) : launch_fwd_tiled<32>(p, s, st);
}

template <int TX, int ND, int NK>
static cudaError_t launch_bwd_tiled(const TiledP& p, const PopeShape& s, cudaStream_t st) {
  const size_t smem = bwd_smem(p.KD, p.DP, ND * TX, NK * TX);
  cudaError_t e = ensure_max_smem<attn_bwd_tiled_kernel<TX, ND, NK>>();
  if (e != cudaSuccess) return e;
  const int nq = s.B * s.H, nk = s.B * s.Hk;
  return launch_clusters(attn_bwd_tiled_kernel<TX, ND, NK>, p.split, dim3((unsigned)((nq + nk) * std::max(p.qt, p.kt) * p.split)), dim3(16 * TX), smem, st, true, p,
                         nq, nk);
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
  p.split = tiled_split((int64_t)p.qt * s.B * s.H + (int64_t)p.kt * s.B * s.Hk, std::min(p.qt, p.kt));
  if (s.d <= 64) return kd <= 64 ? launch_bwd_tiled<8, 8, 8>(p, s, st) : launch_bwd_tiled<8, 8, 16>(p, s, st);
  return kd <= 128 ? launch_bwd_tiled<8, 16, 16>(p, s, st) : kd <= 192 ? launch_bwd_tiled<16, 8, 12>(p, s, st) : launch_bwd_tiled<16, 8, 16>(p, s, st);
}

}  // namespace pope
