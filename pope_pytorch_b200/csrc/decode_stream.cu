// Single-token decode of PoPE attention for 16-bit inputs (sm_100a): one query row per (batch, head) unit against a
// long key / value range.  The work is one pass over K and V (HBM-bound: bytes = K + V), so the kernel is built around
// the copy engine:
//
//   loader warp    : streams tiles of keys through a ring of shared-memory stages with cp.async.bulk (K rows, V rows,
//                    and the fp16 cos / sin rows of the position phase table), completion by mbarrier transaction bytes
//   8 worker warps : LPK lanes share one key; every lane transforms 8-feature chunks of the key straight out of shared
//                    memory (softplus magnitude, table phase) and multiplies them with the query's pre-rotated polar
//                    coordinates, a short shuffle reduction gives the score; every warp keeps its own running
//                    (max, sum, output) over its keys, so no block-wide barrier sits in the loop
//
// With q' = (a_q cos fq, a_q sin fq) and k' = (a_k cos(fk + b), a_k sin(fk + b)) the score term of a rotated feature
// is a_q a_k cos(fq - fk - b) = a_k (Qc cos fk + Qs sin fk), Qc = a_q cos(fq - b), Qs = a_q sin(fq - b): the head's bias
// is folded into the query once per CTA and the key side needs only the bias-free table shared by all units.
// Key ranges are split over CTAs; their partial (o, max, sum) meet in the kernel: in a cluster's shared
// memory, or in the workspace, where the CTA that finishes last merges its unit.
//
// Semantics: PoPE_pytorch/triton_pope_flash_attn.py:52-57,73-80 (transform), :89-91 (mask, True = keep), :96-117
// (softmax, empty rows); the query sits at the LAST table row (PoPE_pytorch/pope.py:64).
//
// Paged cache: the same kernel with K and V in fixed-size pages ([page][key head][page_size][d], page_size a multiple of
// the 64-key tile, so a tile never straddles pages): the page indices of the CTA's key range are read into shared
// memory once, the loader takes each tile's address from them, and every sequence has its own length (the query sits
// at its last cached position).  kv_append_kernel writes new rows into the pages.
#include <algorithm>

#include "kernels.h"
#include "tc_common.cuh"

namespace pope {


struct DecodeStreamP {
  int H, Hk, Nk, r, nsplit, nstages, head_blocks;   // head_blocks: groups of G query heads per key head
  int k_rows_contiguous, v_rows_contiguous;
  float scale_log2;
  const void *q, *k, *v;
  Strides sq, sk, sv, so;
  void* out;
  float* lse;
  const float *freqs, *bias;
  int64_t sfn, bias_sh;
  const __half *ch, *sh;     // fp16 cos / sin of freqs, [Nk][r]
  const uint8_t* mask;
  int64_t msb, msn;
  float *part_o, *part_ml;   // [unit][split][G][D] and [unit][split][G][max (log2 units), sum]
  unsigned int* done;        // [unit] CTAs of the unit that have written their partials; zero when the kernel starts
  unsigned int* status;
  // paged cache (page_table != nullptr): k / v point at the page pools, sk.h / sv.h = page_size * d, sk.n = sv.n = d
  const int32_t* page_table;
  const int32_t* seq_lens;
  int page_size, max_pages, num_pages, npg_smem;
  int64_t page_stride;       // elements per page
};

// two fp32 lanes per instruction (the kernel is bound by instruction issue, not by FMA throughput)
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 x, y, z, w;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmov.b64 z, {%6, %7};\nfma.rn.f32x2 w, x, y, z;\n"
      "mov.b64 {%0, %1}, w;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 x, y, w;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmul.rn.f32x2 w, x, y;\nmov.b64 {%0, %1}, w;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 x, y, w;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nadd.rn.f32x2 w, x, y;\nmov.b64 {%0, %1}, w;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// softplus(x) / ln 2 = max(y, 0) + log2(1 + 2^-|y|), y = x log2(e): the accuracy of softplus_fast; the factor ln 2 is
// part of the query's coordinates
__device__ __forceinline__ float2 softplus2_log2(float2 x) {
  const float2 y = mul2(x, make_float2(LOG2E, LOG2E));
  const float2 t = add2(make_float2(ex2_approx(-fabsf(y.x)), ex2_approx(-fabsf(y.y))), make_float2(1.f, 1.f));
  return add2(make_float2(lg2_approx(t.x), lg2_approx(t.y)), make_float2(fmaxf(y.x, 0.f), fmaxf(y.y, 0.f)));
}

template <typename T, int N2> __device__ __forceinline__ void unpack_words(const void* src, float2 (&x)[N2]) {
  uint32_t u[N2];
  if constexpr (N2 == 4) {
    const uint4 w = *reinterpret_cast<const uint4*>(src);
    u[0] = w.x, u[1] = w.y, u[2] = w.z, u[3] = w.w;
  } else {
    const uint2 w = *reinterpret_cast<const uint2*>(src);
    u[0] = w.x, u[1] = w.y;
  }
#pragma unroll
  for (int e = 0; e < N2; ++e) x[e] = unpack2<T>(u[e]);
}

constexpr int DS_FP32_KEYS = 1024;   // shorter contiguous key ranges keep fp32 phases
constexpr int DS_TILE = 64;       // keys per tile
constexpr int DS_MAX_SPLIT = 64;  // key ranges per unit

// D: head dim (64, 96, 128); G: query heads of one key head that a CTA serves (1, 2, 4) -- each key is transformed once for
// all of them; LPK: lanes per key; E: features of one piece of a key row (8 = 16-byte loads, 4 = 8-byte loads), a lane
// takes pieces t, t + LPK, ...: with half of the features rotated every lane then has as many rotated as plain ones.
// NW: worker warps (+ 1 loader warp): 8, two CTAs per SM; with four heads 16 in one CTA, whose coordinates then are read from
// shared memory (91 against 102 us for 8 warps with everything in registers at (2, 32 / 8, 32768, 128)).
// SHORT: a call of few tiles per CTA, where launches and latency are the cost: the ring brings the fp32 phases themselves and
// the lanes take their cosines and sines (no table kernel), and the splits of a unit form one cluster that merges through
// distributed shared memory (no partials in global memory, no counters).
template <typename T, int D, int G, int LPK, int E, int NW, bool SHORT>
__global__ void __launch_bounds__(32 * (NW + 1), NW == 8 ? 2 : 1) attn_decode_stream_kernel(DecodeStreamP p) {
  constexpr int TILE = DS_TILE;
  constexpr int KPW = 32 / LPK;                   // keys per warp and pass
  constexpr int WK = TILE / NW;           // keys per warp and tile
  constexpr int KPL = WK / KPW;                   // keys per lane and tile
  constexpr int NI = D / (LPK * E);               // pieces per lane
  constexpr int E2 = E / 2;
  constexpr bool QREG = G < 4;                    // the lane's slice of the queries: registers, or read from shared memory per tile
  static_assert(NI * LPK * E == D && KPL * KPW == WK, "pieces must divide over the lanes of a key");
  constexpr int PL = D == 64 ? 8 : 16;            // lanes per row of V, 8 features each
  constexpr int KV = 32 / PL;                     // rows of V per warp and pass
  constexpr int NV = G * KPL, DUP = LPK / NV;     // scores of a lane group; lanes that end up with the same one
  static_assert(NV * DUP == LPK, "the scores of a lane group must divide over its lanes");

  extern __shared__ __align__(128) uint8_t smem[];
  const int r = p.r;
  const int kbytes = TILE * D * 2, tbytes = TILE * r * 2;
  const int stage_bytes = 2 * kbytes + 2 * tbytes;
  float* qcs = reinterpret_cast<float*>(smem + (size_t)p.nstages * stage_bytes);   // [G][2][D] Qc / pass-through q, Qs
  float* red_o = qcs + G * 2 * D;                                                   // [NW][G][D]
  float* red_ml = red_o + NW * G * D;                                       // [NW][G][2]
  float* wgt = red_ml + NW * G * 2;                                         // [G][DS_MAX_SPLIT] weights of the splits
  uint64_t* full = reinterpret_cast<uint64_t*>(wgt + G * DS_MAX_SPLIT);             // [nstages] tile landed
  uint64_t* empty = full + p.nstages;                                               // [nstages] all workers done with it
  unsigned int* last_s = reinterpret_cast<unsigned int*>(empty + p.nstages);        // whether this CTA finished last of its unit
  int* pages_s = reinterpret_cast<int*>(last_s + 2);                                // [npg_smem] pages of this CTA's key range

  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int u = blockIdx.y, hb = u % p.head_blocks, bk = u / p.head_blocks, hk = bk % p.Hk, b = bk / p.Hk;
  auto head = [&](int g) { return hk + (hb * G + g) * p.Hk; };   // query head h reads key head h % Hk
  const T* kbase = (const T*)p.k + b * p.sk.b + hk * p.sk.h;
  const T* vbase = (const T*)p.v + b * p.sv.b + hk * p.sv.h;
  if (tid == 0) {
    for (int s = 0; s < p.nstages; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], NW);
    mbar_init_fence();
  }
  pdl_wait();
  // keys of this sequence (paged cache: its own length, at most the bound the split was planned for), cut evenly
  const int nk = p.seq_lens ? max(0, min(p.seq_lens[b], p.Nk)) : p.Nk;
  const int tiles_all = (nk + TILE - 1) / TILE;
  const int kb = (int)((int64_t)tiles_all * blockIdx.x / p.nsplit) * TILE;
  const int ke = min(nk, (int)((int64_t)tiles_all * (blockIdx.x + 1) / p.nsplit) * TILE);
  const int T_tiles = ke > kb ? (ke - kb + TILE - 1) / TILE : 0;

  if (p.page_table) {
    // page indices of [kb, ke); an index outside the pool is never dereferenced (clamped, status bit 1)
    for (int i = tid; i < p.npg_smem; i += blockDim.x) {
      const int lp = kb / p.page_size + i;
      int pg = 0;
      if ((int64_t)lp * p.page_size < ke) {
        pg = lp < p.max_pages ? p.page_table[(int64_t)b * p.max_pages + lp] : -1;   // a length past the table's reach
        if (pg < 0 || pg >= p.num_pages) pg = 0, atomicOr(p.status, 2u);
      }
      pages_s[i] = pg;
    }
  }
  __syncthreads();
  bool failed = false;

  if (w == NW) {
    // =============================== loader =====================================================
    auto load_kv = [&](int jt, int s) {
      const int key0 = kb + jt * TILE, n = min(TILE, ke - key0);
      uint8_t* st = smem + (size_t)s * stage_bytes;
      if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)(2 * n * D * 2 + 2 * n * r * 2));
      __syncwarp();
      const T *kt = kbase + (int64_t)key0 * p.sk.n, *vt = vbase + (int64_t)key0 * p.sv.n;
      if (p.page_table) {   // the tile lies inside one page
        const int64_t off = (int64_t)pages_s[key0 / p.page_size - kb / p.page_size] * p.page_stride + (int64_t)hk * p.sk.h +
                            (int64_t)(key0 % p.page_size) * p.sk.n;
        kt = (const T*)p.k + off, vt = (const T*)p.v + off;
      }
      if (p.k_rows_contiguous) {
        if (lane == 0) bulk_load(st, kt, n * D * 2, &full[s]);
      } else {
        for (int i = lane; i < n; i += 32) bulk_load(st + i * D * 2, kt + (int64_t)i * p.sk.n, D * 2, &full[s]);
      }
      if (p.v_rows_contiguous) {
        if (lane == 1) bulk_load(st + kbytes, vt, n * D * 2, &full[s]);
      } else {
        for (int i = lane; i < n; i += 32) bulk_load(st + kbytes + i * D * 2, vt + (int64_t)i * p.sv.n, D * 2, &full[s]);
      }
    };
    auto load_phases = [&](int jt, int s) {
      const int key0 = kb + jt * TILE, n = min(TILE, ke - key0);
      uint8_t* st = smem + (size_t)s * stage_bytes + 2 * kbytes;
      if constexpr (SHORT) {   // rows of the phase table itself: as many bytes as the two fp16 rows
        if (r > 0 && lane == 2) bulk_load(st, p.freqs + (int64_t)key0 * r, n * r * 4, &full[s]);
        return;
      }
      if (r > 0 && lane == 2) bulk_load(st, p.ch + (int64_t)key0 * r, n * r * 2, &full[s]);
      if (r > 0 && lane == 3) bulk_load(st + tbytes, p.sh + (int64_t)key0 * r, n * r * 2, &full[s]);
    };
    const int pre = min(T_tiles, p.nstages);
    for (int jt = 0; jt < pre; ++jt) load_kv(jt, jt), load_phases(jt, jt);
    int s = 0;
    uint32_t par = 0;
    for (int jt = pre; jt < T_tiles; ++jt) {
      failed = !mbar_wait(&empty[s], par, WAIT_LIMIT);
      if (failed) { drain_copies(full, p.nstages, jt - p.nstages, jt); break; }
      load_kv(jt, s), load_phases(jt, s);
      if (++s == p.nstages) s = 0, par ^= 1;
    }
    if (failed && lane == 0) atomicOr(p.status, 1u);
    if (SHORT && p.nsplit > 1) cluster_sync(), cluster_sync();
    return;   // nothing below is a block-wide barrier; the workers finish on their own
  }

  // =============================== workers ======================================================
  auto worker_sync = []() { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory"); };
  // the queries' polar coordinates with the key-side bias folded in (exact transform: one row per head and CTA)
  for (int i = tid; i < G * D; i += 32 * NW) {
    const int g = i / D, c = i - g * D;
    const T* qrow = (const T*)p.q + b * p.sq.b + head(g) * p.sq.h;
    const float x = to_f32<T>(qrow[c]);
    float qc = x, qs = 0.f;
    if (c < r) {
      // Cosine and sine of position phase minus bias, each angle by itself: rounded to fp32 the difference would be off by up to
      // 2^-15 rad at a few hundred rad, for every key alike.  (A loop, not two calls in a row: half the code to fetch.)
      const float f = p.freqs[(int64_t)(max(nk, 1) - 1) * p.sfn + c], b_ = p.bias[hk * p.bias_sh + c];
      float cs = 1.f, sn = 0.f;
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        float s1, c1;
        sincosf(i == 0 ? f : -b_, &s1, &c1);
        const float t = cs * c1 - sn * s1;
        sn = fmaf(sn, c1, cs * s1), cs = t;
      }
      const float a = softplus_f(x) * LN2;   // (the keys' magnitudes come in units of ln 2)
      qc = a * cs, qs = a * sn;
    }
    qcs[g * 2 * D + c] = qc, qcs[g * 2 * D + D + c] = qs;
  }
  worker_sync();

  const int kw = lane / LPK, t = lane % LPK;        // key of the warp's group, lane within the key
  const int krow0 = w * WK + kw;                    // first row of the tile this lane works on; the others KPW apart
  float2 qc[QREG ? G : 1][NI][E2], qs[QREG ? G : 1][NI][E2];   // this lane's slice of the queries
  if constexpr (QREG) {
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int e = 0; e < E2; ++e) {
          const int c = (t + LPK * i) * E + 2 * e;
          qc[g][i][e] = *reinterpret_cast<const float2*>(qcs + g * 2 * D + c);
          qs[g][i][e] = *reinterpret_cast<const float2*>(qcs + g * 2 * D + D + c);
        }
  }
  const uint8_t* maskb = p.mask ? p.mask + b * p.msb : nullptr;
  const int vg = lane / PL, vf = (lane % PL) * 8;   // row group and first feature of this lane in the P V step
  // After the reduction over its group a lane holds one score: head my_g, key my_kq of its group.
  const int my_g = t / DUP / KPL, my_kq = t / DUP % KPL;
  auto holder = [](int g, int kq, int kw_) { return kw_ * LPK + (g * KPL + kq) * DUP; };   // first lane with that score
  float m_run = -CUDART_INF_F, l_run = 0.f;         // of head my_g: the warp's maximum, the sum over the lane's own keys
  float2 o[G][4];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[g][e] = make_float2(0.f, 0.f);

  int s = 0;
  uint32_t par = 0;
  for (int jt = 0; jt < T_tiles; ++jt) {
    const int key0 = kb + jt * TILE;
    const uint8_t* st = smem + (size_t)s * stage_bytes;
    const int my_key = key0 + krow0 + my_kq * KPW;
    const bool valid = my_key < ke && (!maskb || maskb[(int64_t)my_key * p.msn] != 0);
    if (!failed) failed = !mbar_wait(&full[s], par, WAIT_LIMIT);
    if (failed) break;
    // (rows past the end of the range hold stale bytes: their scores are dropped by `valid`)
    float2 part[G][KPL];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int kq = 0; kq < KPL; ++kq) part[g][kq] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int c = (t + LPK * i) * E;
      const bool rot = c < r;
      // keys transformed together: one where the queries sit in registers, all where each piece of them is loaded once per tile
      constexpr int KB = QREG ? 1 : KPL;
#pragma unroll
      for (int k0 = 0; k0 < KPL; k0 += KB) {
        float2 kc[KB][E2], ks[KB][E2];   // polar coordinates of the lane's keys (in units of ln 2), or the plain features
#pragma unroll
        for (int m = 0; m < KB; ++m) {
          const int kq = k0 + m;
          const int krow = krow0 + kq * KPW;
          unpack_words<T>(st + krow * (D * 2) + c * 2, kc[m]);
          if (rot) {
            const uint8_t* crow_p = st + 2 * kbytes + krow * (r * (SHORT ? 4 : 2));
            float2 co[E2], si[E2];
            if constexpr (SHORT) {
#pragma unroll
              for (int e = 0; e < E2; ++e) {
                const float2 f = *reinterpret_cast<const float2*>(crow_p + c * 4 + e * 8);
                sincos_reduced(f.x, &si[e].x, &co[e].x), sincos_reduced(f.y, &si[e].y, &co[e].y);
              }
            } else {
              unpack_words<__half>(crow_p + c * 2, co);
              unpack_words<__half>(crow_p + tbytes + c * 2, si);
            }
#pragma unroll
            for (int e = 0; e < E2; ++e) {
              const float2 a = softplus2_log2(kc[m][e]);
              if constexpr (G == 1) {
                part[0][kq] = fma2(a, fma2(qc[0][i][e], co[e], mul2(qs[0][i][e], si[e])), part[0][kq]);
              } else {
                kc[m][e] = mul2(a, co[e]), ks[m][e] = mul2(a, si[e]);
              }
            }
          } else if constexpr (G == 1) {
#pragma unroll
            for (int e = 0; e < E2; ++e) part[0][kq] = fma2(qc[0][i][e], kc[m][e], part[0][kq]);
          }
        }
        if constexpr (G > 1) {
#pragma unroll
          for (int g = 0; g < G; ++g) {
            float2 qv[E2], qw[E2];
#pragma unroll
            for (int e = 0; e < E2; ++e) {
              if constexpr (QREG) qv[e] = qc[g][i][e], qw[e] = qs[g][i][e];
              else qv[e] = *reinterpret_cast<const float2*>(qcs + g * 2 * D + c + 2 * e);
            }
#pragma unroll
            for (int m = 0; m < KB; ++m)
#pragma unroll
              for (int e = 0; e < E2; ++e) part[g][k0 + m] = fma2(qv[e], kc[m][e], part[g][k0 + m]);
            if (rot) {
              if constexpr (!QREG) {
#pragma unroll
                for (int e = 0; e < E2; ++e) qw[e] = *reinterpret_cast<const float2*>(qcs + g * 2 * D + D + c + 2 * e);
              }
#pragma unroll
              for (int m = 0; m < KB; ++m)
#pragma unroll
                for (int e = 0; e < E2; ++e) part[g][k0 + m] = fma2(qw[e], ks[m][e], part[g][k0 + m]);
            }
          }
        }
      }
    }
    // Sum over the lanes of a key, halving the values a lane still carries with every step: NV - 1 + log2(DUP) shuffles for
    // NV scores, and everything that follows is done once per score instead of once per lane.
    float v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = part[i / KPL][i % KPL].x + part[i / KPL][i % KPL].y;
#pragma unroll
    for (int n = NV / 2; n >= 1; n /= 2) {
      const int off = n * DUP;
      const bool hi = (t & off) != 0;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float give = hi ? v[i] : v[i + n], keep = hi ? v[i + n] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
      }
    }
#pragma unroll
    for (int off = DUP / 2; off >= 1; off /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    const float sc = valid ? v[0] * p.scale_log2 : -CUDART_INF_F;     // log2 units
    // the maximum may lag by 2^8: most tiles then need neither a warp reduction nor a rescale
    if (__any_sync(0xffffffffu, sc > m_run + 8.f)) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float old = __shfl_sync(0xffffffffu, m_run, holder(g, 0, 0));
        const float mx = warp_max(my_g == g ? fmaxf(m_run, sc) : -CUDART_INF_F);
        const float alpha = mx == -CUDART_INF_F ? 1.f : ex2_approx(old - mx);    // exp2(-inf) = 0 on the first visible tile
        if (my_g == g) m_run = mx, l_run *= alpha;
#pragma unroll
        for (int e = 0; e < 4; ++e) o[g][e] = mul2(o[g][e], make_float2(alpha, alpha));
      }
    }
    const float pj = ex2_approx(sc - (m_run == -CUDART_INF_F ? 0.f : m_run));   // 0 for masked keys
    l_run += pj;
    const uint8_t* vt = st + kbytes + (w * WK + vg) * (D * 2) + vf * 2;
    const bool clean = !maskb && key0 + TILE <= ke;   // every row of the tile is a key
#pragma unroll
    for (int vk = 0; vk < WK / KV; ++vk) {
      // row vk * KV + vg of the warp = key (row % KPW) of the lane groups, row / KPW of a lane's keys
      float pk[G];
#pragma unroll
      for (int g = 0; g < G; ++g) pk[g] = __shfl_sync(0xffffffffu, pj, holder(g, vk * KV / KPW, vk * KV % KPW + vg));
      bool any = clean;
      if (!clean) {
#pragma unroll
        for (int g = 0; g < G; ++g) any |= pk[g] != 0.f;
      }
      if (any && (D % 64 == 0 || vf < D)) {   // masked / out-of-range rows may hold stale bytes: never touch them
        float2 vv[4];
        unpack_words<T>(vt + vk * KV * (D * 2), vv);
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[g][e] = fma2(make_float2(pk[g], pk[g]), vv[e], o[g][e]);
      }
    }
    fence_async_smem();   // the tile has been read: the loader's next copy may write over it
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (++s == p.nstages) s = 0, par ^= 1;
  }
  if (failed && lane == 0) atomicOr(p.status, 1u);

  // merge the lanes of the warp, then the warps of the CTA
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int off = PL; off < 32; off <<= 1) {
        o[g][e].x += __shfl_xor_sync(0xffffffffu, o[g][e].x, off);
        o[g][e].y += __shfl_xor_sync(0xffffffffu, o[g][e].y, off);
      }
    const float mg = __shfl_sync(0xffffffffu, m_run, holder(g, 0, 0));
    const float lg = warp_sum(my_g == g && t % DUP == 0 ? l_run : 0.f);
    if (lane < PL && vf < D) {
#pragma unroll
      for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(red_o + (w * G + g) * D + vf + 2 * e) = o[g][e];
    }
    if (lane == 0) red_ml[(w * G + g) * 2] = mg, red_ml[(w * G + g) * 2 + 1] = lg;
  }
  worker_sync();
  float* fin = reinterpret_cast<float*>(smem);
  const int64_t slot = ((int64_t)u * p.nsplit + blockIdx.x) * G;
  auto cta_max = [&](int g) {
    float M = -CUDART_INF_F;
#pragma unroll
    for (int ww = 0; ww < NW; ++ww) M = fmaxf(M, red_ml[(ww * G + g) * 2]);
    return M;
  };
  auto cta_sum = [&](int g, float M) {
    float L = 0.f;
#pragma unroll
    for (int ww = 0; ww < NW; ++ww)
      L += red_ml[(ww * G + g) * 2] == -CUDART_INF_F ? 0.f : red_ml[(ww * G + g) * 2 + 1] * ex2_approx(red_ml[(ww * G + g) * 2] - M);
    return L;
  };
  auto write_out = [&](int g, int c, float acc, float L) {
    T* orow = (T*)p.out + b * p.so.b + head(g) * p.so.h;
    orow[c] = from_f32<T>(L > 0.f ? acc / L : 0.f);
  };
  auto write_lse = [&](int g, float M, float L) {
    p.lse[(int64_t)b * p.H + head(g)] = L > 0.f ? M * LN2 + logf(L) : -CUDART_INF_F;
  };
  for (int i = tid; i < G * D; i += 32 * NW) {
    const int g = i / D, c = i - g * D;
    const float M = cta_max(g);
    float acc = 0.f;
#pragma unroll
    for (int ww = 0; ww < NW; ++ww)
      acc += red_ml[(ww * G + g) * 2] == -CUDART_INF_F ? 0.f : red_o[(ww * G + g) * D + c] * ex2_approx(red_ml[(ww * G + g) * 2] - M);
    if (p.nsplit == 1) {
      const float L = cta_sum(g, M);
      write_out(g, c, acc, L);
      if (c == 0) write_lse(g, M, L);
    } else if (SHORT) {   // (every ring stage has been read: the first one takes the CTA's result)
      fin[i] = acc;
      if (c == 0) fin[G * D + 2 * g] = M, fin[G * D + 2 * g + 1] = cta_sum(g, M);
    } else {
      p.part_o[slot * D + i] = acc;
      if (c == 0) p.part_ml[(slot + g) * 2] = M, p.part_ml[(slot + g) * 2 + 1] = cta_sum(g, M);
    }
  }
  if (p.nsplit == 1) return;
  if constexpr (SHORT) {
    // CTA i of the cluster merges every nsplit-th element from the shared memory of all of them
    __syncwarp();
    cluster_sync();
    for (int i = tid * p.nsplit + (int)blockIdx.x; i < G * D; i += 32 * NW * p.nsplit) {
      const int g = i / D, c = i - g * D;
      float m2[8], l2[8], a2[8], M = -CUDART_INF_F, L = 0.f, acc = 0.f;
#pragma unroll
      for (int sp = 0; sp < 8; ++sp) {
        m2[sp] = -CUDART_INF_F, l2[sp] = a2[sp] = 0.f;
        if (sp < p.nsplit) {
          a2[sp] = dsmem_ld(fin + i, sp), m2[sp] = dsmem_ld(fin + G * D + 2 * g, sp), l2[sp] = dsmem_ld(fin + G * D + 2 * g + 1, sp);
        }
        M = fmaxf(M, m2[sp]);
      }
#pragma unroll
      for (int sp = 0; sp < 8; ++sp) {
        const float wt = m2[sp] == -CUDART_INF_F ? 0.f : ex2_approx(m2[sp] - M);
        L = fmaf(wt, l2[sp], L), acc = fmaf(wt, a2[sp], acc);
      }
      write_out(g, c, acc, L);
      if (c == 0) write_lse(g, M, L);
    }
    __syncwarp();
    cluster_sync();   // nobody leaves while its shared memory is read
    return;
  }
  // The CTA that finishes last merges the splits of its unit (one launch less than a kernel of its own, and no wait for the
  // slowest unit of the grid).
  __threadfence();
  worker_sync();
  if (tid == 0) *last_s = atomicAdd(p.done + u, 1u) == (unsigned)p.nsplit - 1u;
  worker_sync();
  if (!*last_s) return;
  __threadfence();
  const int64_t slot0 = (int64_t)u * p.nsplit * G;
  if (w < G) {   // warp g: the weights of head g's splits, relative to their sum
    float m2[DS_MAX_SPLIT / 32], l2[DS_MAX_SPLIT / 32], M = -CUDART_INF_F, L = 0.f;
#pragma unroll
    for (int i = 0; i < DS_MAX_SPLIT / 32; ++i) {
      const int sp = lane + 32 * i;
      const float2 ml = sp < p.nsplit ? __ldcg(reinterpret_cast<const float2*>(p.part_ml + (slot0 + (int64_t)sp * G + w) * 2))
                                      : make_float2(-CUDART_INF_F, 0.f);
      m2[i] = ml.x, l2[i] = ml.y, M = fmaxf(M, ml.x);
    }
    M = warp_max(M);
#pragma unroll
    for (int i = 0; i < DS_MAX_SPLIT / 32; ++i) {
      m2[i] = m2[i] == -CUDART_INF_F ? 0.f : ex2_approx(m2[i] - M);
      L += m2[i] * l2[i];
    }
    L = warp_sum(L);
#pragma unroll
    for (int i = 0; i < DS_MAX_SPLIT / 32; ++i) wgt[w * DS_MAX_SPLIT + lane + 32 * i] = m2[i];
    if (lane == 0) red_ml[w] = L, write_lse(w, M, L);
  }
  worker_sync();
  for (int i = tid; i < G * D; i += 32 * NW) {
    const int g = i / D, c = i - g * D;
    float acc = 0.f;
#pragma unroll 8
    for (int sp = 0; sp < p.nsplit; ++sp) acc = fmaf(wgt[g * DS_MAX_SPLIT + sp], __ldcg(p.part_o + (slot0 + (int64_t)sp * G) * D + i), acc);
    write_out(g, c, acc, red_ml[g]);
  }
}

// ---- host side -----------------------------------------------------------------------------------
// Query heads per CTA: as many of the heads that share a key head as the registers hold (their coordinates live there), so
// that K and V are read and transformed once for all of them.
static int decode_heads(const PopeShape& s) {
  const int groups = s.H / s.Hk;
  return groups % 4 == 0 && s.d != 96 ? 4 : groups % 2 == 0 ? 2 : 1;
}

// Shared memory of a CTA: a ring stage, and everything beside the ring (but the paged cache's page indices)
static size_t decode_stage_bytes(const PopeShape& s) { return (size_t)DS_TILE * (2 * s.d * 2 + 2 * s.r * 2); }
static size_t decode_fixed_bytes(const PopeShape& s, int g, int nw) {
  return ((2 + nw) * g * s.d + nw * g * 2 + g * DS_MAX_SPLIT) * sizeof(float) + 2 * 3 * 8 + 64;
}
constexpr size_t DS_HALF_SM = 112 * 1024;   // what a CTA may take where two share an SM

// CTAs resident at a time: two per SM with 8 worker warps, one with 16 (four heads per CTA), and one where two stages of wide
// rotations do not fit half of the shared memory (counted as two, (1, 8, 30000, 128), r = 128 took 76 us instead of 69,
// (2, 16, 700, 128) 18.5 instead of 12.4)
static int64_t decode_slots(const PopeShape& s) {
  const bool two = decode_heads(s) < 4 && 2 * decode_stage_bytes(s) + decode_fixed_bytes(s, decode_heads(s), 8) <= DS_HALF_SM;
  return (two ? 2 : 1) * 148;
}

// Key ranges per unit.  The time of a grid in units of one 64-key tile: whole waves of resident CTAs times the tiles of a CTA
// plus what a CTA costs beside its tiles (start, ring fill, merge: about four tiles' time); the smallest wins.  SHORT: at
// most a cluster of eight.
static int decode_stream_split(const PopeShape& s, bool shrt) {
  const int tiles = (s.Nk + DS_TILE - 1) / DS_TILE, g = decode_heads(s);
  const int64_t units = (int64_t)s.B * s.H / g, slots = decode_slots(s);
  const int most = std::min(tiles, shrt ? 8 : DS_MAX_SPLIT);
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int n = 1; n <= most; ++n) {
    const int64_t cost = (units * n + slots - 1) / slots * ((tiles + n - 1) / n + 4);
    if (cost < best_cost) best = n, best_cost = cost;
  }
  return best;
}

// The SHORT flavour saves a launch and the trip of the partials through L2, about 2 us, and pays for its own cosines and sines
// with every tile of a CTA, the less the more heads share them: (2, 16, 4000, 128) with 8 tiles per CTA takes 21.6 us
// against 18.9, (4, 32 / 8, 2000, 128) with 8 tiles of four heads 19.9 against 20.7, (2, 16 / 4, 777, 128) 10.0 against 11.8.
// It copies rows of the phase table, which therefore has to be contiguous.  Below DS_FP32_KEYS keys every call takes it, with
// fp32 phases but approximate functions (ex2, lg2, sine and cosine of the special-function unit, 2^-21 absolute and better); a
// call without a usable table goes to the exact family, which took them all before.  Against 64 bits both are off by the rounding
// of the output, 2.066e-4 in fp16 at (2, 16 / 4, 777, 128); the nearest fp16 value is missed in 0.05 % of the outputs here and
// in 1.1 % there.  (Accurate softplus, sine and cosine of the keys changed neither figure and took 11.5 instead of 10.3 us.)
static bool decode_short_possible(const PopeShape& s, const PopeEmbed& e) {
  return s.r == 0 || (e.sf.n == s.r && (reinterpret_cast<uintptr_t>(e.freqs) & 15) == 0);
}
static bool decode_short(const PopeShape& s, const PopeEmbed& e) {
  if (!decode_short_possible(s, e)) return false;
  if (s.Nk < DS_FP32_KEYS) return true;
  const int tiles = (s.Nk + DS_TILE - 1) / DS_TILE, n = decode_stream_split(s, true), g = decode_heads(s);
  const int64_t ctas = (int64_t)s.B * s.H / g * n, slots = decode_slots(s);
  return (ctas + slots - 1) / slots * ((tiles + n - 1) / n) <= 4 + g;
}

bool decode_stream_supported(const PopeAttnArgs& a) {
  const PopeShape& s = a.shape;
  if (s.Nq != 1 || a.causal) return false;
  if (s.Nk < DS_FP32_KEYS && !decode_short_possible(s, a.embed)) return false;
  if (s.dtype != POPE_BF16 && s.dtype != POPE_F16) return false;
  if (s.d != 64 && s.d != 96 && s.d != 128) return false;
  if (s.r % 8 != 0) return false;
  if (s.r > 0 && (a.embed.sf.b != 0 || a.embed.sf.h != 0)) return false;
  auto ok = [&](const void* ptr, const PopeStride3& st) {
    return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && st.b % 8 == 0 && st.h % 8 == 0 && st.n % 8 == 0;
  };
  if (!ok(a.k, a.sk) || !ok(a.v, a.sv)) return false;
  if ((s.Nk > 1 && (a.sk.n < s.d || a.sv.n < s.d))) return false;
  return true;
}

// workspace: [counters][partial outputs][partial max, sum][fp16 cos / sin tables]
struct DecodeWs {
  size_t done, part_o, part_ml, table, total;
};
static DecodeWs decode_ws(const PopeShape& s) {
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t slots = (size_t)s.B * s.H * decode_stream_split(s, false);   // (unit, split, head of the unit)
  DecodeWs w;
  w.done = 0;
  w.part_o = up((size_t)s.B * s.H * sizeof(unsigned int));
  w.part_ml = w.part_o + up(slots * s.d * sizeof(float));
  w.table = w.part_ml + up(slots * 2 * sizeof(float));
  w.total = w.table + up((size_t)s.Nk * s.r * 4);
  return w;
}

size_t decode_stream_workspace(const PopeAttnArgs& a) { return decode_short(a.shape, a.embed) ? 0 : decode_ws(a.shape).total; }

template <typename T, int D, int G, int LPK, int E, int NW, bool SHORT>
static cudaError_t launch_decode_stream(const PopeAttnArgs& a, cudaStream_t st, const PopePagedKV* kv) {
  const PopeShape& s = a.shape;
  DecodeStreamP p = {};
  p.H = s.H, p.Hk = s.Hk, p.Nk = s.Nk, p.r = s.r;
  p.nsplit = decode_stream_split(s, SHORT), p.head_blocks = s.H / s.Hk / G;
  p.scale_log2 = a.softmax_scale * LOG2E;
  p.q = a.q, p.k = a.k, p.v = a.v, p.sq = a.sq, p.sk = a.sk, p.sv = a.sv;
  p.out = a.out, p.so = a.so, p.lse = a.lse;
  p.k_rows_contiguous = a.sk.n == s.d, p.v_rows_contiguous = a.sv.n == s.d;
  p.freqs = a.embed.freqs, p.bias = a.embed.bias, p.sfn = a.embed.sf.n, p.bias_sh = a.embed.bias_stride_h;
  p.mask = a.mask, p.msb = a.mask_stride_b, p.msn = a.mask_stride_n;
  const int tiles = (s.Nk + DS_TILE - 1) / DS_TILE;
  if (kv) {
    p.page_table = kv->page_table, p.seq_lens = kv->seq_lens;
    p.page_size = kv->page_size, p.max_pages = kv->max_pages_per_seq, p.num_pages = kv->num_pages;
    p.page_stride = (int64_t)s.Hk * kv->page_size * s.d;
    p.npg_smem = (tiles + p.nsplit - 1) / p.nsplit * DS_TILE / kv->page_size + 2;
  }
  const DecodeWs ws = decode_ws(s);
  uint8_t* base = static_cast<uint8_t*>(a.workspace);
  p.done = reinterpret_cast<unsigned int*>(base + ws.done);
  p.part_o = reinterpret_cast<float*>(base + ws.part_o), p.part_ml = reinterpret_cast<float*>(base + ws.part_ml);
  __half* ch = reinterpret_cast<__half*>(base + ws.table);
  __half* sh = ch + (size_t)s.Nk * s.r;
  p.ch = ch, p.sh = sh;
  p.status = tc_status_ptr();
  if (!p.status) return cudaErrorInvalidSymbol;
  const size_t stage = decode_stage_bytes(s), fixed = decode_fixed_bytes(s, G, NW) + (size_t)p.npg_smem * sizeof(int);
  // two CTAs per SM: the ring of each takes what half of the shared memory leaves, at most 3 stages
  int nst = (int)(((NW == 8 ? 1 : 2) * (int64_t)DS_HALF_SM - (int64_t)fixed) / (int64_t)stage);
  if (nst < 2) nst = (int)((kMaxDynamicSmem - 1024 - (int64_t)fixed) / (int64_t)stage);   // wide rotations (r = d = 128): one CTA per SM
  nst = nst > 3 ? 3 : nst;
  if (nst < 2) return cudaErrorInvalidValue;
  p.nstages = nst;
  const size_t smem = nst * stage + fixed;
  const auto kernel = attn_decode_stream_kernel<T, D, G, LPK, E, NW, SHORT>;
  cudaError_t e;
  if ((e = ensure_max_smem<attn_decode_stream_kernel<T, D, G, LPK, E, NW, SHORT>>()) != cudaSuccess) return e;
  const unsigned units = (unsigned)(s.B * s.H / G);
  const dim3 grid((unsigned)p.nsplit, units), block(32 * (NW + 1));
  if constexpr (SHORT) {
    return launch_clusters(kernel, p.nsplit, grid, block, smem, st, true, p);
  }
  // behind the table kernel, which also zeroes the counters, the decode kernel starts as its programmatic dependent;
  // without rotated features it is the first launch of the call and an ordinary one
  if (s.r > 0) {
    if ((e = launch_trig_tables(a.embed, s.Nk, s.r, nullptr, nullptr, ch, sh, st, 1, 1, p.done, (int)units)) != cudaSuccess) return e;
    return launch_dependent(kernel, grid, block, smem, st, p);
  }
  if (p.nsplit > 1 && (e = cudaMemsetAsync(p.done, 0, units * sizeof(unsigned int), st)) != cudaSuccess) return e;
  kernel<<<grid, block, smem, st>>>(p);
  return cudaGetLastError();
}

// LPK and E: 8-byte pieces (E = 4) leave a lane few coordinates of many heads, 16-byte ones (E = 8) fewer loads for one head
template <typename T, bool SHORT>
static cudaError_t decode_stream_g(const PopeAttnArgs& a, cudaStream_t st, const PopePagedKV* kv) {
  const int g = decode_heads(a.shape);
  switch (a.shape.d) {
    case 64:
      return g == 4   ? launch_decode_stream<T, 64, 4, 8, 4, 16, SHORT>(a, st, kv)
             : g == 2 ? launch_decode_stream<T, 64, 2, 8, 4, 8, SHORT>(a, st, kv)
                      : launch_decode_stream<T, 64, 1, 8, 4, 8, SHORT>(a, st, kv);
    case 96:
      return g == 2 ? launch_decode_stream<T, 96, 2, 8, 4, 8, SHORT>(a, st, kv) : launch_decode_stream<T, 96, 1, 8, 4, 8, SHORT>(a, st, kv);
    default:
      return g == 4   ? launch_decode_stream<T, 128, 4, 16, 4, 16, SHORT>(a, st, kv)
             : g == 2 ? launch_decode_stream<T, 128, 2, 16, 4, 8, SHORT>(a, st, kv)
                      : launch_decode_stream<T, 128, 1, 8, 8, 8, SHORT>(a, st, kv);
  }
}

template <typename T>
static cudaError_t decode_stream_d(const PopeAttnArgs& a, cudaStream_t st, const PopePagedKV* kv) {
  return decode_short(a.shape, a.embed) ? decode_stream_g<T, true>(a, st, kv) : decode_stream_g<T, false>(a, st, kv);
}

cudaError_t decode_stream(const PopeAttnArgs& a, cudaStream_t st) {
  return a.shape.dtype == POPE_BF16 ? decode_stream_d<__nv_bfloat16>(a, st, nullptr) : decode_stream_d<__half>(a, st, nullptr);
}

// ---- paged cache ---------------------------------------------------------------------------------
// The paged call as the contiguous call sees it: K / V = the page pools, head stride inside a page, rows contiguous.
static PopeAttnArgs paged_as_attn(const PopePagedDecodeArgs& g, float* lse) {
  PopeAttnArgs a = {};
  a.struct_bytes = sizeof(PopeAttnArgs);
  a.causal = 0, a.softmax_scale = g.softmax_scale;
  a.shape = g.shape, a.embed = g.embed;
  a.q = g.q, a.sq = g.sq, a.out = g.out, a.so = g.so, a.lse = lse;
  a.k = g.kv.k_pages, a.v = g.kv.v_pages;
  a.sk.b = 0, a.sk.h = (int64_t)g.kv.page_size * g.shape.d, a.sk.n = g.shape.d;
  a.sv = a.sk;
  a.workspace = g.workspace, a.workspace_bytes = g.workspace_bytes;
  return a;
}

static size_t paged_lse_bytes(const PopeShape& s) { return ((size_t)s.B * s.H * sizeof(float) + 255) & ~(size_t)255; }

bool decode_paged_supported(const PopePagedDecodeArgs& g) {
  const PopeShape& s = g.shape;
  if (s.Nq != 1 || (s.dtype != POPE_BF16 && s.dtype != POPE_F16)) return false;
  if (s.d != 64 && s.d != 96 && s.d != 128) return false;
  if (s.r % 8 != 0) return false;
  if (s.r > 0 && (g.embed.sf.b != 0 || g.embed.sf.h != 0)) return false;
  if (g.kv.page_size < 64 || g.kv.page_size % 64 != 0) return false;
  return true;
}

size_t decode_paged_workspace(const PopePagedDecodeArgs& g) {
  return decode_stream_workspace(paged_as_attn(g, nullptr)) + paged_lse_bytes(g.shape);
}

cudaError_t decode_paged(const PopePagedDecodeArgs& g, cudaStream_t st) {
  // the row statistics go to the caller's lse or, without one, to the end of the workspace
  float* lse = g.lse;
  if (!lse) lse = reinterpret_cast<float*>(static_cast<uint8_t*>(g.workspace) + decode_stream_workspace(paged_as_attn(g, nullptr)));
  const PopeAttnArgs a = paged_as_attn(g, lse);
  return g.shape.dtype == POPE_BF16 ? decode_stream_d<__nv_bfloat16>(a, st, &g.kv) : decode_stream_d<__half>(a, st, &g.kv);
}

struct KvAppendP {
  int Hk, d, n_new, page_size, max_pages, num_pages;
  int64_t page_stride;
  const void *k, *v;
  Strides sk, sv;
  void *k_pages, *v_pages;
  const int32_t* page_table;
  int32_t* seq_lens;
  unsigned int* status;
};

// One thread per 16 bytes of a new row of k and of v.  A position past the table or a page index outside the pool is
// skipped and reported through status bit 1.
template <typename T>
__device__ __forceinline__ void append_group(const KvAppendP& p, int b, int hk, int i, int c, int len) {
  const int pos = len + i, lp = pos / p.page_size;
  if (pos < 0 || lp >= p.max_pages) { atomicOr(p.status, 2u); return; }
  const int pg = p.page_table[(int64_t)b * p.max_pages + lp];
  if (pg < 0 || pg >= p.num_pages) { atomicOr(p.status, 2u); return; }
  const int64_t dst = (int64_t)pg * p.page_stride + ((int64_t)hk * p.page_size + pos % p.page_size) * p.d + c * 8;
  const T* krow = static_cast<const T*>(p.k) + b * p.sk.b + hk * p.sk.h + (int64_t)i * p.sk.n + c * 8;
  const T* vrow = static_cast<const T*>(p.v) + b * p.sv.b + hk * p.sv.h + (int64_t)i * p.sv.n + c * 8;
  *reinterpret_cast<uint4*>(static_cast<T*>(p.k_pages) + dst) = *reinterpret_cast<const uint4*>(krow);
  *reinterpret_cast<uint4*>(static_cast<T*>(p.v_pages) + dst) = *reinterpret_cast<const uint4*>(vrow);
}

template <typename T>
__global__ void __launch_bounds__(256) kv_append_kernel(KvAppendP p) {
  const int cpr = p.d >> 3;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= p.n_new * cpr) return;
  append_group<T>(p, blockIdx.z, blockIdx.y, idx / cpr, idx % cpr, p.seq_lens[blockIdx.z]);
}

// The rows of a few tokens (a decode step): one CTA per sequence, which therefore may advance the length itself when all
// of its threads have read it -- a decode step is bound by its launches.
constexpr int KV_STEP_GROUPS = 4096;   // 16-byte groups of k per sequence that one CTA still copies in a few microseconds
template <typename T>
__global__ void __launch_bounds__(256) kv_append_step_kernel(KvAppendP p, int advance) {
  pdl_wait();
  const int cpr = p.d >> 3, b = blockIdx.x, len = p.seq_lens[b];
  for (int idx = threadIdx.x; idx < p.Hk * p.n_new * cpr; idx += 256) {
    const int row = idx / cpr;
    append_group<T>(p, b, row / p.n_new, row % p.n_new, idx % cpr, len);
  }
  __syncthreads();
  if (advance && threadIdx.x == 0) p.seq_lens[b] = len + p.n_new;
}

__global__ void kv_advance_kernel(int32_t* seq_lens, int B, int n_new) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < B) seq_lens[b] += n_new;
}

cudaError_t kv_append(const PopeKvAppendArgs& g, cudaStream_t st) {
  KvAppendP p = {};
  p.Hk = g.Hk, p.d = g.d, p.n_new = g.n_new;
  p.page_size = g.kv.page_size, p.max_pages = g.kv.max_pages_per_seq, p.num_pages = g.kv.num_pages;
  p.page_stride = (int64_t)g.Hk * g.kv.page_size * g.d;
  p.k = g.k, p.v = g.v, p.sk = Strides(g.sk), p.sv = Strides(g.sv);
  p.k_pages = g.kv.k_pages, p.v_pages = g.kv.v_pages, p.page_table = g.kv.page_table, p.seq_lens = g.kv.seq_lens;
  p.status = tc_status_ptr();
  if (!p.status) return cudaErrorInvalidSymbol;
  // (both 16-bit types move as raw 16-byte groups)
  if ((int64_t)g.Hk * g.n_new * (g.d / 8) <= KV_STEP_GROUPS) {
    return launch_dependent(kv_append_step_kernel<__nv_bfloat16>, dim3(g.B), dim3(256), 0, st, p, (int)g.advance);
  }
  const dim3 grid((unsigned)((g.n_new * (g.d / 8) + 255) / 256), (unsigned)g.Hk, (unsigned)g.B);
  kv_append_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (g.advance) {
    kv_advance_kernel<<<(g.B + 255) / 256, 256, 0, st>>>(g.kv.seq_lens, g.B, g.n_new);
    e = cudaGetLastError();
  }
  return e;
}

constexpr int KV_MAP_BATCH = 128;
struct KvMapBatch {
  int32_t n, index[KV_MAP_BATCH], value[KV_MAP_BATCH];
};
__global__ void kv_map_kernel(const __grid_constant__ KvMapBatch m, int32_t* page_table, int32_t* seq_lens) {
  const int i = threadIdx.x;
  pdl_wait();
  if (i >= m.n) return;
  if (m.index[i] >= 0) page_table[m.index[i]] = m.value[i];
  else seq_lens[-1 - m.index[i]] = m.value[i];
}

cudaError_t kv_map(const PopeKvMapArgs& a, cudaStream_t st) {
  for (int first = 0; first < a.n; first += KV_MAP_BATCH) {
    KvMapBatch m;
    m.n = std::min(a.n - first, KV_MAP_BATCH);
    std::copy_n(a.index + first, m.n, m.index), std::copy_n(a.value + first, m.n, m.value);
    const cudaError_t e = launch_dependent(kv_map_kernel, dim3(1), dim3(KV_MAP_BATCH), 0, st, m, a.page_table, a.seq_lens);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace pope
