// Fused LM-head -> log-softmax -> selected-token log-prob -> GRPO clipped-ratio loss.
//
// Forward never materialises the [tokens, vocab] logits: the tcgen05 pipeline computes
// 128 x 256 logit tiles in TMEM and the epilogue folds each tile into per-row online
// softmax statistics (running max, running sum of exp, the logit of the target token).
// The vocabulary is split across CTAs; a token kernel merges the per-split partials,
// forms logprob = z_target - logsumexp, and evaluates
//     ratio = exp(new - old),  L = -min(ratio*A, clip(ratio, 1-eps, 1+eps_hi)*A)  (+ beta * k3 KL)
// with the per-token weight already folded with mask / normaliser, accumulating the
// loss terms and emitting dLoss/dlogprob for the backward pass.
//
// The gradient is
//     dlogit[t, v] = coef[t] * (onehot(target_t)[v] - exp(logit[t, v] - lse[t]))
// as bf16; a plain TN GEMM against the resident transposed LM head then gives dH.  A training step lets the forward
// write its logits in fp32 for a bounded number of rows and turns them into dlogits in place (dlogits_inplace_kernel);
// a caller that kept no logits recomputes the tiles with the same pipeline (EpiDLogits: the separate forward and backward of
// ops/logprob_loss.py; no training step takes them).
// In a vocab-parallel (TP) layout each rank runs this over its vocabulary shard and
// the 3-float partials are what ranks exchange.
//
// Semantics restated from the reference trainer: chunked matmul + gather + logsumexp at
// src/art/local/train.py:245-281 and the loss arithmetic at src/art/local/train.py:112-151.
#include <math.h>

#include <type_traits>

#include "gemm_pipeline_2cta.cuh"
#include "host_utils.h"
#include "sampling.cuh"

namespace artb {

constexpr int LP_BN = 256;
constexpr int LP_STAGES = 4;

// Work item = (m_blk, vocab split); a CTA walks the n-tiles of its split in order so the
// running statistics stay in registers.  Items with the same split are adjacent so that
// concurrently running CTAs stream the same LM-head tiles through L2.
struct SchedVocabSplit {
  int m_tiles, n_tiles, splits, tiles_per_split;
  __device__ int items_for_cta(int cta, int ncta) const {
    const int total = m_tiles * splits;
    return cta < total ? (total - cta + ncta - 1) / ncta : 0;
  }
  __device__ int tiles_for_cta(int cta, int ncta) const { return items_for_cta(cta, ncta) * tiles_per_split; }
  __device__ TileInfo get(int cta, int ncta, int i) const {
    const int item = cta + (i / tiles_per_split) * ncta;
    const int j = i % tiles_per_split;
    TileInfo ti = make_tile(item % m_tiles, 0);
    ti.group = item / m_tiles;  // split
    ti.n_blk = ti.group * tiles_per_split + j;
    ti.first = (j == 0);
    ti.last = (j == tiles_per_split - 1);
    return ti;
  }
};

// Schedule of the decode-time sampler: one item (128 rows, a span of n-tiles) per CTA, the spans as equal as whole tiles
// allow.  With a fixed number of tiles per split and two items per CTA the longest CTA of a 152 064-token head had 6 tiles
// of 256 where the mean is 4.0.
struct SchedVocabSpan {
  int m_tiles, n_tiles, splits;
  int early = 0;
  __device__ int lo(int s) const { return static_cast<int>(static_cast<long>(s) * n_tiles / splits); }
  __device__ int tiles_for_cta(int cta, int) const {
    const int s = cta / m_tiles;
    return s < splits ? lo(s + 1) - lo(s) : 0;
  }
  __device__ TileInfo get(int cta, int, int i) const {
    const int s = cta / m_tiles, first = lo(s), end = lo(s + 1);
    TileInfo ti = make_tile(cta % m_tiles, first + i);
    ti.group = s;
    ti.first = i == 0;
    ti.last = first + i == end - 1;
    return ti;
  }
};

struct EpiStats {
  static constexpr int COL_SPLIT = 2;   // two warps per lane quarter, each with a partial of its own for its half of the columns
  const int* target;   // [M] target vocabulary id per row (global id, minus vocab_offset locally)
  float* partials;     // [2 splits, M, 4]  (max, sumexp, z_target, unused)
  float* logits;       // [M, ldl] fp32, or null: not kept
  int M, V, ldl, vocab_offset;
  float run_max, run_sum, z;
  int tgt;

  __device__ void tile_begin(const TileInfo& ti, int row) {
    if (ti.first) {
      run_max = -INFINITY;
      run_sum = 0.f;
      z = -INFINITY;
      const int gr = ti.m_blk * GEMM_BM + row;
      tgt = (gr < M) ? target[gr] - vocab_offset : -1;
    }
  }
  __device__ void chunk(const TileInfo& ti, int row, int c, uint32_t (&acc)[32]) {
    const int gc = ti.n_blk * LP_BN + c;
    if (gc >= V) return;
    if (logits) store_logits(ti, row, gc, acc);
    float cmax = -INFINITY;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float v = __uint_as_float(acc[j]);
      if (gc + j >= V) v = -INFINITY;
      acc[j] = __float_as_uint(v);
      cmax = fmaxf(cmax, v);
    }
    const float nmax = fmaxf(run_max, cmax);
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) s += __expf(__uint_as_float(acc[j]) - nmax);
    run_sum = run_sum * __expf(run_max - nmax) + s;
    run_max = nmax;
    const int d = tgt - gc;
    if (d >= 0 && d < 32) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j == d) z = __uint_as_float(acc[j]);
    }
  }
  // 32 rows x 128 bytes of a warp, turned in shared memory so that a store covers whole lines of 4 rows: with a row per lane
  // every store touched 32 lines, and on a K of 896 the tile's main loop is shorter than that (692 us for 1734 rows of the
  // 151 936-token head, against 396 without stores).  Piece p of row r sits at r * 8 + (p ^ (r & 7)): no bank conflicts.
  __device__ __forceinline__ void store_logits(const TileInfo& ti, int row, int gc, const uint32_t (&acc)[32]) {
    __shared__ uint4 s_slab[8][32 * 8];
    const int lane = row & 31, sw = lane & 7;
    uint4* sb = s_slab[epi_warp_slot()];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j) sb[lane * 8 + (j ^ sw)] = make_uint4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
    __syncwarp();
    const int row0 = ti.m_blk * GEMM_BM + (row & ~31), col = gc + 4 * sw;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3);
      if (row0 + r < M && col < ldl)
        *reinterpret_cast<uint4*>(logits + static_cast<size_t>(row0 + r) * ldl + col) = sb[r * 8 + (sw ^ (r & 7))];
    }
  }
  __device__ void tile_end(const TileInfo& ti, int row) {
    if (!ti.last) return;
    const int gr = ti.m_blk * GEMM_BM + row;
    if (gr >= M) return;
    float4 o = make_float4(run_max, run_sum, z, 0.f);
    *reinterpret_cast<float4*>(partials + (static_cast<size_t>(ti.group * 2 + (epi_warp_slot() >> 2)) * M + gr) * 4) = o;
  }
};

struct EpiDLogits {
  const int* target;
  const float* lse;    // [M]
  const float* coef;   // [M] dLoss/dlogprob
  __nv_bfloat16* out;  // [M, ldo]
  int M, V, ldo, vocab_offset;
  float my_lse, my_coef;
  int tgt;

  __device__ void tile_begin(const TileInfo& ti, int row) {
    const int gr = ti.m_blk * GEMM_BM + row;
    if (gr < M) {
      my_lse = lse[gr];
      my_coef = coef[gr];
      tgt = target[gr] - vocab_offset;
    } else {
      my_lse = 0.f;
      my_coef = 0.f;
      tgt = -1;
    }
  }
  __device__ void chunk(const TileInfo& ti, int row, int c, uint32_t (&acc)[32]) {
    const int gr = ti.m_blk * GEMM_BM + row;
    const int gc = ti.n_blk * LP_BN + c;
    if (gr >= M || gc >= ldo) return;
    __nv_bfloat16* o = out + static_cast<size_t>(gr) * ldo + gc;
    uint32_t packed[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      float p0 = __expf(__uint_as_float(acc[j]) - my_lse);
      float p1 = __expf(__uint_as_float(acc[j + 1]) - my_lse);
      float d0 = my_coef * (((gc + j) == tgt ? 1.f : 0.f) - p0);
      float d1 = my_coef * (((gc + j + 1) == tgt ? 1.f : 0.f) - p1);
      if (gc + j >= V) d0 = 0.f;
      if (gc + j + 1 >= V) d1 = 0.f;
      packed[j >> 1] = pack_bf16x2(d0, d1);
    }
    if (gc + 32 <= ldo) {
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<uint4*>(o + 2 * j) = make_uint4(packed[j], packed[j + 1], packed[j + 2], packed[j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (gc + 2 * j + 1 < ldo) *reinterpret_cast<uint32_t*>(o + 2 * j) = packed[j];
    }
  }
  __device__ void tile_end(const TileInfo&, int) {}
};

// Sampling epilogue for the rollout engine: temperature-scaled online softmax statistics plus a
// running Gumbel-max argmax, so one pass over the LM head yields the sampled token and its
// log-probability under the sampling distribution without materialising logits.
//   x = logit * inv_temp ;  sample = argmax_v (x_v + g_v),  g_v = -log(-log(u_v)),  u_v = hash(seed, row, v)
// inv_temp == 0 selects greedy decoding (argmax of the raw logits, log-prob at temperature 1).
// Noise, exponential and arg-max are some 40 dependent instructions per logit: two warps per lane quarter, each with the
// statistics of its half of every tile's columns (a partial of its own).
template <int BN>
struct EpiSample {
  static constexpr int COL_SPLIT = 2;
  float* partials;        // [2 splits, M, 8]: max, sumexp, best_score, best_idx(bits), best_x, -, -, -
  const float* inv_temp;  // [M] per-row 1/temperature (0 = greedy)
  const uint32_t* row_seed;  // [M] per-row seed (request seed mixed with the decode step)
  int M, V, vocab_offset;
  float run_max, run_sum, best_score, best_x, it;
  int best_idx;
  uint32_t seed;

  __device__ void tile_begin(const TileInfo& ti, int row) {
    if (ti.first) {
      run_max = -INFINITY;
      run_sum = 0.f;
      best_score = -INFINITY;
      best_x = 0.f;
      best_idx = -1;
      const int gr = ti.m_blk * GEMM_BM + row;
      it = (gr < M) ? inv_temp[gr] : 0.f;
      seed = (gr < M) ? row_seed[gr] : 0u;
    }
  }
  __device__ void chunk(const TileInfo& ti, int row, int c, uint32_t (&acc)[32]) {
    const int gc = ti.n_blk * BN + c;
    if (gc >= V) return;
    const uint32_t gr = ti.m_blk * GEMM_BM + row;
    const bool greedy = it == 0.f;
    const float sc = greedy ? 1.f : it;
    float cmax = -INFINITY;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float x = __uint_as_float(acc[j]) * sc;
      if (gc + j >= V) x = -INFINITY;
      acc[j] = __float_as_uint(x);
      cmax = fmaxf(cmax, x);
    }
    const float nmax = fmaxf(run_max, cmax);
    float ssum = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float x = __uint_as_float(acc[j]);
      ssum += __expf(x - nmax);
      float score = x;
      if (!greedy) score += gumbel_noise(seed, gr, static_cast<uint32_t>(vocab_offset + gc + j));
      if (score > best_score) {
        best_score = score;
        best_x = x;
        best_idx = vocab_offset + gc + j;
      }
    }
    run_sum = run_sum * __expf(run_max - nmax) + ssum;
    run_max = nmax;
  }
  __device__ void tile_end(const TileInfo& ti, int row) {
    if (!ti.last) return;
    const int gr = ti.m_blk * GEMM_BM + row;
    if (gr >= M) return;
    float* o = partials + (static_cast<size_t>(ti.group * 2 + (epi_warp_slot() >> 2)) * M + gr) * 8;
    *reinterpret_cast<float4*>(o) = make_float4(run_max, run_sum, best_score, __int_as_float(best_idx));
    *reinterpret_cast<float4*>(o + 4) = make_float4(best_x, 0.f, 0.f, 0.f);
  }
};

// Merge sampling partials (over vocabulary splits and, for tensor-parallel heads, over ranks'
// partial buffers laid out back to back): token id and log-prob per row.
// One warp per row: a thread per row walked 200 to 300 partials one after another, 20 to 45 us.
// Of equal scores the lowest token wins, as in sample_restricted.cu and whatever the number of rows: a span's two partials
// hold the left and the right halves of its tiles, so the order of the partials is not the order of the tokens, and it
// changes with the tile width.
__global__ void sample_merge_kernel(const float* __restrict__ partials, int parts, int M, int* __restrict__ token,
                                    float* __restrict__ logprob) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= M) return;
  float mx = -INFINITY, sum = 0.f, best = -INFINITY, bx = 0.f;
  int bi = -1;
  auto take = [&](float score, int id, float x) {      // no token (-1) is behind every token
    if (score > best || (score == best && static_cast<unsigned>(id) < static_cast<unsigned>(bi))) {
      best = score;
      bi = id;
      bx = x;
    }
  };
  for (int s = lane; s < parts; s += 32) {
    const float4* p = reinterpret_cast<const float4*>(partials + (static_cast<size_t>(s) * M + row) * 8);
    const float4 a = p[0];
    const float x = p[1].x;
    const float n = fmaxf(mx, a.x);
    if (n != -INFINITY) sum = sum * __expf(mx - n) + a.y * __expf(a.x - n);
    mx = n;
    take(a.z, __float_as_int(a.w), x);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, mx, o), s2 = __shfl_xor_sync(0xffffffffu, sum, o);
    const float b2 = __shfl_xor_sync(0xffffffffu, best, o), x2 = __shfl_xor_sync(0xffffffffu, bx, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
    const float n = fmaxf(mx, m2);
    if (n != -INFINITY) sum = sum * __expf(mx - n) + s2 * __expf(m2 - n);
    mx = n;
    take(b2, i2, x2);
  }
  if (lane == 0) {
    token[row] = bi;
    logprob[row] = bx - (mx + logf(sum));
  }
}

// Merge vocabulary-split partials and evaluate the per-token GRPO terms.
//   partials [splits, M, 4];  old_lp may hold NaN (= "sampled under the current policy");
//   tok_w = weight * mask / normaliser (already shifted to next-token alignment);
//   accum[0] += sum(pg * tok_w), accum[1] += sum(kl * tok_w), accum[2] += sum(tok_w > 0)
__global__ void grpo_token_kernel(const float* __restrict__ partials, int splits, int M,
                                  const float* __restrict__ old_lp, const float* __restrict__ adv,
                                  const float* __restrict__ tok_w, const float* __restrict__ ref_lp,
                                  float eps_lo, float eps_hi, float beta, float* __restrict__ lse_out,
                                  float* __restrict__ lp_out, float* __restrict__ coef_out,
                                  float* __restrict__ accum) {
  float loc_pg = 0.f, loc_kl = 0.f, loc_n = 0.f;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
    float mx = -INFINITY;
    for (int s = 0; s < splits; ++s) mx = fmaxf(mx, partials[(static_cast<size_t>(s) * M + t) * 4]);
    float sum = 0.f, z = -INFINITY;
    for (int s = 0; s < splits; ++s) {
      const float* p = partials + (static_cast<size_t>(s) * M + t) * 4;
      sum += p[1] * __expf(p[0] - mx);
      z = fmaxf(z, p[2]);
    }
    const float lse = mx + logf(sum);
    const float lp = z - lse;
    lse_out[t] = lse;
    lp_out[t] = lp;
    float c = 0.f;
    if (tok_w) {
      const float w = tok_w[t];
      if (w != 0.f) {
        float old = old_lp[t];
        if (isnan(old)) old = lp;
        const float a = adv[t];
        const float ratio = expf(lp - old);
        const float unclipped = ratio * a;
        const float clipped = fminf(fmaxf(ratio, 1.f - eps_lo), 1.f + eps_hi) * a;
        const float pg = -fminf(unclipped, clipped);
        const bool inside = (ratio >= 1.f - eps_lo) && (ratio <= 1.f + eps_hi);
        float dpg_dlp = (inside || unclipped < clipped) ? -a * ratio : 0.f;
        float kl = 0.f, dkl_dlp = 0.f;
        if (ref_lp && beta > 0.f) {
          const float d = ref_lp[t] - lp;
          const float e = expf(d);
          kl = e - d - 1.f;
          dkl_dlp = 1.f - e;
        }
        loc_pg += pg * w;
        loc_kl += kl * w;
        loc_n += 1.f;
        c = w * (dpg_dlp + beta * dkl_dlp);
      }
    }
    if (coef_out) coef_out[t] = c;
  }
  // block reduce
  __shared__ float red[3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    loc_pg += __shfl_xor_sync(0xffffffffu, loc_pg, o);
    loc_kl += __shfl_xor_sync(0xffffffffu, loc_kl, o);
    loc_n += __shfl_xor_sync(0xffffffffu, loc_n, o);
  }
  if (lane == 0) {
    red[0][warp] = loc_pg;
    red[1][warp] = loc_kl;
    red[2][warp] = loc_n;
  }
  __syncthreads();
  if (warp == 0 && accum) {
    const int nw = blockDim.x >> 5;
    float a = lane < nw ? red[0][lane] : 0.f, b = lane < nw ? red[1][lane] : 0.f, c = lane < nw ? red[2][lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
      atomicAdd(accum + 0, a);
      atomicAdd(accum + 1, b);
      atomicAdd(accum + 2, c);
    }
  }
}

// Logits -> dlogits in place: row t of `buf` holds its V fp32 logits on entry and, from the row's start, ldl bf16 gradients on
// exit (columns V..ldl-1 zero), so the product behind it reads rows of 2 * ldl bf16.  One block per row.  A step loads
// DL_STEP logits, and only when all threads hold theirs does any of them store: the stores of step c end at byte
// 2 (c + 1) DL_STEP, behind every load of step c and below every load of step c + 1 (byte 4 (c + 1) DL_STEP on).
// Bound by HBM: 4 bytes read and 2 written per logit; 1734 rows x 152 064 in 242 us = 6.5 TB/s, where recomputing the tiles
// took 1746 us (K = 3584) and 492 us (K = 896).
constexpr int DL_THREADS = 512;
constexpr int DL_STEP = DL_THREADS * 8;

__global__ void __launch_bounds__(DL_THREADS)
dlogits_inplace_kernel(float* buf, int ldl, const int* __restrict__ target, const float* __restrict__ lse,
                       const float* __restrict__ coef, int V, int vocab_offset) {
  const int t = blockIdx.x;
  float* row = buf + static_cast<size_t>(t) * ldl;
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(row);
  const float l = lse[t], k = coef[t];
  const int tgt = target[t] - vocab_offset;
  float4 a[2];
  auto load = [&](int v) {
    a[0] = a[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (v < V) {                         // ldl is a multiple of 8: the 8 floats are in the row
      a[0] = *reinterpret_cast<const float4*>(row + v);
      a[1] = *reinterpret_cast<const float4*>(row + v + 4);
    }
  };
  int v = threadIdx.x * 8;
  load(v);
  for (int c0 = 0; c0 < ldl; c0 += DL_STEP, v += DL_STEP) {
    const float z[8] = {a[0].x, a[0].y, a[0].z, a[0].w, a[1].x, a[1].y, a[1].z, a[1].w};
    uint32_t packed[4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float d0 = k * ((v + j == tgt ? 1.f : 0.f) - __expf(z[j] - l));
      float d1 = k * ((v + j + 1 == tgt ? 1.f : 0.f) - __expf(z[j + 1] - l));
      if (v + j >= V) d0 = 0.f;
      if (v + j + 1 >= V) d1 = 0.f;
      packed[j >> 1] = pack_bf16x2(d0, d1);
    }
    __syncthreads();                     // every thread's logits of this step are in registers
    load(v + DL_STEP);
    if (v < ldl) *reinterpret_cast<uint4*>(out + v) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  }
}

// From this many token rows on, the LM-head kernels run on CTA pairs (256 x 256 logit tiles, the pair shares each
// LM-head tile in shared memory); below it (decode batches) one CTA per 128 x 256 tile fills the machine better.
static bool lp_pairs(int M) { return M >= 4 * GEMM_BM; }

template <class Epi>
static int launch_lp(const void* H, int ldh, const void* W, int ldw, int M, int V, int K, int splits,
                     const Epi& epi, int* status, cudaStream_t stream) {
  CUtensorMap tA, tB;
  int e;
  int dev = 0;
  cudaGetDevice(&dev);
  SchedVocabSplit sched;
  sched.n_tiles = (V + LP_BN - 1) / LP_BN;
  sched.splits = splits;
  sched.tiles_per_split = (sched.n_tiles + splits - 1) / splits;
  const int kb = (K + GEMM_BK - 1) / GEMM_BK;
  if ((e = make_tmap_bf16_2d(&tA, H, M, K, ldh, GEMM_BM, GEMM_BK))) return e;
  if (lp_pairs(M)) {
    using L = Gemm2SmemLayout<6, LP_BN>;
    auto kern = gemm_tcgen05_2cta_kernel<6, LP_BN, SchedVocabSplit, Epi>;
    static bool configured[64] = {false};
    if (!configured[dev & 63]) {
      cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
      if (ce != cudaSuccess) return static_cast<int>(ce);
      configured[dev & 63] = true;
    }
    if ((e = make_tmap_bf16_2d(&tB, W, V, K, ldw, LP_BN / 2, GEMM_BK))) return e;
    sched.m_tiles = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);      // pair tiles of 256 rows
    int clusters = sched.m_tiles * splits;
    if (clusters > sm_count() / 2) clusters = sm_count() / 2;
    return static_cast<int>(launch_product<2>(kern, dim3(2 * clusters), dim3(gemm_pipe_threads<Epi>()), L::TOTAL, stream, tA, tB,
                                          tA, tB, kb, 0, sched, epi, status, NoComm{}));
  }
  using L = GemmSmemLayout<LP_BN, LP_STAGES>;
  auto kern = gemm_tcgen05_kernel<LP_BN, LP_STAGES, SchedVocabSplit, Epi>;
  static bool configured[64] = {false};
  if (!configured[dev & 63]) {
    cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (ce != cudaSuccess) return static_cast<int>(ce);
    configured[dev & 63] = true;
  }
  if ((e = make_tmap_bf16_2d(&tB, W, V, K, ldw, LP_BN, GEMM_BK))) return e;
  sched.m_tiles = (M + GEMM_BM - 1) / GEMM_BM;
  int grid = sched.m_tiles * splits;
  if (grid > sm_count()) grid = sm_count();
  return static_cast<int>(launch_product<1>(kern, dim3(grid), dim3(gemm_pipe_threads<Epi>()), L::TOTAL, stream, tA, tB, tA, tB, kb,
                                        0, sched, epi, status, NoComm{}));
}

}  // namespace artb

using namespace artb;

// Number of vocabulary splits the forward uses for (M, V): enough (m_blk, split) items to
// fill the machine, never more splits than n-tiles.
static int lp_splits(int M, int V) {
  const bool pairs = lp_pairs(M);
  const int m_tiles = pairs ? (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM) : (M + GEMM_BM - 1) / GEMM_BM;
  const int n_tiles = (V + LP_BN - 1) / LP_BN;
  const int workers = pairs ? sm_count() / 2 : sm_count();
  int splits = (2 * workers + m_tiles - 1) / m_tiles;
  if (splits < 1) splits = 1;
  if (splits > n_tiles) splits = n_tiles;
  // make the last split non-empty
  while (splits > 1 && ((n_tiles + splits - 1) / splits) * (splits - 1) >= n_tiles) --splits;
  return splits;
}

// The partials buffer of artb_logprob_partials is [artb_logprob_parts, M, 4] fp32: two per split.
ARTB_EXPORT int artb_logprob_parts(int M, int V) { return 2 * lp_splits(M, V); }

// Phase 1: per-split online-softmax partials over the vocabulary shard W[V, K]; with `logits` ([M, ldl] fp32, ldl >= V and a
// multiple of 8) the logits are kept for artb_dlogits_inplace.
ARTB_EXPORT int artb_logprob_partials(const void* H, int ldh, const void* W, int ldw, const int* target,
                                      float* partials, float* logits, int ldl, int M, int V, int K, int parts,
                                      int vocab_offset, int* status, cudaStream_t stream) {
  if (M <= 0 || V <= 0 || (K & 7) || parts != artb_logprob_parts(M, V) || (logits && (ldl < V || (ldl & 7)))) return ERR_BAD_SHAPE;
  if (reinterpret_cast<uintptr_t>(logits) & 15) return ERR_BAD_ALIGN;
  EpiStats epi;
  epi.target = target;
  epi.partials = partials;
  epi.logits = logits;
  epi.ldl = ldl;
  epi.M = M;
  epi.V = V;
  epi.vocab_offset = vocab_offset;
  epi.run_max = 0.f;
  epi.run_sum = 0.f;
  epi.z = 0.f;
  epi.tgt = -1;
  return launch_lp(H, ldh, W, ldw, M, V, K, parts / 2, epi, status, stream);
}

// Phase 2: merge partials -> lse, logprob; GRPO terms; coef = dLoss/dlogprob.
// tok_w == nullptr: only lse/logprob are produced (reference-policy pass).
ARTB_EXPORT int artb_grpo_tokens(const float* partials, int splits, int M, const float* old_lp, const float* adv,
                                 const float* tok_w, const float* ref_lp, float eps_lo, float eps_hi, float beta,
                                 float* lse, float* lp, float* coef, float* accum, cudaStream_t stream) {
  if (M <= 0) return 0;
  int grid = (M + 255) / 256;
  if (grid > 1024) grid = 1024;
  grpo_token_kernel<<<grid, 256, 0, stream>>>(partials, splits, M, old_lp, adv, tok_w, ref_lp, eps_lo, eps_hi, beta,
                                              lse, lp, coef, accum);
  return static_cast<int>(cudaGetLastError());
}

// Backward phase 1: dlogits[M, ldo] (bf16) by recomputation.  ldo >= V, multiple of 8;
// columns V..ldo-1 are written as zero.
ARTB_EXPORT int artb_logprob_dlogits(const void* H, int ldh, const void* W, int ldw, const int* target,
                                     const float* lse, const float* coef, void* dlogits, int ldo, int M, int V,
                                     int K, int vocab_offset, int* status, cudaStream_t stream) {
  if (M <= 0 || V <= 0 || (K & 7) || (ldo & 7) || ldo < V) return ERR_BAD_SHAPE;
  EpiDLogits epi;
  epi.target = target;
  epi.lse = lse;
  epi.coef = coef;
  epi.out = reinterpret_cast<__nv_bfloat16*>(dlogits);
  epi.M = M;
  epi.V = V;
  epi.ldo = ldo;
  epi.vocab_offset = vocab_offset;
  epi.my_lse = 0.f;
  epi.my_coef = 0.f;
  epi.tgt = -1;
  // one split per n-tile group is irrelevant here (no cross-tile state): reuse the
  // vocab-split schedule so LM-head tiles are shared through L2 the same way.
  int splits = lp_splits(M, V);
  return launch_lp(H, ldh, W, ldw, M, V, K, splits, epi, status, stream);
}

// Backward phase 1 from kept logits: buf [M, ldl] fp32 -> rows of ldl bf16 dlogits at the start of each row (see the kernel).
ARTB_EXPORT int artb_dlogits_inplace(float* buf, int ldl, const int* target, const float* lse, const float* coef, int M, int V,
                                     int vocab_offset, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (V <= 0 || ldl < V || (ldl & 7)) return ERR_BAD_SHAPE;
  if (reinterpret_cast<uintptr_t>(buf) & 15) return ERR_BAD_ALIGN;
  dlogits_inplace_kernel<<<M, DL_THREADS, 0, stream>>>(buf, ldl, target, lse, coef, V, vocab_offset);
  return static_cast<int>(cudaGetLastError());
}

namespace artb {

template <int BN>
static EpiSample<BN> sample_epi(const float* inv_temp, const uint32_t* row_seed, float* partials, int M, int V,
                                int vocab_offset) {
  EpiSample<BN> epi;
  epi.partials = partials;
  epi.inv_temp = inv_temp;
  epi.row_seed = row_seed;
  epi.M = M;
  epi.V = V;
  epi.vocab_offset = vocab_offset;
  epi.run_max = epi.run_sum = epi.best_score = epi.best_x = epi.it = 0.f;
  epi.best_idx = -1;
  epi.seed = 0;
  return epi;
}

// Decode batches (below the CTA-pair limit): vocabulary spans of whole BN-wide tiles, one per CTA.
struct SamplePlan {
  int bn, n_tiles, m_tiles, splits;
};
// The tile width of 256, 224 or 160 columns whose longest span is the shortest, the widest where they tie: 152 064 tokens
// over 148 CTAs are 5 x 224 columns (the mean is 1027; 5 x 256 would be 14 % more), over 74 (129 to 256 rows) 13 x 160.
static SamplePlan sample_plan(int M, int V) {
  SamplePlan best{0, 0, 0, 0};
  long cost = 0;
  for (int bn : {256, 224, 160}) {
    SamplePlan p{bn, (V + bn - 1) / bn, (M + GEMM_BM - 1) / GEMM_BM, 0};
    p.splits = sm_count() / p.m_tiles;
    if (p.splits > p.n_tiles) p.splits = p.n_tiles;
    if (p.splits < 1) p.splits = 1;
    const long c = static_cast<long>((p.n_tiles + p.splits - 1) / p.splits) * bn;
    if (best.bn == 0 || c < cost) {
      best = p;
      cost = c;
    }
  }
  return best;
}

template <int BN, int STAGES, int AR = GEMM_BM>
static int launch_sample(const void* H, int ldh, const void* W, int ldw, const SamplePlan& p, const EpiSample<BN>& epi, int K,
                         int* status, cudaStream_t stream) {
  using L = GemmSmemLayout<BN, STAGES, AR>;
  static_assert(L::TOTAL <= 227 * 1024, "shared memory");
  CUtensorMap tA, tB;
  int rc;
  if ((rc = make_tmap_bf16_2d(&tA, H, epi.M, K, ldh, AR, GEMM_BK))) return rc;
  if ((rc = make_tmap_bf16_2d(&tB, W, epi.V, K, ldw, BN, GEMM_BK))) return rc;
  auto kern = gemm_tcgen05_kernel<BN, STAGES, SchedVocabSpan, EpiSample<BN>, NoComm, AR>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL);
    if (ce != cudaSuccess) return static_cast<int>(ce);
    configured[dev & 63] = true;
  }
  const SchedVocabSpan sched{p.m_tiles, p.n_tiles, p.splits, weights_early()};
  return static_cast<int>(launch_product<1>(kern, dim3(p.m_tiles * p.splits), dim3(gemm_pipe_threads<EpiSample<BN>>()), L::TOTAL,
                                        stream, tA, tB, tA, tB, (K + GEMM_BK - 1) / GEMM_BK, 0, sched, epi, status, NoComm{}));
}

}  // namespace artb

// Partials of artb_sample_partials for (M, V): two per vocabulary split.
ARTB_EXPORT int artb_sample_parts(int M, int V) {
  return 2 * (lp_pairs(M) ? lp_splits(M, V) : sample_plan(M, V).splits);
}

// Rollout sampling: partials [parts, M, 8] for one vocabulary shard (see EpiSample), parts = artb_sample_parts(M, V).
ARTB_EXPORT int artb_sample_partials(const void* H, int ldh, const void* W, int ldw, const float* inv_temp,
                                     const uint32_t* row_seed, float* partials, int M, int V, int K, int parts,
                                     int vocab_offset, int* status, cudaStream_t stream) {
  if (M <= 0 || V <= 0 || (K & 7) || parts != artb_sample_parts(M, V)) return ERR_BAD_SHAPE;
  auto epi = [&](auto bn) { return sample_epi<decltype(bn)::value>(inv_temp, row_seed, partials, M, V, vocab_offset); };
  using W256 = std::integral_constant<int, 256>;
  if (lp_pairs(M)) return launch_lp(H, ldh, W, ldw, M, V, K, parts / 2, epi(W256{}), status, stream);
  const SamplePlan p = sample_plan(M, V);
  if (p.bn == 256) return launch_sample<256, 4>(H, ldh, W, ldw, p, epi(W256{}), K, status, stream);
  if (p.bn == 224 && M <= 16) return launch_sample<224, 7, 16>(H, ldh, W, ldw, p, epi(std::integral_constant<int, 224>{}), K, status, stream);
  if (p.bn == 224 && M <= 64) return launch_sample<224, 6, 64>(H, ldh, W, ldw, p, epi(std::integral_constant<int, 224>{}), K, status, stream);
  if (p.bn == 224) return launch_sample<224, 5>(H, ldh, W, ldw, p, epi(std::integral_constant<int, 224>{}), K, status, stream);
  return launch_sample<160, 6>(H, ldh, W, ldw, p, epi(std::integral_constant<int, 160>{}), K, status, stream);
}

ARTB_EXPORT int artb_sample_merge(const float* partials, int parts, int M, int* token, float* logprob,
                                  cudaStream_t stream) {
  if (M <= 0) return 0;
  sample_merge_kernel<<<(M + 3) / 4, 128, 0, stream>>>(partials, parts, M, token, logprob);
  return static_cast<int>(cudaGetLastError());
}
