// Paged-KV attention for the rollout engine: cache write, decode attention over block
// tables (GQA, split-KV), and a page gather used by prefill with prefix-cache hits.
//
// Cache layout per layer: k_cache, v_cache  [num_blocks, block_size, Hkv, hd]  bf16.
// A sequence's tokens live in the blocks listed in its row of `block_table`
// [num_seqs, max_blocks]; token t is in block table[t / block_size] at offset t % block_size.
//
// Decode: one new token per sequence.  The G = Hq/Hkv query heads that share a kv head form the rows of one m16 MMA
// tile, so K and V are read once for all of them.  Each of a CTA's 4 warps walks its own 32-key tiles (cp.async into
// private smem stages), keeps private online-softmax state, and the warps are merged through shared memory at the end.
// The op is bandwidth-bound (it streams the KV of every running sequence once per step).  Two ways to share the keys
// out: even shares over the whole chip (the rollout engine's), or a CTA per (sequence, kv head, split), whose partial
// (max, sum, acc) triples a second kernel merges (callers that bring no workspace, or a static one).
//
// This is the in-tree counterpart of the decode/prefill attention the reference delegates to
// its third-party engine (every chat.completions.create ends up there: src/art/local/vllm.py:46-53).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "bounds_check.cuh"
#include "host_utils.h"

namespace artb {

__device__ __forceinline__ void pa_cp16(void* smem, const void* gmem, bool valid) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
}
__device__ __forceinline__ void pa_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void pa_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void pa_ldsm_x4(uint32_t (&r)[4], const void* p) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void pa_ldsm_x4_t(uint32_t (&r)[4], const void* p) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void pa_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pa_pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// ------------------------------------------------------------------ cache write
// qkv [M, ld] holds q | k | v columns (post-RoPE).  slot[m] = block * block_size + offset, or < 0 to skip.
__global__ void kv_write_kernel(const __nv_bfloat16* __restrict__ qkv, int ld, int k_col, int v_col,
                                const int* __restrict__ slot, __nv_bfloat16* __restrict__ k_cache,
                                __nv_bfloat16* __restrict__ v_cache, int M, int kv_width, long num_slots, int* status) {
  const int vec = kv_width >> 3;
  const long total = static_cast<long>(M) * vec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int m = i / vec, c = (i % vec) * 8;
    const int s = slot[m];
    if (s < 0 || !index_ok(s, num_slots, status)) continue;
    const uint4 kv = *reinterpret_cast<const uint4*>(qkv + static_cast<size_t>(m) * ld + k_col + c);
    const uint4 vv = *reinterpret_cast<const uint4*>(qkv + static_cast<size_t>(m) * ld + v_col + c);
    *reinterpret_cast<uint4*>(k_cache + static_cast<size_t>(s) * kv_width + c) = kv;
    *reinterpret_cast<uint4*>(v_cache + static_cast<size_t>(s) * kv_width + c) = vv;
  }
}

// Gather the first n_tok cached tokens of one sequence into contiguous k | v columns of dst [*, ld] (prompt steps take all
// their sequences' rows at once: kv_rows below).
__global__ void kv_gather_kernel(const __nv_bfloat16* __restrict__ k_cache, const __nv_bfloat16* __restrict__ v_cache,
                                 const int* __restrict__ block_table, int block_size, int n_tok,
                                 __nv_bfloat16* __restrict__ dst, int ld, int k_col, int v_col, int kv_width,
                                 long num_blocks, int* status) {
  const int vec = kv_width >> 3;
  const long total = static_cast<long>(n_tok) * vec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int t = i / vec, c = (i % vec) * 8;
    const int blk = block_table[t / block_size];
    if (!index_ok(blk, num_blocks, status)) continue;
    const size_t s = static_cast<size_t>(blk) * block_size + t % block_size;
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(t) * ld + k_col + c) =
        *reinterpret_cast<const uint4*>(k_cache + s * kv_width + c);
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(t) * ld + v_col + c) =
        *reinterpret_cast<const uint4*>(v_cache + s * kv_width + c);
  }
}

// The cached keys and values at a list of slots -> k | v columns of dst [n, ld], one launch for all sequences of a batch;
// rows with a negative slot become zeros.
__global__ void kv_rows_kernel(const __nv_bfloat16* __restrict__ k_cache, const __nv_bfloat16* __restrict__ v_cache,
                               const int* __restrict__ slot, int n, __nv_bfloat16* __restrict__ dst, int ld, int k_col, int v_col,
                               int kv_width, long num_slots, int* status) {
  const int vec = kv_width >> 3;
  const long total = static_cast<long>(n) * vec;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const int t = i / vec, c = (i % vec) * 8;
    const int s = slot[t];
    uint4 k = make_uint4(0, 0, 0, 0), v = k;
    if (s >= 0 && index_ok(s, num_slots, status)) {
      k = *reinterpret_cast<const uint4*>(k_cache + static_cast<size_t>(s) * kv_width + c);
      v = *reinterpret_cast<const uint4*>(v_cache + static_cast<size_t>(s) * kv_width + c);
    }
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(t) * ld + k_col + c) = k;
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(t) * ld + v_col + c) = v;
  }
}

// ------------------------------------------------------------------ decode attention
constexpr int PA_KT = 32;  // keys per warp tile

// Online-softmax state of a warp's share of the keys: rows g and g + 8 of the m16 tile of query heads.
template <int HD>
struct PaState {
  float acc[HD / 8][4];
  float m0, m1, l0, l1;
};

// The CTA's tiles [tile_lo, tile_hi) of keys [0, len) for the G query heads at q_row; warp w takes the tiles tile_lo + w,
// + 4, ..., from a private K and a private V stage.  K of the next tile
// is requested as soon as the scores have been taken from the K stage, V of the next tile once the products are added,
// and the cache slots (one key per lane) one tile ahead of both: a warp always has copies in flight without a second
// stage, which would halve the warps per SM.
template <int HD>
__device__ __forceinline__ void pa_walk(PaState<HD>& st, __nv_bfloat16* sQ, const __nv_bfloat16* q_row, int G, __nv_bfloat16* sKV,
                                        const __nv_bfloat16* kc, const __nv_bfloat16* vc, const int* bt, int len, int block_size,
                                        int kv_width, int tile_lo, int tile_hi, float scale_log2, long num_blocks, int* status) {
  constexpr int LD = HD + 8;
  constexpr int CPR = HD / 8;                 // 16-byte copies per row
  constexpr int RPI = 32 / CPR;               // rows covered by the warp per iteration
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = lane & 3, jm = lane >> 3, rr = lane & 7;
  const int bs_shift = (block_size & (block_size - 1)) == 0 ? 31 - __clz(block_size) : -1;   // power of two: shifts
  __nv_bfloat16* wK = sKV + warp * 2 * PA_KT * LD;
  __nv_bfloat16* wV = wK + PA_KT * LD;
#pragma unroll
  for (int i = 0; i < HD / 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) st.acc[i][j] = 0.f;
  st.m0 = st.m1 = -INFINITY;
  st.l0 = st.l1 = 0.f;
  // the cache slot of this lane's key of a tile, or -1: no such key, zeros are staged
  auto slot_of = [&](int tile) {
    const int kt = tile * PA_KT + lane;
    if (tile >= tile_hi || kt >= len) return -1;
    const int blk = bt[bs_shift >= 0 ? kt >> bs_shift : kt / block_size];
    if (!index_ok(blk, num_blocks, status)) return -1;       // checked build: a bad table entry reads zeros instead
    return blk * block_size + (bs_shift >= 0 ? kt & (block_size - 1) : kt % block_size);
  };
  const int c = (lane % CPR) * 8, r0 = lane / CPR;
  auto stage = [&](__nv_bfloat16* dst, const __nv_bfloat16* src, int slot) {
#pragma unroll
    for (int i = 0; i < PA_KT / RPI; ++i) {
      const int r = r0 + i * RPI, s = __shfl_sync(0xffffffffu, slot, r);
      pa_cp16(dst + r * LD + c, src + static_cast<size_t>(s < 0 ? 0 : s) * kv_width + c, s >= 0);
    }
    pa_commit();
  };
  int tile = tile_lo + warp;
  const int s_cur = slot_of(tile);
  int s_next = slot_of(tile + 4);
  // the query rows are on their way while the table is looked up: G real heads, the other rows zero
  uint4 q_val[HD / 64 ? HD / 64 : 1];
#pragma unroll
  for (int i = 0; i < (HD / 64 ? HD / 64 : 1); ++i) {
    const int v = threadIdx.x + i * 128, r = v / CPR;
    q_val[i] = v < 16 * CPR && r < G ? *reinterpret_cast<const uint4*>(q_row + r * HD + (v % CPR) * 8) : make_uint4(0, 0, 0, 0);
  }
  if (tile < tile_hi) {
    stage(wK, kc, s_cur);
    stage(wV, vc, s_cur);
  }
#pragma unroll
  for (int i = 0; i < (HD / 64 ? HD / 64 : 1); ++i) {
    const int v = threadIdx.x + i * 128;
    if (v < 16 * CPR) *reinterpret_cast<uint4*>(sQ + (v / CPR) * LD + (v % CPR) * 8) = q_val[i];
  }
  __syncthreads();
  if (tile >= tile_hi) return;
  uint32_t qf[HD / 16][4];
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks)
    pa_ldsm_x4(qf[ks], sQ + ((jm & 1) * 8 + rr) * LD + ks * 16 + (jm >> 1) * 8);
  for (; tile < tile_hi; tile += 4) {
    const int k0 = tile * PA_KT, s_after = slot_of(tile + 8);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll
    for (int ks = 0; ks < HD / 16; ++ks) {
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t b[4];
        pa_ldsm_x4(b, wK + (np * 16 + (jm >> 1) * 8 + rr) * LD + ks * 16 + (jm & 1) * 8);
        pa_mma(s[np * 2], qf[ks], b[0], b[1]);
        pa_mma(s[np * 2 + 1], qf[ks], b[2], b[3]);
      }
    }
    __syncwarp();
    if (tile + 4 < tile_hi)
      stage(wK, kc, s_next);
    else
      pa_commit();
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int kt = k0 + i * 8 + 2 * t + j;
        float x0 = s[i][j] * scale_log2, x1 = s[i][2 + j] * scale_log2;
        if (kt >= len) x0 = x1 = -INFINITY;
        s[i][j] = x0;
        s[i][2 + j] = x1;
        mx0 = fmaxf(mx0, x0);
        mx1 = fmaxf(mx1, x1);
      }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float mn0 = fmaxf(st.m0, mx0), mn1 = fmaxf(st.m1, mx1);
    const float ms0 = mn0 == -INFINITY ? 0.f : mn0, ms1 = mn1 == -INFINITY ? 0.f : mn1;
    const float c0 = exp2f(st.m0 - ms0), c1 = exp2f(st.m1 - ms1);
    st.m0 = mn0;
    st.m1 = mn1;
    float rs0 = 0.f, rs1 = 0.f;
    uint32_t pf[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float p00 = exp2f(s[i][0] - ms0), p01 = exp2f(s[i][1] - ms0);
      const float p10 = exp2f(s[i][2] - ms1), p11 = exp2f(s[i][3] - ms1);
      rs0 += p00 + p01;
      rs1 += p10 + p11;
      pf[i >> 1][(i & 1) * 2] = pa_pack2(p00, p01);
      pf[i >> 1][(i & 1) * 2 + 1] = pa_pack2(p10, p11);
    }
    st.l0 = st.l0 * c0 + rs0;
    st.l1 = st.l1 * c1 + rs1;
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) {
      st.acc[i][0] *= c0;
      st.acc[i][1] *= c0;
      st.acc[i][2] *= c1;
      st.acc[i][3] *= c1;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
      for (int dp = 0; dp < HD / 16; ++dp) {
        uint32_t b[4];
        pa_ldsm_x4_t(b, wV + (ks * 16 + (jm & 1) * 8 + rr) * LD + dp * 16 + (jm >> 1) * 8);
        pa_mma(st.acc[dp * 2], pf[ks], b[0], b[1]);
        pa_mma(st.acc[dp * 2 + 1], pf[ks], b[2], b[3]);
      }
    }
    __syncwarp();
    if (tile + 4 < tile_hi)
      stage(wV, vc, s_next);
    else
      pa_commit();
    s_next = s_after;
  }
  pa_wait_all();
  __syncwarp();
  st.l0 += __shfl_xor_sync(0xffffffffu, st.l0, 1);
  st.l0 += __shfl_xor_sync(0xffffffffu, st.l0, 2);
  st.l1 += __shfl_xor_sync(0xffffffffu, st.l1, 1);
  st.l1 += __shfl_xor_sync(0xffffffffu, st.l1, 2);
}

// Publishes the four warps' states and calls put(row, column, max, sum, values) for every four columns of the G rows, the
// values not yet divided by the sum.  The accumulators [16][HD] fp32 go to each warp's own (by then finished) K/V stage,
// which keeps a CTA under a third of the SM's shared memory: three CTAs = twelve warps per SM instead of eight.
template <int HD, class Put>
__device__ __forceinline__ void pa_merge_warps(const PaState<HD>& st, __nv_bfloat16* sKV, float* sM, int G, Put put) {
  constexpr int LD = HD + 8;
  static_assert(16 * HD * 4 <= 2 * PA_KT * LD * 2, "a warp's accumulator slice must fit its K/V staging area");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  auto warp_acc = [&](int w) { return reinterpret_cast<float*>(sKV + w * 2 * PA_KT * LD); };
  // per-warp state (rows g and g + 8; only rows < G matter)
  if (t == 0) {
    sM[warp * 16 + g] = st.m0;
    sM[warp * 16 + g + 8] = st.m1;
    sM[64 + warp * 16 + g] = st.l0;
    sM[64 + warp * 16 + g + 8] = st.l1;
  }
#pragma unroll
  for (int i = 0; i < HD / 8; ++i) {
    float* a0 = warp_acc(warp) + g * HD + i * 8 + 2 * t;
    float* a1 = warp_acc(warp) + (g + 8) * HD + i * 8 + 2 * t;
    a0[0] = st.acc[i][0];
    a0[1] = st.acc[i][1];
    a1[0] = st.acc[i][2];
    a1[1] = st.acc[i][3];
  }
  __syncthreads();
  for (int idx = tid; idx < G * (HD / 4); idx += 128) {
    const int r = idx / (HD / 4);
    float m[4], mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) mm = fmaxf(mm, m[w] = sM[w * 16 + r]);
    float lsum = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mm != -INFINITY) {
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float sc = exp2f(m[w] - mm);
        const float4 v = reinterpret_cast<const float4*>(warp_acc(w))[idx];
        lsum = fmaf(sM[64 + w * 16 + r], sc, lsum);
        o.x = fmaf(v.x, sc, o.x);
        o.y = fmaf(v.y, sc, o.y);
        o.z = fmaf(v.z, sc, o.z);
        o.w = fmaf(v.w, sc, o.w);
      }
    }
    put(r, idx * 4 - r * HD, mm, lsum, o);
  }
}

__device__ __forceinline__ void pa_store4(__nv_bfloat16* dst, const float4& o, float sum) {
  const float inv = sum > 0.f ? 1.f / sum : 0.f;
  *reinterpret_cast<uint2*>(dst) = make_uint2(pa_pack2(o.x * inv, o.y * inv), pa_pack2(o.z * inv, o.w * inv));
}

// One CTA per (sequence, kv head, split) and a split for every 1 / splits of a sequence's keys: the caller chooses.
template <int HD>
__global__ void __launch_bounds__(128)
paged_decode_kernel(const __nv_bfloat16* __restrict__ q, int ldq, const __nv_bfloat16* __restrict__ k_cache,
                    const __nv_bfloat16* __restrict__ v_cache, const int* __restrict__ block_table, int max_blocks,
                    const int* __restrict__ ctx_len, int block_size, int Hq, int Hkv,
                    __nv_bfloat16* __restrict__ out, int ldo, float* __restrict__ ws, int splits,
                    float scale_log2, long num_blocks, int* status) {
  constexpr int LD = HD + 8;
  extern __shared__ __align__(16) uint8_t pa_smem[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(pa_smem);      // [16][LD]
  __nv_bfloat16* sKV = sQ + 16 * LD;                                   // [4 warps][2 (K,V)][PA_KT][LD]
  float* sM = reinterpret_cast<float*>(sKV + 4 * 2 * PA_KT * LD);      // merge: [4][16] max, [4][16] sum

  pdl_wait();                  // q, the cache rows of this step and the block table come from earlier kernels
  pdl_launch_dependents();
  const int seq = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int G = Hq / Hkv;
  const int len = ctx_len[seq];

  // key range of this split, in tiles of PA_KT; warps interleave tiles
  const int tiles_total = (len + PA_KT - 1) / PA_KT;
  const int tiles_per_split = (tiles_total + splits - 1) / splits;
  const int tile_lo = split * tiles_per_split;
  const int tile_hi = min(tiles_total, tile_lo + tiles_per_split);
  PaState<HD> st;
  pa_walk<HD>(st, sQ, q + static_cast<size_t>(seq) * ldq + kvh * G * HD, G, sKV, k_cache + kvh * HD, v_cache + kvh * HD,
              block_table + static_cast<size_t>(seq) * max_blocks, len, block_size, Hkv * HD, tile_lo, tile_hi, scale_log2,
              num_blocks, status);
  pa_merge_warps<HD>(st, sKV, sM, G, [&](int r, int d, float mm, float lsum, const float4& o) {
    const int h = kvh * G + r;
    if (splits == 1) {
      const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
      __nv_bfloat16* dst = out + static_cast<size_t>(seq) * ldo + h * HD + d;
      dst[0] = __float2bfloat16(o.x * inv);
      dst[1] = __float2bfloat16(o.y * inv);
      dst[2] = __float2bfloat16(o.z * inv);
      dst[3] = __float2bfloat16(o.w * inv);
    } else {
      // workspace: [seq, Hq, splits, HD + 2]
      float* w = ws + ((static_cast<size_t>(seq) * Hq + h) * splits + split) * (HD + 2);
      w[d] = o.x;
      w[d + 1] = o.y;
      w[d + 2] = o.z;
      w[d + 3] = o.w;
      if (d == 0) {
        w[HD] = mm;
        w[HD + 1] = lsum;
      }
    }
  });
}

// Even shares.  The sequences are laid end to end, in tiles of PA_KT keys, and cut into equal shares, wherever sequences
// begin and end in them; a share belongs to Hkv neighbouring CTAs, one per kv head, and the shares together fill the chip
// once.  With a CTA per (sequence, kv head) the step took as long as the SM with the longest contexts: 183 us for 48
// contexts of 2000 to 6000 keys with 8 heads of 128, of which the bytes take 122; and 16 CTAs (one context, 2 heads) left
// the chip idle.  The heads of a share walk the same keys at the same time because they lie side by side in the cache: with
// every head cut on its own the same contexts took 403 us.  A pair of sequence and head that lies in several shares is left
// by each as (max, sum, accumulators) in the workspace and merged, in the order of its tiles, by the CTA that finishes
// last.  Bound by the cache's bytes: 145 us for those 48 contexts (845 MB), 125 us instead of 142 for 256 contexts of 512
// to 2032 keys with 4 heads (653 MB), 8.5 us instead of 20.8 for one context of 777 keys with 2 heads.
constexpr int PA_MIN_TILES = 4;          // one per warp: less would idle warps and only add partial results

constexpr int pa_ctas_per_sm(int hd) { return hd == 128 ? 3 : 4; }       // by shared memory and registers
__host__ __device__ constexpr int pa_slot_floats(int G, int hd) { return G * hd + ((2 * G + 3) & ~3); }

template <int HD>
__global__ void __launch_bounds__(128, pa_ctas_per_sm(HD))
paged_decode_even_kernel(const __nv_bfloat16* __restrict__ q, int ldq, const __nv_bfloat16* __restrict__ k_cache,
                         const __nv_bfloat16* __restrict__ v_cache, const int* __restrict__ block_table, int max_blocks,
                         const int* __restrict__ ctx_len, int block_size, int nseq, int Hq, int Hkv,
                         __nv_bfloat16* __restrict__ out, int ldo, float* part, int* count, float scale_log2,
                         long num_blocks, int* status) {
  constexpr int LD = HD + 8;
  extern __shared__ __align__(16) uint8_t pa_smem[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(pa_smem);      // [16][LD]
  __nv_bfloat16* sKV = sQ + 16 * LD;                                   // [4 warps][2 (K,V)][PA_KT][LD]
  float* sM = reinterpret_cast<float*>(sKV + 4 * 2 * PA_KT * LD);      // merge: [4][16] max, [4][16] sum
  __shared__ int s_warp[4], s_at[3], s_done;
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = Hq / Hkv, shares = gridDim.x / Hkv, share = blockIdx.x / Hkv, kvh = blockIdx.x - share * Hkv;
  auto tiles_in = [](int len) { return (len + PA_KT - 1) / PA_KT; };

  // where this share begins: each thread sums the tiles of a run of sequences, then a scan over the threads
  const int run = (nseq + 127) / 128, i0 = min(nseq, tid * run), i1 = min(nseq, i0 + run);
  int own = 0, len = 0;
  for (int i = i0; i < i1; ++i) {
    own += tiles_in(len = max(0, ctx_len[i]));
    if (len == 0 && share == shares - 1) {           // an empty context (the padding of a batch): zeros
      uint2* o = reinterpret_cast<uint2*>(out + static_cast<size_t>(i) * ldo + kvh * G * HD);
      for (int d = 0; d < G * HD / 4; ++d) o[d] = make_uint2(0, 0);
    }
  }
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int total = 0, before = incl - own;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    if (w < warp) before += s_warp[w];
    total += s_warp[w];
  }
  const int per = max(PA_MIN_TILES, (total + shares - 1) / shares);
  int at = share * per;
  if (at >= total) return;                  // the whole CTA
  const int end = min(total, at + per);
  if (before <= at && at < before + own) {
    int i = i0, b = before;
    for (;; ++i) {
      len = max(0, ctx_len[i]);
      const int n = tiles_in(len);
      if (at < b + n) break;
      b += n;
    }
    s_at[0] = i;
    s_at[1] = b;
    s_at[2] = len;
  }
  __syncthreads();
  int seq = s_at[0], first = s_at[1];
  len = s_at[2];
  const int slot_floats = pa_slot_floats(G, HD);
  while (true) {
    const int tiles = tiles_in(len), lo = at - first, hi = min(tiles, end - first);
    PaState<HD> st;
    pa_walk<HD>(st, sQ, q + static_cast<size_t>(seq) * ldq + kvh * G * HD, G, sKV, k_cache + kvh * HD, v_cache + kvh * HD,
                block_table + static_cast<size_t>(seq) * max_blocks, len, block_size, Hkv * HD, lo, hi, scale_log2, num_blocks,
                status);
    // only now may the next product's CTAs come and request their weights: beside the first loads of a short context
    // they made it 13 us instead of 8.5
    if (first + hi >= end) pdl_launch_dependents();
    __nv_bfloat16* o_row = out + static_cast<size_t>(seq) * ldo + kvh * G * HD;
    // a CTA leaves at most two partial results: of the sequence that it begins in the middle of, and of the one it ends in
    auto slot = [&](int sh, bool starts) { return part + static_cast<size_t>((sh * Hkv + kvh) * 2 + starts) * slot_floats; };
    const bool whole = lo == 0 && hi == tiles;
    float* w = slot(share, lo == 0);
    pa_merge_warps<HD>(st, sKV, sM, G, [&](int r, int d, float mm, float lsum, const float4& o) {
      if (whole) {
        pa_store4(o_row + r * HD + d, o, lsum);
      } else {
        *reinterpret_cast<float4*>(w + r * HD + d) = o;
        if (d == 0) {
          w[G * HD + r] = mm;
          w[G * HD + G + r] = lsum;
        }
      }
    });
    if (!whole) {
      __threadfence();
      __syncthreads();
      const int sh0 = first / per, parts = (first + tiles - 1) / per - sh0 + 1;
      if (tid == 0) s_done = atomicAdd(&count[seq * Hkv + kvh], 1) == parts - 1;
      __syncthreads();
      if (s_done) {
        __threadfence();
        for (int idx = tid; idx < G * HD / 4; idx += 128) {
          const int r = idx / (HD / 4);
          float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
          float mx = -INFINITY, sum = 0.f;
          for (int p0 = 0; p0 < parts; p0 += 8) {          // eight partial results' loads in flight
            float m[8], l[8];
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float* sl = slot(sh0 + min(p0 + j, parts - 1), p0 + j == 0);
              m[j] = p0 + j < parts ? __ldcg(sl + G * HD + r) : -INFINITY;
              l[j] = __ldcg(sl + G * HD + G + r);
              v[j] = __ldcg(reinterpret_cast<const float4*>(sl) + idx);
            }
            float mn = mx;
#pragma unroll
            for (int j = 0; j < 8; ++j) mn = fmaxf(mn, m[j]);
            if (mn == -INFINITY) continue;
            const float c = exp2f(mx - mn);
            mx = mn;
            o = make_float4(o.x * c, o.y * c, o.z * c, o.w * c);
            sum *= c;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float sc = exp2f(m[j] - mn);
              sum = fmaf(l[j], sc, sum);
              o.x = fmaf(v[j].x, sc, o.x);
              o.y = fmaf(v[j].y, sc, o.y);
              o.z = fmaf(v[j].z, sc, o.z);
              o.w = fmaf(v[j].w, sc, o.w);
            }
          }
          pa_store4(o_row + idx * 4, o, sum);
        }
        if (tid == 0) count[seq * Hkv + kvh] = 0;            // as the next launch expects it
      }
    }
    at = first + hi;
    if (at >= end) return;
    first = at;                               // the next sequence, from its first tile
    do {
      len = ctx_len[++seq];
    } while (len <= 0);
    __syncthreads();
  }
}

template <int HD>
__global__ void paged_decode_merge_kernel(const float* __restrict__ ws, int splits, int Hq,
                                          __nv_bfloat16* __restrict__ out, int ldo) {
  const int seq = blockIdx.x, h = blockIdx.y, d = threadIdx.x;
  const float* base = ws + (static_cast<size_t>(seq) * Hq + h) * splits * (HD + 2);
  float mm = -INFINITY;
  for (int s = 0; s < splits; ++s) mm = fmaxf(mm, base[s * (HD + 2) + HD]);
  float lsum = 0.f, o = 0.f;
  if (mm != -INFINITY) {
    for (int s = 0; s < splits; ++s) {
      const float sc = exp2f(base[s * (HD + 2) + HD] - mm);
      lsum += base[s * (HD + 2) + HD + 1] * sc;
      o += base[s * (HD + 2) + d] * sc;
    }
  }
  out[static_cast<size_t>(seq) * ldo + h * HD + d] = __float2bfloat16(lsum > 0.f ? o / lsum : 0.f);
}

template <int HD>
static int decode_smem() {
  return (16 * (HD + 8) + 4 * 2 * PA_KT * (HD + 8)) * 2 + (2 * 4 * 16) * 4;
}

}  // namespace artb

using namespace artb;
typedef __nv_bfloat16 bf16;

ARTB_EXPORT int artb_kv_write(const void* qkv, int ld, int k_col, int v_col, const int* slot, void* k_cache,
                              void* v_cache, int M, int kv_width, long num_slots, int* status, cudaStream_t st) {
  if (M <= 0) return 0;
  if ((kv_width & 7) || (ld & 7) || (k_col & 7) || (v_col & 7)) return ERR_BAD_SHAPE;
  long total = (long)M * (kv_width / 8);
  long blocks = (total + 255) / 256;
  if (blocks > 148L * 16) blocks = 148L * 16;
  kv_write_kernel<<<(unsigned)blocks, 256, 0, st>>>((const bf16*)qkv, ld, k_col, v_col, slot, (bf16*)k_cache,
                                                   (bf16*)v_cache, M, kv_width, num_slots, status);
  return (int)cudaGetLastError();
}

ARTB_EXPORT int artb_kv_gather(const void* k_cache, const void* v_cache, const int* block_table, int block_size,
                               int n_tok, void* dst, int ld, int k_col, int v_col, int kv_width, long num_blocks,
                               int* status, cudaStream_t st) {
  if (n_tok <= 0) return 0;
  long total = (long)n_tok * (kv_width / 8);
  long blocks = (total + 255) / 256;
  if (blocks > 148L * 16) blocks = 148L * 16;
  kv_gather_kernel<<<(unsigned)blocks, 256, 0, st>>>((const bf16*)k_cache, (const bf16*)v_cache, block_table,
                                                    block_size, n_tok, (bf16*)dst, ld, k_col, v_col, kv_width,
                                                    num_blocks, status);
  return (int)cudaGetLastError();
}

ARTB_EXPORT int artb_kv_rows(const void* k_cache, const void* v_cache, const int* slot, int n, void* dst, int ld, int k_col,
                             int v_col, int kv_width, long num_slots, int* status, cudaStream_t st) {
  if (n <= 0) return 0;
  if ((kv_width & 7) || (ld & 7) || (k_col & 7) || (v_col & 7)) return ERR_BAD_SHAPE;
  long blocks = (static_cast<long>(n) * (kv_width / 8) + 255) / 256;
  if (blocks > 148L * 16) blocks = 148L * 16;
  kv_rows_kernel<<<(unsigned)blocks, 256, 0, st>>>((const bf16*)k_cache, (const bf16*)v_cache, slot, n, (bf16*)dst, ld, k_col,
                                                  v_col, kv_width, num_slots, status);
  return (int)cudaGetLastError();
}

// Workspace floats needed for `splits` > 1: num_seqs * Hq * splits * (hd + 2).
ARTB_EXPORT int artb_paged_decode(const void* q, int ldq, const void* k_cache, const void* v_cache,
                                  const int* block_table, int max_blocks, const int* ctx_len, int block_size,
                                  int num_seqs, int Hq, int Hkv, int hd, void* out, int ldo, float* ws, int splits,
                                  long num_blocks, int* status, cudaStream_t st) {
  if (num_seqs <= 0) return 0;
  if (Hq <= 0 || Hkv <= 0 || Hq % Hkv || Hq / Hkv > 16 || splits < 1 || (splits > 1 && !ws)) return ERR_BAD_SHAPE;
  int dev_ = 0;
  if (cudaGetDevice(&dev_) != cudaSuccess || dev_ < 0 || dev_ >= 64) return ERR_BAD_SHAPE;
  const float scale_log2 = 1.4426950408889634f / sqrtf((float)hd);
  dim3 grid(num_seqs, Hkv, splits);
#define ARTB_PD(HD_)                                                                                             \
  {                                                                                                              \
    static bool cfgd[64] = {false};   /* the attribute is per device */                                          \
    if (!cfgd[dev_]) {                                                                                           \
      cudaFuncSetAttribute(paged_decode_kernel<HD_>, cudaFuncAttributeMaxDynamicSharedMemorySize, decode_smem<HD_>()); \
      cfgd[dev_] = true;                                                                                         \
    }                                                                                                            \
    launch_kernel(paged_decode_kernel<HD_>, grid, dim3(128), decode_smem<HD_>(), st, (const bf16*)q, ldq,        \
                  (const bf16*)k_cache, (const bf16*)v_cache, block_table, max_blocks, ctx_len, block_size, Hq, Hkv, \
                  (bf16*)out, ldo, ws, splits, scale_log2, num_blocks, status);                                  \
    if (splits > 1) paged_decode_merge_kernel<HD_><<<dim3(num_seqs, Hq), HD_, 0, st>>>(ws, splits, Hq, (bf16*)out, ldo); \
  }
  if (hd == 128) ARTB_PD(128)
  else if (hd == 64) ARTB_PD(64)
  else if (hd == 32) ARTB_PD(32)
  else return ERR_BAD_SHAPE;
#undef ARTB_PD
  return (int)cudaGetLastError();
}

// whole shares: one CTA per kv head in each
static int even_grid(int hd, int Hkv) {
  const int shares = sm_count() * pa_ctas_per_sm(hd) / Hkv;
  return (shares < 1 ? 1 : shares) * Hkv;
}

static int even_part_bytes(int Hq, int Hkv, int hd) { return even_grid(hd, Hkv) * 2 * pa_slot_floats(Hq / Hkv, hd) * 4; }

// Bytes of workspace for artb_paged_decode_even: two partial results per CTA, then counters [num_seqs * Hkv] (zero before the
// first call, zero again after each).  The counters lie behind what does not depend on the batch, so that a call with fewer
// sequences leaves those of a larger one as they are.
ARTB_EXPORT int artb_paged_decode_even_bytes(int num_seqs, int Hq, int Hkv, int hd) {
  if (num_seqs <= 0 || Hkv <= 0 || Hq % Hkv) return 0;
  return even_part_bytes(Hq, Hkv, hd) + ((num_seqs * Hkv + 3) / 4) * 16;
}

// The same result with the keys of all sequences in even shares over the chip.  One call at a time may use a workspace.
ARTB_EXPORT int artb_paged_decode_even(const void* q, int ldq, const void* k_cache, const void* v_cache,
                                       const int* block_table, int max_blocks, const int* ctx_len, int block_size,
                                       int num_seqs, int Hq, int Hkv, int hd, void* out, int ldo, void* ws,
                                       long num_blocks, int* status, cudaStream_t st) {
  if (num_seqs <= 0) return 0;
  if (Hq <= 0 || Hkv <= 0 || Hq % Hkv || Hq / Hkv > 16 || (ldq & 7) || (ldo & 3) || !ws) return ERR_BAD_SHAPE;
  if ((reinterpret_cast<uintptr_t>(ws) & 15) || (reinterpret_cast<uintptr_t>(q) & 15) || (reinterpret_cast<uintptr_t>(out) & 7))
    return ERR_BAD_ALIGN;
  int dev_ = 0;
  if (cudaGetDevice(&dev_) != cudaSuccess || dev_ < 0 || dev_ >= 64) return ERR_BAD_SHAPE;
  const float scale_log2 = 1.4426950408889634f / sqrtf((float)hd);
  float* part = static_cast<float*>(ws);
  int* count = reinterpret_cast<int*>(static_cast<char*>(ws) + even_part_bytes(Hq, Hkv, hd));
#define ARTB_PE(HD_)                                                                                                     \
  {                                                                                                                      \
    static bool cfgd[64] = {false};   /* the attribute is per device */                                                  \
    if (!cfgd[dev_]) {                                                                                                   \
      cudaError_t e =                                                                                                    \
          cudaFuncSetAttribute(paged_decode_even_kernel<HD_>, cudaFuncAttributeMaxDynamicSharedMemorySize, decode_smem<HD_>()); \
      if (e != cudaSuccess) return static_cast<int>(e);                                                                  \
      cfgd[dev_] = true;                                                                                                 \
    }                                                                                                                    \
    return static_cast<int>(launch_kernel(paged_decode_even_kernel<HD_>, dim3(even_grid(HD_, Hkv)), dim3(128), decode_smem<HD_>(), st, \
                                          (const bf16*)q, ldq, (const bf16*)k_cache, (const bf16*)v_cache, block_table,  \
                                          max_blocks, ctx_len, block_size, num_seqs, Hq, Hkv, (bf16*)out, ldo, part, count, \
                                          scale_log2, num_blocks, status));                                              \
  }
  if (hd == 128) ARTB_PE(128)
  if (hd == 64) ARTB_PE(64)
  if (hd == 32) ARTB_PE(32)
#undef ARTB_PE
  return ERR_BAD_SHAPE;
}

// ---------------------------------------------------------------- allocation-free variant
// Split-KV decode whose workspace is a file-scope device array (see include/artb_noalloc.h for
// the contract).  In host code `g_decode_static_ws` is only a handle for the runtime: the device
// address is obtained once per device with cudaGetSymbolAddress and that pointer is what the
// kernels receive.
#include "artb_noalloc.h"

static __device__ __align__(256) float g_decode_static_ws[ARTB_DECODE_STATIC_WS_FLOATS];

static float* decode_static_ws_ptr(int* err) {
  static float* ptrs[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    *err = e != cudaSuccess ? (int)e : ERR_BAD_SHAPE;
    return nullptr;
  }
  if (!ptrs[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_decode_static_ws);   // address on the current device
    if (e != cudaSuccess) {
      *err = (int)e;
      return nullptr;
    }
    ptrs[dev] = static_cast<float*>(p);
  }
  *err = 0;
  return ptrs[dev];
}

ARTB_EXPORT int artb_paged_decode_noalloc(const void* q, int ldq, const void* k_cache, const void* v_cache,
                                          const int* block_table, int max_blocks, const int* ctx_len, int block_size,
                                          int num_seqs, int Hq, int Hkv, int hd, void* out, int ldo, int splits,
                                          cudaStream_t st) {
  if (num_seqs <= 0) return 0;
  if (splits < 1 || hd <= 0 || Hq <= 0 || Hkv <= 0) return ERR_BAD_SHAPE;
  const long need = (long)num_seqs * Hq * splits * (hd + 2);
  if (need > (long)ARTB_DECODE_STATIC_WS_FLOATS) return ERR_TOO_LARGE;
  int err = 0;
  float* ws = decode_static_ws_ptr(&err);
  if (!ws) return err;
  return artb_paged_decode(q, ldq, k_cache, v_cache, block_table, max_blocks, ctx_len, block_size, num_seqs, Hq, Hkv,
                           hd, out, ldo, ws, splits, /*num_blocks: unknown to this entry point*/ (1L << 40), nullptr, st);
}
