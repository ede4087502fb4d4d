// LoRA factor gradients: OUT[C, R] += P[M, C]^T * Q[M, R]   (bf16 in, fp32 accumulate)
//
// Both LoRA weight gradients are contractions over the token dimension between one wide
// activation matrix and one skinny one:
//     dB_cat[N, R]   += dY[M, N]^T * T[M, R]          (T = X A^T, saved by the forward)
//     dA_cat^T[K, R] += X[M, K]^T  * dT[M, R]         (dT = dY (sB))
// R is the padded LoRA width (64), of which the caller says how many columns are used (rank times modules: 8 to 24
// mostly): only those are multiplied and added, in steps of 16.  The op reads the wide matrix exactly once and does
// R/8 times fewer FLOPs than a square GEMM, so it is bandwidth-bound; warp-level
// mma.sync (m16n8k16) with ldmatrix.trans from padded shared tiles is enough to keep up
// with HBM.  Token-dimension splits accumulate with fp32 atomics, two columns each: with all 64 columns added one by
// one they took longer than the loads of short batches (mean of a layer's eight: 18.6 -> 12 us for 2048 rows of the 7B
// shape, 109 -> 68 for 16 384, of which the bytes take 8 and 50).
//
// Counterpart in the reference: autograd through the PEFT/Unsloth LoRA modules
// (src/art/local/state.py:86-92, backward driven from src/art/local/train.py via HF Trainer).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "host_utils.h"

namespace artb {

constexpr int WG_BC = 128;   // columns of P per CTA
constexpr int WG_R = 64;     // columns of Q
constexpr int WG_BM = 32;    // token rows per pipeline chunk
constexpr int WG_PLD = WG_BC + 8;
constexpr int WG_STAGES = 3;
constexpr int WG_CTAS = 5;   // per SM (40 KB of shared memory at most): 80 KB of loads in flight

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct WgArgs {
  const __nv_bfloat16 *P, *Q;
  float* out;
  int ldp, ldq, ldo, C, cblocks, rows_per_split;
};

// NB: 16-column blocks of Q that are used.  Two contractions over the same M rows share a launch: CTAs from a.cblocks on
// belong to b.
template <int NB>
__global__ void __launch_bounds__(128)
lora_wgrad_kernel(const WgArgs a, const WgArgs b, int M, const int* __restrict__ seg_off, long out_stride) {
  constexpr int QLD = NB * 16 + 8;
  __shared__ __align__(16) __nv_bfloat16 sP[WG_STAGES][WG_BM][WG_PLD];
  __shared__ __align__(16) __nv_bfloat16 sQ[WG_STAGES][WG_BM][QLD];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool second = static_cast<int>(blockIdx.x) >= a.cblocks;
  const __nv_bfloat16* __restrict__ P = second ? b.P : a.P;
  const __nv_bfloat16* __restrict__ Q = second ? b.Q : a.Q;
  float* __restrict__ out = second ? b.out : a.out;
  const int ldp = second ? b.ldp : a.ldp, ldq = second ? b.ldq : a.ldq, ldo = second ? b.ldo : a.ldo, C = second ? b.C : a.C;
  const int rows_per_split = second ? b.rows_per_split : a.rows_per_split;
  const int c0 = (blockIdx.x - (second ? a.cblocks : 0)) * WG_BC;
  int m_begin = blockIdx.y * rows_per_split;
  int m_end = min(M, m_begin + rows_per_split);
  if (seg_off) {
    // grouped: blockIdx.z is the expert; its row segment is split evenly over gridDim.y CTAs
    // (clipped to the M rows the operands really have, whatever the offsets say)
    const int lo = min(seg_off[blockIdx.z], M), hi = min(seg_off[blockIdx.z + 1], M);
    const int rows = ((hi - lo + static_cast<int>(gridDim.y) - 1) / static_cast<int>(gridDim.y) + WG_BM - 1) / WG_BM * WG_BM;
    m_begin = lo + blockIdx.y * rows;
    m_end = min(hi, m_begin + rows);
    out += blockIdx.z * out_stride;
  }
  if (m_begin >= m_end) return;
  const int chunks = (m_end - m_begin + WG_BM - 1) / WG_BM;

  auto load_chunk = [&](int chunk, int stage) {
    const int m0 = m_begin + chunk * WG_BM;
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // P: 32 rows x 16 vec
      const int v = tid + i * 128;
      const int r = v >> 4, cv = v & 15;
      const int gm = m0 + r, gc = c0 + cv * 8;
      const bool ok = gm < m_end && gc < C;
      cp_async16(&sP[stage][r][cv * 8], P + (ok ? static_cast<size_t>(gm) * ldp + gc : 0), ok);
    }
    for (int v = tid; v < WG_BM * NB * 2; v += 128) {  // Q: 32 rows x 2 NB vec
      const int r = v / (NB * 2), cv = v % (NB * 2);
      const int gm = m0 + r;
      const bool ok = gm < m_end;
      cp_async16(&sQ[stage][r][cv * 8], Q + (ok ? static_cast<size_t>(gm) * ldq + cv * 8 : 0), ok);
    }
    cp_async_commit();
  };

  float acc[2][2 * NB][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2 * NB; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;

  load_chunk(0, 0);
  if (chunks > 1)
    load_chunk(1, 1);
  else
    cp_async_commit();
  int st = 0;
  for (int ch = 0; ch < chunks; ++ch) {
    cp_async_wait<1>();
    __syncthreads();             // the chunk has arrived, and everyone is done with the stage that is filled next
    if (ch + 2 < chunks)
      load_chunk(ch + 2, st == 0 ? 2 : st - 1);
    else
      cp_async_commit();
    const int j = lane >> 3, rr = lane & 7;  // ldmatrix: lane supplies row rr of matrix j
#pragma unroll
    for (int ks = 0; ks < WG_BM / 16; ++ks) {
      const int k0 = ks * 16;
      uint32_t a[2][4];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        // A = P^T tile: rows = columns c of P, k = token.  smem is [k][c] -> transposed load.
        const int cbase = warp * 32 + mi * 16;
        const int krow = k0 + (j >> 1) * 8 + rr;
        const int ccol = cbase + (j & 1) * 8;
        ldmatrix_x4_trans(a[mi], &sP[st][krow][ccol]);
      }
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        // B = Q tile [k][n] -> transposed load gives the col-major fragments of two n8 blocks.
        uint32_t b[4];
        const int krow = k0 + (j & 1) * 8 + rr;
        const int ncol = nb * 16 + (j >> 1) * 8;
        ldmatrix_x4_trans(b, &sQ[st][krow][ncol]);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          mma_bf16(acc[mi][nb * 2], a[mi], b[0], b[1]);
          mma_bf16(acc[mi][nb * 2 + 1], a[mi], b[2], b[3]);
        }
      }
    }
    st = st == WG_STAGES - 1 ? 0 : st + 1;
  }
  const bool pairs = !(ldo & 1) && !(reinterpret_cast<uintptr_t>(out) & 7);
  auto add2 = [&](float* p, float a, float b) {
    if (pairs) {
      atomicAdd(reinterpret_cast<float2*>(p), make_float2(a, b));
    } else {
      atomicAdd(p, a);
      atomicAdd(p + 1, b);
    }
  };
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int mi = 0; mi < 2; ++mi) {
#pragma unroll
    for (int nj = 0; nj < 2 * NB; ++nj) {
      const int col = nj * 8 + 2 * t;
      const int r0 = c0 + warp * 32 + mi * 16 + g;
      if (r0 < C) add2(out + static_cast<size_t>(r0) * ldo + col, acc[mi][nj][0], acc[mi][nj][1]);
      if (r0 + 8 < C) add2(out + static_cast<size_t>(r0 + 8) * ldo + col, acc[mi][nj][2], acc[mi][nj][3]);
    }
  }
}

static WgArgs wg_args(const void* P, int ldp, const void* Q, int ldq, float* out, int ldo, int C) {
  return WgArgs{reinterpret_cast<const __nv_bfloat16*>(P), reinterpret_cast<const __nv_bfloat16*>(Q), out, ldp, ldq, ldo, C,
                (C + WG_BC - 1) / WG_BC, 0};
}

// rows of a split, so that `ctas` CTAs share a contraction over M rows; a split of 64 rows still has two chunks
static int wg_split(WgArgs& a, int M, int ctas) {
  int splits = (ctas + a.cblocks - 1) / a.cblocks;
  const int max_splits = (M + 2 * WG_BM - 1) / (2 * WG_BM);
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  const int rows = (M + splits - 1) / splits;
  a.rows_per_split = (rows + WG_BM - 1) / WG_BM * WG_BM;
  return (M + a.rows_per_split - 1) / a.rows_per_split;
}

static int launch_wgrad(dim3 grid, const WgArgs& a, const WgArgs& b, int M, int cols, const int* seg_off, long out_stride,
                        cudaStream_t st) {
  auto go = [&](auto kern) {
    kern<<<grid, 128, 0, st>>>(a, b, M, seg_off, out_stride);
    return static_cast<int>(cudaGetLastError());
  };
  if (cols <= 16) return go(lora_wgrad_kernel<1>);
  if (cols <= 32) return go(lora_wgrad_kernel<2>);
  return go(lora_wgrad_kernel<4>);
}

}  // namespace artb

using namespace artb;

// out[C, 64] (fp32, ld = ldo) += P[M, C]^T Q[M, 64].  C % 8 == 0; P, Q 16-byte aligned rows.  Columns of Q from `cols` on are
// zero or not wanted: what is added to their sums is unspecified.
ARTB_EXPORT int artb_lora_wgrad(const void* P, int ldp, const void* Q, int ldq, float* out, int ldo, int M, int C, int cols,
                                cudaStream_t st) {
  if (M <= 0 || C <= 0) return 0;
  if ((C & 7) || (ldp & 7) || (ldq & 7) || ldo < WG_R || cols <= 0 || cols > WG_R) return ERR_BAD_SHAPE;
  WgArgs a = wg_args(P, ldp, Q, ldq, out, ldo, C);
  const int splits = wg_split(a, M, WG_CTAS * sm_count());
  return launch_wgrad(dim3(a.cblocks, splits), a, a, M, cols, nullptr, 0, st);
}

// Both factor gradients of a projection in one launch: out1[C1, 64] += P1^T Q1 and out2[C2, 64] += P2^T Q2 over M rows.
ARTB_EXPORT int artb_lora_wgrad_pair(const void* P1, int ldp1, const void* Q1, int ldq1, float* out1, int ldo1, int C1,
                                     const void* P2, int ldp2, const void* Q2, int ldq2, float* out2, int ldo2, int C2, int M,
                                     int cols, cudaStream_t st) {
  if (M <= 0) return 0;
  if (C1 <= 0 || C2 <= 0 || (C1 & 7) || (C2 & 7) || (ldp1 & 7) || (ldq1 & 7) || (ldp2 & 7) || (ldq2 & 7) || ldo1 < WG_R ||
      ldo2 < WG_R || cols <= 0 || cols > WG_R)
    return ERR_BAD_SHAPE;
  WgArgs a = wg_args(P1, ldp1, Q1, ldq1, out1, ldo1, C1), b = wg_args(P2, ldp2, Q2, ldq2, out2, ldo2, C2);
  // splits of about the same number of rows on both sides
  const int all = a.cblocks + b.cblocks, ctas = WG_CTAS * sm_count();
  const int sa = wg_split(a, M, static_cast<int>(static_cast<long>(ctas) * a.cblocks / all));
  const int sb = wg_split(b, M, static_cast<int>(static_cast<long>(ctas) * b.cblocks / all));
  return launch_wgrad(dim3(all, sa > sb ? sa : sb), a, b, M, cols, nullptr, 0, st);
}

// Grouped form for expert-sorted rows: out[e][C, 64] += P[seg_e, C]^T Q[seg_e, 64] for every expert e,
// seg_e = rows seg_off[e] .. seg_off[e+1] (device array, padded rows are zero).  One launch covers all experts.
ARTB_EXPORT int artb_lora_wgrad_grouped(const void* P, int ldp, const void* Q, int ldq, float* out, int ldo,
                                        long out_stride, const int* seg_off, int num_experts, int C, int splits,
                                        int rows, int cols, cudaStream_t st) {
  if (num_experts <= 0 || C <= 0 || rows <= 0) return 0;
  if ((C & 7) || (ldp & 7) || (ldq & 7) || ldo < WG_R || splits < 1 || cols <= 0 || cols > WG_R) return ERR_BAD_SHAPE;
  const WgArgs a = wg_args(P, ldp, Q, ldq, out, ldo, C);
  return launch_wgrad(dim3(a.cblocks, splits, num_experts), a, a, rows, cols, seg_off, out_stride, st);
}
