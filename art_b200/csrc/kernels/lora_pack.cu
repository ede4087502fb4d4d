// LoRA bookkeeping of a whole model in one launch per direction.
//
// Masters and gradients are flat fp32 buffers of per-module A [r, K] and B [n, r]; the products read bf16 operands that hold
// the factors of one fused linear side by side, plain and transposed (A_cat [kpad, K], A_catT [K, kpad], B_cat [N, kpad],
// B_catT [kpad, N]), and accumulate fp32 gradients dA [K, kpad], dB [N, kpad].  The arithmetic is one rounding or one product
// per element; what bounds it is launches: 14 to 30 library calls per linear and step, about 1700 for 24 layers, 5.8 ms of
// kernel time and more of the host's (0.5B preset).  So all members of all linears go through one grid: a block finds its
// member and its 64 rows (of B) or columns (of A) in a table that is written once per model.  The 168 members of those 24
// layers take 45 us for the copies and 27 us for the gradients.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "host_utils.h"

namespace artb {

struct LoraItem {
  const float* a;          // [r, K] master
  const float* b;          // [n, r] master
  float* ga;               // gradients, laid out as the masters
  float* gb;
  __nv_bfloat16* A_cat;
  __nv_bfloat16* A_catT;
  __nv_bfloat16* B_cat;
  __nv_bfloat16* B_catT;
  const float* dA;
  const float* dB;
  const long long* rows;   // row of the fused weight that output n of this module is
  int K, n, N, kpad, c0;   // c0: first of the r columns that are this module's
  int pad_;
};

constexpr int LP_TILE = 64;
constexpr int LP_THREADS = 256;   // 64 rows or columns x 4 groups of 8 ranks

// Thread (x, g) takes row / column x of the tile and ranks g * 8 .. g * 8 + 7, then 32 further on: lanes run along x, so the
// accesses of [r, K] and of the transposed operands are contiguous, those of [K, kpad] are runs of 8 ranks.
template <bool EXPORT>
__global__ void __launch_bounds__(LP_THREADS) lora_pack_kernel(const LoraItem* __restrict__ items, const int2* __restrict__ blocks,
                                                               int r, float scale) {
  const int2 where = blocks[blockIdx.x];
  const LoraItem it = items[where.x];
  const int tiles_a = (it.K + LP_TILE - 1) / LP_TILE;
  const int x = threadIdx.x & (LP_TILE - 1), g = threadIdx.x / LP_TILE;
  if (where.y < tiles_a) {
    const int k = where.y * LP_TILE + x;
    if (k >= it.K) return;
    for (int i0 = g * 8; i0 < r; i0 += 32)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = i0 + j;
        if (i >= r) break;
        const size_t flat = static_cast<size_t>(i) * it.K + k, wide = static_cast<size_t>(k) * it.kpad + it.c0 + i;
        if (EXPORT) {
          it.ga[flat] = it.dA[wide];
        } else {
          const __nv_bfloat16 v = __float2bfloat16(it.a[flat]);
          it.A_cat[static_cast<size_t>(it.c0 + i) * it.K + k] = v;
          it.A_catT[wide] = v;
        }
      }
    return;
  }
  const int o = (where.y - tiles_a) * LP_TILE + x;
  if (o >= it.n) return;
  const size_t row = static_cast<size_t>(it.rows[o]);
  for (int i0 = g * 8; i0 < r; i0 += 32)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j;
      if (i >= r) break;
      const size_t flat = static_cast<size_t>(o) * r + i, wide = row * it.kpad + it.c0 + i;
      if (EXPORT) {
        it.gb[flat] = it.dB[wide] * scale;
      } else {
        const __nv_bfloat16 v = __float2bfloat16(it.b[flat] * scale);
        it.B_cat[wide] = v;
        it.B_catT[static_cast<size_t>(it.c0 + i) * it.N + row] = v;
      }
    }
}

}  // namespace artb

using namespace artb;

ARTB_EXPORT int artb_lora_item_bytes() { return static_cast<int>(sizeof(LoraItem)); }

// export_grads = 0: masters -> bf16 operands; 1: accumulated gradients -> flat gradients.  `blocks` [n_blocks] pairs
// (item, tile): tiles of 64 columns of A first, then tiles of 64 rows of B.
ARTB_EXPORT int artb_lora_pack(const void* items, const void* blocks, int n_blocks, int r, float scale, int export_grads,
                               cudaStream_t stream) {
  if (n_blocks <= 0) return 0;
  if (r <= 0) return ERR_BAD_SHAPE;
  auto i = reinterpret_cast<const LoraItem*>(items);
  auto b = reinterpret_cast<const int2*>(blocks);
  if (export_grads)
    lora_pack_kernel<true><<<n_blocks, LP_THREADS, 0, stream>>>(i, b, r, scale);
  else
    lora_pack_kernel<false><<<n_blocks, LP_THREADS, 0, stream>>>(i, b, r, scale);
  return static_cast<int>(cudaGetLastError());
}
