// bf16 transpose of some columns of a token matrix, for the operands that attention wants along the tokens.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace artb {

// dst[c, token] = src[token, c0 + c] for c < width: 64 x 64 tiles, 16-byte loads and stores (M % 8 == 0, width % 64 == 0).
// Bound by the bytes.  Vector v of row r lies at v ^ (r / 8): the eight rows of tokens that a warp gathers a column from are
// 1024 bytes apart, and with padded rows they met in one bank.  16 384 tokens: 64 us a
// transpose before (mean of 3584, 3584 and 512 columns), 33 now.
static __global__ void __launch_bounds__(256)
attn_tc_transpose_kernel(const __nv_bfloat16* __restrict__ src, int ld, int c0, __nv_bfloat16* __restrict__ dst, long M) {
  __shared__ __align__(16) __nv_bfloat16 tile[64 * 64];
  const long t0 = static_cast<long>(blockIdx.x) * 64;
  const int cb = blockIdx.y * 64;
  const int tid = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int v = tid + i * 256;          // 512 vectors: 64 tokens x 8
    const int r = v >> 3, cv = v & 7;
    const long t = t0 + r;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (t < M) x = *reinterpret_cast<const uint4*>(src + t * ld + c0 + cb + cv * 8);
    *reinterpret_cast<uint4*>(tile + r * 64 + (cv ^ (r >> 3)) * 8) = x;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int v = tid + i * 256;          // 512 vectors: 64 columns x 8 token groups
    const int c = v >> 3, tv = v & 7;
    __align__(16) __nv_bfloat16 e[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = tile[(tv * 8 + j) * 64 + ((c >> 3) ^ tv) * 8 + (c & 7)];
    const long t = t0 + tv * 8;
    if (t < M) *reinterpret_cast<uint4*>(dst + static_cast<size_t>(cb + c) * M + t) = *reinterpret_cast<const uint4*>(e);
  }
}

}  // namespace artb
