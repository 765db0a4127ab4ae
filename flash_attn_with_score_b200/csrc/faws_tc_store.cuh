// Plain-store counterparts of the score kernels' TMA stores, for score tensors whose rows do not start on 16-byte
// boundaries (odd lengths): TMA cannot address those.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace faws {

// Whether TMA can write a (.., rows, cols) score tensor of `esize`-byte elements at `base`.
inline bool tma_score_rows(const void* base, int cols, int esize) {
  return (int64_t)cols * esize % 16 == 0 && reinterpret_cast<uintptr_t>(base) % 16 == 0;
}

// A box of 32 rows x 128 bytes that the warp has staged in the layout of the 128-byte swizzle goes to global memory one
// row per instruction, lane l writing the l-th 4-byte word: 128 contiguous bytes, whatever the row's alignment.
// `rows` / `cols`: what the tensor's edges leave of the box (cols <= 0: nothing).  ESIZE 2: a word is a pair of columns,
// stored as one where `pairs` says that the tensor's rows keep pairs on 4-byte boundaries.
template <int ESIZE>
__device__ __forceinline__ void store_box_direct(const unsigned char* box, char* dst, int64_t row_bytes, int rows, int cols,
                                                 int lane, bool pairs) {
  const int col = lane * (4 / ESIZE);
  if (col >= cols) return;
  dst += lane * 4;
  const int chunk = lane >> 2, off = (lane & 3) << 2;
#pragma unroll 1
  for (int r0 = 0; r0 < rows; r0 += 8) {
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e] = *reinterpret_cast<const uint32_t*>(box + (r0 + e) * 128 + ((chunk ^ e) << 4) + off);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (r0 + e < rows) {
        if (ESIZE == 4 || pairs) *reinterpret_cast<uint32_t*>(dst) = w[e];
        else {
          *reinterpret_cast<uint16_t*>(dst) = (uint16_t)w[e];
          if (col + 1 < cols) *reinterpret_cast<uint16_t*>(dst + 2) = (uint16_t)(w[e] >> 16);
        }
      }
      dst += row_bytes;
    }
  }
}

// `n` elements of ESIZE bytes from `dst` on are set to the repeated pattern `word` by one warp: elements up to the first
// 16-byte boundary, 16 bytes a lane, the rest.
template <int ESIZE>
__device__ __forceinline__ void fill_row_direct(char* dst, int n, uint32_t word, int lane) {
  using E = typename std::conditional<ESIZE == 4, uint32_t, uint16_t>::type;
  const int lead = min(n, (int)((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15) / ESIZE);
  E* d = reinterpret_cast<E*>(dst);
  if (lane < lead) d[lane] = (E)word;
  const int vec = (n - lead) / (16 / ESIZE);
  uint4* v = reinterpret_cast<uint4*>(d + lead);
  const uint4 w4 = make_uint4(word, word, word, word);
  for (int x = lane; x < vec; x += 32) v[x] = w4;
  const int done = lead + vec * (16 / ESIZE);
  if (done + lane < n) d[done + lane] = (E)word;
}

}  // namespace faws
