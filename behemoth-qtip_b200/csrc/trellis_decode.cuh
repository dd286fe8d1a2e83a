// Decode of trellis windows from the 32-copy table in shared memory: shared by the register kernel of few tokens and the
// tensor-core kernel of batches.
#pragma once
#include "common.cuh"

namespace qb {

constexpr int kLutBytes = 1024 * 32 * 4;  // 128 KiB, 32 copies

// Dynamic shared memory of these kernels, named at namespace scope so that every access is known to be a
// shared-memory access at a constant base (a pointer carried through a struct is not): words [0, 32768) hold the
// replicated LUT.
extern __shared__ __align__(16) uint32_t gemm_smem_words[];

// Decodes the two windows that one 32-bit word pair holds: o = word c of tiles (i1 = 1 : i1 = 0) of one tile column,
// p = word c + 1 of the same tiles. State t of a window is its 16 bits starting at bit 4 t; bits above 15 of a state
// register never reach the table index, so a state is cut with ONE funnel shift from the two source registers (the first
// state of the low tile is `o` itself), doubled, hashed with one multiply-add (2 v (v + 1), entry in bits 7..16) and
// turned into the byte address of the lane's own copy (entry e, copy l at byte 128 e + 4 l) with one three-input logic
// operation: shift, add, multiply-add, and-or, load per state.
__device__ __forceinline__ uint32_t lut_word(uint32_t v, uint32_t lane4) {
  const uint32_t v2 = v + v;
  uint32_t y2;
  asm("mad.lo.u32 %0, %1, %2, %2;" : "=r"(y2) : "r"(v), "r"(v2));
  const uint32_t at = (y2 & 0x1ff80u) | lane4;
  return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const unsigned char*>(gemm_smem_words) + at);
}
__device__ __forceinline__ void decode_pair(uint32_t o, uint32_t p, uint32_t lane4, uint32_t (&lo)[4],
                                            uint32_t (&hi)[4]) {
  const uint32_t pl = p << 16, oh = o >> 16;
  lo[0] = lut_word(o, lane4);
  hi[0] = lut_word(oh, lane4);
#pragma unroll
  for (int k = 1; k < 4; ++k) {
    lo[k] = lut_word(__funnelshift_l(pl, o, 4 * k), lane4);
    hi[k] = lut_word(__funnelshift_l(p, oh, 4 * k), lane4);
  }
}
// One of the two windows only: `upper` (the same for the whole warp) takes the tile i1 = 1.
__device__ __forceinline__ void decode_half(uint32_t o, uint32_t p, bool upper, uint32_t lane4, uint32_t (&v)[4]) {
  const uint32_t first = upper ? o >> 16 : o, next = upper ? p : p << 16;
  v[0] = lut_word(first, lane4);
#pragma unroll
  for (int k = 1; k < 4; ++k) v[k] = lut_word(__funnelshift_l(next, first, 4 * k), lane4);
}

}  // namespace qb
