// Shared-memory layout of fft_strided_kernel (fft.cu), in words: the tile, then each warp's twiddle
// tables. Constant expressions without CUDA types, so that a host compiler can check them.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CS_LAYOUT __host__ __device__ __forceinline__ constexpr
#else
#define CS_LAYOUT constexpr
#endif

namespace cs {

// A strided tile holds [m][e] with 8 (EB = 3) or 16 pad words per stage row (2^TA values of m), so
// that the rows of a warp fall on distinct banks.
template <int TA, int EB>
CS_LAYOUT uint32_t strided_pad(uint32_t L) {
  return L + ((L >> (TA + EB)) << EB);
}
template <int T, int EB>
CS_LAYOUT uint32_t strided_tile_words() {
  return (1u << (EB + T)) + (1u << (EB + T - T / 2));
}
template <int T, int EB>
CS_LAYOUT uint32_t strided_warps() {
  return ((1u << EB) << (T / 2)) / 32;
}
// A warp reads its tables behind a warp barrier only, so the tables it reads are those it wrote: the
// high stage's (one group of 2^TB words, the same in every warp of the block) and those of its own low
// stage rows (32 >> EB of them, twice as many where TB > TA).
template <int T, int EB>
CS_LAYOUT uint32_t strided_high_table(uint32_t warp) {
  return strided_tile_words<T, EB>() + warp * (1u << (T - T / 2));
}
template <int T, int EB>
CS_LAYOUT uint32_t strided_low_table(uint32_t warp) {
  return strided_high_table<T, EB>(strided_warps<T, EB>()) + warp * ((32u >> EB) << (T - T / 2));
}
template <int T, int EB>
CS_LAYOUT uint32_t strided_smem_words() {
  return strided_low_table<T, EB>(strided_warps<T, EB>());
}

}  // namespace cs

#undef CS_LAYOUT
