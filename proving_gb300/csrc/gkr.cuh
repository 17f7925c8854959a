// What the GKR kernels share: secure columns, QM31 helpers and the eq column (gkr.cu, gkr_prove.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "common.cuh"
#include "field.cuh"

namespace cs {

// One instance of cs_gkr_prove_batch: its input layer's columns (num[1..3] null for multiplicities,
// num null for a product or LogUp singles).
struct GkrInput {
  uint32_t kind = 0, n_vars = 0;
  const uint32_t* num[4] = {nullptr, nullptr, nullptr, nullptr};
  const uint32_t* den[4] = {nullptr, nullptr, nullptr, nullptr};
};
cs_status gkr_prove_on_device(const std::vector<GkrInput>& inputs, uint32_t chan[9], std::vector<uint64_t>& out,
                              cudaStream_t st);

namespace {

struct QIn {
  const uint32_t* c[4];
};
struct QOut {
  uint32_t* c[4];
};

__device__ __forceinline__ qm31 q_one() { return qm31_make(1, 0, 0, 0); }
__device__ __forceinline__ qm31 q_zero() { return qm31_make(0, 0, 0, 0); }
__device__ __forceinline__ qm31 q_double(qm31 x) { return qm31_add(x, x); }

__device__ __forceinline__ qm31 q_load(const QIn& s, uint32_t i) {
  return qm31_make(s.c[0][i], s.c[1][i], s.c[2][i], s.c[3][i]);
}
__device__ __forceinline__ void q_store(const QOut& d, uint32_t i, qm31 v) {
  d.c[0][i] = v.a.a;
  d.c[1][i] = v.a.b;
  d.c[2][i] = v.b.a;
  d.c[3][i] = v.b.b;
}
// values 2i and 2i + 1 of a secure column (8-byte loads: 2i is even)
__device__ __forceinline__ void q_load_pair(const QIn& s, uint32_t i, qm31& a, qm31& b) {
  uint2 w[4];
#pragma unroll
  for (int k = 0; k < 4; k++) w[k] = reinterpret_cast<const uint2*>(s.c[k])[i];
  a = qm31_make(w[0].x, w[1].x, w[2].x, w[3].x);
  b = qm31_make(w[0].y, w[1].y, w[2].y, w[3].y);
}

__device__ __forceinline__ qm31 q_shfl_add(qm31 v, int off) {
  return qm31_make(m31_add(v.a.a, __shfl_xor_sync(0xffffffffu, v.a.a, off)),
                   m31_add(v.a.b, __shfl_xor_sync(0xffffffffu, v.a.b, off)),
                   m31_add(v.b.a, __shfl_xor_sync(0xffffffffu, v.b.a, off)),
                   m31_add(v.b.b, __shfl_xor_sync(0xffffffffu, v.b.b, off)));
}

constexpr uint32_t kEqLowBits = 10;    // index bits of the per-block table
constexpr uint32_t kEqChunkBits = 14;  // values written per block
constexpr uint32_t kEqMaxVars = 28;

// evals[i] = v * prod_j eq(x_j, y_j), x_j = bit n-1-j of i (gen_eq_evals,
// cpu/lookups/gkr.rs:230-246: the loop over y in reverse doubles the table, so
// y[n-1] is index bit 0). Each block builds the factor of the low kEqLowBits
// bits as a table in shared memory by the same doubling, the factor of its own
// high bits directly, and writes their products.
__device__ __forceinline__ void eq_evals_block(uint32_t block, const qm31 v, const qm31* y, uint32_t n, const QOut& out) {
  __shared__ qm31 low[1u << kEqLowBits];
  __shared__ qm31 high[1u << (kEqChunkBits - kEqLowBits)];
  const uint32_t k = min(n, kEqLowBits);
  const uint32_t chunk = min(n, kEqChunkBits);
  if (threadIdx.x == 0) low[0] = q_one();
  __syncthreads();
  for (uint32_t t = 0; t < k; t++) {
    const qm31 yt = y[n - 1 - t];
    for (uint32_t j = threadIdx.x; j < (1u << t); j += blockDim.x) {
      const qm31 lj = low[j];
      const qm31 tmp = qm31_mul(lj, yt);
      low[j + (1u << t)] = tmp;
      low[j] = qm31_sub(lj, tmp);
    }
    __syncthreads();
  }
  const uint32_t first = block << chunk;
  if (threadIdx.x < (1u << (chunk - k))) {
    const uint32_t hi = (first >> k) + threadIdx.x;
    qm31 h = v;
    for (uint32_t t = k; t < n; t++) {
      const qm31 yt = y[n - 1 - t];
      h = qm31_mul(h, ((hi >> (t - k)) & 1u) ? yt : qm31_sub(q_one(), yt));
    }
    high[threadIdx.x] = h;
  }
  __syncthreads();
  const uint32_t low_mask = (1u << k) - 1;
  for (uint32_t e = threadIdx.x; e < (1u << chunk); e += blockDim.x)
    q_store(out, first + e, qm31_mul(high[e >> k], low[e & low_mask]));
}

}  // namespace
}  // namespace cs
