// The GKR batch prover on the device: prove_batch (crates/stwo/src/prover/lookups/gkr_prover.rs)
// and its sum-check (crates/stwo/src/prover/lookups/sumcheck.rs) with the Fiat-Shamir channel, the
// round polynomials and the claims in device memory, so that the host enqueues the whole protocol
// and reads the proof back once.
//
// Before, the host ran the protocol over the kernels of gkr.cu: about five launches, their
// allocations and a synchronising read-back per sum-check round, 60 us a round whatever its size
// (14.4 ms for the 231 rounds of 2^22 fractions beside 2^20 products; now 3.7). A round's own chain is
// short: fix, sums, one product per coefficient, three dependent Blake2s compressions. Here a round of many
// terms is one launch: it fixes the previous variable, writes the halved columns, sums the next
// round's terms from the same registers, and the last block to finish turns the sums into the round
// polynomial, mixes it and draws the next challenge. The last kTailRounds rounds of a layer, the
// layer's masks and the next layer's claims and constants (and whole layers while they are that
// small) are one single-block launch. The launches of one proof are a chain of programmatic dependent
// launches.
//
// Bound: latency (7.3 us a round in the single-block kernel, 13 in a launch of its own: 4.6 for the
// terms, 1.5 for the blocks' sums, 4.7 to end the round, 0.7 to the next launch). A QM31 product is
// 155-220 cycles for a lone warp and a compression about 1,900, so the block spreads a round's products over
// its threads in as few levels as they need: one product per element to fix, two per part of a term, one per
// (coefficient, sum), and what only the next round needs (claims, corrections, coefficient tables) runs in
// other warps beside the next fix.
#include <algorithm>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <vector>

#include "blake2s.cuh"
#include "channel.cuh"
#include "common.cuh"
#include "field.cuh"
#include "gkr.cuh"

namespace cs {
namespace {

// Rounds of up to 2^(kTailRounds - 1) terms run in the single-block kernel: 64 terms are 1,024 items of
// two products for its 512 threads, about 8 us a round; at 128 and 256 terms a round there takes 15 and
// 25 us and a launch over several blocks 13 (2^22 + 2^20 with a limit of 6, 7, 8 rounds: 3.78, 3.75,
// 3.75 ms; 9 before the launches overlapped: 4.30).
constexpr uint32_t kTailRounds = 7;
constexpr uint32_t kTailThreads = 512;
constexpr uint32_t kTailTerms = 1u << (kTailRounds - 1);
constexpr uint32_t kRoundThreads = 128;
constexpr uint32_t kMaxVars = 32;
constexpr uint32_t kSharedInst = 64;  // instances whose state is kept in shared memory
constexpr uint32_t kSharedCols = 4;   // instances whose tail columns are kept in shared memory

// An instance's layer during its sum-check. Round 0 reads num / den; the first fix reads them and
// writes fnum / fden, later ones work in fnum / fden in place (an element's or term's thread reads
// and writes its own values only).
struct LayerCols {
  const uint32_t *num[4], *den[4];
  uint32_t *fnum[4], *fden[4];
  uint32_t kind;
  uint32_t n_vars;  // variables of the layer; 0 before the instance joins
};

// The round polynomial is linear in the sums f0, f2 at t = 0, 2 and the claim:
// coefficient t = corr f0 u[t] + corr f2 v[t] + claim w[t] with the row of the k variables left
// (correct_sum_as_poly_in_first_variable; RoundConstants of proving_gb300/gkr.py).
struct GkrState {
  uint32_t chan[9];
  uint32_t err;  // a round constant divides by zero
  uint32_t pad[6];
  qm31 lam, alpha, x;
  qm31 y[kMaxVars], sc[kMaxVars];  // the point of the layer's claims, this sum-check's challenges
  struct {
    qm31 u[4], v[4], w[4];
  } row[kMaxVars];  // k variables left
};

struct InstState {
  qm31 claim, corr;
  qm31 apow;                        // alpha^(instances that joined before)
  qm31 poly[4], pa[4];              // the round polynomial, and times apow
  qm31 cu[4], lcu[4], cv[4], lcv[4];  // corr u, lambda corr u (a product: corr u), the same for v
  qm31 out[2];                      // the layer claims, from masks or the output layer
  uint32_t n_out, poly_size;
  uint32_t delta;  // layers before the instance joins
  uint32_t product;
};

struct GkrProgram {
  GkrState* state;
  InstState* inst;
  unsigned long long* acc;      // [instance][A0, C0, A2, C2][coordinate], zero between rounds
  const LayerCols* cols;        // [layer][instance], valid from the layer at which an instance joins
  const uint32_t* const* out0;  // [instance][8]: the output layer's num / den (num null: a product)
  uint32_t n_inst, n_layers;
  uint32_t* partial;
  uint32_t* counter;
  uint32_t* polys;    // [l (l - 1) / 2 + round][17]: size, coefficients
  uint32_t* masks;    // [layer][instance][16]
  uint32_t* outputs;  // [instance][8]
  const uint32_t* eq;  // the layer's eq column: 4 coordinates of 2^(l - 1)
};

__device__ __forceinline__ qm31 q_make4(const uint32_t* w) { return qm31_make(w[0], w[1], w[2], w[3]); }
__device__ __forceinline__ void q_put(uint32_t* w, qm31 v) { w[0] = v.a.a, w[1] = v.a.b, w[2] = v.b.a, w[3] = v.b.b; }
__device__ __forceinline__ bool q_is_zero(qm31 v) { return (v.a.a | v.a.b | v.b.a | v.b.b) == 0; }

// ------------------------------------------------------------ channel (one warp)

// SIGMA (RFC 7693 section 2.7) by round and lane: the two words of lane q's column step, then those of
// its diagonal step.
__device__ const uint8_t kSigma[160] = {
    0, 1, 8, 9, 2, 3, 10, 11, 4, 5, 12, 13, 6, 7, 14, 15, 14, 10, 1, 12, 4, 8, 0, 2, 9, 15, 11, 7, 13, 6, 5, 3,
    11, 8, 10, 14, 12, 0, 3, 6, 5, 2, 7, 1, 15, 13, 9, 4, 7, 9, 2, 6, 3, 1, 5, 10, 13, 12, 4, 0, 11, 14, 15, 8,
    9, 0, 14, 1, 5, 7, 11, 12, 2, 4, 6, 8, 10, 15, 3, 13, 2, 12, 4, 13, 6, 10, 7, 5, 0, 11, 15, 14, 8, 3, 1, 9,
    12, 5, 0, 7, 1, 15, 6, 3, 14, 13, 9, 2, 4, 10, 8, 11, 13, 11, 5, 0, 7, 14, 15, 4, 12, 1, 8, 6, 3, 9, 2, 10,
    6, 15, 12, 2, 14, 9, 13, 7, 11, 3, 1, 4, 0, 8, 10, 5, 10, 2, 15, 11, 8, 4, 9, 14, 7, 6, 3, 12, 1, 5, 13, 0};

struct Hash {
  __align__(16) uint32_t sched[160];  // the message in kSigma's order
  uint32_t msg[16], out[8];
  uint32_t sigma[160];
};

// Compresses the block in H.msg into the chaining value in H.out, by one warp: every four lanes alike,
// lane q the state's column q (h0 = v[q], h1 = v[4 + q]), the diagonals by rotating the rows among the
// four. 56 instructions a half round, 40 of them on the ALU pipe, hold a lone lane's compression at
// 1,672 cycles (2,430 as a loop that reads the message from shared memory, 2,630 unrolled where other
// code ran in between and its 18 KB are fetched anew); a lane's 14 leave the latency of the step and
// of three shuffles, and the loop's few instructions stay in the cache. init: start from the
// parameter block.
__device__ __forceinline__ void warp_compress(Hash& H, bool init, uint32_t t, bool last) {
  const uint32_t lane = threadIdx.x & 31, q = lane & 3;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 5; j++) H.sched[lane + 32 * j] = H.msg[H.sigma[lane + 32 * j]];
  const uint32_t iv0 = q < 2 ? (q == 0 ? b2s_iv(0) : b2s_iv(1)) : (q == 2 ? b2s_iv(2) : b2s_iv(3));
  const uint32_t iv1 = q < 2 ? (q == 0 ? b2s_iv(4) : b2s_iv(5)) : (q == 2 ? b2s_iv(6) : b2s_iv(7));
  const uint32_t h0 = init ? iv0 ^ (q == 0 ? 0x01010020u : 0u) : H.out[q], h1 = init ? iv1 : H.out[4 + q];
  uint32_t a = h0, b = h1, c = iv0, d = iv1 ^ (q == 0 ? t : q == 2 && last ? 0xffffffffu : 0u);
  __syncwarp();
  const uint4* sched = reinterpret_cast<const uint4*>(H.sched) + q;
  const int up = (int)((lane & 28) | ((q + 1) & 3)), across = (int)(lane ^ 2), down = (int)((lane & 28) | ((q + 3) & 3));
  uint4 m = sched[0];
#pragma unroll 2
  for (int r = 1; r <= 10; r++) {
    const uint4 n = sched[r < 10 ? 4 * r : 0];
    CS_B2S_G_CHAIN(a, b, c, d, m.x, m.y)
    b = __shfl_sync(0xffffffffu, b, up);
    c = __shfl_sync(0xffffffffu, c, across);
    d = __shfl_sync(0xffffffffu, d, down);
    CS_B2S_G_CHAIN(a, b, c, d, m.z, m.w)
    b = __shfl_sync(0xffffffffu, b, down);
    c = __shfl_sync(0xffffffffu, c, across);
    d = __shfl_sync(0xffffffffu, d, up);
    m = n;
  }
  if (lane < 4) {
    H.out[q] = h0 ^ a ^ c;
    H.out[4 + q] = h1 ^ b ^ d;
  }
  __syncwarp();
}

// digest <- Blake2s(digest || n felts), n <= 4; the draw counter restarts (Blake2sChannel::mix_felts).
__device__ __noinline__ void warp_mix(GkrState& S, Hash& H, const qm31* felts, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31, words = 4 * n, len = 32 + 16 * n;
  const uint32_t* f = reinterpret_cast<const uint32_t*>(felts);
  if (lane < 16) H.msg[lane] = lane < 8 ? S.chan[lane] : lane - 8 < words ? f[lane - 8] : 0;
  const bool two = len > 64;
#pragma unroll 1
  for (int block = 0; block < (two ? 2 : 1); block++) {
    if (block == 1 && lane < 16) H.msg[lane] = lane < 8 && 8 + lane < words ? f[8 + lane] : 0;
    const bool last = block == (two ? 1 : 0);
    warp_compress(H, block == 0, last ? len : 64, last);
  }
  if (lane < 9) S.chan[lane] = lane < 8 ? H.out[lane] : 0;
  __syncwarp();
}

__device__ __noinline__ qm31 warp_draw(GkrState& S, Hash& H) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t h[8], state[9], felt[4];
  if (lane < 16) H.msg[lane] = lane < 9 ? S.chan[lane] : 0;
  warp_compress(H, true, kChannelDrawBytes, true);
#pragma unroll
  for (int i = 0; i < 8; i++) h[i] = H.out[i];
  state[8] = 0;
  channel_after_draw(state, h, felt);
  __syncwarp();
  if (lane == 0) S.chan[8] += 1;
  __syncwarp();
  return q_make4(felt);
}

__device__ void hash_setup(Hash& H) {
  for (uint32_t e = threadIdx.x; e < 160; e += blockDim.x) H.sigma[e] = kSigma[e];
}

// One copy of the product's code for the latency-bound parts (their inlined products together would
// not stay in the instruction cache).
__device__ __noinline__ qm31 mul(qm31 a, qm31 b) { return qm31_mul(a, b); }
__device__ __forceinline__ qm31 q_shfl(qm31 v, int lane) {
  return qm31_make(__shfl_sync(0xffffffffu, v.a.a, lane), __shfl_sync(0xffffffffu, v.a.b, lane),
                   __shfl_sync(0xffffffffu, v.b.a, lane), __shfl_sync(0xffffffffu, v.b.b, lane));
}
__device__ __forceinline__ qm31 q_lerp(qm31 l, qm31 h, qm31 x) { return qm31_add(mul(x, qm31_sub(h, l)), l); }

// ------------------------------------------------------------ a round's end, a layer's ends

// The tables of corr u and corr v for k variables left, by one warp (lanes 4..7 and 8..11); v is
// corr u[t] or corr v[t] in those lanes.
__device__ __forceinline__ void put_tables(InstState& I, qm31 v, qm31 lam) {
  const uint32_t lane = threadIdx.x & 31;
  const qm31 l = mul(v, lam);
  if (lane >= 4 && lane < 8) {
    I.cu[lane - 4] = v;
    I.lcu[lane - 4] = I.product ? v : l;
  } else if (lane >= 8 && lane < 12) {
    I.cv[lane - 8] = v;
    I.lcv[lane - 8] = I.product ? v : l;
  }
}

// One instance's round polynomial from its sums, by one warp: lane 4 s + t has the s-th product of
// coefficient t.
__device__ __forceinline__ void make_poly(const GkrState& S, InstState& I, unsigned long long* acc, uint32_t layer,
                                          uint32_t round) {
  const uint32_t lane = threadIdx.x & 31, s = lane >> 2, t = lane & 3;
  qm31 p = q_zero();
  if (round >= I.delta) {
    qm31 a = q_zero(), b = q_zero();
    if (s < 4) {
      // volatile: sums in global memory (many instances) are added to past L1
      const volatile unsigned long long* w = acc + 4 * s;
      a = qm31_make(m31_reduce64(w[0]), m31_reduce64(w[1]), m31_reduce64(w[2]), m31_reduce64(w[3]));
      b = s == 0 ? I.cu[t] : s == 1 ? I.lcu[t] : s == 2 ? I.cv[t] : I.lcv[t];
    } else if (s == 4) {
      a = I.claim;
      b = S.row[layer - round].w[t];
    }
    p = mul(a, b);
    p = qm31_add(qm31_add(qm31_add(p, q_shfl(p, (lane + 4) & 31)), qm31_add(q_shfl(p, (lane + 8) & 31), q_shfl(p, (lane + 12) & 31))),
                 q_shfl(p, (lane + 16) & 31));
  } else if (lane == 0) {
    p = qm31_mul_m31(I.claim, (P + 1) / 2);
  }
  __syncwarp();
  if (lane < 16) acc[lane] = 0;
  const uint32_t nz = __ballot_sync(0xffffffffu, lane < 4 && !q_is_zero(p));
  const qm31 pa = mul(p, I.apow);
  if (lane < 4) {
    I.poly[lane] = p;
    I.pa[lane] = pa;
  }
  if (lane == 0) I.poly_size = nz == 0 ? 0 : 32 - __clz(nz);
}

// The round's polynomials from the sums, their combination into the channel and the next challenge
// (sumcheck::prove_batch's loop body), by the block; the sums are in acc and visible to it.
__device__ void finish_round(const GkrProgram& g, GkrState& S, InstState* inst, unsigned long long* acc, Hash& H,
                             uint32_t layer, uint32_t round) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t i = warp; i < g.n_inst; i += blockDim.x >> 5)
    if (inst[i].delta <= layer) make_poly(S, inst[i], acc + 16 * i, layer, round);
  __syncthreads();
  if (warp == 0) {
    __shared__ qm31 comb[4];
    uint32_t top = 0;
    qm31 c = q_zero();
    for (uint32_t i = 0; i < g.n_inst; i++) {
      if (inst[i].delta > layer) continue;
      top = max(top, inst[i].poly_size);
      if (lane < 4) c = qm31_add(c, inst[i].pa[lane]);
    }
    if (lane < 4) {
      comb[lane] = c;
      uint32_t* o = g.polys + 17 * ((size_t)layer * (layer - 1) / 2 + round);
      q_put(o + 1 + 4 * lane, c);
      if (lane == 0) o[0] = top;
    }
    __syncwarp();
    warp_mix(S, H, comb, top);
    const qm31 x = warp_draw(S, H);
    if (lane == 0) {
      S.sc[round] = x;
      S.x = x;
    }
  }
  __syncthreads();
}

// What the next round needs of an instance: its claim at the challenge, the eq correction and the
// tables scaled by it. One warp.
__device__ __forceinline__ void advance(const GkrState& S, InstState& I, uint32_t layer, uint32_t round) {
  const uint32_t lane = threadIdx.x & 31, k = layer - round - 1;
  const qm31 x = S.x, y = S.y[round];
  const qm31 m1 = mul(x, lane == 0 ? x : y);
  const qm31 x2 = q_shfl(m1, 0), xy = q_shfl(m1, 1);
  const qm31 e = qm31_add(qm31_sub(qm31_sub(q_one(), x), y), q_double(xy));  // eq(x, y)
  const qm31 m2 = mul(lane == 0 ? x2 : I.corr, lane == 0 ? x : e);
  const qm31 x3 = q_shfl(m2, 0);
  const qm31 corr = round >= I.delta ? q_shfl(m2, 1) : I.corr;
  qm31 a = corr, b = q_zero();
  if (lane < 4) {
    a = I.poly[lane];
    b = lane == 1 ? x : lane == 2 ? x2 : x3;
  } else if (lane < 8) {
    b = S.row[k].u[lane - 4];
  } else if (lane < 12) {
    b = S.row[k].v[lane - 8];
  }
  const qm31 m3 = mul(a, b);
  const qm31 claim = qm31_add(qm31_add(I.poly[0], q_shfl(m3, 1)), qm31_add(q_shfl(m3, 2), q_shfl(m3, 3)));
  __syncwarp();
  put_tables(I, m3, S.lam);
  if (lane == 0) {
    I.claim = claim;
    I.corr = corr;
  }
}

// advance for every instance, from the block's last warp down (the first ones have the next fix's
// elements).
__device__ __forceinline__ void advance_all(const GkrProgram& g, const GkrState& S, InstState* inst, uint32_t layer,
                                            uint32_t round) {
  const uint32_t warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
  for (uint32_t i = warps - 1 - warp; i < g.n_inst; i += warps)
    if (inst[i].delta <= layer) advance(S, inst[i], layer, round);
}

// The round tables of the point y (lane j: the row of k = layer - j, from y[j]). One warp.
__device__ void layer_tables(GkrState& S, uint32_t layer) {
  const uint32_t lane = threadIdx.x & 31;
  const bool on = lane < layer;
  const qm31 y = on ? S.y[lane] : q_zero();
  const qm31 one_y = qm31_sub(q_one(), y);
  qm31 prefix = one_y;  // prod_{t <= j} (1 - y_t)
#pragma unroll 1
  for (int off = 1; off < 32; off <<= 1) {
    const qm31 m = mul(prefix, q_shfl(prefix, (lane - off) & 31));
    if (lane >= (uint32_t)off) prefix = m;
  }
  const qm31 d = qm31_sub(one_y, y);
  const qm31 pd = mul(prefix, d);
  const qm31 inv = qm31_inv(pd);
  const qm31 a = mul(inv, d);                   // 1 / prefix
  const qm31 b = mul(one_y, mul(inv, prefix));  // (1 - y) / (1 - 2 y)
  const qm31 x0 = qm31_neg(b), x1 = qm31_sub(q_one(), b), x2 = qm31_add_m31(x1, 1);
  const qm31 x01 = mul(x0, x1), x012 = mul(x01, x2);
  const qm31 inv3 = qm31_inv(x012);
  const qm31 inv01 = mul(inv3, x2);
  const qm31 i0 = mul(inv01, x1), i1 = mul(inv01, x0), i2 = mul(inv3, x01);  // 1 / (x - b)
  const qm31 e0 = mul(a, one_y);                                             // a eq(0, y)
  const qm31 e2 = mul(a, qm31_add_m31(qm31_add(q_double(y), y), P - 1));     // a eq(2, y)
  // q0 = f0 al, q1 = claim i1 - f0 be, q2 = f2 ga; c2 = (q2 - 2 q1 + q0) / 2, c1 = q1 - q0 - c2;
  // the polynomial is (t - b) (q0 + c1 t + c2 t^2)
  const qm31 al = mul(e0, i0), be = mul(e0, i1), ga = mul(e2, i2);
  const uint32_t half = (P + 1) / 2;
  const qm31 al2 = qm31_mul_m31(al, half), ga2 = qm31_mul_m31(ga, half), be2 = q_double(be), i1x2 = q_double(i1);
  auto put = [&](qm31* o, qm31 q0, qm31 c1, qm31 c2) {
    const qm31 o0 = qm31_neg(mul(b, q0)), o1 = qm31_sub(q0, mul(b, c1)), o2 = qm31_sub(c1, mul(b, c2));
    if (on) o[0] = o0, o[1] = o1, o[2] = o2, o[3] = c2;
  };
  auto& row = S.row[on ? layer - lane : 0];
  put(row.u, al, qm31_neg(qm31_add(be2, qm31_add(al, al2))), qm31_add(al2, be));
  put(row.v, q_zero(), qm31_neg(ga2), ga2);
  put(row.w, q_zero(), i1x2, qm31_neg(i1));
  if (on && (q_is_zero(pd) || q_is_zero(x012))) S.err = 1;
}

// The layer's first half: the claims of the instances that join (their output layer's values), every
// claim into the channel and the two draws by one warp, the round tables by another, then the
// sum-check claims. The block (two warps at least); ends with a barrier.
__device__ void begin_layer(const GkrProgram& g, GkrState& S, InstState* inst, Hash& H, uint32_t layer) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 1) layer_tables(S, layer);
  if (warp == 0) {
    for (uint32_t i = lane; i < g.n_inst; i += 32) {
      InstState& I = inst[i];
      if (I.delta != layer) continue;
      const uint32_t* const* c = g.out0 + 8 * i;
      uint32_t n = 0;
      if (c[0] != nullptr) I.out[n++] = qm31_make(*c[0], *c[1], *c[2], *c[3]);
      I.out[n++] = qm31_make(*c[4], *c[5], *c[6], *c[7]);
      I.n_out = n;
      for (uint32_t t = 0; t < n; t++) q_put(g.outputs + 8 * i + 4 * t, I.out[t]);
    }
    __syncwarp();
    for (uint32_t i = 0; i < g.n_inst; i++)
      if (inst[i].delta <= layer) warp_mix(S, H, inst[i].out, inst[i].n_out);
    const qm31 alpha = warp_draw(S, H);
    const qm31 lam = warp_draw(S, H);
    if (lane == 0) {
      S.alpha = alpha;
      S.lam = lam;
    }
    qm31 apow = q_one();
    for (uint32_t i = 0; i < g.n_inst; i++) {
      InstState& I = inst[i];
      if (I.delta > layer) continue;
      qm31 c = I.out[I.n_out - 1];
      if (I.n_out == 2) c = qm31_add(mul(c, lam), I.out[0]);
      // an instance that joined delta layers late counts every point 2^delta times
      c = qm31_mul_m31(c, 1u << I.delta);
      if (lane == 0) {
        I.claim = c;
        I.corr = q_one();
        I.apow = apow;
      }
      if (i + 1 < g.n_inst) apow = mul(apow, alpha);
    }
  }
  __syncthreads();
  for (uint32_t i = warp; i < g.n_inst; i += blockDim.x >> 5)
    if (inst[i].delta <= layer)
      put_tables(inst[i],
                 lane >= 4 && lane < 8 ? S.row[layer].u[lane - 4] : lane >= 8 && lane < 12 ? S.row[layer].v[lane - 8] : q_zero(),
                 S.lam);
  __syncthreads();
}

// ------------------------------------------------------------ the sums of a round

struct Quad {
  qm31 v00, v01, v10, v11;  // a column at 2i, 2i + 1, 2 (T + i), 2 (T + i) + 1
};

__device__ __forceinline__ void load_pair(const uint32_t* const c[4], uint32_t pair, qm31& a, qm31& b) {
  uint2 w[4];
#pragma unroll
  for (int k = 0; k < 4; k++) w[k] = reinterpret_cast<const uint2*>(c[k])[pair];
  a = qm31_make(w[0].x, w[1].x, w[2].x, w[3].x);
  b = qm31_make(w[0].y, w[1].y, w[2].y, w[3].y);
}
__device__ __forceinline__ void load_base_pair(const uint32_t* c, uint32_t pair, qm31& a, qm31& b) {
  const uint2 w = reinterpret_cast<const uint2*>(c)[pair];
  a = qm31_make(w.x, 0, 0, 0);
  b = qm31_make(w.y, 0, 0, 0);
}
__device__ __forceinline__ void store_pair(uint32_t* const c[4], uint32_t pair, qm31 a, qm31 b) {
  reinterpret_cast<uint2*>(c[0])[pair] = make_uint2(a.a.a, b.a.a);
  reinterpret_cast<uint2*>(c[1])[pair] = make_uint2(a.a.b, b.a.b);
  reinterpret_cast<uint2*>(c[2])[pair] = make_uint2(a.b.a, b.b.a);
  reinterpret_cast<uint2*>(c[3])[pair] = make_uint2(a.b.b, b.b.b);
}

// Term i's values of one column: read, or with FIX folded by the challenge from the twice longer
// column src (element e from e and e + 4T) and written to dst.
template <bool FIX, bool BASE>
__device__ __forceinline__ Quad column_quad(const uint32_t* const src[4], uint32_t* const dst[4], uint32_t T, uint32_t i,
                                            const qm31_const& x) {
  Quad q;
  auto pair = [&](uint32_t at, qm31& a, qm31& b) {
    if (BASE)
      load_base_pair(src[0], at, a, b);
    else
      load_pair(src, at, a, b);
  };
  pair(i, q.v00, q.v01);
  pair(T + i, q.v10, q.v11);
  if (FIX) {
    Quad h;
    pair(2 * T + i, h.v00, h.v01);
    pair(3 * T + i, h.v10, h.v11);
    q.v00 = qm31_add(qm31_mul_const(qm31_sub(h.v00, q.v00), x), q.v00);
    q.v01 = qm31_add(qm31_mul_const(qm31_sub(h.v01, q.v01), x), q.v01);
    q.v10 = qm31_add(qm31_mul_const(qm31_sub(h.v10, q.v10), x), q.v10);
    q.v11 = qm31_add(qm31_mul_const(qm31_sub(h.v11, q.v11), x), q.v11);
    store_pair(dst, i, q.v00, q.v01);
    store_pair(dst, T + i, q.v10, q.v11);
  }
  return q;
}

// The sums of one instance's round: A = sum eq (numerator), C = sum eq (denominator) at t = 0 and 2 (a
// product has C alone); lambda C is added once per round instead of once per term.
struct Sums {
  qm31 a0, c0, a2, c2;
};

// Adds term i's share (sum_poly_kernel of gkr.cu).
template <int KIND, bool FIX, bool BASE>
__device__ __forceinline__ void add_term(const LayerCols& L, bool in_place, uint32_t T, uint32_t i, qm31 e,
                                         const qm31_const& x, Sums& s) {
  const Quad d = column_quad<FIX, false>(in_place ? L.fden : L.den, L.fden, T, i, x);
  const qm31 d20 = qm31_sub(q_double(d.v10), d.v00), d21 = qm31_sub(q_double(d.v11), d.v01);
  s.c0 = qm31_add(s.c0, qm31_mul(e, qm31_mul(d.v00, d.v01)));
  s.c2 = qm31_add(s.c2, qm31_mul(e, qm31_mul(d20, d21)));
  if constexpr (KIND == CS_GKR_LOGUP_SINGLES) {
    // 1/a + 1/b = (a + b) / (a b) (Reciprocal, crates/stwo/src/prover/lookups/utils.rs)
    s.a0 = qm31_add(s.a0, qm31_mul(e, qm31_add(d.v00, d.v01)));
    s.a2 = qm31_add(s.a2, qm31_mul(e, qm31_add(d20, d21)));
  } else if constexpr (KIND != CS_GKR_GRAND_PRODUCT) {
    const Quad n = column_quad<FIX, BASE>(in_place ? L.fnum : L.num, L.fnum, T, i, x);
    const qm31 n20 = qm31_sub(q_double(n.v10), n.v00), n21 = qm31_sub(q_double(n.v11), n.v01);
    s.a0 = qm31_add(s.a0, qm31_mul(e, qm31_add(qm31_mul(d.v01, n.v00), qm31_mul(d.v00, n.v01))));
    s.a2 = qm31_add(s.a2, qm31_mul(e, qm31_add(qm31_mul(d21, n20), qm31_mul(d20, n21))));
  }
}

// The sums over the terms i = first, first + step, ... < T of one instance's round; fixes: how many
// variables of the layer are fixed once this round's are.
__device__ __forceinline__ Sums round_terms(const LayerCols& L, uint32_t fixes, uint32_t T, uint32_t first, uint32_t step,
                                            const uint32_t* eq, uint32_t eq_stride, qm31 challenge) {
  const qm31_const x = qm31_const_of(challenge);
  const bool in_place = fixes >= 2;
  Sums s{q_zero(), q_zero(), q_zero(), q_zero()};
  auto e = [&](uint32_t i) {
    return qm31_make(eq[i], eq[eq_stride + i], eq[2 * (size_t)eq_stride + i], eq[3 * (size_t)eq_stride + i]);
  };
#define CS_GKR_TERMS(KIND, FIX, BASE) \
  for (uint32_t i = first; i < T; i += step) add_term<KIND, FIX, BASE>(L, in_place, T, i, e(i), x, s);
  if (L.kind == CS_GKR_GRAND_PRODUCT) {
    if (fixes) { CS_GKR_TERMS(CS_GKR_GRAND_PRODUCT, true, false) }
    else { CS_GKR_TERMS(CS_GKR_GRAND_PRODUCT, false, false) }
  } else if (L.kind == CS_GKR_LOGUP_SINGLES) {
    if (fixes) { CS_GKR_TERMS(CS_GKR_LOGUP_SINGLES, true, false) }
    else { CS_GKR_TERMS(CS_GKR_LOGUP_SINGLES, false, false) }
  } else if (L.kind == CS_GKR_LOGUP_MULTIPLICITIES && !in_place) {
    if (fixes) { CS_GKR_TERMS(CS_GKR_LOGUP_GENERIC, true, true) }
    else { CS_GKR_TERMS(CS_GKR_LOGUP_GENERIC, false, true) }
  } else {
    if (fixes) { CS_GKR_TERMS(CS_GKR_LOGUP_GENERIC, true, false) }
    else { CS_GKR_TERMS(CS_GKR_LOGUP_GENERIC, false, false) }
  }
#undef CS_GKR_TERMS
  return s;
}

// The block's state in dynamic shared memory: the program's, its instances' (up to kSharedInst) and
// their sums.
struct Block {
  GkrState* S;
  Hash* H;
  InstState* inst;
  unsigned long long* acc;
  unsigned char* rest;
};
__host__ __device__ inline size_t block_bytes(uint32_t n_inst) {
  const size_t per = sizeof(InstState) + 16 * sizeof(unsigned long long);
  return sizeof(GkrState) + sizeof(Hash) + (n_inst <= kSharedInst ? n_inst * per : 0);
}
__device__ __forceinline__ void copy_words(void* dst, const void* src, size_t bytes) {
  for (uint32_t k = threadIdx.x; k < bytes / 4; k += blockDim.x)
    static_cast<uint32_t*>(dst)[k] = static_cast<const uint32_t*>(src)[k];
}
__device__ Block load_block(const GkrProgram& g, unsigned char* smem) {
  Block B;
  B.S = reinterpret_cast<GkrState*>(smem);
  B.H = reinterpret_cast<Hash*>(smem + sizeof(GkrState));
  B.inst = g.inst;
  B.acc = g.acc;
  copy_words(B.S, g.state, sizeof(GkrState));
  hash_setup(*B.H);
  if (g.n_inst <= kSharedInst) {
    unsigned char* p = smem + sizeof(GkrState) + sizeof(Hash);
    B.acc = reinterpret_cast<unsigned long long*>(p);
    B.inst = reinterpret_cast<InstState*>(p + 16 * sizeof(unsigned long long) * g.n_inst);
    copy_words(B.inst, g.inst, sizeof(InstState) * g.n_inst);
    for (uint32_t k = threadIdx.x; k < 16 * g.n_inst; k += blockDim.x) B.acc[k] = 0;
  }
  B.rest = smem + block_bytes(g.n_inst);
  __syncthreads();
  return B;
}
__device__ void store_block(const GkrProgram& g, const Block& B) {
  __syncthreads();
  copy_words(g.state, B.S, sizeof(GkrState));
  if (B.inst != g.inst) copy_words(g.inst, B.inst, sizeof(InstState) * g.n_inst);
}

// Programmatic dependent launch: a kernel of the chain may start while the one before it drains, and
// waits here for its end before it reads what that one wrote. Released to the next kernel right after.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void copy_async(void* dst, const void* src, size_t bytes) {  // multiples of 16 bytes
  for (uint32_t k = threadIdx.x; k < bytes / 16; k += blockDim.x)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(
                     static_cast<unsigned char*>(dst) + 16 * k)),
                 "l"(static_cast<const unsigned char*>(src) + 16 * k));
}
// The part of the state that ending a round reads, fetched while the block sums its terms.
__device__ Block prefetch_block(const GkrProgram& g, unsigned char* smem, uint32_t layer, uint32_t round) {
  Block B;
  B.S = reinterpret_cast<GkrState*>(smem);
  B.H = reinterpret_cast<Hash*>(smem + sizeof(GkrState));
  B.inst = g.inst;
  B.acc = g.acc;
  const uint32_t k = layer - round;
  copy_async(B.S, g.state, offsetof(GkrState, y));
  copy_async(&B.S->y[round], &g.state->y[round], sizeof(qm31));
  copy_async(&B.S->row[k - 1], &g.state->row[k - 1], 2 * sizeof(B.S->row[0]));
  if (g.n_inst <= kSharedInst) {
    unsigned char* p = smem + sizeof(GkrState) + sizeof(Hash);
    B.acc = reinterpret_cast<unsigned long long*>(p);
    B.inst = reinterpret_cast<InstState*>(p + 16 * sizeof(unsigned long long) * g.n_inst);
    copy_async(B.inst, g.inst, sizeof(InstState) * g.n_inst);
    for (uint32_t j = threadIdx.x; j < 16 * g.n_inst; j += blockDim.x) B.acc[j] = 0;
  }
  B.rest = nullptr;
  return B;
}
// What ending a round changed.
__device__ void store_round(const GkrProgram& g, const Block& B, uint32_t round) {
  __syncthreads();
  copy_words(g.state, B.S, offsetof(GkrState, y));
  copy_words(&g.state->sc[round], &B.S->sc[round], sizeof(qm31));
  if (B.inst != g.inst) copy_words(g.inst, B.inst, sizeof(InstState) * g.n_inst);
}

__device__ __forceinline__ void add_to(unsigned long long* acc, qm31 v) {
  atomicAdd(acc + 0, (unsigned long long)v.a.a);
  atomicAdd(acc + 1, (unsigned long long)v.a.b);
  atomicAdd(acc + 2, (unsigned long long)v.b.a);
  atomicAdd(acc + 3, (unsigned long long)v.b.b);
}
__device__ __forceinline__ qm31 warp_sum(qm31 v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = q_shfl_add(v, off);
  return v;
}

// One round of many terms over the whole chip: blockIdx.x is the instance (any number of them; those
// that have not joined or wait for their first round are counted all the same), blockIdx.y its block.
// The last block to finish ends the round.
__global__ void __launch_bounds__(kRoundThreads) gkr_round_kernel(const GkrProgram g, uint32_t layer, uint32_t round) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ bool last;
  __shared__ qm31 part[4][kRoundThreads / 32];
  const uint32_t i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // how late the instance joins, from the table that no launch of the chain writes (InstState, which the
  // launch before this one writes back, may only be read after the wait)
  const LayerCols& L = g.cols[(size_t)layer * g.n_inst + i];
  const uint32_t delta = layer + 1 - L.n_vars;
  hash_setup(*reinterpret_cast<Hash*>(smem + sizeof(GkrState)));
  chain_wait();
  const Block B = prefetch_block(g, smem, layer, round);
  if (delta <= round) {
    const Sums s = round_terms(L, round - delta, 1u << (layer - round - 1),
                               blockIdx.y * blockDim.x + threadIdx.x, gridDim.y * blockDim.x, g.eq, 1u << (layer - 1),
                               g.state->x);
    const qm31 w[4] = {warp_sum(s.a0), warp_sum(s.c0), warp_sum(s.a2), warp_sum(s.c2)};
    if (lane == 0)
      for (int k = 0; k < 4; k++) part[k][warp] = w[k];
    __syncthreads();
    if (threadIdx.x < 4) {
      qm31 v = part[threadIdx.x][0];
      for (int k = 1; k < (int)kRoundThreads / 32; k++) v = qm31_add(v, part[threadIdx.x][k]);
      q_put(g.partial + 16 * ((size_t)i * gridDim.y + blockIdx.y) + 4 * threadIdx.x, v);
      __threadfence();
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(g.counter, 1u) == gridDim.x * gridDim.y - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (uint32_t j = 0; j < g.n_inst; j++) {
    if (B.inst[j].delta > round) continue;
    // thread 4 b + k adds sum k of the blocks b, b + 32, ...
    qm31 v = q_zero();
    for (uint32_t b = threadIdx.x >> 2; b < gridDim.y; b += kRoundThreads / 4) {
      const uint4 u = __ldcg(reinterpret_cast<const uint4*>(g.partial + 16 * ((size_t)j * gridDim.y + b)) + (threadIdx.x & 3));
      v = qm31_add(v, qm31_make(u.x, u.y, u.z, u.w));
    }
#pragma unroll
    for (int off = 16; off >= 4; off >>= 1) v = q_shfl_add(v, off);
    if (lane < 4) add_to(B.acc + 16 * j + 4 * lane, v);
  }
  __syncthreads();
  finish_round(g, *B.S, B.inst, B.acc, *B.H, layer, round);
  advance_all(g, *B.S, B.inst, layer, round);
  store_round(g, B, round);
  if (threadIdx.x == 0) *g.counter = 0;
}

// ------------------------------------------------------------ the single-block kernel

// Where an instance's columns are during the tail.
struct TailCols {
  const LayerCols* L;
  uint32_t* shared;  // [2 columns][4 coordinates][4 kTailTerms], or null: L's fnum / fden
  uint32_t fixes;    // including this round's
  bool entered;      // the tail's first round
  // coordinate k of column c (0: numerators) before and after this round's fix
  __device__ __forceinline__ const uint32_t* original(int c, int k) const { return c ? L->den[k] : L->num[k]; }
  __device__ __forceinline__ uint32_t* current(int c, int k) const {
    return shared ? shared + (4 * c + k) * (4 * kTailTerms) : c ? L->fden[k] : L->fnum[k];
  }
  __device__ __forceinline__ const uint32_t* before(int c, int k) const {
    if (fixes <= 1) return original(c, k);
    return entered ? (c ? L->fden[k] : L->fnum[k]) : current(c, k);
  }
  __device__ __forceinline__ const uint32_t* now(int c, int k) const {
    return fixes == 0 ? original(c, k) : current(c, k);
  }
  __device__ __forceinline__ bool has(int c) const {
    return c == 1 || L->kind == CS_GKR_LOGUP_GENERIC || L->kind == CS_GKR_LOGUP_MULTIPLICITIES;
  }
  __device__ __forceinline__ bool base(int c) const { return c == 0 && L->kind == CS_GKR_LOGUP_MULTIPLICITIES; }
};
__device__ __forceinline__ TailCols tail_cols(const GkrProgram& g, uint32_t* shared, uint32_t layer, uint32_t i,
                                              uint32_t fixes, bool entered) {
  return {g.cols + ((size_t)layer * g.n_inst + i), shared ? shared + (size_t)i * 32 * kTailTerms : nullptr, fixes,
          entered};
}

// A round's fix and sums, by the block: element e of every column folds to itself, then every part of
// a term (numerator's two products, denominator, at t = 0 and 2) is one item.
__device__ void tail_round(const GkrProgram& g, const Block& B, uint32_t* shared, const uint32_t* eq, uint32_t layer,
                           uint32_t round, bool entered) {
  const uint32_t log_t = layer - round - 1, T = 1u << log_t;
  const qm31 x = B.S->x;
  if (round > 0 && !entered) advance_all(g, *B.S, B.inst, layer, round - 1);
  for (uint32_t idx = threadIdx.x; idx < (g.n_inst << (log_t + 3)); idx += blockDim.x) {
    const uint32_t e = idx & (4 * T - 1), c = (idx >> (log_t + 2)) & 1, i = idx >> (log_t + 3);
    const uint32_t delta = B.inst[i].delta;
    if (delta >= round) continue;  // not joined, or nothing to fix yet
    const TailCols C = tail_cols(g, shared, layer, i, round - delta, entered);
    if (!C.has(c)) continue;
    qm31 v;
    if (C.fixes == 1 && C.base(c)) {
      const uint32_t l = C.before(c, 0)[e], h = C.before(c, 0)[e + 4 * T];
      v = qm31_add_m31(qm31_mul_m31(x, m31_sub(h, l)), l);
    } else {
      qm31 l, h;
      l = qm31_make(C.before(c, 0)[e], C.before(c, 1)[e], C.before(c, 2)[e], C.before(c, 3)[e]);
      h = qm31_make(C.before(c, 0)[e + 4 * T], C.before(c, 1)[e + 4 * T], C.before(c, 2)[e + 4 * T],
                    C.before(c, 3)[e + 4 * T]);
      v = q_lerp(l, h, x);
    }
    C.current(c, 0)[e] = v.a.a;
    C.current(c, 1)[e] = v.a.b;
    C.current(c, 2)[e] = v.b.a;
    C.current(c, 3)[e] = v.b.b;
  }
  __syncthreads();
  const uint32_t items = g.n_inst << (log_t + 3);  // 8 slots a term, 6 of them used
  for (uint32_t first = threadIdx.x & ~31u; first < items; first += blockDim.x) {
    const uint32_t idx = first + (threadIdx.x & 31);
    const uint32_t i = idx >> (log_t + 3), slot = (idx >> log_t) & 7, t = idx & (T - 1), at = slot >> 2, part = slot & 3;
    qm31 v = q_zero();
    bool on = idx < items && part < 3 && B.inst[i].delta <= round;
    if (on) {
      const TailCols C = tail_cols(g, shared, layer, i, round - B.inst[i].delta, entered);
      auto value = [&](int c, uint32_t j) {  // the column at 2 t + j and its t = 0 or 2 point
        const bool base = C.fixes == 0 && C.base(c);
        uint32_t w[4] = {0, 0, 0, 0}, z[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (k > 0 && base) break;
          const uint32_t* p = C.now(c, k);
          w[k] = p[2 * t + j];
          if (at) z[k] = p[2 * (T + t) + j];
        }
        const qm31 v0 = q_make4(w);
        return at ? qm31_sub(q_double(q_make4(z)), v0) : v0;
      };
      const bool num = C.has(0);
      on = part == 2 || num || (part == 0 && C.L->kind == CS_GKR_LOGUP_SINGLES);
      if (on) {
        const qm31 a = value(1, part == 0 ? 1 : 0);
        const qm31 b = part == 2 || !num ? value(1, part == 2 ? 1 : 0) : value(0, part);
        v = part < 2 && !num ? qm31_add(a, b) : mul(a, b);
        v = mul(v, qm31_make(eq[t], eq[kTailTerms + t], eq[2 * kTailTerms + t], eq[3 * kTailTerms + t]));
      }
    }
    for (uint32_t off = min(T, 32u) >> 1; off > 0; off >>= 1) v = q_shfl_add(v, off);
    if (on && (t & 31) == 0) add_to(B.acc + 16 * i + 8 * at + (part == 2 ? 4 : 0), v);
  }
  __syncthreads();
}

// The layer's second half: the masks (the two values of every column left after the last challenge),
// their mix, the draw that extends the point and the claims at it. One warp.
__device__ void end_layer(const GkrProgram& g, const Block& B, uint32_t* shared, uint32_t layer) {
  const uint32_t lane = threadIdx.x & 31;
  GkrState& S = *B.S;
  // a lane per (instance, column, value); a mask without numerators has the denominators first
  for (uint32_t idx = lane; idx < 4 * g.n_inst; idx += 32) {
    const uint32_t i = idx >> 2, c = (idx >> 1) & 1, j = idx & 1;
    InstState& I = B.inst[i];
    if (I.delta > layer) continue;
    const TailCols C = tail_cols(g, shared, layer, i, layer - I.delta, false);
    const bool ones = C.L->kind == CS_GKR_LOGUP_SINGLES;
    if (j == 0 && c == 1) I.n_out = C.has(0) || ones ? 2 : 1;
    qm31 m = q_one();
    if (C.has(c)) {
      qm31 v[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 4; k++)
          if ((k == 0 || !(C.base(c) && C.fixes == 1)) && (h == 0 || C.fixes > 0)) w[k] = C.before(c, k)[j + 2 * h];
        v[h] = q_make4(w);
      }
      m = C.fixes > 0 ? q_lerp(v[0], v[1], S.x) : v[0];
    } else if (!ones) {
      continue;
    }
    const uint32_t t = C.has(0) || ones ? idx & 3 : j;
    I.poly[t] = m;
    q_put(g.masks + 16 * ((size_t)layer * g.n_inst + i) + 4 * t, m);
  }
  __syncwarp();
  for (uint32_t i = 0; i < g.n_inst; i++)
    if (B.inst[i].delta <= layer) warp_mix(S, *B.H, B.inst[i].poly, 2 * B.inst[i].n_out);
  const qm31 x = warp_draw(S, *B.H);
  if (lane == 0) S.x = x;
  if (lane < layer) S.y[lane] = S.sc[lane];
  if (lane == layer) S.y[lane] = x;
  for (uint32_t i = lane; i < g.n_inst; i += 32) {
    InstState& I = B.inst[i];
    if (I.delta > layer) continue;
    I.out[0] = q_lerp(I.poly[0], I.poly[1], x);
    if (I.n_out == 2) I.out[1] = q_lerp(I.poly[2], I.poly[3], x);
  }
  __syncwarp();
}

size_t tail_smem(uint32_t n_inst) {
  return block_bytes(n_inst) + (n_inst <= kSharedCols ? (size_t)n_inst * 32 * kTailTerms * sizeof(uint32_t) : 0);
}

// Rounds [round, layer) of `layer` and its masks, and the whole of the layers that follow while they
// have at most kTailRounds rounds. begin: start with the layer's claims.
__global__ void __launch_bounds__(kTailThreads) gkr_tail_kernel(const GkrProgram g, uint32_t layer, uint32_t round,
                                                                uint32_t begin) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t eq[4][kTailTerms];
  chain_wait();
  const Block B = load_block(g, smem);
  uint32_t* shared = g.n_inst <= kSharedCols ? reinterpret_cast<uint32_t*>(B.rest) : nullptr;
  if (begin) {
    begin_layer(g, *B.S, B.inst, *B.H, layer);
  }
  for (;;) {
    const uint32_t entry = round;
    if (layer > kTailRounds) {
      for (uint32_t k = threadIdx.x; k < 4 * kTailTerms; k += blockDim.x)
        eq[k / kTailTerms][k % kTailTerms] = g.eq[((size_t)(k / kTailTerms) << (layer - 1)) + k % kTailTerms];
    } else if (layer > 0) {
      // eq(x, (y_1, ..)) eq(0, y_0): the doubling of gen_eq_evals; y_1 is the highest index bit
      if (threadIdx.x == 0) {
        const qm31 v = qm31_sub(q_one(), B.S->y[0]);
        eq[0][0] = v.a.a, eq[1][0] = v.a.b, eq[2][0] = v.b.a, eq[3][0] = v.b.b;
      }
      __syncthreads();
      for (uint32_t t = 0; t + 1 < layer; t++) {
        const uint32_t n = 1u << t, j = threadIdx.x;
        if (j < n) {
          const qm31 l = qm31_make(eq[0][j], eq[1][j], eq[2][j], eq[3][j]);
          const qm31 hi = mul(l, B.S->y[layer - 1 - t]), lo = qm31_sub(l, hi);
          eq[0][j] = lo.a.a, eq[1][j] = lo.a.b, eq[2][j] = lo.b.a, eq[3][j] = lo.b.b;
          eq[0][j + n] = hi.a.a, eq[1][j + n] = hi.a.b, eq[2][j + n] = hi.b.a, eq[3][j + n] = hi.b.b;
        }
        __syncthreads();
      }
    }
    __syncthreads();
    for (; round < layer; round++) {
      tail_round(g, B, shared, &eq[0][0], layer, round, round == entry);
      finish_round(g, *B.S, B.inst, B.acc, *B.H, layer, round);
    }
    if (threadIdx.x < 32) end_layer(g, B, shared, layer);
    layer++;
    round = 0;
    if (layer == g.n_layers || layer > kTailRounds) break;
    __syncthreads();
    begin_layer(g, *B.S, B.inst, *B.H, layer);
  }
  store_block(g, B);
}

// A long layer's start: block 0 makes the claims and tables, the others the layer's eq column from the
// point in the state (eq_evals_kernel), 2^kEqChunkBits values each.
__global__ void __launch_bounds__(256) gkr_start_kernel(const GkrProgram g, uint32_t layer, const QOut eq) {
  extern __shared__ __align__(16) unsigned char smem[];
  chain_wait();
  if (blockIdx.x == 0) {
    const Block B = load_block(g, smem);
    begin_layer(g, *B.S, B.inst, *B.H, layer);
    // the point stays as it is: the other blocks read it
    copy_words(g.state, B.S, offsetof(GkrState, y));
    copy_words(g.state->row, B.S->row, sizeof(B.S->row));
    if (B.inst != g.inst) copy_words(g.inst, B.inst, sizeof(InstState) * g.n_inst);
    return;
  }
  eq_evals_block(blockIdx.x - 1, qm31_sub(q_one(), g.state->y[0]), g.state->y + 1, layer - 1, eq);
}

// ------------------------------------------------------------ host

// Raises a kernel's dynamic shared memory limit (a per-device attribute) once per device.
template <typename Kernel>
cs_status allow_smem(Kernel kernel, size_t bytes, int which) {
  static std::mutex mu;
  static bool done[3][kMaxDevices] = {};
  int dev = 0;
  CS_CUDA(cudaGetDevice(&dev));
  CS_CHECK_ARG(dev >= 0 && dev < kMaxDevices, "gkr_prove_batch: device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!done[which][dev]) {
    CS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[which][dev] = true;
  }
  return CS_OK;
}

// Device memory of one proof, freed in stream order.
struct Buffers {
  cudaStream_t st;
  std::vector<void*> ptrs;
  ~Buffers() {
    for (void* p : ptrs) cudaFreeAsync(p, st);
  }
  template <typename T>
  cs_status get(T*& out, size_t n) {
    void* p = nullptr;
    const cudaError_t e = stream_alloc(&p, std::max<size_t>(16, n * sizeof(T)), st);
    if (e != cudaSuccess) return from_cuda(e, "gkr_prove_batch: allocation");
    ptrs.push_back(p);
    out = static_cast<T*>(p);
    return CS_OK;
  }
};

void put_q(std::vector<uint64_t>& out, const uint32_t* w) {
  for (int k = 0; k < 4; k++) out.push_back(w[k]);
}

}  // namespace

// The protocol over `inputs` from the channel state `chan` (advanced); the proof and artifact are
// appended to `out` in the layout of cs_gkr_prove_batch.
cs_status gkr_prove_on_device(const std::vector<GkrInput>& inputs, uint32_t chan[9], std::vector<uint64_t>& out,
                              cudaStream_t st) {
  const uint32_t n_inst = (uint32_t)inputs.size();
  uint32_t n_layers = 0;
  for (const GkrInput& in : inputs) {
    n_layers = std::max(n_layers, in.n_vars);
    // such an instance's only layer is never fixed, so its masks would be base values
    CS_CHECK_ARG(in.kind != CS_GKR_LOGUP_MULTIPLICITIES || in.n_vars > 1,
                 "gkr_prove_batch: mask of a multiplicities layer");
  }
  Buffers mem{st, {}};

  // every instance's layers above its input, 2^(n - 1) values down to one, one after another
  std::vector<LayerCols> cols((size_t)n_layers * n_inst);
  std::vector<const uint32_t*> out0(8 * (size_t)n_inst, nullptr);
  struct Stack {
    uint32_t *num = nullptr, *den = nullptr;
  };
  std::vector<Stack> stacks(n_inst);
  auto coords = [](uint32_t* base, uint32_t n, uint32_t vars, uint32_t* c[4]) {
    // layer of 2^vars values in a stack whose first layer has 2^(n - 1)
    uint32_t* p = base + 4 * (((size_t)1 << n) - ((size_t)2 << vars));
    for (int k = 0; k < 4; k++) c[k] = p + ((size_t)k << vars);
  };
  for (uint32_t i = 0; i < n_inst; i++) {
    const GkrInput& in = inputs[i];
    const bool product = in.kind == CS_GKR_GRAND_PRODUCT;
    const size_t words = (size_t)4 << in.n_vars;
    Stack& s = stacks[i];
    // the input's first fix goes to scratch of half its size, behind the stack
    const size_t half = (size_t)4 << (in.n_vars - 1);
    const bool fix_num = in.kind == CS_GKR_LOGUP_GENERIC || in.kind == CS_GKR_LOGUP_MULTIPLICITIES;
    cs_status a = mem.get(s.den, words + half);
    if (a == CS_OK && !product) a = mem.get(s.num, words + (fix_num ? half : 0));
    if (a != CS_OK) return a;
    const uint32_t* num[4] = {in.num[0], in.num[1], in.num[2], in.num[3]};
    const uint32_t* den[4] = {in.den[0], in.den[1], in.den[2], in.den[3]};
    uint32_t kind = in.kind;
    const uint32_t delta = n_layers - in.n_vars;
    for (uint32_t vars = in.n_vars;; vars--) {
      if (vars > 0) {
        LayerCols& L = cols[(size_t)(delta + vars - 1) * n_inst + i];
        L.kind = kind;
        L.n_vars = vars;
        const bool input = vars == in.n_vars;
        for (int k = 0; k < 4; k++) {
          L.num[k] = num[k];
          L.den[k] = den[k];
          L.fnum[k] = input ? (fix_num ? s.num + words + ((size_t)k << (vars - 1)) : nullptr)
                            : const_cast<uint32_t*>(num[k]);
          L.fden[k] = input ? s.den + words + ((size_t)k << (vars - 1)) : const_cast<uint32_t*>(den[k]);
        }
      } else {
        for (int k = 0; k < 4; k++) {
          out0[8 * (size_t)i + k] = product ? nullptr : num[k];
          out0[8 * (size_t)i + 4 + k] = den[k];
        }
        break;
      }
      uint32_t *on[4] = {nullptr, nullptr, nullptr, nullptr}, *od[4];
      coords(s.den, in.n_vars, vars - 1, od);
      if (!product) coords(s.num, in.n_vars, vars - 1, on);
      const cs_status r = cs_gkr_next_layer(kind, kind == CS_GKR_GRAND_PRODUCT || kind == CS_GKR_LOGUP_SINGLES ? nullptr : num,
                                            den, vars, product ? nullptr : on, od, reinterpret_cast<cs_stream>(st));
      if (r != CS_OK) return r;
      for (int k = 0; k < 4; k++) num[k] = on[k], den[k] = od[k];
      if (!product) kind = CS_GKR_LOGUP_GENERIC;
    }
  }

  // tables and state up, results back: one buffer each way
  const size_t n_polys = (size_t)n_layers * (n_layers - 1) / 2;
  const uint32_t max_terms_log = n_layers >= 2 ? n_layers - 2 : 0;
  const uint32_t max_blocks = std::min<uint64_t>(((1ull << max_terms_log) + kRoundThreads - 1) / kRoundThreads, 152 * 8);
  struct Up {
    std::vector<unsigned char> bytes;
    size_t add(const void* p, size_t n) {
      const size_t at = (bytes.size() + 15) & ~(size_t)15;
      bytes.resize(at + n);
      if (p != nullptr) std::memcpy(bytes.data() + at, p, n);
      return at;
    }
  } up;
  GkrState state{};
  for (int k = 0; k < 9; k++) state.chan[k] = chan[k];
  std::vector<InstState> inst(n_inst, InstState{});
  for (uint32_t i = 0; i < n_inst; i++) {
    inst[i].delta = n_layers - inputs[i].n_vars;
    inst[i].product = inputs[i].kind == CS_GKR_GRAND_PRODUCT;
  }
  const std::vector<unsigned long long> acc(16 * (size_t)n_inst, 0);
  const size_t at_state = up.add(&state, sizeof(state));
  const size_t at_inst = up.add(inst.data(), sizeof(InstState) * n_inst);
  const size_t at_acc = up.add(acc.data(), sizeof(acc[0]) * acc.size());
  const size_t at_cols = up.add(cols.data(), sizeof(LayerCols) * cols.size());
  const size_t at_out0 = up.add(out0.data(), sizeof(void*) * out0.size());
  const uint32_t zero = 0;
  const size_t at_counter = up.add(&zero, sizeof(zero));
  // results, right after the state and the instances (read back together)
  const size_t at_polys = up.add(nullptr, 0), polys_bytes = 4 * 17 * n_polys;
  const size_t at_masks = (at_polys + polys_bytes + 15) & ~(size_t)15, masks_bytes = 4 * 16 * (size_t)n_layers * n_inst;
  const size_t at_outputs = (at_masks + masks_bytes + 15) & ~(size_t)15, outputs_bytes = 4 * 8 * (size_t)n_inst;
  const size_t at_partial = (at_outputs + outputs_bytes + 15) & ~(size_t)15;
  const size_t total = at_partial + 4 * 16 * (size_t)n_inst * max_blocks;
  unsigned char* dev = nullptr;
  uint32_t* eq = nullptr;
  cs_status a = mem.get(dev, total);
  if (a == CS_OK) a = mem.get(eq, (size_t)4 << max_terms_log);
  if (a != CS_OK) return a;
  CS_CUDA(cudaMemcpyAsync(dev, up.bytes.data(), up.bytes.size(), cudaMemcpyHostToDevice, st));

  GkrProgram g;
  g.state = reinterpret_cast<GkrState*>(dev + at_state);
  g.inst = reinterpret_cast<InstState*>(dev + at_inst);
  g.cols = reinterpret_cast<const LayerCols*>(dev + at_cols);
  g.out0 = reinterpret_cast<const uint32_t* const*>(dev + at_out0);
  g.counter = reinterpret_cast<uint32_t*>(dev + at_counter);
  g.polys = reinterpret_cast<uint32_t*>(dev + at_polys);
  g.masks = reinterpret_cast<uint32_t*>(dev + at_masks);
  g.outputs = reinterpret_cast<uint32_t*>(dev + at_outputs);
  g.acc = reinterpret_cast<unsigned long long*>(dev + at_acc);
  g.partial = reinterpret_cast<uint32_t*>(dev + at_partial);
  g.n_inst = n_inst;
  g.n_layers = n_layers;
  g.eq = eq;

  const size_t round_bytes = block_bytes(n_inst), tail_bytes = tail_smem(n_inst);
  // the tail's largest: tail columns of kSharedCols instances, or the state of kSharedInst
  cs_status attr = allow_smem(gkr_tail_kernel, std::max(tail_smem(kSharedCols), tail_smem(kSharedInst)), 0);
  if (attr == CS_OK) attr = allow_smem(gkr_round_kernel, block_bytes(kSharedInst), 1);
  if (attr != CS_OK) return attr;
  attr = allow_smem(gkr_start_kernel, block_bytes(kSharedInst), 2);
  if (attr != CS_OK) return attr;
  gkr_tail_kernel<<<1, kTailThreads, tail_bytes, st>>>(g, 0, 0, 1);
  CS_LAUNCHED("gkr_tail_kernel");
  // the rest is one chain of dependent launches
  cudaLaunchAttribute dependent;
  dependent.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  dependent.val.programmaticStreamSerializationAllowed = 1;
  auto config = [&](dim3 grid, uint32_t threads, size_t smem) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &dependent;
    c.numAttrs = 1;
    return c;
  };
  for (uint32_t l = kTailRounds + 1; l < n_layers; l++) {
    QOut e;
    for (int k = 0; k < 4; k++) e.c[k] = eq + ((size_t)k << (l - 1));
    cudaLaunchConfig_t c = config(dim3(1 + (1u << (l - 1 - std::min(l - 1, kEqChunkBits)))), 256, round_bytes);
    CS_CUDA(cudaLaunchKernelEx(&c, gkr_start_kernel, (const GkrProgram)g, l, (const QOut)e));
    note_launch();
    for (uint32_t r = 0; r + kTailRounds < l; r++) {
      const uint64_t terms = 1ull << (l - r - 1);
      const uint32_t blocks = (uint32_t)std::min<uint64_t>((terms + kRoundThreads - 1) / kRoundThreads, 152 * 8);
      c = config(dim3(n_inst, blocks), kRoundThreads, round_bytes);
      CS_CUDA(cudaLaunchKernelEx(&c, gkr_round_kernel, (const GkrProgram)g, l, r));
      note_launch();
    }
    c = config(dim3(1), kTailThreads, tail_bytes);
    CS_CUDA(cudaLaunchKernelEx(&c, gkr_tail_kernel, (const GkrProgram)g, l, l - kTailRounds, 0u));
    note_launch();
  }
  std::vector<unsigned char> back(at_partial);
  CS_CUDA(cudaMemcpyAsync(back.data(), dev, back.size(), cudaMemcpyDeviceToHost, st));
  CS_CUDA(cudaStreamSynchronize(st));
  const GkrState& S = *reinterpret_cast<const GkrState*>(back.data() + at_state);
  const InstState* I = reinterpret_cast<const InstState*>(back.data() + at_inst);
  // (a round polynomial agrees with its claim by construction: it is interpolated through
  // r(1) = claim - r(0))
  CS_CHECK_ARG(S.err == 0, "gkr_prove_batch: division by zero in the round constants");
  const uint32_t* polys = reinterpret_cast<const uint32_t*>(back.data() + at_polys);
  const uint32_t* masks = reinterpret_cast<const uint32_t*>(back.data() + at_masks);
  const uint32_t* outputs = reinterpret_cast<const uint32_t*>(back.data() + at_outputs);
  out.push_back(n_layers);
  for (uint32_t l = 0; l < n_layers; l++) {
    out.push_back(l);
    for (uint32_t r = 0; r < l; r++) {
      const uint32_t* p = polys + 17 * ((size_t)l * (l - 1) / 2 + r);
      out.push_back(p[0]);
      for (uint32_t t = 0; t < p[0]; t++) put_q(out, p + 1 + 4 * t);
    }
  }
  auto columns = [&](uint32_t i, uint32_t l) { return cols[(size_t)l * n_inst + i].kind == CS_GKR_GRAND_PRODUCT ? 1u : 2u; };
  out.push_back(n_inst);
  for (uint32_t i = 0; i < n_inst; i++) {
    out.push_back(inputs[i].n_vars);
    for (uint32_t l = I[i].delta; l < n_layers; l++) {
      out.push_back(columns(i, l));
      for (uint32_t t = 0; t < 2 * columns(i, l); t++) put_q(out, masks + 16 * ((size_t)l * n_inst + i) + 4 * t);
    }
  }
  for (uint32_t i = 0; i < n_inst; i++) {
    const uint32_t n = inputs[i].kind == CS_GKR_GRAND_PRODUCT ? 1 : 2;
    out.push_back(n);
    for (uint32_t t = 0; t < n; t++) put_q(out, outputs + 8 * (size_t)i + 4 * t);
  }
  out.push_back(n_layers);
  for (uint32_t l = 0; l < n_layers; l++) put_q(out, reinterpret_cast<const uint32_t*>(&S.y[l]));
  for (uint32_t i = 0; i < n_inst; i++) {
    out.push_back(columns(i, n_layers - 1));
    for (uint32_t t = 0; t < columns(i, n_layers - 1); t++) put_q(out, reinterpret_cast<const uint32_t*>(&I[i].out[t]));
  }
  for (uint32_t i = 0; i < n_inst; i++) out.push_back(inputs[i].n_vars);
  for (int k = 0; k < 9; k++) chan[k] = S.chan[k];
  return CS_OK;
}

}  // namespace cs
