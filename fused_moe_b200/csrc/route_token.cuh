// Routing of one token by one warp (the rules are stated at the top of routing.cu), shared by the routing kernels and the
// decode path.
#pragma once
#include "common.cuh"

namespace b200moe {

// exp(-x) and the sigmoid are built from individually rounded IEEE operations only (no fast-math, no contraction
// left to the compiler), so that a host restatement with fmaf() produces the same bits.
__device__ __forceinline__ float exp_neg_exact_ops(float x) {
  float z = fminf(fmaxf(-x, -87.0f), 88.0f);
  float t = __fmul_rn(z, 1.44269504088896341f);
  float n = rintf(t);
  float r = __fmaf_rn(n, -0.693145751953125f, z);           // ln2 high part (exact product for |n| < 2^11)
  r = __fmaf_rn(n, -1.42860682030941723e-6f, r);            // ln2 low part
  float p = 1.0f / 5040.0f;
  p = __fmaf_rn(p, r, 1.0f / 720.0f);
  p = __fmaf_rn(p, r, 1.0f / 120.0f);
  p = __fmaf_rn(p, r, 1.0f / 24.0f);
  p = __fmaf_rn(p, r, 1.0f / 6.0f);
  p = __fmaf_rn(p, r, 0.5f);
  p = __fmaf_rn(p, r, 1.0f);
  p = __fmaf_rn(p, r, 1.0f);
  float scale = __int_as_float((static_cast<int>(n) + 127) << 23);
  return __fmul_rn(p, scale);
}
__device__ __forceinline__ float sigmoid_exact_ops(float x) {
  return __fdiv_rn(1.0f, __fadd_rn(1.0f, exp_neg_exact_ops(x)));
}

// float <-> unsigned key with the same ordering (larger float = larger key); key 0 is below every float.
__device__ __forceinline__ uint32_t f2key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key2f(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Routing of one token by one warp.  Lane k < 8 returns the k-th selected expert in `my_idx` and its final weight in
// `my_w` (other lanes return 0).
__device__ __forceinline__ void route_token(const float* logits_row, const uint16_t* bias,
                                            float scale_factor, int lane, int& my_idx, float& my_w) {
  float s[N_GROUP];
  uint32_t key[N_GROUP];
#pragma unroll
  for (int g = 0; g < N_GROUP; ++g) {
    float x = ld_dep(logits_row + g * 32 + lane);
    float b = bf16_bits_to_float(ld_dep(bias + g * 32 + lane));
    s[g] = sigmoid_exact_ops(x);
    key[g] = f2key(__fadd_rn(s[g], b));
  }
  // group scores (warp-uniform)
  float gs[N_GROUP];
#pragma unroll
  for (int g = 0; g < N_GROUP; ++g) {
    uint32_t m1 = __reduce_max_sync(0xffffffffu, key[g]);
    uint32_t hit = __ballot_sync(0xffffffffu, key[g] == m1);
    int first = __ffs(hit) - 1;
    uint32_t m2 = __reduce_max_sync(0xffffffffu, lane == first ? 0u : key[g]);
    gs[g] = __fadd_rn(key2f(m1), key2f(m2));
  }
  // top-4 groups, lower index wins ties
  uint32_t gmask = 0;
#pragma unroll
  for (int r = 0; r < TOPK_GROUP; ++r) {
    int best = -1;
    float bv = 0.f;
#pragma unroll
    for (int g = 0; g < N_GROUP; ++g) {
      bool free_g = !((gmask >> g) & 1u);
      if (free_g && (best < 0 || gs[g] > bv)) { best = g; bv = gs[g]; }
    }
    gmask |= 1u << best;
  }
#pragma unroll
  for (int g = 0; g < N_GROUP; ++g)
    if (!((gmask >> g) & 1u)) key[g] = 0u;

  // top-8 experts by repeated arg-max with removal
  my_idx = 0;
  float my_s = 0.f;
  float sum = 0.f;
#pragma unroll
  for (int k = 0; k < TOP_K; ++k) {
    uint32_t bk = key[0];
    int bg = 0;
#pragma unroll
    for (int g = 1; g < N_GROUP; ++g)
      if (key[g] > bk) { bk = key[g]; bg = g; }
    uint32_t vmax = __reduce_max_sync(0xffffffffu, bk);
    uint32_t cand = (bk == vmax) ? static_cast<uint32_t>(bg * 32 + lane) : 0xffffu;
    uint32_t widx = __reduce_min_sync(0xffffffffu, cand);
    int owner = widx & 31, slot = widx >> 5;
    float sv = 0.f;
#pragma unroll
    for (int g = 0; g < N_GROUP; ++g)
      if (g == slot) {
        sv = s[g];
        if (lane == owner) key[g] = 0u;
      }
    sv = __shfl_sync(0xffffffffu, sv, owner);
    sum = __fadd_rn(sum, sv);
    if (lane == k) { my_idx = static_cast<int>(widx); my_s = sv; }
  }
  my_w = __fmul_rn(__fdiv_rn(my_s, __fadd_rn(sum, 1e-20f)), scale_factor);
}

}  // namespace b200moe
