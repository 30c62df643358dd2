// What the kernels of LinearInt8Scaled share: parameters, epilogue arithmetic, the kernels of few rows.
#pragma once

#include "common.cuh"

namespace difb200 {

enum : uint32_t { kEpiBias = 1u, kEpiGeluTanh = 2u };

struct GemmParams {
  const float *row_scales;
  const float *col_scales;
  const uint16_t *bias;
  uint16_t *out;
  int32_t *acc_out;
  uint32_t M, N, K;
  uint32_t epilogue;
  uint32_t a_rows;  // rows of a load of x
  uint32_t split;   // CTAS = 1: CTAs of a cluster that share one tile's k-blocks (1 = no cluster)
  uint32_t tma_store; // 1: outputs leave through TMA stores (needs N % 8 == 0, aligned out)
  uint32_t weights_first; // 1: w is not written by the kernel in front, its first blocks are requested before that one is done
  uint32_t withhold_kb; // test aid: the loads of this k-block are never issued (0xffffffff = none)
  unsigned long long wait_ns; // limit of every bounded wait
  DeviceStatus *status;
};

// Whether the kernels of few rows take a problem, and their launch (weights and codes start on 16 bytes, K % 16 == 0).
bool few_rows(uint64_t M, uint64_t N, uint64_t K, bool weights_first);
int launch_few_rows(const int8_t *x, const int8_t *w, const GemmParams &p, cudaStream_t stream);

#ifdef __CUDACC__

__device__ __forceinline__ float gelu_tanh(float v) {
  // Reference form (cpu_executor.cpp:93-113): 0.5 * v * (1 + tanh(u)), u = 0.79788456 * (v +
  // 0.044715 * v^3). The reference's fp32 sum 1 + tanh(u) cancels for negative v, and that
  // rounding is part of its result, so the same three roundings are kept here and only tanh
  // itself is computed differently: tanh|u| = 1 - 2 / (e^(2|u|) + 1) with two MUFU ops
  // (ex2, rcp), absolute error below one ulp of 1.
  constexpr float kA = 0.7978845608028654f * 2.0f * 1.4426950408889634f;
  constexpr float kB = kA * 0.044715f;
  const float t = fmaf(kB, v * v, kA) * v; // 2u * log2(e), same sign as v
  float e, r;
  asm("ex2.approx.f32 %0, %1;" : "=f"(e) : "f"(fabsf(t)));
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(e + 1.0f));
  const float th = copysignf(fmaf(-2.0f, r, 1.0f), v);
  return __fmul_rn(__fmul_rn(0.5f, v), __fadd_rn(1.0f, th));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t packed;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(hi), "f"(lo));
  return packed;
}

#endif // __CUDACC__

} // namespace difb200
