// Shared by the QuantizeInt8Rows kernels: parameters, the radix-4 butterfly, exact divisions.
#pragma once

#include "common.cuh"
#include "glue.h"

namespace difb200 {

constexpr int kMaxParts = 8;

struct QuantParams {
  const uint16_t *part[kMaxParts];
  uint32_t width[kMaxParts];
  uint32_t part_count;
  uint32_t wide;  // every part starts on 32 bytes
  uint32_t columns;
  uint64_t rows;
  float clip;
  const float *clip_device;
  int8_t *codes;
  float *scales;
  int8_t *rcodes;
  float *rscales;
  uint32_t mse;   // weight rows: choose the row scale by the offline packer's MSE search
  const uint16_t *equalise; // weight rows: bf16 [columns], every element is divided by its entry first
  // RmsNormModulate in front of the quantiser (explicit scale / shift layout), all bf16:
  const uint16_t *norm_weight; // [columns] or nullptr
  const uint16_t *norm_scale;  // [rows, columns]; nullptr = no prologue
  const uint16_t *norm_shift;  // [rows, columns]
  const uint16_t *norm_bias;   // [columns]: LayerNormModulate (mean removed, weight and bias); nullptr = RMS
  uint64_t norm_rows_per_mod;  // rows that share one row of scale / shift
  Divisor norm_mod;            // by their number, where rows and it are below 2^31 (else 0)
  glue::RowStats norm_stats;   // per row (mean, inverse deviation)
  // Two fp32 -0, added to products of the norm. The assembler contracts mul.rn.f32x2 followed by add.rn.f32x2
  // into one fused operation (seen as single codes off by one), and an fma with a constant -0 as well; with
  // a -0 it cannot see, the product keeps its own rounding (x + -0 = x for every x, signed zeros included).
  uint64_t minus_zero2;
  uint32_t linear_follows; // the next kernel may start at once: a GEMM, which has its set-up (and weights) to do meanwhile
  unsigned long long wait_ns; // limit of a bounded wait, and where it is reported
  DeviceStatus *status;
  uint32_t withhold; // test aid: the first CTA waits for one announcement more of its second row than its warps make
};

// The 256-wide variants (2, 3, 5, 6), with or without residual outputs, weight packing or a norm in front.
int launch_convrot256(const QuantParams &p, int implementation, cudaStream_t stream);
int launch_convrot256_pack(const QuantParams &p, bool is_signed, bool f32, cudaStream_t stream);

#ifdef __CUDACC__

// Fixed Rademacher diagonal of the signed variants (reference cpu_executor.cpp:183-189).
__device__ __forceinline__ uint32_t sign_bit(uint32_t column) {
  uint32_t hash = column + 0x9e3779b9u;
  hash = (hash ^ (hash >> 16)) * 0x7feb352du;
  hash = (hash ^ (hash >> 15)) * 0x846ca68bu;
  hash ^= hash >> 16;
  return hash & 1u;
}

// One radix-4 butterfly on packed pairs, without the reference's exact factor 0.5.
__device__ __forceinline__ void bfly(uint64_t &x0, uint64_t &x1, uint64_t &x2, uint64_t &x3) {
  const uint64_t s = add2(x0, x1);
  const uint64_t t = sub2(x0, x1);
  const uint64_t y0 = sub2(add2(s, x2), x3);
  const uint64_t y1 = add2(sub2(s, x2), x3);
  const uint64_t y2 = add2(add2(t, x2), x3);
  // the reference forms (x1 - x0) + x2: x1 - x0 = -t exactly, and (-t) + x2 = x2 - t
  const uint64_t y3 = add2(sub2(x2, t), x3);
  x0 = y0;
  x1 = y1;
  x2 = y2;
  x3 = y3;
}

__device__ __forceinline__ float absmax2(float m, uint64_t v) {
  float lo, hi;
  unpack2(v, lo, hi);
  asm("max.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(lo)), "f"(fabsf(hi))); // one three-input maximum
  return m;
}

// Correctly rounded fp32 quotient a/b from y = RN(1/b): two Markstein refinements.
__device__ __forceinline__ uint64_t div2_exact(uint64_t a, uint64_t y, uint64_t negb) {
  uint64_t q = mul2(a, y);
  uint64_t r = fma2(negb, q, a);
  q = fma2(r, y, q);
  r = fma2(negb, q, a);
  return fma2(r, y, q);
}
// bf16(a / b) for bf16 values a and b (8 significant bits each, integers V and S in [128, 255]
// times powers of two) needs no refinement at all: a rounding boundary of the quotient is M / 2^k
// with M odd in [257, 511], and |V / S - M / 2^k| = |2^k V - M S| / (S 2^k) is either 0 -- which
// would need the odd M > 255 to divide V <= 255, impossible -- or at least 2^-17 of the quotient,
// while a * RN(1 / b) is within 2^-23 of it. So the plain product rounds to the same bf16 value
// as the IEEE quotient, ties cannot occur, and a zero numerator gives zero.
__device__ __forceinline__ uint64_t div2_bf16(uint64_t a, uint64_t y) { return mul2(a, y); }

__device__ __forceinline__ uint32_t pack_bf16_pair(float lo, float hi) {
  uint32_t packed;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(hi), "f"(lo));
  return packed;
}
__device__ __forceinline__ uint32_t pack_bf16_pair(uint64_t v) {
  float lo, hi;
  unpack2(v, lo, hi);
  return pack_bf16_pair(lo, hi);
}
__device__ __forceinline__ uint64_t unpack_bf16_pair(uint32_t packed) {
  return pack2(__uint_as_float(packed << 16), __uint_as_float(packed & 0xffff0000u));
}
__device__ __forceinline__ uint64_t round_bf16_2(uint64_t v) { return unpack_bf16_pair(pack_bf16_pair(v)); }

// Quotients of packed bf16 pairs by one bf16 divisor, as bf16: v r1 + v r2 with the two bf16 parts of r = (1 + 6 / 2^23) / divisor,
// a product and a fused sum that rounds once. For every pair of 8-bit significands that is the rounded quotient, with the
// reciprocal anywhere between 1 + 2^-25 and 1 + 43 / 2^25 times the exact one, and the approximate one is within 2^-23.
// Beside the fp32 product and its rounding it saves the conversions on either side.
struct SplitReciprocal {
  uint32_t r1 = 0x3f803f80u, r2 = 0u; // 1 and 0: quotients made before
  // False where the divisor leaves no room for the low part, or quotients (of values up to `maximum`) could overflow.
  __device__ __forceinline__ bool of(float divisor, float maximum) {
    if (!(divisor < 0x1p110f && maximum < divisor * 0x1p40f))
      return false;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(divisor));
    r *= 0x1.00000cp+0f;
    r1 = pack_bf16_pair(r, r);
    const float low = r - __uint_as_float(r1 << 16);
    r2 = pack_bf16_pair(low, low);
    return true;
  }
  __device__ __forceinline__ uint32_t quotients(uint32_t v) const {
    uint32_t q;
    asm("{\n.reg .b32 t;\nmul.rn.bf16x2 t, %1, %3;\nfma.rn.bf16x2 %0, %1, %2, t;\n}" : "=r"(q) : "r"(v), "r"(r1), "r"(r2));
    return q;
  }
};
// The fp32 product's quotients, within +-1024 (NaN stays NaN): what codes are made of saturates long before.
__device__ __forceinline__ uint32_t bounded_quotients(uint32_t v, float recip) {
  uint32_t q = pack_bf16_pair(mul2(unpack_bf16_pair(v), pack2(recip, recip)));
  asm("min.NaN.bf16x2 %0, %0, %1;" : "+r"(q) : "r"(0x44804480u));
  asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(q) : "r"(0xc480c480u));
  return q;
}

__device__ __forceinline__ int sat_s8(float v) {
  int r;
  asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(r) : "f"(v));
  return r;
}

// INT8 codes of two quotients in the low 16 bits: round to nearest even, saturate, NaN gives 0. Two conversions to 32-bit integers
// and the saturating pack are one operation at half the issue rate; a conversion to 8 bits alone runs at an eighth of it.
// `above`: codes whose low 16 bits become the high ones.
__device__ __forceinline__ uint32_t code_bytes(float q0, float q1, uint32_t above = 0u) {
  uint32_t codes;
  asm("{\n.reg .b32 c0, c1;\ncvt.rni.s32.f32 c0, %1;\ncvt.rni.s32.f32 c1, %2;\ncvt.pack.sat.s8.s32.b32 %0, c1, c0, %3;\n}"
      : "=r"(codes)
      : "f"(q0), "f"(q1), "r"(above));
  return codes;
}
__device__ __forceinline__ uint32_t code_bytes(uint32_t q) { // of a packed pair of bf16 quotients
  return code_bytes(__uint_as_float(q << 16), __uint_as_float(q & 0xffff0000u));
}
__device__ __forceinline__ uint32_t code_bytes_127(float q0, float q1) { // not below -127
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(q0) : "f"(-127.0f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(q1) : "f"(-127.0f));
  return code_bytes(q0, q1);
}

// INT8 codes of a pair of bf16 quotients that are not NaN as (the bits of) two floats kCodeBias + code: clamped to
// [-128, 127], then rounded to the nearest even integer by the addition of 1.5 * 2^23.
constexpr float kCodeBias = 12582912.0f;
__device__ __forceinline__ void code_words(uint32_t q, uint32_t &c0, uint32_t &c1) {
  float f0, f1;
  asm("max.bf16x2 %0, %0, %1;" : "+r"(q) : "r"(0xc300c300u));
  asm("min.bf16x2 %0, %0, %1;" : "+r"(q) : "r"(0x42fe42feu));
  asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %2;\nadd.rn.f32.bf16 %0, lo, %3;\nadd.rn.f32.bf16 %1, hi, %3;\n}"
      : "=f"(f0), "=f"(f1)
      : "r"(q), "f"(kCodeBias));
  c0 = __float_as_uint(f0);
  c1 = __float_as_uint(f1);
}

// max * clip / 127 as the reference rounds it (IEEE product, IEEE quotient, then the guard): one
// Markstein step from RN(1/127) gives the correctly rounded quotient for every fp32 mantissa
// (checked exhaustively), and below 2^-90, where the residual could underflow, the guard decides.
__device__ __forceinline__ float row_scale(float maximum, float clip) {
  constexpr float kInv127 = 1.0f / 127.0f;
  const float a = __fmul_rn(maximum, clip);
  float q = __fmul_rn(a, kInv127);
  q = __fmaf_rn(__fmaf_rn(-127.0f, q, a), kInv127, q);
  if (!(a < 3.0e38f)) // inf and NaN as the plain division treats them
    q = a / 127.0f;
  return fmaxf(q, 1.0e-30f);
}

// QuantizeInt8Rows(Direct, clip 1) codes of 2 N neighbouring bf16 values v of a row whose largest magnitude is `maximum`, N even:
// the nearest even integer to the IEEE quotient RN(v / scale), scale = RN(maximum / 127), four codes per word. With V and M
// the significands (integers up to 255) of v and the maximum, v / scale is 127 V / (M 2^k) but for the rounding of the scale.
// * Where that is not the middle n + 1/2 of two integers it is at least 1 / (510 * 2^k) away from it, 2^-17 of the quotient:
//   any product v y with y within 2^-19 of 1 / scale rounds to the same integer.
// * It is the middle for v = +-maximum / 2, 63.5, and (127 being prime) for no other v unless M = 254. Whether the rounded
//   scale leaves the quotient at 63.5 or above (code 64) or below it (63) shows in 127 scale - maximum, which is exact; y
//   is moved by 2^-21 to that side.
// * M = 254 makes the scale a power of two: quotients, reciprocal and products are exact.
// One product and half a conversion per pair in the place of a division; rows that are not finite, or so small that the scale
// is the guard, are divided. (With a check of every product's distance from the middle instead: attention operands,
// B2 S4608 H24, 34 us, now 30; rotation of q and k with codes, 33272 x 24 rows, 144 and 125.)
template <int N>
__device__ __forceinline__ void direct_codes(const uint64_t (&v)[N], float maximum, float scale, uint32_t (&words)[N / 2]) {
  if (maximum < 3.0e38f && maximum > 1.3e-28f) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(scale));
    y = __fmaf_rn(__fmaf_rn(-scale, y, 1.0f), y, y);
    const float apart = __fmaf_rn(127.0f, scale, -maximum);
    y = __fmaf_rn(y, apart == 0.0f ? 0.0f : apart <= maximum * 3.0e-8f ? 0x1p-21f : -0x1p-21f, y);
    const uint64_t y2 = pack2(y, y);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      float q[4];
      unpack2(mul2(v[i], y2), q[0], q[1]);
      unpack2(mul2(v[i + 1], y2), q[2], q[3]);
      words[i >> 1] = code_bytes(q[0], q[1], code_bytes(q[2], q[3]));
    }
  } else {
    const float recip = __frcp_rn(scale);
    const uint64_t y2 = pack2(recip, recip), nb2 = pack2(-scale, -scale);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      float q[4];
      unpack2(div2_exact(v[i], y2, nb2), q[0], q[1]);
      unpack2(div2_exact(v[i + 1], y2, nb2), q[2], q[3]);
      words[i >> 1] = code_bytes_127(q[0], q[1]) | code_bytes_127(q[2], q[3]) << 16;
    }
  }
}

// ---- shared-memory access through 32-bit shared addresses (cheap address arithmetic) ----
__device__ __forceinline__ void sts128(uint32_t addr, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(x), "f"(y), "f"(z), "f"(w)
               : "memory");
}
template <int OFF>
__device__ __forceinline__ uint64_t lds64(uint32_t addr) {
  uint64_t v;
  asm volatile("ld.shared.b64 %0, [%1+%2];" : "=l"(v) : "r"(addr), "n"(OFF) : "memory");
  return v;
}
template <int OFF>
__device__ __forceinline__ void sts8(uint32_t addr, int v) {
  asm volatile("st.shared.u8 [%0+%1], %2;" ::"r"(addr), "n"(OFF), "r"(v) : "memory");
}
template <int OFF>
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u16 [%0+%1], %2;" ::"r"(addr), "n"(OFF), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ float lds32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// ---- 256-wide rotation: a warp's 1024 columns, 16 packed pairs per thread (layout: convrot256.cuh) ----
// Shared memory per warp: 4 groups x 256 fp32, two 16x32-word transposes whose rows are padded, so that every access is
// free of conflicts at a constant offset.
constexpr uint32_t kRowPitch = 144;             // bytes of a row of 16 pairs in the transpose
constexpr uint32_t kHalfBytes = 16 * kRowPitch; // a half-warp's area
constexpr int kWarpBytes256 = 2 * kHalfBytes;

// From 16 consecutive elements of two groups to elements 16 j + a of both, rotated and scaled by 16. Thread a of a half-warp
// writes its pairs as row a (wr_addr = area + kRowPitch a) and reads pair a of every row (rd_addr = area + 8 a).
__device__ __forceinline__ void rotate_pairs(uint64_t (&P)[16], uint32_t wr_addr, uint32_t rd_addr) {
  // stage 0 (stride 1) and stage 1 (stride 4)
#pragma unroll
  for (int q = 0; q < 4; ++q)
    bfly(P[4 * q], P[4 * q + 1], P[4 * q + 2], P[4 * q + 3]);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    bfly(P[q], P[q + 4], P[q + 8], P[q + 12]);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float x0, x1, x2, x3;
    unpack2(P[2 * c], x0, x1);
    unpack2(P[2 * c + 1], x2, x3);
    sts128(wr_addr + 16u * c, x0, x1, x2, x3);
  }
  __syncwarp();
#define DIFB200_READ_PAIR(J) P[J] = lds64<(J) * kRowPitch>(rd_addr);
  DIFB200_READ_PAIR(0) DIFB200_READ_PAIR(1) DIFB200_READ_PAIR(2) DIFB200_READ_PAIR(3)
  DIFB200_READ_PAIR(4) DIFB200_READ_PAIR(5) DIFB200_READ_PAIR(6) DIFB200_READ_PAIR(7)
  DIFB200_READ_PAIR(8) DIFB200_READ_PAIR(9) DIFB200_READ_PAIR(10) DIFB200_READ_PAIR(11)
  DIFB200_READ_PAIR(12) DIFB200_READ_PAIR(13) DIFB200_READ_PAIR(14) DIFB200_READ_PAIR(15)
#undef DIFB200_READ_PAIR
  __syncwarp();
  // Now P[j] = element 16*j + a of both groups. stage 2 (stride 16), stage 3 (stride 64).
#pragma unroll
  for (int q = 0; q < 4; ++q)
    bfly(P[4 * q], P[4 * q + 1], P[4 * q + 2], P[4 * q + 3]);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    bfly(P[q], P[q + 4], P[q + 8], P[q + 12]);
}

#endif // __CUDACC__

} // namespace difb200
