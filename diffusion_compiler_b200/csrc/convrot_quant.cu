// QuantizeInt8Rows for sm_100a: the entry point, the 4096-wide ConvRot variants and the Direct variant
// (the 256-wide variants are in convrot256.cuh). Semantics follow the reference opcode bit for bit
// (reference src/runtime/cpu_executor.cpp:124-307; generated GPU kernel src/compiler/compiler.cpp:635-845).
#include "glue.h"
#include "ops.h"
#include "quant_common.cuh"

#include <cstdio>

namespace difb200 {
namespace {

// ---------------------------------------------------------------------------------------
// 4096-wide ConvRot: six radix-4 stages. A warp runs stages 0-3 on four 256-wide groups as the
// 256-wide kernel does (16 packed fp32x2 values per thread, one transpose per group through shared
// memory); a second, CTA-wide transpose across the 16 groups of a block gives every thread the
// elements of stages 4-5. One row per CTA.
// ---------------------------------------------------------------------------------------
constexpr int kWarpBytes = 4096;

// MAXT bounds the block, and with it the registers: 256 threads -> 3 blocks per SM, 384 -> 2, 512 -> 1.
template <bool F32, bool RESIDUAL, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT == 256 ? 3 : (MAXT == 384 ? 2 : 1))
convrot4096_kernel(const QuantParams p) {
  extern __shared__ __align__(128) uint32_t smem[];
  // The loads below are plain ones, which stay behind the wait; with the wait in the address of __ldg's the same
  // kernel took longer, from a graph: 700 x 4096 fp32 6.3 us, 5.5 so, 9216 x 12288 150 and 145.
  grid_dependency_wait();
  if (p.linear_follows)
    grid_dependents_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = lane >> 4, a = lane & 15;
  const int warps = blockDim.x >> 5;
  const uint32_t smem_addr = smem_u32(smem), warp_addr = smem_addr + warp * kWarpBytes;
  float *red = reinterpret_cast<float *>(smem + warps * (kWarpBytes / 4)); // [2][2][warps]
  const float clip = p.clip_device ? *p.clip_device : p.clip;
  constexpr float kCarry = 64.0f; // the values carried through the rotation are scaled by 2^stages
  const uint32_t columns = p.columns, col0 = 1024u * warp + 512u * h + 16u * a;

  // transpose addressing inside a group: see convrot256.cuh
  const uint32_t half_addr = warp_addr + h * 2048u;
  const uint32_t wr_addr = half_addr + 128u * a + ((a & 7u) << 4);
  const uint32_t rd_addr = half_addr + ((uint32_t)(a >> 1) << 4) + 8u * (a & 1u);
  // natural order of the row (fp32), and the two element positions whose 16 groups this thread combines
  const uint32_t nat_a = smem_addr + 4u * (1024u * warp + 512u * h + a), nat_b = nat_a + 1024u;
  const uint32_t u0 = threadIdx.x, u1 = threadIdx.x + (columns >> 5);
  const uint32_t c0 = (u0 >> 8) * 4096u + (u0 & 255u), c1 = (u1 >> 8) * 4096u + (u1 & 255u);
  const uint32_t rowbuf_a = smem_addr + 4u * c0, rowbuf_b = smem_addr + 4u * c1;
  const uint32_t code_a = smem_addr + c0 + ((c0 >> 9) << 6), code_b = smem_addr + c1 + ((c1 >> 9) << 6);
  const uint32_t copy_addr = smem_addr + (uint32_t)warp * 1152u + 16u * lane, copy_col = 1024u * warp + 16u * lane;

  // sign flips as XOR masks on the packed bf16 pairs, four 16-byte vectors per thread
  const uint32_t mask_addr = smem_addr + (uint32_t)warps * (kWarpBytes + 16u) + 64u + threadIdx.x * 16u;
  const uint32_t mask_step = blockDim.x * 16u;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    const uint32_t c = col0 + (uint32_t)(q >> 1) * 256u + 8u * (q & 1);
    uint32_t m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      m[i] = (sign_bit(c + 2 * i) << 15) | (sign_bit(c + 2 * i + 1) << 31);
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(mask_addr + q * mask_step), "r"(m[0]), "r"(m[1]),
                 "r"(m[2]), "r"(m[3])
                 : "memory");
  }
  auto fetch = [&](uint64_t row, uint4 (&v)[4]) {
    v[0] = v[1] = v[2] = v[3] = make_uint4(0, 0, 0, 0);
    if (row < p.rows) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t c = col0 + 256u * g, i = 0;
        while (c >= p.width[i])
          c -= p.width[i++];
        const uint4 *src = reinterpret_cast<const uint4 *>(p.part[i] + row * p.width[i] + c);
        v[2 * g] = src[0];
        v[2 * g + 1] = src[1];
      }
    }
  };
  uint4 next[4];
  fetch(blockIdx.x, next);
  uint32_t parity = 0;
  for (uint64_t row = blockIdx.x; row < p.rows; row += gridDim.x, parity ^= 1u) {
    uint64_t P[16];
    {
      uint32_t wa[8] = {next[0].x, next[0].y, next[0].z, next[0].w, next[1].x, next[1].y, next[1].z, next[1].w};
      uint32_t wb[8] = {next[2].x, next[2].y, next[2].z, next[2].w, next[3].x, next[3].y, next[3].z, next[3].w};
      fetch(row + gridDim.x, next); // the next row is requested before this one is processed
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint4 ma4 = lds128(mask_addr + q * mask_step), mb4 = lds128(mask_addr + (2 + q) * mask_step);
        const uint32_t ma[4] = {ma4.x, ma4.y, ma4.z, ma4.w}, mb[4] = {mb4.x, mb4.y, mb4.z, mb4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          wa[4 * q + i] ^= ma[i];
          wb[4 * q + i] ^= mb[i];
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        P[2 * i] = pack2(__uint_as_float(wa[i] << 16), __uint_as_float(wb[i] << 16));
        P[2 * i + 1] = pack2(__uint_as_float(wa[i] & 0xffff0000u), __uint_as_float(wb[i] & 0xffff0000u));
      }
    }
    auto two_stages = [&]() { // strides s and 4 s of the 16 values a thread holds
#pragma unroll
      for (int q = 0; q < 4; ++q)
        bfly(P[4 * q], P[4 * q + 1], P[4 * q + 2], P[4 * q + 3]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        bfly(P[q], P[q + 4], P[q + 8], P[q + 12]);
    };
    two_stages();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float x0, x1, x2, x3;
      unpack2(P[2 * c], x0, x1);
      unpack2(P[2 * c + 1], x2, x3);
      sts128(wr_addr ^ (uint32_t)(c << 4), x0, x1, x2, x3);
    }
    __syncwarp();
#define DIFB200_READ_PAIR(J) P[J] = lds64<(J) * 128>(rd_addr ^ (uint32_t)(((J) & 7) << 4));
    DIFB200_READ_PAIR(0) DIFB200_READ_PAIR(1) DIFB200_READ_PAIR(2) DIFB200_READ_PAIR(3)
    DIFB200_READ_PAIR(4) DIFB200_READ_PAIR(5) DIFB200_READ_PAIR(6) DIFB200_READ_PAIR(7)
    DIFB200_READ_PAIR(8) DIFB200_READ_PAIR(9) DIFB200_READ_PAIR(10) DIFB200_READ_PAIR(11)
    DIFB200_READ_PAIR(12) DIFB200_READ_PAIR(13) DIFB200_READ_PAIR(14) DIFB200_READ_PAIR(15)
#undef DIFB200_READ_PAIR
    __syncwarp();
    two_stages(); // P[j] = element 16*j + a of both groups
    // second transpose: this warp's 1024 columns in natural order, then 16 groups of one element position
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float x0, x1;
      unpack2(P[j], x0, x1);
      sts32(nat_a + 64u * j, x0);
      sts32(nat_b + 64u * j, x1);
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < 16; ++g)
      P[g] = pack2(lds32(rowbuf_a + 1024u * g), lds32(rowbuf_b + 1024u * g));
    two_stages();

    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      m = absmax2(m, P[j]);
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    float *redp = red + parity * 2 * warps;
    if (lane == 0)
      redp[warp] = m;
    __syncthreads(); // also: every read of the natural-order row is done before codes overwrite it
    m = lane < warps ? redp[lane] : 0.0f;
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    const float scale = row_scale(m * (1.0f / kCarry), clip), scale_bf16 = round_bf16_number(scale);
    const float stored = F32 ? scale : scale_bf16, divisor = stored * kCarry;
    constexpr bool kSplitQuotient = !F32 && !RESIDUAL; // the rotated values are packed as bf16 pairs for it
    uint32_t V[kSplitQuotient ? 16 : 1];
    if (kSplitQuotient)
#pragma unroll
      for (int j = 0; j < 16; ++j)
        V[kSplitQuotient ? j : 0] = pack_bf16_pair(P[j]);
    float recip = 0.0f;
    SplitReciprocal split;
    if (!kSplitQuotient || !split.of(divisor, m)) {
      recip = __frcp_rn(divisor);
      if (kSplitQuotient)
#pragma unroll
        for (int j = 0; j < 16; ++j)
          V[kSplitQuotient ? j : 0] = bounded_quotients(V[kSplitQuotient ? j : 0], recip);
    }
    const uint64_t y2 = pack2(recip, recip), nb2 = pack2(-divisor, -divisor);
    if (threadIdx.x == 0)
      p.scales[row] = stored;

    auto code_pair = [&](int i) { // the codes of both positions, the first's in the low byte
      if (F32) {
        float q0, q1;
        unpack2(div2_exact(P[i], y2, nb2), q0, q1);
        return code_bytes_127(q0, q1);
      }
      return code_bytes(kSplitQuotient ? split.quotients(V[kSplitQuotient ? i : 0]) : pack_bf16_pair(div2_bf16(round_bf16_2(P[i]), y2)));
    };
    auto flush_codes = [&](int8_t *dst) { // every lane copies 2 x 16 bytes of its warp's 1024 columns
      __syncthreads();
#pragma unroll
      for (int part = 0; part < 2; ++part)
        *reinterpret_cast<uint4 *>(dst + row * columns + copy_col + part * 512u) = lds128(copy_addr + part * 576u);
      __syncthreads();
    };
    // group J of a block sits 256 J columns on; one byte per column with a 64-byte skew per 512 columns
#define DIFB200_STAGE(J)                          \
  {                                               \
    const uint32_t codes = emit(J);               \
    sts8<256 * (J) + 64 * ((J) >> 1)>(code_a, (int)codes); \
    sts8<256 * (J) + 64 * ((J) >> 1)>(code_b, (int)(codes >> 8)); \
  }
#define DIFB200_STAGE_ALL                                                                                   \
  DIFB200_STAGE(0) DIFB200_STAGE(1) DIFB200_STAGE(2) DIFB200_STAGE(3) DIFB200_STAGE(4) DIFB200_STAGE(5)     \
  DIFB200_STAGE(6) DIFB200_STAGE(7) DIFB200_STAGE(8) DIFB200_STAGE(9) DIFB200_STAGE(10) DIFB200_STAGE(11)   \
  DIFB200_STAGE(12) DIFB200_STAGE(13) DIFB200_STAGE(14) DIFB200_STAGE(15)
    float rm = 0.0f;
    auto residual_pair = [&](int i, uint32_t codes, float &r0, float &r1) { // cpu_executor.cpp:262-305
      float x0, x1;
      unpack2(F32 ? P[i] : round_bf16_2(P[i]), x0, x1);
      r0 = __fmaf_rn(-(float)(int8_t)codes, stored, x0 * (1.0f / kCarry));
      r1 = __fmaf_rn(-(float)(int8_t)(codes >> 8), stored, x1 * (1.0f / kCarry));
    };
    {
      auto emit = [&](int i) {
        const uint32_t codes = code_pair(i);
        if (RESIDUAL) {
          float r0, r1;
          residual_pair(i, codes, r0, r1);
          asm("max.f32 %0, %0, %1, %2;" : "+f"(rm) : "f"(fabsf(r0)), "f"(fabsf(r1)));
        }
        return codes;
      };
      DIFB200_STAGE_ALL
    }
    flush_codes(p.codes);
    if (RESIDUAL) {
      rm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(rm)));
      if (lane == 0)
        redp[warps + warp] = rm;
      __syncthreads();
      rm = lane < warps ? redp[warps + lane] : 0.0f;
      rm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(rm)));
      const float rscale = row_scale(rm, 1.0f), rstored = F32 ? rscale : round_bf16_number(rscale);
      if (threadIdx.x == 0)
        p.rscales[row] = rstored;
      const float rrecip = __frcp_rn(rstored);
      const uint64_t ry2 = pack2(rrecip, rrecip), rnb2 = pack2(-rstored, -rstored);
      auto emit = [&](int i) {
        float r0, r1;
        residual_pair(i, code_pair(i), r0, r1);
        if (F32) {
          float q0, q1;
          unpack2(div2_exact(pack2(r0, r1), ry2, rnb2), q0, q1);
          return code_bytes_127(q0, q1);
        }
        return code_bytes(pack_bf16_pair(div2_bf16(round_bf16_2(pack2(r0, r1)), ry2)));
      };
      DIFB200_STAGE_ALL
      flush_codes(p.rcodes);
    }
#undef DIFB200_STAGE_ALL
#undef DIFB200_STAGE
  }
}

template <bool F32>
int launch_convrot4096(const QuantParams &p, cudaStream_t stream) {
  if (p.mse || p.equalise || p.norm_scale)
    return fail(kUnsupported, "QuantizeInt8Rows: weight packing (MSE scale, input equalisation) exists for "
                              "the 256-wide variants without residual outputs");
  const int warps = (int)(p.columns >> 10), threads = 32 * warps;
  const size_t smem = (size_t)warps * (kWarpBytes + 16 + 32 * 64) + 64;
  auto kernel = threads <= 256   ? (p.rcodes ? convrot4096_kernel<F32, true, 256> : convrot4096_kernel<F32, false, 256>)
                : threads <= 384 ? (p.rcodes ? convrot4096_kernel<F32, true, 384> : convrot4096_kernel<F32, false, 384>)
                                 : (p.rcodes ? convrot4096_kernel<F32, true, 512> : convrot4096_kernel<F32, false, 512>);
  int resident = 1;
  if (int rc = resident_blocks(reinterpret_cast<const void *>(kernel), threads, smem, &resident))
    return rc;
  uint64_t grid = (uint64_t)sm_count() * resident;
  grid = grid > p.rows ? p.rows : grid;
  return launch_ahead("convrot4096_kernel launch", kernel, grid, threads, smem, stream, p);
}

// ---------------------------------------------------------------------------------------
// Direct variant (no rotation; reference cpu_executor.cpp:232-260): one warp per row, any
// width. Used for activations of plain W8A8 linears and for the per-token-per-head
// quantisation of attention Q/K (rows of width 128).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float load_logical(const QuantParams &p, uint64_t after, uint64_t row, uint32_t column) {
  uint32_t c = column;
  for (uint32_t i = 0; i < p.part_count; ++i) {
    if (c < p.width[i])
      return bf16_bits_to_f32(load_global(p.part[i] + after + row * p.width[i] + c));
    c -= p.width[i];
  }
  return 0.0f;
}

template <bool VEC8>
__global__ void __launch_bounds__(256)
direct_quant_kernel(const QuantParams p) {
  const uint64_t after = grid_dependency_wait_zero();
  if (p.linear_follows)
    grid_dependents_launch();
  const int lane = threadIdx.x & 31;
  const uint64_t warp_global = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint64_t warp_count = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const float clip = p.clip_device ? load_global(p.clip_device + after) : p.clip;
  const uint32_t K = p.columns;
  for (uint64_t row = warp_global; row < p.rows; row += warp_count) {
    float m = 0.0f;
    if (VEC8) { // single part, width % 8 == 0, 16-byte aligned rows
      const uint4 *src = reinterpret_cast<const uint4 *>(p.part[0] + after + row * K);
      for (uint32_t c = lane; c < (K >> 3); c += 32) {
        const uint4 v = load_global(src + c);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          m = fmaxf(m, fabsf(__uint_as_float(w[i] << 16)));
          m = fmaxf(m, fabsf(__uint_as_float(w[i] & 0xffff0000u)));
        }
      }
    } else {
      for (uint32_t c = lane; c < K; c += 32)
        m = fmaxf(m, fabsf(load_logical(p, after, row, c)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float scale = fmaxf(__fdiv_rn(__fmul_rn(m, clip), 127.0f), 1.0e-30f);
    if (lane == 0)
      p.scales[row] = scale;
    const bool residual = p.rcodes != nullptr;
    float rm = 0.0f;
    if (VEC8) {
      const uint4 *src = reinterpret_cast<const uint4 *>(p.part[0] + after + row * K);
      uint2 *dst = reinterpret_cast<uint2 *>(p.codes + row * K);
      for (uint32_t c = lane; c < (K >> 3); c += 32) {
        const uint4 v = load_global(src + c);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t out[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float x0 = __uint_as_float(w[i] << 16), x1 = __uint_as_float(w[i] & 0xffff0000u);
          const int c0 = max(sat_s8(__fdiv_rn(x0, scale)), -127);
          const int c1 = max(sat_s8(__fdiv_rn(x1, scale)), -127);
          out[i >> 1] |= ((uint32_t)(c0 & 0xff) << (16 * (i & 1))) |
                         ((uint32_t)(c1 & 0xff) << (16 * (i & 1) + 8));
          if (residual) {
            rm = fmaxf(rm, fabsf(__fmaf_rn(-(float)c0, scale, x0)));
            rm = fmaxf(rm, fabsf(__fmaf_rn(-(float)c1, scale, x1)));
          }
        }
        dst[c] = make_uint2(out[0], out[1]);
      }
    } else {
      for (uint32_t c = lane; c < K; c += 32) {
        const float x = load_logical(p, after, row, c);
        const int code = max(sat_s8(__fdiv_rn(x, scale)), -127);
        p.codes[row * K + c] = (int8_t)code;
        if (residual)
          rm = fmaxf(rm, fabsf(__fmaf_rn(-(float)code, scale, x)));
      }
    }
    if (residual) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        rm = fmaxf(rm, __shfl_xor_sync(0xffffffffu, rm, o));
      const float rscale = fmaxf(__fdiv_rn(rm, 127.0f), 1.0e-30f);
      if (lane == 0)
        p.rscales[row] = rscale;
      __syncwarp();
      for (uint32_t c = lane; c < K; c += 32) {
        const float x = load_logical(p, after, row, c);
        const float r = __fmaf_rn(-(float)p.codes[row * K + c], scale, x);
        p.rcodes[row * K + c] = (int8_t)max(sat_s8(__fdiv_rn(r, rscale)), -127);
      }
    }
  }
}

} // namespace

int quantize_int8_rows(const void *const *parts, const uint64_t *part_widths, uint32_t part_count,
                       uint64_t rows, int implementation, float clip, const float *clip_device,
                       int8_t *codes, float *scales, int8_t *rcodes, float *rscales,
                       cudaStream_t stream, bool mse_weight_scale, const void *equalise_bf16,
                       const NormPrologue *norm, bool linear_follows, DeviceStatus *status_words) {
  if (part_count == 0 || part_count > kMaxParts)
    return fail(kUnsupported, "QuantizeInt8Rows: 1..8 concatenated inputs are supported");
  if (!codes || !scales || (rcodes == nullptr) != (rscales == nullptr))
    return fail(kInvalidArgument, "QuantizeInt8Rows: missing output pointer");
  if (!(clip > 0.0f) && !clip_device)
    return fail(kInvalidArgument, "QuantizeInt8Rows: clip ratio must be positive");
  QuantParams p{};
  uint64_t columns = 0;
  bool aligned16 = true, aligned8 = true;
  p.wide = 1;
  for (uint32_t i = 0; i < part_count; ++i) {
    if (!parts[i] || part_widths[i] == 0 || part_widths[i] > 0xffffffffull)
      return fail(kInvalidArgument, "QuantizeInt8Rows: bad input part");
    p.part[i] = static_cast<const uint16_t *>(parts[i]);
    p.width[i] = (uint32_t)part_widths[i];
    columns += part_widths[i];
    p.wide = p.wide && (reinterpret_cast<uintptr_t>(parts[i]) & 31) == 0;
    aligned16 = aligned16 && part_widths[i] % 16 == 0 && (reinterpret_cast<uintptr_t>(parts[i]) & 15) == 0;
    aligned8 = aligned8 && part_widths[i] % 8 == 0 && (reinterpret_cast<uintptr_t>(parts[i]) & 15) == 0;
  }
  if (columns > 0xffffffffull)
    return fail(kUnsupported, "QuantizeInt8Rows: row too wide");
  p.part_count = part_count;
  p.columns = (uint32_t)columns;
  p.rows = rows;
  p.clip = clip;
  p.clip_device = clip_device;
  p.codes = codes;
  p.scales = scales;
  p.rcodes = rcodes;
  p.rscales = rscales;
  p.linear_follows = linear_follows ? 1u : 0u;
  p.status = status_words;
  p.mse = mse_weight_scale ? 1u : 0u;
  p.equalise = static_cast<const uint16_t *>(equalise_bf16);
  if (norm) {
    if (!norm->scale || !norm->shift)
      return fail(kInvalidArgument, "QuantizeInt8Rows: norm prologue without scale / shift");
    if (implementation < 2 || implementation == 4 || implementation == 7 || part_count != 1 || rcodes ||
        ((reinterpret_cast<uintptr_t>(norm->scale) | reinterpret_cast<uintptr_t>(norm->shift) |
          reinterpret_cast<uintptr_t>(norm->weight) | reinterpret_cast<uintptr_t>(norm->bias)) & 15) ||
        norm->rows_per_modulation == 0 || (norm->bias && !norm->weight))
      return fail(kUnsupported, "QuantizeInt8Rows: the norm prologue needs one input, a 256-wide ConvRot variant, no "
                                "residual outputs and 16-byte aligned pointers");
    p.norm_weight = static_cast<const uint16_t *>(norm->weight);
    p.norm_scale = static_cast<const uint16_t *>(norm->scale);
    p.norm_shift = static_cast<const uint16_t *>(norm->shift);
    p.norm_bias = static_cast<const uint16_t *>(norm->bias);
    p.minus_zero2 = 0x8000000080000000ull;
    p.norm_rows_per_mod = norm->rows_per_modulation;
    if (rows < (1ull << 31) && norm->rows_per_modulation < (1ull << 31))
      p.norm_mod = divisor(norm->rows_per_modulation);
  }
  if (rows == 0)
    return kOk;
  if ((mse_weight_scale || equalise_bf16) && (implementation == 1 || clip_device || part_count != 1))
    return fail(kUnsupported, "QuantizeInt8Rows: weight packing applies to one input, the ConvRot variants and a "
                              "static clip");
  if (equalise_bf16 && (reinterpret_cast<uintptr_t>(equalise_bf16) & 15))
    return fail(kUnsupported, "QuantizeInt8Rows: the equalisation vector must be 16-byte aligned");
  if (implementation == 1) {
    const int threads = 256;
    uint64_t blocks = (rows + 7) / 8;
    const uint64_t cap = (uint64_t)sm_count() * 16;
    if (blocks > cap)
      blocks = cap;
    if (part_count == 1 && columns == 128 && !rcodes && !clip_device) { // per token-head rows: a thread per row
      int rc = 0;
      if (glue::direct_quant_rows128(parts[0], codes, scales, rows, clip, stream, &rc))
        return rc;
    }
    const bool vec = part_count == 1 && aligned8 && (reinterpret_cast<uintptr_t>(codes) & 7) == 0;
    return launch_ahead("direct_quant_kernel launch", vec ? direct_quant_kernel<true> : direct_quant_kernel<false>, blocks, threads, 0, stream, p);
  }
  if (implementation < 2 || implementation > 7)
    return fail(kInvalidArgument, "QuantizeInt8Rows: unknown implementation");
  const bool h4096 = implementation == 4 || implementation == 7;
  if (columns % (h4096 ? 4096u : 256u) != 0)
    return fail(kInvalidArgument, "QuantizeInt8Rows: width is not a multiple of the rotation group");
  if (columns > 16384) // 16 warps of 1024 columns: one limit for every form, whatever the number of rows
    return fail(kUnsupported, "QuantizeInt8Rows: ConvRot width above 16384 is not supported");
  if (!aligned16 || (reinterpret_cast<uintptr_t>(codes) & 15) != 0 ||
      (rcodes && (reinterpret_cast<uintptr_t>(rcodes) & 15) != 0))
    return fail(kUnsupported,
                "QuantizeInt8Rows: ConvRot path needs 16-byte aligned pointers and part widths "
                "that are multiples of 16");
  StreamScratch scratch(stream);
  if (norm) { // the row statistic, by its own kernel in front: only now that nothing above refuses the call
    const uint64_t vector = columns * 2, mods = (rows + norm->rows_per_modulation - 1) / norm->rows_per_modulation * vector;
    if (int rc = glue::row_stats(parts[0], rows, columns, norm->epsilon, norm->bias != nullptr, true, codes, columns,
                                 {{norm->weight, vector}, {norm->bias, vector}, {norm->scale, mods}, {norm->shift, mods}},
                                 scratch, &p.norm_stats, stream))
      return rc;
  }
  if (!h4096)
    return launch_convrot256(p, implementation, stream);
  return implementation == 4 ? launch_convrot4096<false>(p, stream) : launch_convrot4096<true>(p, stream);
}

} // namespace difb200
