// QuantizeInt8Rows for sm_100a, the 256-wide ConvRot variants: orthogonal block rotation fused with
// per-row absmax INT8 quantisation. Semantics follow the reference opcode bit for bit (reference
// src/runtime/cpu_executor.cpp:124-307; generated GPU kernel src/compiler/compiler.cpp:635-845).
// bf16 is read once from HBM, codes and scales are written once.
//
// A 256-wide group is the Kronecker product H4 (x) H4 (x) H4 (x) H4, applied as four radix-4 stages with
// strides 1, 4, 16, 64 in exactly the reference's fp32 association order ((x0+x1)+x2)-x3 etc. The
// reference multiplies every stage by 0.5; a multiplication by a power of two commutes with fp32
// rounding, so the kernel skips it and carries values scaled by 16, folding the factor into the
// divisor. Results are bit-identical unless an intermediate leaves the normal fp32 range.
//
// Layout. A warp works on 4 groups (1024 columns) at a time; each thread owns 16 consecutive elements of
// two neighbouring groups as 16 packed fp32x2 registers (lane 0 of the pair = first group, lane 1 =
// second group), so every butterfly is one packed add/sub for two groups. Stages 0-1 run on the
// thread's own 16 elements; a 16x16 transpose through shared memory (padded rows, conflict-free)
// gives the thread the 16 elements of stride 16, on which stages 2-3 run.
//
// What bounds it: nothing alone. A warp's 1024 elements are about 430 instructions (13.5 per element and lane, 5 of them packed
// additions of two clocks), and with 24 warps per SM the FMA pipe is 57 % busy, the issue slots 63 % and the L1 and shared-memory
// pipe 69 % (9216 x 8192): 64 of its 112 accesses per block are the transpose, which fp32 sums between the stages need whole. Between
// rotation and quantisation the bf16 variants keep the values as packed bf16 (their result is defined on the rounded
// values), half the registers of fp32. The codes of a pair are made by one conversion and leave as 16 bits; as a
// conversion and a byte store per element they kept the quarter-rate unit busy for 256 clocks of a block, and a warp took three
// blocks at a time to save per-row work. Before -> now, us: 33272 x 3072 83.9 -> 71.8 (4.3 TB/s), 33272 x 8192 220.6 -> 181.7,
// 9216 x 12288 100.4 -> 78.8, 4608 x (3072 + 12288) 70.0 -> 54.2, 2 x 3072 2.8 -> 2.6, the scale search of the weight form
// 12288 x 3072 64.7 -> 56.5 (all lanes evaluate samples, in doubles only where candidates are close), with input
// equalisation 94.2 -> 63.1 (a table of reciprocals, packed sums), RmsNormModulate in front of 16384 x 3072 92.0 -> 85.3 with its
// statistic. Staging the input with bulk copies through shared memory instead of registers gave nothing, nor (3 to 8 % slower) did
// scale and shift of a norm's next row prefetched into L2.
#pragma once
#include "ptx.cuh"
#include "quant_common.cuh"

namespace difb200 {
namespace {

// Shared memory per warp: the rotation's transpose, reused for the code pairs and the sampled elements of the scale search.
constexpr int kWarpBytes = kWarpBytes256;
constexpr uint32_t kCodeHalfBytes = 544, kCodeBytes = 2 * kCodeHalfBytes; // code pairs of a half-warp's two groups, of a block

// kPack: weight rows with the scale search, kEqualise: with input equalisation, kPackEqualise: with both, kPackTable: with both
// and a table of the equalisation's reciprocals. kNorm: RmsNormModulate in front, kLayer: LayerNormModulate (one kernel that looked
// at its parameters for which it is took 473 us for 33272 x 8192 in the RMS form, 449 so, 8318 x 3072 49.2 and 47.2).
enum Extra { kPlain = 0, kPack = 1, kNorm = 2, kEqualise = 3, kPackEqualise = 4, kPackTable = 5, kLayer = 6 };
__host__ __device__ constexpr bool searches(int extra) { return extra == kPack || extra == kPackEqualise || extra == kPackTable; }
__host__ __device__ constexpr bool norms(int extra) { return extra == kNorm || extra == kLayer; }
__host__ __device__ constexpr bool equalises(int extra) { return extra == kEqualise || extra == kPackEqualise || extra == kPackTable; }

// Shared memory of a CTA: per warp the transpose / staging area and the row maxima; for the signed variants 16 XOR masks per
// thread and block (with input equalisation the signs are in its table); the sums of the scale search; that table.
template <bool SIGNED, int EXTRA, int NIT>
__host__ __device__ constexpr uint32_t sums_offset(uint32_t warps) {
  return warps * kWarpBytes + warps * 16u + 64u + (SIGNED && EXTRA != kPackTable ? warps * 32u * 64u * NIT : 0u);
}
template <bool SIGNED, int EXTRA, int NIT>
__host__ __device__ constexpr uint32_t table_offset(uint32_t warps) {
  return (sums_offset<SIGNED, EXTRA, NIT>(warps) + (searches(EXTRA) ? warps * 7u * (uint32_t)(sizeof(double) + sizeof(float)) : 0u) + 15u) & ~15u;
}
constexpr uint32_t kTableBlockBytes = 8192; // of 1024 columns: [16][32 lanes] x 16 bytes, pairs of high parts, then of low parts

// 32 bytes of one thread: one 256-bit load where every run starts on 32 bytes, else two of 128 bits.
__device__ __forceinline__ void load_run(const uint4 *src, bool wide, uint4 &a, uint4 &b) {
  if (wide) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "l"(src));
  } else {
    a = load_global(src);
    b = load_global(src + 1);
  }
}

// AHEAD: the next row is rotated before one is finished.
template <bool SIGNED, bool F32, bool RESIDUAL, int EXTRA, int NIT, bool PREFETCH, int MAXT, int MINB, bool AHEAD>
__global__ void __launch_bounds__(MAXT, MINB)
convrot256_kernel(const QuantParams p, const int warps_per_row, const int rows_per_cta) {
  static_assert(!norms(EXTRA) || NIT == 1, "the row's barrier separates reading its statistic from writing its codes");
  static_assert(!F32 || NIT == 1, "the fp32 variants keep fp32 values: one block per warp");
  extern __shared__ __align__(128) uint32_t smem[];
  const uint64_t after = grid_dependency_wait_zero(); // in the address of every load
  if (p.linear_follows || p.rows <= (uint64_t)gridDim.x * rows_per_cta)
    grid_dependents_launch();
  constexpr bool kEqualised = equalises(EXTRA), kTable = EXTRA == kPackTable, kFlips = SIGNED && !kTable;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = warp / warps_per_row;         // which row of this CTA's batch
  const int wrow = warp - slot * warps_per_row;  // warp index inside the row
  const int h = lane >> 4, a = lane & 15;
  const int total_warps = blockDim.x >> 5;
  const uint32_t smem_addr = smem_u32(smem);
  const uint32_t warp_addr = smem_addr + warp * kWarpBytes;
  float *red = reinterpret_cast<float *>(smem + total_warps * (kWarpBytes / 4)); // [2][2][total_warps], AHEAD [4][total_warps]
  const float clip = p.clip_device ? load_global(p.clip_device + after) : p.clip;
  constexpr float kCarry = 16.0f; // the values carried through the rotation are scaled by 2^stages
  const uint32_t columns = p.columns;
  const uint32_t col_warp = (uint32_t)wrow * (NIT * 1024u);
  const uint32_t col0 = col_warp + 512u * h + 16u * a; // this thread's run in the first group of block 0

  // Rows of more than 12 blocks are one CTA per SM, whose 13 to 16 warps a barrier per row would stop together. With AHEAD a warp
  // announces its maximum (an mbarrier for each of four rows) and looks for the others' when it has rotated its block of the next row.
  static_assert(!AHEAD || (EXTRA == kPlain && PREFETCH && !F32 && !RESIDUAL && NIT == 1), "");
  if (AHEAD) {
    if (threadIdx.x == 0) {
      for (uint32_t i = 0; i < 4u; ++i)
        ptx::mbar_init(smem_addr + (uint32_t)total_warps * (kWarpBytes + 16u) + 8u * i,
                       (uint32_t)total_warps + (p.withhold != 0u && blockIdx.x == 0u && i == 1u ? 1u : 0u));
      ptx::fence_barrier_init();
    }
    __syncthreads();
  }

  // Transpose: thread a writes its 16 pairs as row a and reads pair a of every row j.
  const uint32_t wr_addr = warp_addr + h * kHalfBytes + kRowPitch * a; // + 16 c
  const uint32_t rd_addr = warp_addr + h * kHalfBytes + 8u * a;        // + kRowPitch j
  // The two codes that belong together, of the same element of both groups, are staged as 16 bits: element 16 j + a in
  // row j of 32 bytes, whose two 16-byte chunks change places in rows 4-7 and 12-15 (a thread reads whole rows).
  const uint32_t code_wr = warp_addr + h * kCodeHalfBytes + ((uint32_t)(a >> 3) << 4) + 2u * (a & 7u); // ^ 16, + 32 j
  const uint32_t code_rd = warp_addr + h * kCodeHalfBytes + 32u * a + (((uint32_t)a >> 2 & 1u) << 4);  // ^ 16 c

  // Sign flips of this thread's columns as XOR masks on the packed bf16 pairs (bits 15 and 31 of
  // word i: elements 2i and 2i+1), kept in shared memory: per block four 16-byte vectors per thread
  // (two per group), vector q of all threads contiguous.
  const uint32_t mask_step = blockDim.x * 16u;
  const uint32_t mask_addr = smem_addr + (uint32_t)total_warps * (kWarpBytes + 16u) + 64u + threadIdx.x * 16u;
  if (kFlips) {
#pragma unroll 1
    for (int q = 0; q < 4 * NIT; ++q) {
      const uint32_t c = col0 + (uint32_t)(q >> 2) * 1024u + (uint32_t)((q >> 1) & 1) * 256u + 8u * (q & 1);
      uint32_t m[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        m[i] = (sign_bit(c + 2 * i) << 15) | (sign_bit(c + 2 * i + 1) << 31);
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(mask_addr + q * mask_step), "r"(m[0]), "r"(m[1]),
                   "r"(m[2]), "r"(m[3])
                   : "memory");
    }
  }
  // Input equalisation divides every row by the same vector e: the CTA's rows share a table of 1 / e as the sum of two fp32 numbers,
  // good to 2^-48, so that w / e is a product and a fused sum. (The quotient of two 8-bit significands is never within 2^-33 of a
  // rounding boundary of fp32.) Reciprocal, residual and correction in every row: packing 12288 x 3072 with
  // the search 70.0 us, with the table and the prefetch that its registers allow 63.1 (16384 rows, seven full rounds, 91.0 and 77.4).
  const uint32_t table_addr = smem_addr + table_offset<SIGNED, EXTRA, NIT>((uint32_t)total_warps);
  bool equalise_fast = true; // this warp's entries are of ordinary magnitude
  if (kTable) {
    for (uint32_t i = threadIdx.x; i < ((columns + 1023u) >> 10) * 32u; i += blockDim.x) { // one lane's runs of one block
      const uint32_t c = (i >> 5) * 1024u + 512u * ((i >> 4) & 1u) + 16u * (i & 15u), to = table_addr + (i >> 5) * kTableBlockBytes + (i & 31u) * 16u;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint4 one = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
        const uint4 *ep = reinterpret_cast<const uint4 *>(p.equalise + after + c) + half;
        const uint4 ea4 = c < columns ? load_global(ep) : one, eb4 = c + 256u < columns ? load_global(ep + 32) : one;
        const uint32_t ea[4] = {ea4.x, ea4.y, ea4.z, ea4.w}, eb[4] = {eb4.x, eb4.y, eb4.z, eb4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float e[4] = {__uint_as_float(ea[k] << 16), __uint_as_float(eb[k] << 16), __uint_as_float(ea[k] & 0xffff0000u),
                              __uint_as_float(eb[k] & 0xffff0000u)};
          float high[4], low[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (SIGNED && sign_bit(c + 256u * (j & 1u) + 8u * half + 2u * k + (j >> 1)))
              e[j] = -e[j];
            high[j] = __frcp_rn(e[j]);
            low[j] = __fmul_rn(__fmaf_rn(-e[j], high[j], 1.0f), high[j]);
          }
          sts128(to + (4u * half + k) * 512u, high[0], high[1], high[2], high[3]);
          sts128(to + (8u + 4u * half + k) * 512u, low[0], low[1], low[2], low[3]);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8 * NIT; ++q) {
      if (col0 + 1024u * (q >> 3) < columns) {
        const uint4 h = lds128(table_addr + ((uint32_t)wrow * NIT + (q >> 3)) * kTableBlockBytes + (q & 7u) * 512u + lane * 16u);
        const uint32_t high[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          equalise_fast = equalise_fast && fabsf(__uint_as_float(high[i])) > 1.0e-9f && fabsf(__uint_as_float(high[i])) < 1.0e9f;
      }
    }
    equalise_fast = __all_sync(0xffffffffu, equalise_fast);
  } else if (kEqualised) {
#pragma unroll
    for (int q = 0; q < 2 * NIT; ++q) {
      const uint32_t c = col0 + (uint32_t)(q >> 1) * 1024u + (uint32_t)(q & 1) * 256u;
      if (c < columns) {
        const uint4 *ep = reinterpret_cast<const uint4 *>(p.equalise + after + c);
        const uint4 e0 = load_global(ep), e1 = load_global(ep + 1);
        const uint32_t w[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float lo = fabsf(__uint_as_float(w[i] << 16)), hi = fabsf(__uint_as_float(w[i] & 0xffff0000u));
          equalise_fast = equalise_fast && lo > 1.0e-9f && lo < 1.0e9f && hi > 1.0e-9f && hi < 1.0e9f;
        }
      }
    }
    equalise_fast = __all_sync(0xffffffffu, equalise_fast);
  }

  // The 64 bytes of a thread's two runs in block `it` of a row. Widths of concatenated inputs are
  // multiples of 16, so a run never straddles two of them.
  auto run_of = [&](uint64_t row, uint32_t c) {
    if (p.part_count == 1)
      return reinterpret_cast<const uint4 *>(p.part[0] + after + row * columns + c);
    uint32_t i = 0;
    while (c >= p.width[i])
      c -= p.width[i++];
    return reinterpret_cast<const uint4 *>(p.part[i] + after + row * p.width[i] + c);
  };
  // With one block per warp the runs of a thread are in the same place of every row: looked up once. (Not where
  // registers are short: the fp32 form with 64 of them spills, 9216 x 15360 147 -> 156 us.)
  constexpr bool kPlaced = NIT == 1 && EXTRA == kPlain && !RESIDUAL && !(F32 && !SIGNED && MAXT * MINB > 768);
  const uint16_t *src_a = p.part[0] + after + col0, *src_b = src_a + 256;
  uint32_t pitch_a = columns, pitch_b = columns;
  if (kPlaced && p.part_count > 1) {
    auto place = [&](uint32_t c, const uint16_t *&src, uint32_t &pitch) {
      uint32_t i = 0;
      while (c >= p.width[i])
        c -= p.width[i++];
      src = p.part[i] + after + c;
      pitch = p.width[i];
    };
    if (col0 < columns)
      place(col0, src_a, pitch_a);
    if (col0 + 256u < columns)
      place(col0 + 256u, src_b, pitch_b);
  }
  auto fetch = [&](uint64_t row, int it, uint4 (&v)[4]) {
    v[0] = v[1] = v[2] = v[3] = make_uint4(0, 0, 0, 0);
    const uint32_t c = col0 + 1024u * it;
    if (row < p.rows) {
      // A prefetch must not wait for what it requests: its loads are predicated, without a branch that they would have
      // to return from (one width, places known).
      constexpr bool kPredicated = PREFETCH && kPlaced;
      if (c < columns)
        load_run(kPlaced ? reinterpret_cast<const uint4 *>(src_a + row * pitch_a) : run_of(row, c),
                 !kPredicated && p.wide != 0, v[0], v[1]);
      if (c + 256u < columns)
        load_run(kPlaced ? reinterpret_cast<const uint4 *>(src_b + row * pitch_b) : run_of(row, c + 256u),
                 !kPredicated && p.wide != 0, v[2], v[3]);
    }
  };
  auto row_barrier = [&]() { // the warps of one row only; rows in flight do not wait for each other
    if (kTable && warps_per_row == 1)
      __syncwarp();
    else if (NIT == 1 || warps_per_row > 1)
      asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "r"(warps_per_row * 32) : "memory");
  };

  const uint64_t row_step = (uint64_t)gridDim.x * rows_per_cta;
  // Where a CTA has all rows of an SM, those of a last round are spread over the SMs (12288 x 3072 with the table 66.5 -> 63.1 us);
  // of smaller CTAs every SM gets its share of a last round anyway.
  uint64_t row = kTable ? (uint64_t)slot * gridDim.x + blockIdx.x : (uint64_t)blockIdx.x * rows_per_cta + slot;
  uint4 next[4];
  if (PREFETCH)
    fetch(row, 0, next);
  auto modulation_of = [&](uint64_t row) -> uint64_t {
    return p.norm_mod.by ? p.norm_mod.quotient((uint32_t)row) : row / p.norm_rows_per_mod;
  };
  // This warp's part of a row rotated: PF (fp32 variants) or V (bf16 variants, as bf16 pairs), and its largest magnitude.
  auto rotate_row = [&](uint64_t row, uint64_t(&PF)[F32 ? 16 : 1], uint32_t(&V)[F32 ? 1 : 16 * NIT]) {
    float m = 0.0f;
    float mean = 0.0f, inv = 0.0f;
    if (norms(EXTRA)) {
      // stands where this row's codes go: written behind the barrier of the row maximum, when all its warps have read it
      const float2 st = glue::row_stat(p.norm_stats, row);
      mean = st.x;
      inv = st.y;
    }
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      uint64_t P[16];
      {
        if (!PREFETCH)
          fetch(row, it, next);
        uint32_t wa[8] = {next[0].x, next[0].y, next[0].z, next[0].w, next[1].x, next[1].y, next[1].z, next[1].w};
        uint32_t wb[8] = {next[2].x, next[2].y, next[2].z, next[2].w, next[3].x, next[3].y, next[3].z, next[3].w};
        // software pipeline: the next block is requested before this one is processed
        if (PREFETCH) {
          if (it + 1 < NIT)
            fetch(row, it + 1, next);
          else
            fetch(row + row_step, 0, next);
        }
        const uint32_t c = col0 + 1024u * it;
        const bool act_a = c < columns, act_b = c + 256u < columns;
        if (norms(EXTRA)) {
          // The norm in front (reference cpu_executor.cpp:1241-1264 RmsNormModulate, :1108-1148
          // LayerNormModulate): the words are replaced by the bf16 result the unfused op would have
          // stored, rounding for rounding, two groups per packed operation.
          const uint64_t at = modulation_of(row) * columns + c + after;
          constexpr bool layer = EXTRA == kLayer;
          const bool weighted = p.norm_weight != nullptr;
          auto product = [&](uint64_t u, uint64_t v) { return fma2(u, v, p.minus_zero2); };
          const uint64_t inv2 = pack2(inv, inv), mean2 = pack2(mean, mean), one2 = pack2(1.0f, 1.0f);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const uint4 zero = make_uint4(0, 0, 0, 0), one = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
            auto pick = [&](const uint16_t *base, uint64_t index, bool active, const uint4 &other) {
              return active ? load_global(reinterpret_cast<const uint4 *>(base + index) + half) : other;
            };
            const uint4 sa4 = pick(p.norm_scale, at, act_a, zero), sb4 = pick(p.norm_scale, at + 256u, act_b, zero);
            const uint4 ha4 = pick(p.norm_shift, at, act_a, zero), hb4 = pick(p.norm_shift, at + 256u, act_b, zero);
            const uint4 ga4 = pick(p.norm_weight, c + after, act_a && weighted, one),
                        gb4 = pick(p.norm_weight, c + 256u + after, act_b && weighted, one);
            const uint4 ba4 = pick(p.norm_bias, c + after, act_a && layer, zero),
                        bb4 = pick(p.norm_bias, c + 256u + after, act_b && layer, zero);
            const uint32_t sa[4] = {sa4.x, sa4.y, sa4.z, sa4.w}, sb[4] = {sb4.x, sb4.y, sb4.z, sb4.w};
            const uint32_t ha[4] = {ha4.x, ha4.y, ha4.z, ha4.w}, hb[4] = {hb4.x, hb4.y, hb4.z, hb4.w};
            const uint32_t ga[4] = {ga4.x, ga4.y, ga4.z, ga4.w}, gb[4] = {gb4.x, gb4.y, gb4.z, gb4.w};
            const uint32_t ba[4] = {ba4.x, ba4.y, ba4.z, ba4.w}, bb[4] = {bb4.x, bb4.y, bb4.z, bb4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                auto pair_of = [&](uint32_t wa_, uint32_t wb_) {
                  return k ? pack2(__uint_as_float(wa_ & 0xffff0000u), __uint_as_float(wb_ & 0xffff0000u))
                           : pack2(__uint_as_float(wa_ << 16), __uint_as_float(wb_ << 16));
                };
                const uint64_t x2 = pair_of(wa[4 * half + i], wb[4 * half + i]);
                const uint64_t s2 = pair_of(sa[i], sb[i]), h2 = pair_of(ha[i], hb[i]), g2 = pair_of(ga[i], gb[i]);
                uint64_t y2;
                if (layer) { // intermediate bf16 roundings of the reference's LayerNormModulate
                  const uint64_t b2 = pair_of(ba[i], bb[i]);
                  const uint64_t n2 = round_bf16_2(add2(product(product(sub2(x2, mean2), inv2), g2), b2));
                  y2 = add2(round_bf16_2(product(n2, round_bf16_2(add2(one2, s2)))), h2);
                } else {
                  const uint64_t n2 = product(product(x2, inv2), g2);
                  y2 = add2(product(n2, add2(one2, s2)), h2);
                }
                P[8 * half + 2 * i + k] = y2;
              }
            }
          }
          // the bf16 result, and the sign flips of the signed variants on it
#pragma unroll
          for (int e = 0; e < 16; ++e)
            P[e] = round_bf16_2(P[e]);
          if ((columns & 1023u) != 0) { // groups that do not exist hold -mean / deviation: not for the row's maximum
            const uint64_t keep = (act_a ? 0xffffffffull : 0ull) | (act_b ? 0xffffffff00000000ull : 0ull);
#pragma unroll
            for (int e = 0; e < 16; ++e)
              P[e] &= keep;
          }
          if (SIGNED) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const uint4 ma4 = lds128(mask_addr + (4 * it + q) * mask_step), mb4 = lds128(mask_addr + (4 * it + 2 + q) * mask_step);
              const uint32_t ma[4] = {ma4.x, ma4.y, ma4.z, ma4.w}, mb[4] = {mb4.x, mb4.y, mb4.z, mb4.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                P[8 * q + 2 * i] ^= ((uint64_t)(mb[i] << 16) << 32) | (uint64_t)(ma[i] << 16);
                P[8 * q + 2 * i + 1] ^= ((uint64_t)(mb[i] & 0xffff0000u) << 32) | (uint64_t)(ma[i] & 0xffff0000u);
              }
            }
          }
        } else {
          if (kFlips) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const uint4 ma4 = lds128(mask_addr + (4 * it + q) * mask_step), mb4 = lds128(mask_addr + (4 * it + 2 + q) * mask_step);
              const uint32_t ma[4] = {ma4.x, ma4.y, ma4.z, ma4.w}, mb[4] = {mb4.x, mb4.y, mb4.z, mb4.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                wa[4 * q + i] ^= ma[i];
                wb[4 * q + i] ^= mb[i];
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            P[2 * i] = pack2(__uint_as_float(wa[i] << 16), __uint_as_float(wb[i] << 16));
            P[2 * i + 1] = pack2(__uint_as_float(wa[i] & 0xffff0000u), __uint_as_float(wb[i] & 0xffff0000u));
          }
          if (kEqualised) {
            // weight rows with input equalisation: w / e in fp32 before anything else (reference
            // tools/difflux2sample.cpp:3005-3014; the sign flip commutes with the division). Where a result is not finite
            // the division decides. Results below 2^-100 may be off by 2^-149: the row scale is at least 1e-30.
            auto number = [](const uint32_t(&w)[8], int i) { return __uint_as_float((i & 1) ? (w[i >> 1] & 0xffff0000u) : (w[i >> 1] << 16)); };
            auto entries = [&](uint32_t(&ea)[8], uint32_t(&eb)[8]) {
              const uint4 z = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u); // bf16 ones
              const uint4 *ep = reinterpret_cast<const uint4 *>(p.equalise + after + c);
              const uint4 e4[4] = {act_a ? load_global(ep) : z, act_a ? load_global(ep + 1) : z, act_b ? load_global(ep + 32) : z, act_b ? load_global(ep + 33) : z};
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint4 &va = e4[i >> 2], &vb = e4[2 + (i >> 2)];
                ea[i] = (i & 3) == 0 ? va.x : (i & 3) == 1 ? va.y : (i & 3) == 2 ? va.z : va.w;
                eb[i] = (i & 3) == 0 ? vb.x : (i & 3) == 1 ? vb.y : (i & 3) == 2 ? vb.z : vb.w;
              }
            };
            uint32_t ea[8], eb[8];
            if constexpr (kTable) {
              float most = 0.0f;
              if (equalise_fast) { // (of the warp)
                const uint32_t at = table_addr + ((uint32_t)wrow * NIT + it) * kTableBlockBytes + lane * 16u;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  const uint4 h = lds128(at + q * 512u), l = lds128(at + (8u + q) * 512u);
                  auto of = [](uint32_t a_, uint32_t b_) { return pack2(__uint_as_float(a_), __uint_as_float(b_)); };
                  P[2 * q] = fma2(P[2 * q], of(h.x, h.y), mul2(P[2 * q], of(l.x, l.y)));
                  P[2 * q + 1] = fma2(P[2 * q + 1], of(h.z, h.w), mul2(P[2 * q + 1], of(l.z, l.w)));
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  float lo, hi;
                  unpack2(P[i], lo, hi);
                  asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(fabsf(lo)), "f"(fabsf(hi)));
                }
              }
              if (!equalise_fast || !(most < INFINITY)) { // the words once more: they are not kept for this
                uint4 again[4];
                fetch(row, it, again);
                const uint32_t xa[8] = {again[0].x, again[0].y, again[0].z, again[0].w, again[1].x, again[1].y, again[1].z, again[1].w};
                const uint32_t xb[8] = {again[2].x, again[2].y, again[2].z, again[2].w, again[3].x, again[3].y, again[3].z, again[3].w};
                entries(ea, eb);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  P[i] = pack2(__fdiv_rn(number(xa, i), number(ea, i)), __fdiv_rn(number(xb, i), number(eb, i)));
                  if (SIGNED)
                    P[i] ^= (uint64_t)sign_bit(c + i) << 31 | (uint64_t)sign_bit(c + 256u + i) << 63;
                }
              }
            } else {
              // without a table: a reciprocal and one Markstein step, 2^-44 at most off, and a choice per result instead of a test of all
              entries(ea, eb);
              if (equalise_fast) { // (of the warp: a branch for every pair cost packing 12288 x 3072 a tenth)
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const float e0 = number(ea, i), e1 = number(eb, i);
                  float y0, y1;
                  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(e0));
                  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(e1));
                  const uint64_t y2 = pack2(y0, y1), q2 = mul2(P[i], y2);
                  float q0, q1, x0, x1;
                  unpack2(q2, q0, q1);
                  unpack2(fma2(fma2(pack2(-e0, -e1), q2, P[i]), y2, q2), x0, x1);
                  P[i] = pack2(x0 == x0 ? x0 : q0, x1 == x1 ? x1 : q1);
                }
              } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  float w0, w1;
                  unpack2(P[i], w0, w1);
                  P[i] = pack2(__fdiv_rn(w0, number(ea, i)), __fdiv_rn(w1, number(eb, i)));
                }
              }
            }
          }
        }
      }
      rotate_pairs(P, wr_addr, rd_addr);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        m = absmax2(m, P[j]);
        if (F32)
          PF[F32 ? j : 0] = P[j];
        else
          V[F32 ? 0 : 16 * it + j] = pack_bf16_pair(P[j]);
      }
    }

    // (the bits of a non-negative float order like integers)
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
  };
  auto maximum_of = [&](const float *maxima) { // of the row's warps
    const float m = lane < warps_per_row ? maxima[lane] : 0.0f;
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
  };
  // Scale, codes and residual outputs of a row whose largest rotated value is m.
  auto finish_row = [&](uint64_t row, uint64_t(&PF)[F32 ? 16 : 1], uint32_t(&V)[F32 ? 1 : 16 * NIT], float m, float *redp) {
    const float maximum = m * (1.0f / kCarry);
    float scale = row_scale(maximum, clip);
    if (searches(EXTRA)) {
      // The scale is the one of seven clipped candidates with the lowest squared error over every
      // fourth rotated element, the offline packer's rule (reference tools/difflux2sample.cpp:
      // 1225-1259). Those elements sit in the lanes with a % 4 == 0; they go through shared memory
      // so that all 32 lanes take an equal share. The reference evaluates in double: value and candidate have 8 significant bits and the code 8,
      // so value - code * candidate is exact in fp32 (15 bits at the granularity of either term)
      // and only its square and the sum need double. The sum's order differs from the reference's
      // sequential one, which matters only for candidates that tie to 1e-15.
      constexpr float factors[7] = {1.0f, 0.96f, 0.92f, 0.88f, 0.84f, 0.80f, 0.76f};
      const int samples = F32 ? 16 : 16 * NIT; // pairs per sampled lane
      if ((a & 3) == 0) {
#pragma unroll
        for (int i = 0; i < (F32 ? 16 : 16 * NIT); ++i)
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(warp_addr + 4u * (uint32_t)((lane >> 2) * samples + i)),
                       "r"(F32 ? pack_bf16_pair(PF[F32 ? i : 0]) : V[F32 ? 0 : i])
                       : "memory");
      }
      __syncwarp();
      float candidate[7], reciprocal[7];
#pragma unroll
      for (int f = 0; f < 7; ++f) {
        candidate[f] = round_bf16_number(row_scale(maximum, factors[f])) * kCarry;
        reciprocal[f] = __frcp_rn(candidate[f]);
      }
      // sums of the row's warps: doubles, then floats in an area of their own (rows of a CTA are not in step)
      double *errors = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(smem) +
                                                  sums_offset<SIGNED, EXTRA, NIT>((uint32_t)total_warps));
      float *sums = reinterpret_cast<float *>(errors + 7 * total_warps);
      auto sample = [&](int i) {
        uint32_t pair;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(pair) : "r"(warp_addr + 4u * i) : "memory");
        return pair;
      };
      // First in fp32: the value minus code times candidate is exact, and the at most 48 additions of squares leave a
      // sum within 3e-6 of the exact one. Where one candidate is better than the others by 1e-4 it is the answer;
      // else, and where the sums left the range of fp32, the doubles decide. (Doubles for every row -> this:
      // 12288 x 3072 78 -> 69 us, with input equalisation 110 -> 99 us.) Both barriers are passed on either way.
      float chosen = candidate[0];
      bool decided;
      {
        uint64_t e2[7] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
        const uint64_t bias2 = pack2(kCodeBias, kCodeBias);
#pragma unroll 1
        for (int i = lane; i < 8 * samples; i += 32) {
          const uint64_t v2 = unpack_bf16_pair(sample(i));
#pragma unroll
          for (int f = 0; f < 7; ++f) {
            uint32_t t0, t1;
            code_words(pack_bf16_pair(mul2(v2, pack2(reciprocal[f], reciprocal[f]))), t0, t1);
            const uint64_t minus2 = sub2(bias2, pack2(__uint_as_float(t0), __uint_as_float(t1)));
            const uint64_t d2 = fma2(minus2, pack2(candidate[f], candidate[f]), v2);
            e2[f] = fma2(d2, d2, e2[f]);
          }
        }
        float e[7];
#pragma unroll
        for (int f = 0; f < 7; ++f) {
          float lo, hi;
          unpack2(e2[f], lo, hi);
          e[f] = lo + hi;
        }
        // Halving: with every exchange a lane keeps half of its sums, so that lane l ends with candidate l / 4's (7: none).
        // 9 exchanges in the place of 35, and what follows is per lane instead of per candidate.
        float four[4], two[2];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const float upper = f < 3 ? e[f + 4] : 0.0f;
          four[f] = (lane & 16 ? upper : e[f]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? e[f] : upper, 16);
        }
#pragma unroll
        for (int f = 0; f < 2; ++f)
          two[f] = (lane & 8 ? four[f + 2] : four[f]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? four[f] : four[f + 2], 8);
        float own = (lane & 4 ? two[1] : two[0]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? two[0] : two[1], 4);
        own += __shfl_xor_sync(0xffffffffu, own, 2);
        own += __shfl_xor_sync(0xffffffffu, own, 1);
        const int mine = lane >> 2;
        if (warps_per_row > 1) {
          if ((lane & 3) == 0 && mine < 7)
            sums[mine * total_warps + warp] = own;
          row_barrier();
          own = 0.0f;
          for (int v = 0; v < warps_per_row; ++v)
            own += sums[(mine < 7 ? mine : 0) * total_warps + slot * warps_per_row + v];
        }
        const bool finite = own < INFINITY; // (sums of squares: not negative, or NaN)
        if (mine == 7 || !finite)
          own = INFINITY;
        const float best = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(own)));
        const uint32_t close = __ballot_sync(0xffffffffu, (lane & 3) == 0 && mine < 7 && own <= best * 1.0001f);
        const uint32_t all_finite = __ballot_sync(0xffffffffu, finite || mine == 7);
        const int which = close ? (__ffs((int)close) - 1) >> 2 : 0;
#pragma unroll
        for (int f = 1; f < 7; ++f)
          chosen = which == f ? candidate[f] : chosen;
        decided = __popc(close) == 1 && best > 1.0e-30f && all_finite == 0xffffffffu; // the same for every thread of the row
      }
      double e[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      if (!decided) {
#pragma unroll 1
        for (int i = lane; i < 8 * samples; i += 32) {
          const uint32_t pair = sample(i);
          const float v0 = __uint_as_float(pair << 16), v1 = __uint_as_float(pair & 0xffff0000u);
#pragma unroll
          for (int f = 0; f < 7; ++f) {
            const uint32_t q = pack_bf16_pair(__fmul_rn(v0, reciprocal[f]), __fmul_rn(v1, reciprocal[f]));
            // nearest-even integer by the magic constant 1.5 * 2^23 (|q| < 2^9)
            const float n0 = __fadd_rn(fminf(fmaxf(__uint_as_float(q << 16), -128.0f), 127.0f), 12582912.0f) - 12582912.0f;
            const float n1 =
                __fadd_rn(fminf(fmaxf(__uint_as_float(q & 0xffff0000u), -128.0f), 127.0f), 12582912.0f) - 12582912.0f;
            const double d0 = (double)__fmaf_rn(-n0, candidate[f], v0), d1 = (double)__fmaf_rn(-n1, candidate[f], v1);
            e[f] = fma(d0, d0, e[f]); // the square is exact in double: one rounding, as multiply then add
            e[f] = fma(d1, d1, e[f]);
          }
        }
#pragma unroll
        for (int f = 0; f < 7; ++f) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
            e[f] = __dadd_rn(e[f], __shfl_xor_sync(0xffffffffu, e[f], o));
          if (warps_per_row > 1 && lane == 0)
            errors[f * total_warps + warp] = e[f];
        }
      }
      if (warps_per_row > 1)
        row_barrier(); // (also: every warp has read the sums; the barriers of the next row keep the errors until they are read)
      if (!decided) {
        if (warps_per_row > 1) {
#pragma unroll
          for (int f = 0; f < 7; ++f) {
            e[f] = 0.0;
            for (int w = 0; w < warps_per_row; ++w)
              e[f] = __dadd_rn(e[f], errors[f * total_warps + slot * warps_per_row + w]);
          }
        }
        double best = e[0];
        chosen = candidate[0];
#pragma unroll
        for (int f = 1; f < 7; ++f)
          if (e[f] < best) {
            best = e[f];
            chosen = candidate[f];
          }
      }
      scale = maximum == 0.0f ? 1.0e-30f : chosen * (1.0f / kCarry);
      __syncwarp(); // the samples are read before the codes overwrite them
    }
    const float scale_bf16 = round_bf16_number(scale);
    const float stored = ((SIGNED || searches(EXTRA)) && !F32) ? scale_bf16 : scale;
    const float divisor = (F32 ? scale : scale_bf16) * kCarry;
    if (wrow == 0 && lane == 0)
      p.scales[row] = stored;
    constexpr bool kSplitQuotient = !F32 && !RESIDUAL;
    float recip = 0.0f;
    SplitReciprocal split;
    if (!kSplitQuotient || !split.of(divisor, maximum)) {
      recip = __frcp_rn(divisor);
      if (kSplitQuotient)
#pragma unroll
        for (int i = 0; i < (F32 ? 1 : 16 * NIT); ++i)
          V[i] = bounded_quotients(V[i], recip);
    }
    const uint64_t y2 = pack2(recip, recip), nb2 = pack2(-divisor, -divisor);

    // codes of pair i (block i / 16, element 16 (i % 16) + a), the first group's in the low byte
    auto code_pair = [&](int i) {
      if (F32) {
        float q0, q1;
        unpack2(div2_exact(PF[F32 ? i : 0], y2, nb2), q0, q1);
        return code_bytes_127(q0, q1);
      }
      const uint32_t v = V[F32 ? 0 : i];
      const uint32_t q = kSplitQuotient ? split.quotients(v) : pack_bf16_pair(div2_bf16(unpack_bf16_pair(v), y2));
      return code_bytes(q);
    };
    auto flush_codes = [&](int8_t *dst) { // every thread copies row a of both its groups
      __syncwarp();
      int8_t *to = dst + row * columns + col0;
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const uint4 x = lds128(code_rd + kCodeBytes * it), y = lds128((code_rd ^ 16u) + kCodeBytes * it);
        if (col0 + 1024u * it < columns)
          *reinterpret_cast<uint4 *>(to + 1024u * it) = make_uint4(__byte_perm(x.x, x.y, 0x6420), __byte_perm(x.z, x.w, 0x6420),
                                                                   __byte_perm(y.x, y.y, 0x6420), __byte_perm(y.z, y.w, 0x6420));
        if (col0 + 1024u * it + 256u < columns)
          *reinterpret_cast<uint4 *>(to + 1024u * it + 256u) = make_uint4(__byte_perm(x.x, x.y, 0x7531), __byte_perm(x.z, x.w, 0x7531),
                                                                          __byte_perm(y.x, y.y, 0x7531), __byte_perm(y.z, y.w, 0x7531));
      }
      __syncwarp();
    };
#define DIFB200_STAGE(J) sts16<32 * (J)>(((J) & 4) ? code_wr_odd : code_wr_even, emit(16 * it + (J)));
#define DIFB200_STAGE_ALL                                                                                     \
  _Pragma("unroll") for (int it = 0; it < NIT; ++it) {                                                        \
    const uint32_t code_wr_even = code_wr + kCodeBytes * it, code_wr_odd = (code_wr ^ 16u) + kCodeBytes * it; \
    DIFB200_STAGE(0) DIFB200_STAGE(1) DIFB200_STAGE(2) DIFB200_STAGE(3) DIFB200_STAGE(4) DIFB200_STAGE(5)     \
    DIFB200_STAGE(6) DIFB200_STAGE(7) DIFB200_STAGE(8) DIFB200_STAGE(9) DIFB200_STAGE(10) DIFB200_STAGE(11)   \
    DIFB200_STAGE(12) DIFB200_STAGE(13) DIFB200_STAGE(14) DIFB200_STAGE(15)                                   \
  }
    float rm = 0.0f;
    // Residuals of a pair (reference cpu_executor.cpp:262-305): r = fma(-code, stored, value).
    auto residual_pair = [&](int i, uint32_t codes, float &r0, float &r1) {
      float x0, x1;
      unpack2(F32 ? PF[F32 ? i : 0] : unpack_bf16_pair(V[F32 ? 0 : i]), x0, x1);
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
        redp[total_warps + warp] = rm;
      row_barrier();
      rm = lane < warps_per_row ? redp[total_warps + slot * warps_per_row + lane] : 0.0f;
      rm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(rm)));
      const float rscale = row_scale(rm, 1.0f);
      const float rscale_bf16 = round_bf16_number(rscale);
      if (wrow == 0 && lane == 0)
        p.rscales[row] = (SIGNED && !F32) ? rscale_bf16 : rscale;
      const float rdivisor = F32 ? rscale : rscale_bf16, rrecip = __frcp_rn(rdivisor);
      const uint64_t ry2 = pack2(rrecip, rrecip), rnb2 = pack2(-rdivisor, -rdivisor);
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
  };

  if constexpr (AHEAD) {
    const uint32_t bar = smem_addr + (uint32_t)total_warps * (kWarpBytes + 16u);
    uint64_t PF[1];
    uint32_t V[2][16];
    uint64_t before = 0; // the row that is rotated and not finished
    uint32_t turn = 0;
    auto step = [&](uint32_t(&mine)[16], uint32_t(&other)[16]) {
      const bool more = row < p.rows;
      if (more) {
        const float m = rotate_row(row, PF, mine);
        if (lane == 0) {
          red[(turn & 3u) * total_warps + warp] = m;
          ptx::mbar_arrive(bar + 8u * (turn & 3u));
        }
      }
      if (turn != 0u) {
        const uint32_t of = turn - 1u;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(bar + 8u * (of & 3u), (of >> 2) & 1u, p.wait_ns))) {
          if (lane == 0 && atomicExch(&p.status->flag, 1u) == 0u) {
            p.status->kernel = 1u;
            p.status->role = (uint32_t)warp;
            p.status->detail = of;
          }
          return false;
        }
        finish_row(before, PF, other, maximum_of(red + (of & 3u) * total_warps), red);
      }
      before = row;
      row += row_step;
      ++turn;
      return more;
    };
    while (step(V[0], V[1]) && step(V[1], V[0])) {
    }
    return;
  }
  for (uint32_t parity = 0; row < p.rows; row += row_step, parity ^= 1u) {
    uint64_t PF[F32 ? 16 : 1];
    uint32_t V[F32 ? 1 : 16 * NIT];
    float m = rotate_row(row, PF, V);
    float *redp = red + parity * 2 * total_warps;
    if (NIT == 1 || warps_per_row > 1) {
      if (lane == 0)
        redp[warp] = m;
      row_barrier();
      m = maximum_of(redp + slot * warps_per_row);
    }
    finish_row(row, PF, V, m, redp);
  }
}

template <bool SIGNED, bool F32, bool RESIDUAL, int EXTRA, int NIT, bool PREFETCH, int MAXT, int MINB, bool AHEAD = false>
int launch_form(const QuantParams &p, cudaStream_t stream) {
  const uint32_t groups = p.columns >> 8;
  const int warps_per_row = (int)((groups + 4u * NIT - 1u) / (4u * NIT));
  if (warps_per_row > MAXT / 32)
    return fail(kInternalError, "QuantizeInt8Rows: row too wide for this form");
  int rows_per_cta = (MAXT / 32 < 8 || EXTRA == kPackTable ? MAXT / 32 : 8) / warps_per_row;
  rows_per_cta = rows_per_cta < 1 ? 1 : rows_per_cta;
  if ((uint64_t)rows_per_cta > p.rows)
    rows_per_cta = (int)p.rows;
  if (EXTRA == kPackTable) { // all rows in flight on an SM share its table, as far as the rows go round
    const uint64_t share = (p.rows + sm_count() - 1) / sm_count();
    rows_per_cta = (uint64_t)rows_per_cta > share ? (int)share : rows_per_cta;
  }
  const int warps = warps_per_row * rows_per_cta, threads = warps * 32;
  const size_t smem = table_offset<SIGNED, EXTRA, NIT>((uint32_t)warps) +
                      (EXTRA == kPackTable ? (size_t)((p.columns + 1023u) >> 10) * kTableBlockBytes : 0);
  auto kernel = convrot256_kernel<SIGNED, F32, RESIDUAL, EXTRA, NIT, PREFETCH, MAXT, MINB, AHEAD>;
  int resident = 1;
  if (int rc = resident_blocks(reinterpret_cast<const void *>(kernel), threads, smem, &resident))
    return rc;
  const uint64_t batches = (p.rows + rows_per_cta - 1) / rows_per_cta;
  uint64_t grid = (uint64_t)sm_count() * resident; // persistent: as many CTAs as are resident at once
  grid = grid > batches ? batches : grid;
  return launch_ahead("convrot256_kernel launch", kernel, grid, threads, smem, stream, p, warps_per_row, rows_per_cta);
}

// The form of a row of `blocks` blocks of 1024 columns, one per warp: threads and CTAs per SM, and whether a warp requests
// its next row before it works on this one. Up to 8 blocks several rows share a CTA; wider rows are a CTA each, and two or
// three CTAs per SM hide one another's barriers. us per call, one block per warp with 80 registers, 24 warps per SM and a
// prefetch / 64 registers, 32 warps and none / 80 registers and none:
//   33272 x 3072 72.8 / 78.5 / 76.6, 16384 x 8192 91.9 / 99.0 / 102.4, 4608 x 12288 42.1 / 49.2 / 48.2,
//   9216 x 15360 (one CTA of 128 registers with a prefetch) 105.8 / 117.4 / -; signed 98.3 / 107.3 / 108.1 (8192),
//   fp32 106.5 / 112.1 / 111.5 (8192), but 13.0 / 13.1 / 12.3 (4159 x 3072). Three blocks per warp, which save per-row work, were
//   the best form before the codes were converted in pairs, and are no longer (9216 x 3072 23.2, now 21.5).
// Signed rows that are all resident at once want the shortest path (333 x 3072 4.1 / 4.4 / 4.4).
// A norm in front needs its registers for three tensors in flight (33272 x 3072 176 / 189 / 168), residual outputs
// are arithmetic (4000 x 8192 46.8 / 43.0 / 41.6).
template <bool SIGNED, bool F32, bool RESIDUAL, int EXTRA>
int launch_single(const QuantParams &p, cudaStream_t stream) {
  const uint32_t blocks = ((p.columns >> 8) + 3u) / 4u;
  // us without / with the next row rotated ahead: 4608 x 15360 55.8 / 54.2, 1000 14.4 / 13.6, 2000 x 16384 27.1 / 25.6, signed 28.8 / 27.4,
  // 13312 24.6 / 24.6; 200 x 15360 5.5 / 5.5, but 16 rows 3.4 / 3.6. (In fp32 the registers do not hold two rows.)
  if constexpr (EXTRA == kPlain && !RESIDUAL && !F32)
    if (blocks > 12u && p.rows > 2ull * (uint64_t)sm_count()) {
      QuantParams q = p;
      if (!q.status)
        q.status = device_status_words();
      const unsigned long long withheld = take_withheld_row_maximum();
      q.withhold = withheld != 0 ? 1u : 0u;
      q.wait_ns = withheld != 0 ? withheld : wait_limit_ns();
      if (q.status)
        return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, true, 512, 1, true>(q, stream);
    }
  if (blocks > 12u)
    return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, true, 512, 1>(p, stream);
  constexpr bool kArithmetic = EXTRA != kPlain || RESIDUAL;
  if (blocks > 8u)
    return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, !kArithmetic, 384, 2>(p, stream);
  if constexpr (!kArithmetic && SIGNED)
    if (p.rows * blocks <= (uint64_t)sm_count() * 16u)
      return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, true, 256, 2>(p, stream);
  if constexpr (!kArithmetic && F32 && !SIGNED)
    if (blocks <= 3u)
      return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, false, 256, 3>(p, stream);
  // Rows of 7 and 8 blocks are a CTA each: from as many as three CTAs per SM hold up to five for each SM the second round is
  // short, and its few CTAs want the shortest path. us with three / as here: 700 rows of 8192 columns 7.6 / 6.8, fp32 8.2 / 7.3,
  // signed 9.4 / 8.2, both 10.0 / 8.6; 592 of 7168 6.2 / 5.6, 6.8 / 5.9, 7.8 / 7.1, 8.6 / 7.4; 740 of 8192 7.4 / 7.2, 8.2 / 7.8,
  // 9.4 / 9.1, 10.2 / 9.8; at 445 within 3 %. Beyond, three hide more (4159 x 8192 26.6, four 28.0).
  if constexpr (!kArithmetic) {
    const uint64_t sms = (uint64_t)sm_count();
    if (blocks > 6u && p.rows > 3u * sms && p.rows <= 5u * sms) {
      if constexpr (SIGNED)
        return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, true, 256, 2>(p, stream);
      else
        return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, false, 256, 4>(p, stream);
    }
  }
  return launch_form<SIGNED, F32, RESIDUAL, EXTRA, 1, !kArithmetic, 256, 3>(p, stream);
}

} // namespace
} // namespace difb200
