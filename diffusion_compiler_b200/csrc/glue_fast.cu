// bf16 fast paths of the block-glue kernels that carry most of a DiT block's non-GEMM,
// non-attention time: every access is 16 bytes (8 bf16), rows stay in registers between the
// statistic and the normalisation, and the per-(token, head) operators give one thread a whole
// 128-wide row. Arithmetic and rounding points are those of the generic kernels in glue.cu (and
// therefore of the reference CPU executor; file:line per kernel, paths in the reference project).
// glue.cu selects these when dtype, widths and alignment allow and falls back otherwise.
#include "glue.h"

#include "common.cuh"
#include "quant_common.cuh"

#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace difb200 {
namespace glue {
namespace {

__device__ __forceinline__ void unpack8(const uint4 v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t packed;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(hi), "f"(lo));
  return packed;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                    pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

#define GRID_STRIDE(i, n)                                                                     \
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n);                 \
       i += (uint64_t)gridDim.x * blockDim.x)

// ---- ResidualGate (cpu_executor.cpp:1703-1719): out = res + gate * branch ----
__global__ void __launch_bounds__(256)
k_residual_gate_bf16(const uint4 *res, const uint4 *branch, const uint4 *gate, uint4 *o, uint64_t groups,
                     uint64_t width8, uint64_t rows_per_gate) {
  const uint64_t after = grid_dependency_wait_zero();
  res += after;
  branch += after;
  gate += after;
  GRID_STRIDE(i, groups) {
    const uint64_t row = i / width8, col = i - row * width8;
    float r[8], b[8], g[8], y[8];
    unpack8(load_global(res + i), r);
    unpack8(load_global(branch + i), b);
    unpack8(load_global(gate + (row / rows_per_gate) * width8 + col), g);
#pragma unroll
    for (int e = 0; e < 8; ++e)
      y[e] = __fadd_rn(r[e], __fmul_rn(g[e], b[e]));
    o[i] = pack8(y);
  }
}

// ---- SwiGlu (cpu_executor.cpp:1267-1286): out = value * (gate / (1 + exp(-gate))) ----
// Near HBM's rate, with the issue slots next (an exponential and a division per element), of which a 64-bit division per
// group of 8 elements took its share: 33272 x 8192 296 us, so 272 = 6.0 TB/s; 4608 x 12288 67 -> 61. The launch makes a
// reciprocal where that holds, for less than 2^31 groups. (ResidualGate, whose time is its bytes, gains nothing by it.)
struct Wide {
  uint64_t by;
  __device__ __forceinline__ uint64_t quotient(uint64_t n) const { return n / by; }
};
template <class D>
__global__ void __launch_bounds__(256)
k_swiglu_bf16(const uint4 *x, uint4 *o, uint64_t groups, const D width, uint64_t in_width8, uint64_t start8, int gate_first) {
  x += grid_dependency_wait_zero();
  const uint64_t width8 = width.by;
  GRID_STRIDE(i, groups) {
    const uint64_t row = width.quotient(i), col = i - row * width8, base = row * in_width8 + start8 + col;
    float value[8], gate[8], y[8];
    unpack8(load_global(x + base + (gate_first ? width8 : 0)), value);
    unpack8(load_global(x + base + (gate_first ? 0 : width8)), gate);
#pragma unroll
    for (int e = 0; e < 8; ++e)
      y[e] = __fmul_rn(value[e], __fdiv_rn(gate[e], __fadd_rn(1.0f, expf(-gate[e]))));
    o[i] = pack8(y);
  }
}


// ---- row statistics in the reference's sequential order ----
// The reference sums a row's squares (or values, then squared deviations) in one fp32 chain, column
// by column (cpu_executor.cpp:1051-1062 RmsNorm, 1119-1129 LayerNormModulate, 1250-1256
// RmsNormModulate). A parallel sum differs from that chain in the last bit of about one row in
// three, which flips one bf16 output in a few thousand -- and every ConvRot quantiser behind the
// norm amplifies such a flip across its 256-wide group. So the statistic is computed here in the
// reference's order: one lane per row walks its row sequentially. A warp owns 32 rows and moves them
// through shared memory 64 columns at a time (asynchronous 16-byte copies in coalesced 128-byte
// runs, rows 9 x 16 bytes apart so that lanes read their own rows without bank conflicts), four or eight
// chunks deep: a chunk takes a warp about 0.17 us, so seven in flight cover the HBM latency even with
// one or two warps on an SM.
// Squares of bf16 values are exact in fp32, so the
// fused multiply-add equals the reference's multiply followed by add; the deviations of the layer
// form are not, and get the two roundings. The mixed-precision adds and fused multiply-adds take the bf16
// operand as it is, so an element of the chain is one instruction (the layer form's second pass: three)
// and the kernel is bound by that chain -- cols dependent operations of about four clocks -- for few
// rows and by HBM for many.
constexpr int kStatCols = 64, kStatPitch = 9; // uint4 per row in shared memory (8 + 1 pad)
constexpr int kStatWarps = 2;                 // warps per CTA

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid) {
  // 16 bytes global -> shared, asynchronously; zero-filled when the row does not exist
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// acc after the two bf16 elements of a word, low half first. KIND 0: acc + x; 1: acc + x * x (exact
// square, one rounding).
template <int KIND>
__device__ __forceinline__ float accumulate_word(uint32_t word, float acc) {
  if (KIND == 0) {
    asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; add.rn.f32.bf16 %0, lo, %0; add.rn.f32.bf16 %0, hi, %0; }"
        : "+f"(acc) : "r"(word));
  } else {
    asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; fma.rn.f32.bf16 %0, lo, lo, %0; fma.rn.f32.bf16 %0, hi, hi, %0; }"
        : "+f"(acc) : "r"(word));
  }
  return acc;
}
// The squared deviations of a word's two elements, with the roundings of subtract and multiply. (volatile: stays where
// it is written, between the dependent sums)
__device__ __forceinline__ void deviations(uint32_t word, float mean, float &d0, float &d1) {
  asm volatile("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %2; sub.rn.f32.bf16 %0, lo, %3; sub.rn.f32.bf16 %1, hi, %3; }"
               : "=f"(d0), "=f"(d1) : "r"(word), "f"(mean));
}
__device__ __forceinline__ float square_in_place(float d) {
  float q;
  asm volatile("mul.rn.f32 %0, %1, %1;" : "=f"(q) : "f"(d));
  return q;
}
__device__ __forceinline__ void add_in_place(float &acc, float v) {
  asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(acc) : "f"(v));
}

// What the sequential kernel computes: the RMS statistic, the layer form's two, or of these the mean alone.
enum RowSums { kRms, kLayer, kMean };
__device__ __forceinline__ float inverse_deviation(float sum, uint32_t cols, float eps) {
  return __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(sum, (float)cols), eps)));
}
template <int SUMS, int STAGES>
__global__ void __launch_bounds__(32 * kStatWarps)
k_row_stats_sequential(const uint4 *x, const RowStats stats, uint64_t rows, uint32_t cols, float eps) {
  extern __shared__ uint4 stat_smem[];
  auto tile = reinterpret_cast<uint4 (*)[STAGES][32 * kStatPitch]>(stat_smem); // [kStatWarps]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t cols8 = cols >> 3, chunks = cols / kStatCols;
  for (uint64_t row0 = ((uint64_t)blockIdx.x * kStatWarps + warp) * 32; row0 < rows;
       row0 += (uint64_t)gridDim.x * kStatWarps * 32) {
    const uint64_t row = row0 + lane;
    // lane l copies, for j = 0..7, the 16 bytes (row0 + 4 j + l / 8, chunk column l % 8) of a chunk
    const uint4 *src = x + (row0 + (lane >> 3)) * cols8 + (lane & 7);
    const uint32_t slot = smem_u32(&tile[warp][0][(lane >> 3) * kStatPitch + (lane & 7)]);
    auto issue = [&](uint32_t chunk) { // no branch: past the last chunk the copies only zero-fill
      const uint32_t dst = slot + (chunk % STAGES) * (uint32_t)sizeof(tile[0][0]);
      const uint4 *from = src + chunk * (kStatCols / 8);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool valid = chunk < chunks && row0 + 4 * j + (lane >> 3) < rows;
        cp_async16(dst + 64u * j * kStatPitch, valid ? from + 4ull * j * cols8 : x, valid);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto read = [&](uint32_t chunk, uint4 (&v)[8]) {
      const uint4 *stage = tile[warp][chunk % STAGES] + lane * kStatPitch;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        v[c] = stage[c];
    };
    float mean = 0.0f, acc = 0.0f;
    auto pass = [&](auto kind) {
      auto chain = [&](const uint4 (&v)[8]) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          acc = accumulate_word<decltype(kind)::value>(v[c].x, acc);
          acc = accumulate_word<decltype(kind)::value>(v[c].y, acc);
          acc = accumulate_word<decltype(kind)::value>(v[c].z, acc);
          acc = accumulate_word<decltype(kind)::value>(v[c].w, acc);
        }
      };
      // The chunk after the one being summed is already in registers, and the requests sit between the
      // dependent sums, so that nothing but the chain itself takes time.
      auto advance = [&](uint32_t chunk, const uint4 (&v)[8], uint4 (&next)[8]) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 3) : "memory");
        __syncwarp();                 // chunk + 1 has landed for every lane, chunk - 1 has been summed by all
        issue(chunk + STAGES - 1);    // into the stage of chunk - 1
        read(chunk + 1, next);
        chain(v);
      };
      acc = 0.0f;
      __syncwarp();
      for (uint32_t c = 0; c < (uint32_t)STAGES - 1; ++c)
        issue(c);
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      __syncwarp();
      uint4 a[8], b[8];
      read(0, a);
      uint32_t chunk = 0;
#pragma unroll 1
      for (; chunk + 1 < chunks; chunk += 2) {
        advance(chunk, a, b);
        advance(chunk + 1, b, a);
      }
      if (chunk < chunks)
        chain(a);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    };
    // The second pass of the layer form, acc + (x - mean)^2: the squares of the next chunk are made between the sums of
    // this one, which alone depend on one another. (Subtract, multiply and add of an element one behind the other took
    // 16 us for 3072 columns, the chain of sums takes 7.)
    auto deviation_pass = [&]() {
      auto squares_of = [&](const uint4 (&v)[8], int w, float &q0, float &q1) {
        const uint32_t word = (w & 3) == 0 ? v[w >> 2].x : (w & 3) == 1 ? v[w >> 2].y : (w & 3) == 2 ? v[w >> 2].z : v[w >> 2].w;
        float d0, d1;
        deviations(word, mean, d0, d1);
        q0 = square_in_place(d0);
        q1 = square_in_place(d1);
      };
      auto advance = [&](uint32_t chunk, const float (&q)[64], float (&next)[64]) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 3) : "memory");
        __syncwarp();
        uint4 v[8];
        read(chunk + 1, v);
        issue(chunk + STAGES - 1);
#pragma unroll
        for (int w = 0; w < 32; ++w) {
          add_in_place(acc, q[2 * w]);
          if (w >= 4)
            squares_of(v, w - 4, next[2 * w - 8], next[2 * w - 7]);
          add_in_place(acc, q[2 * w + 1]);
        }
#pragma unroll
        for (int w = 28; w < 32; ++w)
          squares_of(v, w, next[2 * w], next[2 * w + 1]);
      };
      acc = 0.0f;
      __syncwarp();
      for (uint32_t c = 0; c < (uint32_t)STAGES - 1; ++c)
        issue(c);
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      __syncwarp();
      float a[64], b[64];
      {
        uint4 v[8];
        read(0, v);
#pragma unroll
        for (int w = 0; w < 32; ++w)
          squares_of(v, w, a[2 * w], a[2 * w + 1]);
      }
      uint32_t chunk = 0;
#pragma unroll 1
      for (; chunk + 1 < chunks; chunk += 2) {
        advance(chunk, a, b);
        advance(chunk + 1, b, a);
      }
      if (chunk < chunks)
#pragma unroll
        for (int e = 0; e < 64; ++e)
          add_in_place(acc, a[e]);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    };
    if (SUMS != kRms) {
      pass(std::integral_constant<int, 0>{});
      mean = __fdiv_rn(acc, (float)cols);
      if (SUMS == kLayer)
        deviation_pass();
    } else {
      pass(std::integral_constant<int, 1>{});
    }
    if (row < rows)
      *reinterpret_cast<float2 *>(stats.at + row * stats.pitch) = make_float2(mean, SUMS == kMean ? 0.0f : inverse_deviation(acc, cols, eps));
  }
}

// ---- the same sums of squares in 16 parts per row, for few rows ----
// A chain of cols dependent additions takes 7 us for 3072, however few rows there are. Its terms are not negative, so that
// it can be cut: of two chains of the same terms that start at t and r, in one binade and a multiple of four units of its last place
// apart, each step adds the same number to both, by round to nearest even on the same grid, and one crossing into the next
// binade changes nothing as long as both cross it in the same step, since the grid there is twice as wide. So every lane runs the
// chain of its part of the row from a guess r of where the row's chain will arrive (the sum of what lies in front), for each value
// of the guess's last two bits, and the row's chain t then steps from lane to lane: it takes the chain with its own last two
// bits and adds the distance t - r that it has from that one's start. Every lane says between which distances that holds (the
// same binade at the start, at most one crossing, in a step whose sums on either side are further from the boundary than t and r from
// one another); where it does not, in one row of ten as a part's numbers cross several binades at once, or where numbers are not
// finite, the part's terms are added one by one. Compared with the sequential kernel, all bits of the statistics: 4.8e8 rows of 1024 to
// 8192 numbers, normal ones and others built to meet boundaries, ties and many binades, the same (tests/test_gpu_norm_streams.py has a few).
// It is bound by the operations of five chains (about 750 per row and warp at IPC 0.5), so that many rows are better off with the
// sequential kernel, whose lanes have a row each: row_stats has the line. 32 parts per row took the same time for few rows and
// a fifth more for many, 8 more for few; rows kept for a second pass in registers (unrolled: 168 of them) the same.
constexpr int kSquareWarps = 4, kSquareParts = 16; // warps of a CTA, parts of a row
struct SquareParams {
  const uint4 *x;
  RowStats stats; // the layer form's mean stands there
  uint64_t rows;
  uint32_t cols, groups; // groups of 8 columns in a part of a row
  float eps;
  Divisor by_groups;
};
__host__ __device__ constexpr uint32_t square_pitch(uint32_t groups) { return (groups | 1u) * 16u; } // of a part in shared memory

// The terms of a word's two elements, and a step of the chain.
__device__ __forceinline__ void square_terms(uint32_t word, float mean, float &q0, float &q1) {
  float d0, d1;
  asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %2; sub.rn.f32.bf16 %0, lo, %3; sub.rn.f32.bf16 %1, hi, %3; }"
      : "=f"(d0), "=f"(d1) : "r"(word), "f"(mean));
  q0 = __fmul_rn(d0, d0);
  q1 = __fmul_rn(d1, d1);
}
// CHAINS sums after the eight elements of a group; `after` sees each of them.
template <bool LAYER, int CHAINS, class F>
__device__ __forceinline__ void square_chain(const uint4 &v, float mean, float (&acc)[CHAINS], F &&after) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (LAYER) {
      float q0, q1;
      square_terms(w[i], mean, q0, q1);
#pragma unroll
      for (int c = 0; c < CHAINS; ++c)
        acc[c] = __fadd_rn(acc[c], q0);
      after();
#pragma unroll
      for (int c = 0; c < CHAINS; ++c)
        acc[c] = __fadd_rn(acc[c], q1);
      after();
    } else {
#pragma unroll
      for (int c = 0; c < CHAINS; ++c)
        asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; fma.rn.f32.bf16 %0, lo, lo, %0; }" : "+f"(acc[c]) : "r"(w[i]));
      after();
#pragma unroll
      for (int c = 0; c < CHAINS; ++c)
        asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %1; fma.rn.f32.bf16 %0, hi, hi, %0; }" : "+f"(acc[c]) : "r"(w[i]));
      after();
    }
  }
}

// A lane per part, two rows per warp at a time. GROUPS: p.groups as a constant, or 0. The constant of 3072 columns makes the copies'
// addresses and the layout of shared memory known: norm and quantiser from a graph, us, constant / general: RMS, 1 row 6.1 / 6.3, 77
// 6.7 / 7.0, 300 8.5 / 8.9, 1500 13.5 / 13.7, 2900 21.2 / 21.4; layer form, 77 18.5 / 18.6, 600 21.7 / 21.7, 2900 34.9 / 34.7.
template <bool LAYER, int GROUPS>
__global__ void __launch_bounds__(32 * kSquareWarps)
k_row_squares(const SquareParams p) {
  extern __shared__ uint4 square_smem[];
  grid_dependency_wait(); // (what it reads comes by asynchronous copies and, the mean, by plain loads: both stay behind)
  constexpr uint32_t kParts = kSquareParts, kRows = 32 / kParts;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, part = lane % kParts, groups = GROUPS ? GROUPS : p.groups;
  const uint32_t pitch = square_pitch(groups), cols8 = groups * kParts;
  unsigned char *buffer = reinterpret_cast<unsigned char *>(square_smem) + warp * 32u * pitch;
  const uint4 *mine = reinterpret_cast<const uint4 *>(buffer + lane * pitch);
  const uint32_t to = smem_u32(buffer);
  for (uint64_t row0 = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + warp) * kRows; row0 < p.rows; row0 += (uint64_t)gridDim.x * (blockDim.x >> 5) * kRows) {
    const uint64_t row = row0 + lane / kParts;
    { // the rows are neighbours: 32 parts one behind the other
      const uint32_t valid = (uint32_t)min((uint64_t)kRows, p.rows - row0) * cols8;
      const uint4 *from = p.x + row0 * cols8;
#pragma unroll
      for (uint32_t k = 0; k < groups; ++k) {
        const uint32_t c = lane + 32u * k, of = GROUPS ? c / groups : p.by_groups.quotient(c);
        cp_async16(to + of * pitch + (c - of * groups) * 16u, c < valid ? from + c : p.x, c < valid);
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
      __syncwarp();
    }
    const float mean = LAYER && row < p.rows ? row_stat(p.stats, row).x : 0.0f;
    // the guess: the sum of the parts in front (each in order, so that the second part starts from the row's very chain: it
    // is the one that most often crosses several binades)
    float sum[1] = {0.0f};
#pragma unroll 4
    for (uint32_t k = 0; k < groups; ++k)
      square_chain<LAYER>(mine[k], mean, sum, [] {});
    float front = sum[0];
#pragma unroll
    for (int o = 1; o < (int)kParts; o <<= 1) {
      const float other = __shfl_up_sync(0xffffffffu, front, o, kParts);
      if (part >= (uint32_t)o)
        front += other;
    }
    front = __shfl_up_sync(0xffffffffu, front, 1, kParts);
    const uint32_t start = part == 0u ? 0u : __float_as_uint(front) & ~3u;
    const float bound = __uint_as_float(((start >> 23) + 1u) << 23);
    // the four chains, and the group in which the first of them crosses into the next binade
    float acc[4], before = 0.0f, behind = 0.0f;
    uint32_t crossing = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      acc[c] = __uint_as_float(start + c);
#pragma unroll 4
    for (uint32_t k = 0; k < groups; ++k) {
      if (acc[0] < bound) {
        before = acc[0];
        crossing = k;
      }
      square_chain<LAYER>(mine[k], mean, acc, [] {});
    }
    if (acc[0] >= bound) { // (also where the chain has crossed more than once: the ends will tell)
      float one[1] = {before}, sums[8];
      int at = 0;
      square_chain<LAYER>(mine[crossing], mean, one, [&] { sums[at++] = one[0]; });
      behind = INFINITY;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        before = fmaxf(before, sums[i] < bound ? sums[i] : 0.0f);
        behind = fminf(behind, sums[i] < bound ? INFINITY : sums[i]);
      }
    }
    // Distances t - r with which the row's chain goes the way of these: it stays below the boundary where they do; where they
    // cross it, it is below it in front of the same step and above it behind, and meets no other.
    float above = INFINITY, below = -INFINITY; // none
    {
      const uint32_t binade = start >> 23;
      const float four_units = __uint_as_float((binade - 21u) << 23), room = bound - before - four_units;
      if (binade >= 25u && binade < 253u) {
        if (acc[3] < bound) {
          above = -INFINITY;
          below = bound - acc[3];
        } else if (acc[0] >= bound && acc[3] < 2.0f * bound && room > 0.0f && behind > bound && behind < INFINITY) {
          above = bound - behind;
          below = fminf(room, 2.0f * bound - acc[3]);
        }
      }
    }
    // the row's chain from part to part
    bool done = false; // this part's end is known
    float total = 0.0f;
    for (;;) {
      bool open = false;
#pragma unroll
      for (uint32_t s = 0; s < kParts; ++s) {
        const float in = s == 0u ? 0.0f : __shfl_sync(0xffffffffu, total, s - 1u, kParts);
        const uint32_t t = __float_as_uint(in), last = t & 3u, from = start | last;
        const float end = last & 2u ? (last & 1u ? acc[3] : acc[2]) : (last & 1u ? acc[1] : acc[0]);
        const float apart = in - __uint_as_float(from); // where they hold, a multiple of four units
        const bool holds = t == from || ((t ^ from) < 0x800000u && apart > above && apart < below);
        if (part == s && !done) {
          total = t == from ? end : end + apart; // (infinite ones have no distance)
          open = !holds;
        }
      }
      uint32_t all_open = __ballot_sync(0xffffffffu, open && row < p.rows);
      if (all_open == 0u)
        break;
      // The first open part of every row, term by term and by all lanes; what is in front of it is final.
      constexpr uint32_t kPartsMask = (1u << kParts) - 1u;
#pragma unroll 1
      for (uint32_t r = 0; r < kRows; ++r) {
        const uint32_t of_row = all_open >> (r * kParts) & kPartsMask;
        if (of_row == 0u)
          continue;
        const uint32_t at = r * kParts + (uint32_t)__ffs((int)of_row) - 1u;
        const float in = __shfl_sync(0xffffffffu, total, at == 0u ? 0u : at - 1u);
        float one[1] = {at % kParts == 0u ? 0.0f : in};
        const float row_mean = __shfl_sync(0xffffffffu, mean, at);
        const uint4 *terms = reinterpret_cast<const uint4 *>(buffer + at * pitch);
        for (uint32_t k = 0; k < groups; ++k)
          square_chain<LAYER>(terms[k], row_mean, one, [] {});
        if (lane == at)
          total = one[0];
        if (lane / kParts == r && lane <= at)
          done = true;
      }
    }
    if (part == kParts - 1u && row < p.rows)
      *reinterpret_cast<float2 *>(p.stats.at + row * p.stats.pitch) = make_float2(mean, inverse_deviation(total, p.cols, p.eps));
    __syncwarp(); // the rows are read: the next ones may come
  }
}

// The statistics as parallel sums, one warp per row.
__global__ void __launch_bounds__(256)
k_row_stats_parallel(const uint4 *x, const RowStats stats, uint64_t rows, uint32_t cols, float eps, int layer) {
  x += grid_dependency_wait_zero();
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t cols8 = cols >> 3;
  for (uint64_t r = warp; r < rows; r += (uint64_t)gridDim.x * (blockDim.x >> 5)) {
    float mean = 0.0f, sum = 0.0f;
    if (layer) {
      for (uint32_t c = lane; c < cols8; c += 32) {
        float f[8];
        unpack8(load_global(x + r * cols8 + c), f);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          mean += f[e];
      }
      mean = __fdiv_rn(warp_sum(mean), (float)cols);
    }
    for (uint32_t c = lane; c < cols8; c += 32) {
      float f[8];
      unpack8(load_global(x + r * cols8 + c), f);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = __fsub_rn(f[e], mean);
        sum = __fmaf_rn(d, d, sum);
      }
    }
    sum = warp_sum(sum);
    if (lane == 0)
      *reinterpret_cast<float2 *>(stats.at + r * stats.pitch) =
          make_float2(mean, __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(sum, (float)cols), eps))));
  }
}

// ---- RmsNormModulate, explicit scale / shift (cpu_executor.cpp:1241-1264) ----
// One warp per row; lane l owns the 8-element groups l, l + 32, ... CHUNKS > 0: the row has
// CHUNKS * 256 columns and stays in registers; CHUNKS == 0: any multiple of 256, read twice. Stores hold back the loads behind them, so
// scale, shift and weight of a row in registers are all requested first: 16384 x 3072 158 us a chunk at a time, 84 so.
template <int CHUNKS>
__global__ void __launch_bounds__(256)
k_rms_norm_modulate_bf16(const uint4 *x, const uint4 *w, const uint4 *a, const uint4 *b, uint4 *o, uint64_t rows,
                         uint32_t cols, float eps, const RowStats stats) {
  const uint64_t after = grid_dependency_wait_zero();
  x += after;
  w += after;
  a += after;
  b += after;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint32_t cols8 = cols >> 3, chunks = CHUNKS > 0 ? (uint32_t)CHUNKS : cols >> 8;
  for (uint64_t r = warp; r < rows; r += nwarps) {
    const uint4 *xr = x + r * cols8;
    uint4 kept[CHUNKS > 0 ? CHUNKS : 1];
    float sum = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < chunks; ++k) {
      const uint4 v = load_global(xr + lane + 32u * k);
      if (CHUNKS > 0)
        kept[CHUNKS > 0 ? k : 0] = v;
      float f[8];
      unpack8(v, f);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        sum = __fmaf_rn(f[e], f[e], sum);
    }
    sum = warp_sum(sum);
    // `stats`: the statistic in the reference's sequential order (row_stats), which
    // makes every output bit the reference's; else the warp's parallel sum (last bit may differ)
    const float inv = stats.at ? row_stat(stats, r).y
                               : __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(sum, (float)cols), eps)));
    __syncwarp(); // every lane has its copy: the row may be written
    constexpr uint32_t kBatch = CHUNKS > 0 ? CHUNKS : 1; // chunks whose loads go out before the first is stored
#pragma unroll
    for (uint32_t k0 = 0; k0 < chunks; k0 += kBatch) {
      uint4 as[kBatch], bs[kBatch], ws[kBatch];
#pragma unroll
      for (uint32_t j = 0; j < kBatch; ++j) {
        const uint32_t c = lane + 32u * (k0 + j);
        as[j] = load_global(a + r * cols8 + c);
        bs[j] = load_global(b + r * cols8 + c);
        if (w)
          ws[j] = load_global(w + c);
      }
#pragma unroll
      for (uint32_t j = 0; j < kBatch; ++j) {
        const uint32_t c = lane + 32u * (k0 + j);
        float f[8], wv[8], av[8], bv[8], y[8];
        unpack8(CHUNKS > 0 ? kept[CHUNKS > 0 ? k0 + j : 0] : load_global(xr + c), f);
        unpack8(as[j], av);
        unpack8(bs[j], bv);
        if (w)
          unpack8(ws[j], wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float normalized = __fmul_rn(__fmul_rn(f[e], inv), w ? wv[e] : 1.0f);
          y[e] = __fadd_rn(__fmul_rn(normalized, __fadd_rn(1.0f, av[e])), bv[e]);
        }
        o[r * cols8 + c] = pack8(y);
      }
    }
  }
}

// ---- LayerNormModulate (cpu_executor.cpp:1108-1148): rounds to bf16 after the affine norm,
// after 1 + scale and after their product; scale / shift rows broadcast over rows_per_mod rows ----
template <int CHUNKS>
__global__ void __launch_bounds__(256)
k_layer_norm_modulate_bf16(const uint4 *x, const uint4 *w, const uint4 *b, const uint4 *scale, const uint4 *shift,
                           uint4 *o, uint64_t rows, uint32_t cols, uint64_t rows_per_mod, float eps,
                           const RowStats stats) {
  const uint64_t after = grid_dependency_wait_zero();
  x += after;
  w += after;
  b += after;
  scale += after;
  shift += after;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint32_t cols8 = cols >> 3, chunks = CHUNKS > 0 ? (uint32_t)CHUNKS : cols >> 8;
  for (uint64_t r = warp; r < rows; r += nwarps) {
    const uint4 *xr = x + r * cols8;
    uint4 kept[CHUNKS > 0 ? CHUNKS : 1];
    float mean = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < chunks; ++k) {
      const uint4 v = load_global(xr + lane + 32u * k);
      if (CHUNKS > 0)
        kept[CHUNKS > 0 ? k : 0] = v;
      float f[8];
      unpack8(v, f);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        mean += f[e];
    }
    const float2 given = stats.at ? row_stat(stats, r) : make_float2(0.0f, 0.0f);
    __syncwarp(); // every lane has its copy: the row may be written
    mean = stats.at ? given.x : __fdiv_rn(warp_sum(mean), (float)cols);
    float var = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < chunks; ++k) {
      float f[8];
      unpack8(CHUNKS > 0 ? kept[CHUNKS > 0 ? k : 0] : load_global(xr + lane + 32u * k), f);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = __fsub_rn(f[e], mean);
        var = __fmaf_rn(d, d, var);
      }
    }
    var = warp_sum(var);
    const float inv = stats.at ? given.y : __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(var, (float)cols), eps)));
    const uint64_t mrow = (r / rows_per_mod) * cols8;
#pragma unroll
    for (uint32_t k = 0; k < chunks; ++k) {
      const uint32_t c = lane + 32u * k;
      float f[8], wv[8], bv[8], sc[8], sh[8], y[8];
      unpack8(CHUNKS > 0 ? kept[CHUNKS > 0 ? k : 0] : load_global(xr + c), f);
      unpack8(load_global(w + c), wv);
      unpack8(load_global(b + c), bv);
      unpack8(load_global(scale + mrow + c), sc);
      unpack8(load_global(shift + mrow + c), sh);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float normalized =
            round_bf16(__fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(f[e], mean), inv), wv[e]), bv[e]));
        const float one_plus = round_bf16(__fadd_rn(1.0f, sc[e]));
        y[e] = __fadd_rn(round_bf16(__fmul_rn(normalized, one_plus)), sh[e]);
      }
      o[r * cols8 + c] = pack8(y);
    }
  }
}

// ---- QkNormPartialRope on 128-wide heads (cpu_executor.cpp:1741-1837), optionally followed by
// QuantizeInt8Rows(Direct) of the result (cpu_executor.cpp:124-307, Direct branch) ----
// A warp takes ROWS (token, head) rows of 256 bytes through shared memory. First a lane sums the squares of a row
// in the reference's sequential order (squares of bf16 values are exact, so the fused operation is the reference's
// multiply then add): the statistic has the reference's bits. Then 8 lanes share a row, two runs of 8 elements
// each, chosen so that rotation partners are in the same lane: every access to HBM is a full 128-byte line, and
// the codes come from direct_codes. HBM-bound by its bytes (3 per element), by its arithmetic in practice:
// 33272 x 24 rows with rotary 96 and codes take 125 us (230 us as one thread per row with
// IEEE divisions), 4096 x 24 with rotary 128 in pairs 21 us (37 us). Few rows take 8 per warp, for more warps in flight
// (256 x 24: 12.6 -> 6.3 us a call).
struct RowRopeParams {
  const uint4 *x;
  const uint4 *w;       // [128] bf16
  const void *cosv, *sinv;
  uint4 *o;             // bf16 output or nullptr
  int8_t *codes;        // Direct codes or nullptr
  float *scales;
  uint64_t rows, heads, input_seq, table_seq, table_start;
  uint64_t in_token_stride16, in_offset16; // where a token's heads start in x, in 16-byte units
  uint64_t out_seq, out_start;            // output token = (token / input_seq) * out_seq + out_start + token % input_seq
  uint32_t table_width, table_f32;
  float eps;
};

__device__ __forceinline__ void load_table8(const void *table, uint32_t f32, uint64_t index, float (&v)[8]) {
  if (f32) {
    const float4 *p = reinterpret_cast<const float4 *>(static_cast<const float *>(table) + index);
    const float4 lo = load_global(p), hi = load_global(p + 1);
    v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
  } else {
    unpack8(load_global(reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(table) + index)), v);
  }
}
constexpr int kRopePitch = 17;  // uint4 per row in shared memory (16 + 1 pad)
constexpr int kRopeWarps = 4;

template <int ROTARY, bool V2, int ROWS>
__global__ void __launch_bounds__(32 * kRopeWarps)
k_qk_norm_rope_row128(const RowRopeParams p) {
  __shared__ uint4 tile[kRopeWarps][ROWS * kRopePitch];
  const uint64_t after = grid_dependency_wait_zero();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t row0 = ((uint64_t)blockIdx.x * kRopeWarps + warp) * ROWS;
  if (row0 >= p.rows)
    return;
  // this lane's row of the first pass
  const uint64_t mine = row0 + (lane % ROWS) < p.rows ? row0 + (lane % ROWS) : p.rows - 1;
  const uint64_t token = mine / p.heads, head = mine - token * p.heads, sequence = token / p.input_seq;
  const uint64_t in_sequence = token - sequence * p.input_seq;
  const uint64_t src = token * p.in_token_stride16 + p.in_offset16 + head * 16;
  const uint64_t out_row = (sequence * p.out_seq + p.out_start + in_sequence) * p.heads + head;
  const uint64_t trow = (sequence * p.table_seq + p.table_start + in_sequence) * p.table_width + after;
#pragma unroll
  for (int i = 0; i < ROWS; i += 2) { // half a warp copies a row
    const int r = i + (lane >> 4);
    const uint64_t from = __shfl_sync(0xffffffffu, src, r) + (lane & 15);
    cp_async16(smem_u32(&tile[warp][r * kRopePitch + (lane & 15)]), p.x + from, true);
  }
  // runs of 8 elements of this lane in the second pass: partners of a half-split rotation are ROTARY / 2 apart
  constexpr int kRun = ROTARY / 8; // runs that rotate
  const int j = lane & 7;
  const bool rotates = V2 ? 2 * j < kRun : j < kRun / 2;
  const int c0 = V2 ? 2 * j : j < kRun / 2 ? j : kRun + 2 * (j - kRun / 2);
  const int c1 = V2 || !rotates ? c0 + 1 : j + kRun / 2;
  uint64_t w[8];
  {
    const uint4 a = load_global(p.w + after + c0), b = load_global(p.w + after + c1);
    const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
      w[i] = unpack_bf16_pair(u[i]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  float sum = 0.0f;
  {
    const uint4 *row = tile[warp] + (lane % ROWS) * kRopePitch;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 v = row[c];
      sum = accumulate_word<1>(v.x, sum);
      sum = accumulate_word<1>(v.y, sum);
      sum = accumulate_word<1>(v.z, sum);
      sum = accumulate_word<1>(v.w, sum);
    }
  }
  const float inv_mine = __fdiv_rn(1.0f, sqrtf(__fadd_rn(__fdiv_rn(sum, 128.0f), p.eps)));
#pragma unroll 1
  for (int it = 0; it < ROWS; it += 4) { // rows it .. it + 3
    const int r = it + (lane >> 3);
    const float inv = __shfl_sync(0xffffffffu, inv_mine, r);
    const uint64_t out = __shfl_sync(0xffffffffu, out_row, r), at = __shfl_sync(0xffffffffu, trow, r);
    const bool exists = row0 + r < p.rows;
    uint64_t n[8]; // run c0, then run c1
    {
      const uint4 a = tile[warp][r * kRopePitch + c0], b = tile[warp][r * kRopePitch + c1];
      const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      const uint64_t inv2 = pack2(inv, inv);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t scaled = mul2(unpack_bf16_pair(u[i]), inv2);
        n[i] = V2 ? round_bf16_2(mul2(round_bf16_2(scaled), w[i])) : mul2(scaled, w[i]);
      }
    }
    if (rotates) {
      float a[8], b[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        unpack2(n[i], a[2 * i], a[2 * i + 1]);
        unpack2(n[4 + i], b[2 * i], b[2 * i + 1]);
      }
      if (V2) { // interleaved pairs (2 i, 2 i + 1), one table entry per pair: 8 entries for the two runs
        float c[8], s[8];
        load_table8(p.cosv, p.table_f32, at + 4 * c0, c);
        load_table8(p.sinv, p.table_f32, at + 4 * c0, s);
        auto rotate = [&](float (&x)[8], int first) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float even = x[2 * e], odd = x[2 * e + 1];
            x[2 * e] = __fsub_rn(__fmul_rn(even, c[first + e]), __fmul_rn(odd, s[first + e]));
            x[2 * e + 1] = __fadd_rn(__fmul_rn(even, s[first + e]), __fmul_rn(odd, c[first + e]));
          }
        };
        rotate(a, 0);
        rotate(b, 4);
      } else { // half-split pairs (d, d + ROTARY / 2)
        const uint64_t second = at + 8 * c0 + (p.table_width == (uint32_t)ROTARY ? ROTARY / 2 : 0); // its own entries, or the same
        float c[8], s[8], first[8];
        load_table8(p.cosv, p.table_f32, at + 8 * c0, c);
        load_table8(p.sinv, p.table_f32, at + 8 * c0, s);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          first[e] = __fsub_rn(__fmul_rn(a[e], c[e]), __fmul_rn(b[e], s[e]));
        load_table8(p.cosv, p.table_f32, second, c);
        load_table8(p.sinv, p.table_f32, second, s);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          b[e] = __fadd_rn(__fmul_rn(b[e], c[e]), __fmul_rn(a[e], s[e]));
          a[e] = first[e];
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        n[i] = pack2(a[2 * i], a[2 * i + 1]);
        n[4 + i] = pack2(b[2 * i], b[2 * i + 1]);
      }
    }
    // the stored bf16 values (what a consumer of the unfused op would read back)
    uint32_t bits[8], most = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      bits[i] = pack_bf16_pair(n[i]);
      asm("max.bf16x2 %0, %0, %1;" : "+r"(most) : "r"(bits[i] & 0x7fff7fffu)); // NaN does not count
    }
    float m = fmaxf(__uint_as_float(most << 16), __uint_as_float(most & 0xffff0000u));
    if (p.o && exists) {
      p.o[out * 16 + c0] = make_uint4(bits[0], bits[1], bits[2], bits[3]);
      p.o[out * 16 + c1] = make_uint4(bits[4], bits[5], bits[6], bits[7]);
    }
    if (p.codes) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      const float scale = row_scale(m, 1.0f); // clip 1: max * 1 / 127
      uint32_t words[4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        n[i] = unpack_bf16_pair(bits[i]);
      direct_codes(n, m, scale, words);
      if (exists) {
        *reinterpret_cast<uint2 *>(p.codes + out * 128 + 8 * c0) = make_uint2(words[0], words[1]);
        *reinterpret_cast<uint2 *>(p.codes + out * 128 + 8 * c1) = make_uint2(words[2], words[3]);
        if (j == 0)
          p.scales[out] = scale;
      }
    }
  }
}

// ---- QuantizeInt8Rows(Direct) of 128-wide rows, one thread per row (same arithmetic as the
// warp-per-row kernel in convrot_quant.cu) ----
__global__ void __launch_bounds__(128)
k_direct_quant_row128(const uint4 *x, int8_t *codes, float *scales, uint64_t rows, float clip) {
  x += grid_dependency_wait_zero();
  const uint64_t row = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows)
    return;
  float n[128], m = 0.0f;
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    float f[8];
    unpack8(load_global(x + row * 16 + c), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      n[8 * c + e] = f[e];
      m = fmaxf(m, fabsf(f[e]));
    }
  }
  const float scale = fmaxf(__fdiv_rn(__fmul_rn(m, clip), 127.0f), 1.0e-30f);
  scales[row] = scale;
  uint4 *dst = reinterpret_cast<uint4 *>(codes + row * 128);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint32_t word[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t packed = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        packed |= (uint32_t)(max(sat_s8(__fdiv_rn(n[16 * c + 4 * q + e], scale)), -127) & 0xff) << (8 * e);
      word[q] = packed;
    }
    dst[c] = make_uint4(word[0], word[1], word[2], word[3]);
  }
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline unsigned blocks_for(uint64_t n, int threads) {
  uint64_t b = (n + threads - 1) / threads;
  const uint64_t cap = (uint64_t)sm_count() * 32;
  return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

} // namespace

bool residual_gate_fast(const void *res, const void *branch, const void *gate, void *o, uint32_t dt, uint64_t n,
                        uint64_t width, uint64_t rows_per_gate, cudaStream_t s, int *rc) {
  if (dt != 2 || width % 8 != 0 || !aligned16(res) || !aligned16(branch) || !aligned16(gate) || !aligned16(o))
    return false;
  *rc = launch_ahead("k_residual_gate_bf16", k_residual_gate_bf16, blocks_for(n / 8, 256), 256, 0, s,
                     static_cast<const uint4 *>(res), static_cast<const uint4 *>(branch), static_cast<const uint4 *>(gate),
                     static_cast<uint4 *>(o), n / 8, width / 8, rows_per_gate);
  return true;
}

bool swiglu_fast(const void *x, void *o, uint32_t dt, uint64_t rows, uint64_t width, uint64_t in_width,
                 uint64_t start, bool gate_first, cudaStream_t s, int *rc) {
  if (dt != 2 || width % 8 != 0 || in_width % 8 != 0 || start % 8 != 0 || !aligned16(x) || !aligned16(o))
    return false;
  const uint64_t groups = rows * (width / 8);
  auto launch = [&](auto kernel, auto by) {
    *rc = launch_ahead("k_swiglu_bf16", kernel, blocks_for(groups, 256), 256, 0, s, static_cast<const uint4 *>(x),
                       static_cast<uint4 *>(o), groups, by, in_width / 8, start / 8, gate_first ? 1 : 0);
  };
  if (groups != 0 && groups < (1ull << 31))
    launch(k_swiglu_bf16<Divisor>, divisor(width / 8));
  else
    launch(k_swiglu_bf16<Wide>, Wide{width / 8});
  return true;
}

int row_stats(const void *x, uint64_t rows, uint64_t cols, float eps, bool layer, bool always, void *out,
              uint64_t out_pitch, std::initializer_list<Span> reads, StreamScratch &scratch, RowStats *stats,
              cudaStream_t s) {
  *stats = RowStats{};
  if (always && (!aligned16(x) || cols == 0 || cols % 8 != 0 || cols > 0xffffff00ull)) // 16 bytes at a time
    return fail(kUnsupported, "row statistics: rows must start on 16 bytes");
  const char *exact = std::getenv("DIFB200_EXACT_NORM");
  const bool sequential = !(exact && exact[0] == '0') && cols != 0 && cols % kStatCols == 0 && cols <= 0xffffff00ull &&
                          aligned16(x);
  if (rows == 0 || (!sequential && !always))
    return kOk;
  const uintptr_t begin = reinterpret_cast<uintptr_t>(out), end = begin + rows * out_pitch;
  auto meets = [&](const Span &r) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(r.start);
    return r.start && b < end && begin < b + r.bytes;
  };
  bool shared = begin % 8 != 0 || out_pitch % 8 != 0 || out_pitch < sizeof(float2) || meets({x, rows * cols * 2});
  for (const Span &r : reads)
    shared = shared || meets(r);
  if (shared) {
    if (int rc = scratch.allocate(rows * sizeof(float2), "row statistics scratch"))
      return rc;
    *stats = RowStats{static_cast<unsigned char *>(scratch.get()), sizeof(float2)};
  } else {
    *stats = RowStats{static_cast<unsigned char *>(out), out_pitch};
  }
  const auto *X = static_cast<const uint4 *>(x);
  if (!sequential) {
    uint64_t blocks = (rows + 7) / 8;
    const uint64_t cap = (uint64_t)sm_count() * 8;
    blocks = blocks > cap ? cap : blocks;
    return launch_ahead("k_row_stats_parallel", k_row_stats_parallel, blocks, 256, 0, s, X, *stats, rows, (uint32_t)cols, eps, layer ? 1 : 0);
  }
  auto squares = [&]() {
    constexpr int kGroups3072 = 3072 / (8 * kSquareParts);
    const uint32_t groups = (uint32_t)(cols / (8 * kSquareParts)), warp_bytes = 32u * square_pitch(groups);
    const SquareParams p{X, *stats, rows, (uint32_t)cols, groups, eps, divisor(groups)};
    const uint64_t sms = (uint64_t)sm_count(), wanted = (rows + 32 / kSquareParts - 1) / (32 / kSquareParts);
    const uint32_t warps = (uint32_t)std::min<uint64_t>(kSquareWarps, (wanted + sms - 1) / sms);
    auto kernel = groups == kGroups3072 ? (layer ? k_row_squares<true, kGroups3072> : k_row_squares<false, kGroups3072>)
                                        : (layer ? k_row_squares<true, 0> : k_row_squares<false, 0>);
    int resident = 1;
    if (int rc = resident_blocks(reinterpret_cast<const void *>(kernel), 32 * (int)warps, warps * warp_bytes, &resident))
      return rc;
    const uint64_t blocks = std::min<uint64_t>((wanted + warps - 1) / warps, sms * resident);
    if (layer || rows <= sms)
      return launch_ahead("k_row_squares", kernel, blocks, 32 * (int)warps, warps * warp_bytes, s, p);
    kernel<<<(unsigned)blocks, 32 * warps, warps * warp_bytes, s>>>(p);
    return launched(cudaGetLastError(), "k_row_squares");
  };
  // The statistic is launched plainly. Launched ahead, behind a kernel that lets dependents start (a quantiser, as a rule), its few CTAs
  // gather on the SMs that have room, and what is bound by a warp's chain takes longer: norm and quantiser from a graph, 5000 x 3072
  // 33.9 / 38.0 ahead, layer form 48.7 / 60.5, 300 x 12288 43.8 / 61.7; in parts 300 x 3072 9.0 / 12.3, 1500 14.4 / 16.8, but up to a
  // row per SM 150 8.5 / 7.9. (The second kernel of the layer form follows one that says nothing.)
  // Norm and quantiser from a graph, us, sequential / in parts: RMS, 3072 columns, 1 row 12.8 / 6.3, 150 14.0 / 7.9, 600 16.0 / 10.4, 1500
  // 18.9 / 14.4, 3000 25.0 / 22.8, 4700 33.6 / 33.2; 8192 columns, 600 33.6 / 18.7, 3000 62.2 / 62.3, 4700 83.1 / 88.5; 1024 columns, 150
  // 8.6 / 6.9, 590 8.6 / 8.0. Of the layer form, whose mean stays a chain, the deviations: 3072 columns, 150 26.0 / 19.7, 1500 31.7 / 27.4,
  // 3000 39.1 / 36.1; 8192 columns, 3000 97.5 / 93.0, 4700 120 / 124; 1024 columns, 590 13.7 / 12.8.
  const bool in_parts = cols % (8 * kSquareParts) == 0 && cols >= 1024 && cols <= 8192 && rows <= (cols >= 2048 ? 20ull : 4ull) * (uint64_t)sm_count();
  if (in_parts && !layer)
    return squares();
  // Eight chunks in flight where a few warps per SM have to cover the latency alone, four where the rows
  // give an SM more than six warps (33272 x 3072: one wave of resident CTAs instead of two).
  const uint64_t warps = (rows + 31) / 32;
  const bool deep = warps <= (uint64_t)sm_count() * 6;
  auto kernel = !layer     ? (deep ? k_row_stats_sequential<kRms, 8> : k_row_stats_sequential<kRms, 4>)
                : in_parts ? (deep ? k_row_stats_sequential<kMean, 8> : k_row_stats_sequential<kMean, 4>)
                           : (deep ? k_row_stats_sequential<kLayer, 8> : k_row_stats_sequential<kLayer, 4>);
  const size_t smem = sizeof(uint4) * kStatWarps * (deep ? 8 : 4) * 32 * kStatPitch;
  int resident = 1;
  if (int rc = resident_blocks(reinterpret_cast<const void *>(kernel), 32 * kStatWarps, smem, &resident))
    return rc;
  uint64_t blocks = (warps + kStatWarps - 1) / kStatWarps;
  const uint64_t cap = (uint64_t)sm_count() * resident;
  blocks = blocks > cap ? cap : blocks;
  kernel<<<(unsigned)blocks, 32 * kStatWarps, smem, s>>>(X, *stats, rows, (uint32_t)cols, eps);
  if (int rc = launched(cudaGetLastError(), "k_row_stats_sequential"))
    return rc;
  return in_parts ? squares() : kOk;
}

bool rms_norm_modulate_fast(const void *x, const void *w, const void *a, const void *b, void *o, uint32_t dt,
                            uint64_t rows, uint64_t cols, float eps, cudaStream_t s, int *rc) {
  if (dt != 2 || cols == 0 || cols % 256 != 0 || cols > 0xffffff00ull || !aligned16(x) || (w && !aligned16(w)) ||
      !aligned16(a) || !aligned16(b) || !aligned16(o))
    return false;
  uint64_t blocks = (rows + 7) / 8;
  const uint64_t cap = (uint64_t)sm_count() * 16;
  blocks = blocks < 1 ? 1 : (blocks > cap ? cap : blocks);
  const auto X = static_cast<const uint4 *>(x), W = static_cast<const uint4 *>(w), A = static_cast<const uint4 *>(a),
             B = static_cast<const uint4 *>(b);
  RowStats stats;
  StreamScratch scratch(s);
  const uint64_t row_bytes = cols * 2;
  if ((*rc = row_stats(x, rows, cols, eps, false, false, o, row_bytes, {{w, row_bytes}, {a, rows * row_bytes}, {b, rows * row_bytes}},
                       scratch, &stats, s)))
    return true;
  *rc = launch_ahead("k_rms_norm_modulate_bf16", cols == 3072 ? k_rms_norm_modulate_bf16<12> : k_rms_norm_modulate_bf16<0>, blocks, 256, 0,
                     s, X, W, A, B, static_cast<uint4 *>(o), rows, (uint32_t)cols, eps, stats);
  return true;
}

bool layer_norm_modulate_fast(const void *x, const void *w, const void *b, const void *scale, const void *shift,
                              void *o, uint32_t dt, uint64_t rows, uint64_t cols, uint64_t rows_per_mod, float eps,
                              cudaStream_t s, int *rc) {
  if (dt != 2 || cols == 0 || cols % 256 != 0 || cols > 0xffffff00ull || !aligned16(x) || !aligned16(w) ||
      !aligned16(b) || !aligned16(scale) || !aligned16(shift) || !aligned16(o))
    return false;
  uint64_t blocks = (rows + 7) / 8;
  const uint64_t cap = (uint64_t)sm_count() * 16;
  blocks = blocks < 1 ? 1 : (blocks > cap ? cap : blocks);
  const auto X = static_cast<const uint4 *>(x), W = static_cast<const uint4 *>(w), B = static_cast<const uint4 *>(b),
             SC = static_cast<const uint4 *>(scale), SH = static_cast<const uint4 *>(shift);
  RowStats stats;
  StreamScratch scratch(s);
  const uint64_t row_bytes = cols * 2, mod_bytes = (rows + rows_per_mod - 1) / rows_per_mod * row_bytes;
  if ((*rc = row_stats(x, rows, cols, eps, true, false, o, row_bytes,
                       {{w, row_bytes}, {b, row_bytes}, {scale, mod_bytes}, {shift, mod_bytes}}, scratch, &stats, s)))
    return true;
  *rc = launch_ahead("k_layer_norm_modulate_bf16", cols == 3072 ? k_layer_norm_modulate_bf16<12> : k_layer_norm_modulate_bf16<0>, blocks,
                     256, 0, s, X, W, B, SC, SH, static_cast<uint4 *>(o), rows, (uint32_t)cols, rows_per_mod, eps, stats);
  return true;
}

// QkNormPartialRope (+ optional Direct quantisation) for bf16 rows of 128; false when the shape is
// not covered (the caller then runs the generic kernel).
bool qk_norm_rope_fast(const void *x, const void *w, const void *cosv, const void *sinv, void *o, int8_t *codes,
                       float *scales, uint32_t dt, uint32_t dt_table, uint64_t tokens, uint64_t heads, uint64_t dim,
                       uint64_t rotary, uint64_t table_width, uint64_t input_seq, uint64_t table_seq,
                       uint64_t table_start, float eps, bool interleaved_v2, const RopeLayout *layout, cudaStream_t s,
                       int *rc) {
  const RopeLayout dense{heads * 128, 0, input_seq, 0};
  const RopeLayout &l = layout ? *layout : dense;
  if (l.in_token_stride % 8 != 0 || l.in_offset % 8 != 0)
    return false;
  if (dt != 2 || dim != 128 || (dt_table != 1 && dt_table != 2) || !aligned16(x) || !aligned16(w) ||
      !aligned16(cosv) || !aligned16(sinv) || (o && !aligned16(o)) || (codes && !aligned16(codes)))
    return false;
  if (rotary != 64 && rotary != 96 && rotary != 128)
    return false;
  // table rows must start on 16 bytes and hold what the layout reads
  const uint64_t entry = dt_table == 1 ? 4 : 2;
  if ((table_width * entry) % 16 != 0)
    return false;
  if (interleaved_v2 ? table_width != rotary / 2 : (table_width != rotary && table_width != rotary / 2))
    return false;
  RowRopeParams p{static_cast<const uint4 *>(x), static_cast<const uint4 *>(w), cosv, sinv, static_cast<uint4 *>(o),
                  codes, scales, tokens * heads, heads, input_seq, table_seq, table_start, l.in_token_stride / 8,
                  l.in_offset / 8, l.out_seq, l.out_start, (uint32_t)table_width, dt_table == 1 ? 1u : 0u, eps};
  if (p.rows == 0) { // nothing to launch
    *rc = kOk;
    return true;
  }
  const bool few = p.rows <= (uint64_t)sm_count() * 12 * 32; // less than three warps of 32 rows per scheduler
  const uint64_t blocks = (p.rows + (few ? 8 : 32) * kRopeWarps - 1) / ((few ? 8 : 32) * kRopeWarps);
  if (blocks > 0x7fffffffull)
    return false;
#define DIFB200_ROPE_CASE(R, V)                                                                   \
  if (rotary == R && interleaved_v2 == V) {                                                       \
    *rc = launch_ahead("k_qk_norm_rope_row128", few ? k_qk_norm_rope_row128<R, V, 8> : k_qk_norm_rope_row128<R, V, 32>, blocks, \
                       32 * kRopeWarps, 0, s, p);                                                 \
    return true;                                                                                  \
  }
  DIFB200_ROPE_CASE(64, false)
  DIFB200_ROPE_CASE(96, false)
  DIFB200_ROPE_CASE(128, false)
  DIFB200_ROPE_CASE(64, true)
  DIFB200_ROPE_CASE(96, true)
  DIFB200_ROPE_CASE(128, true)
#undef DIFB200_ROPE_CASE
  return false;
}

bool direct_quant_rows128(const void *x, int8_t *codes, float *scales, uint64_t rows, float clip, cudaStream_t s,
                          int *rc) {
  if (!aligned16(x) || !aligned16(codes) || rows + 127 > 0x7fffffffull * 128ull)
    return false;
  *rc = launch_ahead("k_direct_quant_row128", k_direct_quant_row128, (rows + 127) / 128, 128, 0, s, static_cast<const uint4 *>(x), codes,
                     scales, rows, clip);
  return true;
}

} // namespace glue
} // namespace difb200
