// LinearInt8Scaled and the whole W8A8 linear for problems of few rows (sm_100a).
//
// A problem of at most 32 rows reads every weight for next to no arithmetic, and what the tile kernel spends around its
// main loop (tensor memory, barriers, the first loads' latency, a chain of k-blocks, a cluster's exchange) is most of its
// time. Here a CTA takes 16 columns, whose weights go from global memory straight into the registers of warp-wide integer MMAs
// (16 columns x 32 k x 8 rows; which k stands in which slot is the same for both operands and otherwise free, so every lane
// loads 16 contiguous bytes), all of a warp's first loads before it waits for the quantiser. Eight warps share the k
// range in turns of 64 bytes and add their INT32 sums through shared memory. INT32 sums are exact: the bits are those of the
// tile kernel, whose epilogue arithmetic this one shares.
//
// The smallest problems are one launch: every CTA rotates and quantises the rows itself, while its weights are on their way. It
// is launched ahead and waits at its start: the time between two kernels, not their work, was a third of a call (2 x 3072 x 3072,
// calls one behind the other, weights not in L2: 8.0 us launched plainly, 5.4 so).
// That costs a CTA about 1.5 us and saves a launch, 3 us of the host. 2 x 3072 x 3072 from a graph, weights not in L2, all launched
// plainly, one launch / two / the tile kernel and a quantiser: 6.2 / 5.4 / 11.0 us, of the host 5.1 / 8.0 / 8.5. Launched ahead: one
// 4.9, the two of 4 rows 4.8.
#include "gemm_common.cuh"
#include "ops.h"
#include "quant_common.cuh"

#include <cstdlib>

namespace difb200 {
namespace {

constexpr int kFewWarps = 8, kFewBatch = 6; // chunks of 64 bytes of k that a warp requests at once
struct FewParams {
  const int8_t *x, *w;
  GemmParams g;
};

__device__ __forceinline__ void mma_s8_16x8x32(int32_t (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// This warp's sums of eight rows to shared memory, [row][16 columns].
__device__ __forceinline__ void store_sums(int32_t *sums, const int32_t (&c)[4]) {
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  sums[32 * t + g] = c[0];
  sums[32 * t + 16 + g] = c[1];
  sums[32 * t + g + 8] = c[2];
  sums[32 * t + 16 + g + 8] = c[3];
}

__device__ __forceinline__ void write_output(const GemmParams &p, uint32_t row, uint32_t n, int32_t acc, float row_scale) {
  if (p.acc_out)
    p.acc_out[(size_t)row * p.N + n] = acc;
  const float y = __fmul_rn(__fmul_rn((float)acc, row_scale), load_produced(p.col_scales + n));
  uint32_t bits = pack_bf16x2(y, 0.0f);
  if (p.epilogue & kEpiBias)
    bits = pack_bf16x2(__fadd_rn(__uint_as_float(bits << 16), bf16_bits_to_f32(load_produced(p.bias + n))), 0.0f);
  if (p.epilogue & kEpiGeluTanh)
    bits = pack_bf16x2(gelu_tanh(__uint_as_float(bits << 16)), 0.0f);
  p.out[(size_t)row * p.N + n] = (uint16_t)bits;
}

// The 16 columns from n0 on: lane (g, t) has columns g and g + 8.
struct Columns {
  const int8_t *low, *high;
  bool low_ok, high_ok;
  __device__ __forceinline__ Columns(const int8_t *w, uint32_t n0, uint32_t N, uint32_t K) {
    const uint32_t g = (threadIdx.x & 31) >> 2;
    low_ok = n0 + g < N;
    high_ok = n0 + 8u + g < N;
    low = w + (size_t)(low_ok ? n0 + g : 0) * K;
    high = w + (size_t)(high_ok ? n0 + 8u + g : 0) * K;
  }
};

// k of this lane's 16 bytes in a warp's u-th chunk of the batch that starts with chunk `first`
__device__ __forceinline__ uint32_t k_of(uint32_t first, int u) {
  return (first + (threadIdx.x >> 5) + kFewWarps * u) * 64u + 16u * (threadIdx.x & 3u);
}

// A batch of this warp's chunks of 16 columns' weights.
struct Weights {
  uint4 low[kFewBatch], high[kFewBatch];
  template <bool READY>
  __device__ __forceinline__ void load(const Columns &columns, uint32_t K, uint32_t first) {
    auto from = [](const int8_t *at) { return READY ? load_streamed(at) : load_produced_once(at); };
#pragma unroll
    for (int u = 0; u < kFewBatch; ++u) {
      const uint32_t k = k_of(first, u);
      low[u] = high[u] = make_uint4(0, 0, 0, 0);
      if (k < K) {
        if (columns.low_ok)
          low[u] = from(columns.low + k);
        if (columns.high_ok)
          high[u] = from(columns.high + k);
      }
    }
  }
  __device__ __forceinline__ void multiply(int32_t (&c)[4], const uint4 (&x)[kFewBatch]) const {
#pragma unroll
    for (int u = 0; u < kFewBatch; ++u) {
      mma_s8_16x8x32(c, low[u].x, high[u].x, low[u].y, high[u].y, x[u].x, x[u].y);
      mma_s8_16x8x32(c, low[u].z, high[u].z, low[u].w, high[u].w, x[u].z, x[u].w);
    }
  }
};

// GROUPS: of 8 rows. READY: no kernel that may still run writes the weights (GemmParams::weights_first). Otherwise they are
// read like everything that the kernel in front produces: the non-coherent path is for what nobody writes meanwhile. (With
// the same hint, no line in L1, they take the same time: 2 x 3072 x 12288, weights not in L2, 10.3 us both ways, with .cg 10.6.)
template <int GROUPS, bool READY>
__global__ void __launch_bounds__(32 * kFewWarps, 2)
gemm_i8_few_rows_kernel(const FewParams f) {
  const GemmParams &p = f.g;
  const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2;
  const uint32_t n0 = blockIdx.x * 16u, chunks = (p.K + 63u) / 64u;
  const Columns columns(f.w, n0, p.N, p.K);
  Weights w;
  if (READY)
    w.load<READY>(columns, p.K, 0);
  grid_dependency_wait();
  if (!READY)
    w.load<READY>(columns, p.K, 0);
  int32_t c[GROUPS][4] = {};
  for (uint32_t first = 0; first < chunks; first += kFewWarps * kFewBatch) {
    if (first != 0u)
      w.load<READY>(columns, p.K, first);
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
      const uint32_t row = 8u * q + g;
      uint4 x[kFewBatch];
#pragma unroll
      for (int u = 0; u < kFewBatch; ++u) {
        const uint32_t k = k_of(first, u);
        x[u] = make_uint4(0, 0, 0, 0);
        if (k < p.K && row < p.M)
          x[u] = load_produced(reinterpret_cast<const uint4 *>(f.x + (size_t)row * p.K + k));
      }
      w.multiply(c[q], x);
    }
  }
  __shared__ int32_t sums[kFewWarps][GROUPS * 8][16]; // [warp][row][column]
#pragma unroll
  for (int q = 0; q < GROUPS; ++q)
    store_sums(&sums[warp][8 * q][0], c[q]);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 16u * p.M; i += 32 * kFewWarps) {
    const uint32_t row = i >> 4, n = n0 + (i & 15u);
    if (n >= p.N)
      continue;
    int32_t acc = 0;
#pragma unroll
    for (int v = 0; v < kFewWarps; ++v)
      acc += sums[v][row][i & 15u];
    write_output(p, row, n, acc, load_produced(p.row_scales + row));
  }
}

// QuantizeInt8Rows (the unsigned 256-wide rotation on bf16) and the linear in one launch: rows of at most 8 blocks of 1024
// columns in all, one for each warp (two for each take longer than a quantiser in front: 5 x 3072 x 3072 7.9 and 5.1 us). Every
// CTA makes the same codes; the first one also writes them and the row scales to the caller's scratch. A CTA then takes every
// gridDim.x-th tile of 16 columns.
struct FusedParams {
  const uint16_t *x;
  const int8_t *w;
  int8_t *codes;
  float *scales, clip;
  uint32_t row_blocks; // of 1024 columns
  GemmParams g;
};
constexpr uint32_t kFusedRows = 8, kFusedBlocks = kFewWarps;
uint32_t fused_smem(uint32_t M, uint32_t K) {
  return kFewWarps * kWarpBytes256 + M * (K + 16u) + (kFusedBlocks + kFusedRows) * (uint32_t)sizeof(float);
}

__global__ void __launch_bounds__(32 * kFewWarps, 2)
w8a8_few_rows_kernel(const FusedParams f) {
  const GemmParams &p = f.g;
  extern __shared__ __align__(128) uint8_t few_smem[];
  const uint64_t after = grid_dependency_wait_zero();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t K = p.K, tiles = (p.N + 15u) / 16u, chunks = (K + 63u) / 64u, pitch = K + 16u;
  Weights w;
  w.load<false>(Columns(f.w, blockIdx.x * 16u, p.N, K), K, 0); // (the grid has no more CTAs than tiles)

  uint8_t *codes = few_smem + kFewWarps * kWarpBytes256;
  float *maxima = reinterpret_cast<float *>(codes + p.M * pitch), *scales = maxima + kFusedBlocks;
  {
    const int h = lane >> 4, a = lane & 15;
    const uint32_t area = smem_u32(few_smem) + warp * kWarpBytes256 + h * kHalfBytes;
    const uint32_t row = warp / f.row_blocks, block = warp - row * f.row_blocks, column = block * 1024u + 512u * h;
    const bool act_a = row < p.M && column + 16u * a < K, act_b = row < p.M && column + 16u * a + 256u < K; // (groups exist whole or not at all)
    uint32_t V[16];
    {
      const uint4 zero = make_uint4(0, 0, 0, 0);
      const uint4 *src = reinterpret_cast<const uint4 *>(f.x + after + (size_t)row * K + column + 16u * a);
      const uint4 v[4] = {act_a ? load_global(src) : zero, act_a ? load_global(src + 1) : zero, act_b ? load_global(src + 32) : zero,
                          act_b ? load_global(src + 33) : zero};
      const uint32_t wa[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
      const uint32_t wb[8] = {v[2].x, v[2].y, v[2].z, v[2].w, v[3].x, v[3].y, v[3].z, v[3].w};
      uint64_t P[16];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        P[2 * e] = pack2(__uint_as_float(wa[e] << 16), __uint_as_float(wb[e] << 16));
        P[2 * e + 1] = pack2(__uint_as_float(wa[e] & 0xffff0000u), __uint_as_float(wb[e] & 0xffff0000u));
      }
      rotate_pairs(P, area + kRowPitch * a, area + 8u * a);
      float m = 0.0f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        m = absmax2(m, P[j]);
        V[j] = pack_bf16_pair(P[j]);
      }
      m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
      if (lane == 0)
        maxima[warp] = m;
    }
    __syncthreads();
    if (row < p.M) {
      constexpr float kCarry = 16.0f; // of the rotation
      float m = (uint32_t)lane < f.row_blocks ? maxima[row * f.row_blocks + lane] : 0.0f;
      m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
      const float maximum = m * (1.0f / kCarry), scale = row_scale(maximum, f.clip), divisor = round_bf16_number(scale) * kCarry;
      if (block == 0u && lane == 0)
        scales[row] = scale;
      SplitReciprocal split;
      if (!split.of(divisor, maximum)) {
        const float recip = __frcp_rn(divisor);
#pragma unroll
        for (int j = 0; j < 16; ++j)
          V[j] = bounded_quotients(V[j], recip);
      }
      uint8_t *to = codes + row * pitch + column + a;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const uint32_t pair = code_bytes(split.quotients(V[j]));
        if (act_a)
          to[16 * j] = (uint8_t)pair;
        if (act_b)
          to[16 * j + 256] = (uint8_t)(pair >> 8);
      }
    }
    __syncthreads();
  }
  if (blockIdx.x == 0) {
    for (uint32_t i = threadIdx.x; i < p.M * (K / 16u); i += 32 * kFewWarps) {
      const uint32_t row = i / (K / 16u), at = i - row * (K / 16u);
      reinterpret_cast<uint4 *>(f.codes)[i] = *reinterpret_cast<const uint4 *>(codes + row * pitch + 16u * at);
    }
    if (threadIdx.x < p.M)
      f.scales[threadIdx.x] = scales[threadIdx.x];
  }

  const int g = lane >> 2;
  int32_t *sums = reinterpret_cast<int32_t *>(few_smem); // [warp][8 rows][16 columns]
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    int32_t c[4] = {};
    for (uint32_t first = 0; first < chunks; first += kFewWarps * kFewBatch) {
      if (first != 0u)
        w.load<false>(Columns(f.w, tile * 16u, p.N, K), K, first);
      uint4 x[kFewBatch];
#pragma unroll
      for (int u = 0; u < kFewBatch; ++u) {
        const uint32_t k = k_of(first, u);
        x[u] = k < K && (uint32_t)g < p.M ? *reinterpret_cast<const uint4 *>(codes + g * pitch + k) : make_uint4(0, 0, 0, 0);
      }
      w.multiply(c, x);
    }
    if (tile + gridDim.x < tiles)
      w.load<false>(Columns(f.w, (tile + gridDim.x) * 16u, p.N, K), K, 0);
    store_sums(sums + warp * 128, c);
    __syncthreads();
    const uint32_t row = threadIdx.x >> 4, n = tile * 16u + (threadIdx.x & 15u);
    if (row < p.M && n < p.N) { // at most 8 rows: the first 128 threads
      int32_t acc = 0;
#pragma unroll
      for (int v = 0; v < kFewWarps; ++v)
        acc += sums[v * 128 + threadIdx.x];
      write_output(p, row, n, acc, scales[row]);
    }
    __syncthreads();
  }
}

template <int GROUPS>
int launch_groups(const FewParams &f, cudaStream_t stream) {
  return launch_ahead("gemm_i8_few_rows_kernel launch",
                      f.g.weights_first ? gemm_i8_few_rows_kernel<GROUPS, true> : gemm_i8_few_rows_kernel<GROUPS, false>,
                      (f.g.N + 15u) / 16u, 32 * kFewWarps, 0, stream, f);
}

// Waves of the few-rows kernels: two CTAs of 16 columns per SM.
uint64_t few_waves(uint64_t N) {
  const uint64_t columns = 32ull * (uint64_t)sm_count();
  return (N + columns - 1) / columns;
}
bool tile_form_is_forced() { return std::getenv("DIFB200_GEMM_FORM") || std::getenv("DIFB200_GEMM_CTAS"); }

} // namespace

// Whether the few-rows kernel takes a linear from the tile kernel. Every CTA reads all rows' codes and pays its start, its sums
// and its outputs for 16 columns: the time grows with the waves of CTAs, and with 9 and 17 rows by an MMA per chunk, where the
// tile kernel's hardly does. So the line is one of waves (4736 columns each on 148 SMs), and of K where both come close. Tile
// kernel / this one, us, weights not in L2:
//   1 to 8 rows    two waves   8 x 128 x 9216 3.9 / 3.7, 8 x 3072 x 9216 10.4 / 9.1, 8 x 8192 x 9216 18.3 / 18.6
//                  three       8 x 3072 x 12288 11.4 / 11.8, 4 x 8192 x 12288 24.1 / 23.7; 8 x 512 x 16384 5.8 / 7.8; with a
//                              quantiser in front, behind which this one has its first weights already, 8 x 512 x 12288 8.0 / 9.0,
//                              8 x 2048 x 12288 11.9 / 11.7, 4 x 3072 x 12288 13.8 / 13.2
//   9 to 16 rows   one wave    16 x 128 x 4736 3.9 / 2.7, 16 x 12288 x 3072 13.9 / 12.7
//                  two         16 x 3072 x 9216 10.5 / 10.4, 16 x 128 x 9216 3.9 / 4.4, 16 x 4096 x 9216 12.3 / 14.0
//   17 to 32 rows  one wave    32 x 256 x 4736 4.1 / 4.0, 32 x 3072 x 4736 8.8 / 7.8, 32 x 12288 x 1024 11.5 / 11.2
//                  two         32 x 512 x 5120 6.0 / 6.1, 17 x 512 x 12288 5.4 / 10.5
// The limits on N K end what was measured: beyond them the two are within a few percent.
bool few_rows(uint64_t M, uint64_t N, uint64_t K, bool weights_first) {
  if (M > 32 || tile_form_is_forced())
    return false;
  const uint64_t waves = few_waves(N);
  if (M <= 8)
    return waves <= 2 || (waves == 3 && K >= (weights_first ? 2048u : 8192u));
  if (M <= 16)
    return waves == 1 ? N * K <= (5ull << 23) : waves == 2 && K >= 256 && K <= 3072;
  return waves == 1 && N * K <= (1ull << 24);
}

namespace {
// The same for the whole linear in one launch, which has the quantiser's launch to save and stays for further tiles. Quantiser and
// tile kernel / this one, us: 8 x 1024 x 16384 10.0 / 9.8, 2 x 3072 x 16384 15.6 / 13.3, 2 x 3072 x 32768 24.5 / 19.8; but
// 8 x 256 x 32768 9.7 / 11.5, 8 x 1024 x 32768 13.1 / 14.8.
bool few_rows_in_one_launch(uint64_t M, uint64_t N, uint64_t K) {
  return M <= kFusedRows && !tile_form_is_forced() && (few_waves(N) <= 4 || K >= 2048);
}
} // namespace

int launch_few_rows(const int8_t *x, const int8_t *w, const GemmParams &p, cudaStream_t stream) {
  const FewParams f{x, w, p};
  return p.M <= 8 ? launch_groups<1>(f, stream) : p.M <= 16 ? launch_groups<2>(f, stream) : launch_groups<4>(f, stream);
}

bool w8a8_few_rows(const void *x_bf16, const int8_t *w, const float *col_scales, const void *bias_bf16, uint32_t epilogue,
                   int implementation, float clip, uint64_t M, uint64_t N, uint64_t K, int8_t *codes, float *scales,
                   void *out_bf16, cudaStream_t stream, int *rc) {
  const uint64_t row_blocks = (K + 1023) / 1024;
  const uintptr_t aligned = reinterpret_cast<uintptr_t>(x_bf16) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(codes);
  if (implementation != 2 || M == 0 || N == 0 || N > 0x7fffffffull || K == 0 || K % 256 != 0 ||
      M * row_blocks > kFusedBlocks || !(clip > 0.0f) || !x_bf16 || !w || !col_scales || !codes || !scales || !out_bf16 ||
      (epilogue & ~(kEpiBias | kEpiGeluTanh)) || ((epilogue & kEpiBias) && !bias_bf16) || (aligned & 15) ||
      gemm_load_is_withheld() || !few_rows_in_one_launch(M, N, K))
    return false;
  // Every CTA reads all of x, and other CTAs write meanwhile: not where a call is in place.
  const uintptr_t begin = reinterpret_cast<uintptr_t>(x_bf16), end = begin + M * K * 2;
  auto meets = [&](const void *start, uint64_t bytes) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(start);
    return b < end && begin < b + bytes;
  };
  if (meets(out_bf16, M * N * 2) || meets(codes, M * K) || meets(scales, M * 4))
    return false;
  FusedParams f{};
  f.x = static_cast<const uint16_t *>(x_bf16);
  f.w = w;
  f.codes = codes;
  f.scales = scales;
  f.clip = clip;
  f.row_blocks = (uint32_t)row_blocks;
  f.g.col_scales = col_scales;
  f.g.bias = static_cast<const uint16_t *>(bias_bf16);
  f.g.out = static_cast<uint16_t *>(out_bf16);
  f.g.M = (uint32_t)M;
  f.g.N = (uint32_t)N;
  f.g.K = (uint32_t)K;
  f.g.epilogue = epilogue;
  const uint32_t smem = fused_smem((uint32_t)M, (uint32_t)K);
  int resident = 1;
  if ((*rc = resident_blocks(reinterpret_cast<const void *>(w8a8_few_rows_kernel), 32 * kFewWarps, smem, &resident)))
    return true;
  const uint64_t tiles = (N + 15) / 16, most = (uint64_t)sm_count() * resident;
  *rc = launch_ahead("w8a8_few_rows_kernel launch", w8a8_few_rows_kernel, tiles < most ? tiles : most, 32 * kFewWarps, smem, stream, f);
  return true;
}

} // namespace difb200
