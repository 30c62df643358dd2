// INT8 attention for sm_100a: INT8 Q.K^T on tcgen05 (kind::i8, INT32 scores in tensor memory),
// fp32 online softmax with a power-of-two running maximum, bf16 P.V on tcgen05 (kind::f16, fp32
// output accumulator in tensor memory), flash-style over 128-key tiles with TMA K/V staging.
// Grouped-query attention and a key-validity mask are supported; non-causal.
//
// Semantics. The op replaced is DiffIR Attention (reference src/runtime/cpu_executor.cpp:
// 1839-1910; GQA head mapping :1853-1863, all-masked-row rule :1881-1887; key mask as produced by
// BooleanMaskToBias with MaskQueries=false, :627-650) in the INT8 lowering that the reference
// only ships for sm_86 (src/runtime/h3_owned_attention.cu:646-929). Numerical contract (per
// query row i of head h, kv head h / (H / KV)):
//   acc_j = sum_d q8[i,d] * k8[j,d]                 INT32, exact
//   u_j   = float(acc_j) * ks'_j                    one fp32 rounding; ks'_j = the key scale rounded
//                                                   (nearest-even) to 22 significant bits;
//                                                   u_j = -inf for masked keys
//   A     = qs_i * (scale * log2(e))
//   m     = an integer >= ceil(max_j u_j * A)       (any such integer gives the same result up
//                                                    to the rounding of the fma below: bf16
//                                                    rounding commutes with powers of two). The
//                                                    kernel takes the Cauchy-Schwarz bound
//                                                    ceil(A * |q8_i| * max_j(|k8_j| * ks'_j)) when
//                                                    that is at most 60 (one pass, no running
//                                                    maximum, no rescaling of the output), else a
//                                                    running maximum, which moves to 24 above the
//                                                    scores where they exceed it
//   p_j   = exp2(fma(u_j, A, -m)),  P_j = bf16(p_j)   (never above 1)
//   out   = bf16((sum_j P_j * v_j) / (sum_j p_j))   fp32 accumulation; all keys masked -> 0
// q8/qs and k8/ks are QuantizeInt8Rows(Direct) of the [B,S,H,128] / [B,S,KV,128] tensors.
//
// Structure: one CTA per (batch, head, 256 queries) = two 128-query tiles that share every K/V
// tile. Warp 0 = TMA producer, warps 1 and 2 = MMA issuers of query tile 0 / 1 (warp 3 idle). Warps 4-11 and 12-19:
// softmax + epilogue of query tile 0 / 1, two threads per query row that take 32 columns of a step each (a thread's
// scores live in registers, so no shuffles). K/V arrive in 128-key stages; the score / softmax / P.V pipeline
// works in 64-key steps. Scores and P have their own columns of tensor memory, so the scores of step g + 1 are
// made while those of step g are worked on in registers: at the end of a step a warp takes the next scores,
// leaves its P and arrives once; the MMA warp then issues P.V of the step and Q.K^T of the one after the next.
// Tensor memory per query tile (256 columns): scores of one step (64), P (32 columns of bf16 pairs, the A operand
// of P.V), Q codes (32 columns, the A operand of Q.K^T: read from shared memory for every 64 keys they alone took its
// bandwidth for 128 clocks, 387 against 259 clocks for the Q.K^T of both tiles), output (fp32, 128). Items that would
// not fill a last wave are shared by clusters of CTAs that take a part of the keys each (plan_split).
//
// Chunked form (the token-sharded block, where keys arrive from other GPUs one slice at a time):
// a launch covers up to two ranges of 128-key tiles and may carry the unnormalised state of every
// query row -- m, l and the fp32 output accumulator -- in from an earlier launch and out to a
// later one. Every m is an integer, so moving a row from one m to a larger one multiplies l, O
// and every p by an exact power of two: a sequence of launches over disjoint key ranges gives the
// single launch's result up to the order of the fp32 sums.
#include "common.cuh"
#include "ops.h"
#include "ptx.cuh"
#include "quant_common.cuh"

#include <mutex>

namespace difb200 {
namespace {

constexpr int kTile = 128;          // queries per tile, keys per tile, head dim
constexpr int kStages = 4;          // K/V ring depth (Q passes through stages 2 and 3 first)
constexpr uint32_t kKBytes = 128 * 128;        // int8 [128 keys x 128]
constexpr uint32_t kVBytes = 128 * 128 * 2;    // bf16 [128 keys x 128] as two 64-wide halves
constexpr uint32_t kKsBytes = 128 * 8;         // the tile's 128 key scales, then its 128 mask entries
constexpr uint32_t kStageBytes = kKBytes + kVBytes + kKsBytes;
constexpr int kThreads = 640;      // 4 control warps, 2 x 8 softmax warps
constexpr uint32_t kPartialBytes = 32 * 32 * 4; // split form: a [32 rows x 32 columns] fp32 partial output
constexpr uint32_t kOutBoxBytes = 32 * 128;    // a warp's output staging: two [32 rows x 64 bf16] boxes
constexpr float kHeadroom = 24.0f;  // powers of two that the running maximum goes beyond a row's scores when it moves
constexpr float kLeastSum = 1.0f / (1u << 25); // of a running maximum: its largest p is above 2^-(kHeadroom + 1)
constexpr uint32_t kPairBytes = 4096;          // [2 phases][2 tiles][2 halves][128 rows] fp32
constexpr size_t kSmemBytes = 1024 + kStages * kStageBytes + 256 + kPairBytes;

struct AttnParams {
  const int8_t *q8;      // [B,Sq,H,128]
  const float *qs;       // [B,Sq,H]
  const float *table;    // [B,KV,S_pad/128] x (128 key scales ks'_j, 128 mask entries)
  const float *tile_bound; // [B,KV,S_pad/128] max over the tile's valid keys of |k8_j| * ks'_j
  uint32_t B, Sq, Sk, H, KV, S_pad; // Sq query tokens, Sk key tokens (S_pad = Sk rounded up to 128)
  uint16_t *out;         // [B,Sq,H,128] bf16
  float scale_log2e;     // scale * log2(e)
  unsigned long long wait_ns; // limit of every bounded wait
  DeviceStatus *status;
  // key tiles of this launch: [tile_begin[0], +tile_count[0]) then [tile_begin[1], +tile_count[1])
  uint32_t tile_begin[2], tile_count[2];
  // The state carried between launches. The unnormalised outputs (fp32) of 32 neighbouring rows, or what is left of
  // them, stand together as [32 float4 of a row][rows]: a warp's accesses are whole lines. With 16 bytes of 32 rows each
  // per instruction, 4096 queries over 512 keys in two launches took 101 us, so 72.
  float *o_state;        // [B,H,Sq,128]
  float2 *ml_state;      // [B,H,Sq] m, l of the even half of the columns
  float *l2_state;       // [B,H,Sq] l of the other half: a sequence of launches continues the very same sums
  uint32_t carry_in, carry_out;
  uint32_t behind_whole; // 1: launched behind the items that are not split, whose operands this launch shares
  uint32_t split_follows; // 1: such a launch comes next
  uint32_t item0, split; // first (batch, head, query block) of this launch; CTAs of a cluster that share its keys
  Divisor q_blocks, heads, group; // blocks of 256 queries, H, H / KV
};

__device__ __forceinline__ void report(DeviceStatus *status, uint32_t role, uint32_t detail) {
  if (atomicExch(&status->flag, 1u) == 0u) {
    status->kernel = 3u;
    status->role = role;
    status->detail = detail;
  }
}

// The scale of one key, rounded to the 22 significant bits of the contract, and the key's contribution to its tile's
// bound, from the key scale and the sum of squares of its codes.
__device__ __forceinline__ void key_entry(float ks, int n2, float &k22, float &bound) {
  uint32_t bits = __float_as_uint(ks);
  bits = (bits + 1u + ((bits >> 2) & 1u)) & ~3u; // nearest-even to 22 significant bits
  k22 = __uint_as_float(bits);
  bound = __fmul_rn(__fsqrt_rn((float)n2), k22);
  if (!(fabsf(k22) < INFINITY))
    k22 = __int_as_float(0x7fc00000); // whatever the score, such a key makes its rows NaN
}

// Builds the key table [B,KV,S_pad/128]: per 128-key tile its key scales, re-laid from the [B,S,KV] row order to be
// contiguous along keys, then its mask entries. u = RN(float(acc) * ks') is the conversion and one multiplication; a
// 16-byte load brings the scales of four keys. (An integer addition of the bits of 1.5 * 2^23 in the place of the
// conversion, with -1.5 * 2^23 ks' beside every scale, takes twice the loads: B2 S4608 H24 390 us, now 382.) Masked and padding keys carry the scale 0 and the mask entry -inf, which
// is added: u = -inf. The others' entry is 0, and a segment of 32 keys (what a softmax thread takes of a step) says in
// its first entry whether it has such keys at all: +0 there means none, and the softmax leaves the entries unread. In
// a segment that has some, the first key's entry is -inf or -0.
// Also writes, per 128-key tile, the largest |k8_j|_2 * ks'_j of its valid keys: with |q8_i|_2 it
// bounds every score of the tile (Cauchy-Schwarz on the integer codes).
// One block of 128 threads per (batch, kv head, key tile), one thread per key.
__global__ void __launch_bounds__(128)
key_table_kernel(const int8_t *k8, const float *ks, const uint8_t *key_valid, float *table,
                 float *tile_bound, uint32_t S, uint32_t KV, uint32_t S_pad, uint32_t begin0, uint32_t count0,
                 uint32_t begin1, uint32_t count1) {
  const uint64_t after = grid_dependency_wait_zero();
  grid_dependents_launch();
  const uint32_t tiles = S_pad / kTile;     // tiles of the whole key axis (table layout)
  const uint32_t mine = count0 + count1;    // tiles this launch covers
  const uint32_t local = blockIdx.x % mine;
  const uint32_t tile = local < count0 ? begin0 + local : begin1 + (local - count0);
  const uint32_t kvh = (blockIdx.x / mine) % KV;
  const uint32_t b = blockIdx.x / (mine * KV);
  const uint32_t j = tile * kTile + threadIdx.x;
  float k22 = 0.0f, mask = -INFINITY, bound = 0.0f;
  if (j < S && (key_valid == nullptr || key_valid[(uint64_t)b * S + j] != 0)) {
    const uint4 *row = reinterpret_cast<const uint4 *>(k8 + after + (((uint64_t)b * S + j) * KV + kvh) * kTile);
    int n2 = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint4 w = load_global(row + c);
      n2 = __dp4a((int)w.x, (int)w.x, n2);
      n2 = __dp4a((int)w.y, (int)w.y, n2);
      n2 = __dp4a((int)w.z, (int)w.z, n2);
      n2 = __dp4a((int)w.w, (int)w.w, n2);
    }
    key_entry(ks[((uint64_t)b * S + j) * KV + kvh], n2, k22, bound);
    mask = 0.0f;
  }
  if (__any_sync(0xffffffffu, mask != 0.0f) && (threadIdx.x & 31) == 0 && mask == 0.0f)
    mask = -0.0f;
  float *t = table + (((uint64_t)b * KV + kvh) * tiles + tile) * (2u * kTile) + threadIdx.x;
  t[0] = k22;
  t[kTile] = mask;
  __shared__ float warp_max[4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    bound = fmaxf(bound, __shfl_xor_sync(0xffffffffu, bound, o));
  if ((threadIdx.x & 31) == 0)
    warp_max[threadIdx.x >> 5] = bound;
  __syncthreads();
  if (threadIdx.x == 0)
    tile_bound[((uint64_t)b * KV + kvh) * tiles + tile] =
        fmaxf(fmaxf(warp_max[0], warp_max[1]), fmaxf(warp_max[2], warp_max[3]));
}

// QuantizeInt8Rows(Direct, clip 1) of 128-wide bf16 rows for the attention's operands, and the key table
// from the same pass: the codes, row scales and (for keys) the table entries and tile bounds that the
// quantiser and key_table_kernel would give one after the other, bit for bit. 8 lanes hold a row
// (16 elements each), so every access is a full 32-byte sector; HBM-bound (3 bytes per element). The first
// `key_blocks` CTAs each take the 128 keys of one (batch, kv head, tile), the others 128 query rows each.
// (Two thread-per-row quantiser launches and the table's own pass over the codes: B2 S4608 H24 81 us.)
struct OperandParams {
  const uint4 *q, *k;
  int8_t *q8, *k8;
  float *qs, *ks;
  const uint8_t *key_valid;
  float *table, *tile_bound;
  uint64_t q_rows;
  uint32_t S, KV, S_pad, key_blocks;
};
// STEPS: rows of a lane, in a CTA of 1024 / STEPS threads. Two where all CTAs are resident at once, whose time is a lane's chain
// (1101 tokens, 24 heads over 8: attention and operands 23.9 us with four, 23.4; 300 tokens 13.6 and 13.1), four where rows
// are many (1101 over 24, 423 CTAs: 25.5, with two 25.9).
template <int STEPS>
__global__ void __launch_bounds__(1024 / STEPS)
attention_operands_kernel(const OperandParams p) {
  const uint64_t after = grid_dependency_wait_zero();
  grid_dependents_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane & 7;
  // The four rows of a lane are requested before the first is worked on (behind one another, each waited for its load:
  // B2 S4608 H24 41 us against 34).
  uint4 lows[STEPS], highs[STEPS];
  constexpr uint32_t kStepRows = 128u / STEPS;
  auto request = [&](int step, const uint4 *row, bool valid) {
    lows[step] = highs[step] = make_uint4(0, 0, 0, 0);
    if (valid) {
      lows[step] = load_global(row + 2 * part);
      highs[step] = load_global(row + 2 * part + 1);
    }
  };
  // codes of this lane's 16 elements of a row and the row's scale (in every lane)
  auto quantise = [&](int step, uint4 &codes, float &scale) {
    const uint4 lo = lows[step], hi = highs[step];
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint64_t v[8];
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = unpack_bf16_pair(w[i]);
      m = absmax2(m, v[i]);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    scale = row_scale(m, 1.0f);
    uint32_t out[4];
    direct_codes(v, m, scale, out);
    codes = make_uint4(out[0], out[1], out[2], out[3]);
  };
  if (blockIdx.x < p.key_blocks) {
    const uint32_t tiles = p.S_pad / kTile, tile = blockIdx.x % tiles, kvh = (blockIdx.x / tiles) % p.KV,
                   b = blockIdx.x / (tiles * p.KV);
    auto key_of = [&](int step) { return tile * kTile + step * kStepRows + warp * 4u + (lane >> 3); };
    auto row_of = [&](int step) { return ((uint64_t)b * p.S + (key_of(step) < p.S ? key_of(step) : 0)) * p.KV + kvh; };
#pragma unroll
    for (int step = 0; step < STEPS; ++step)
      request(step, p.k + after + row_of(step) * 16, key_of(step) < p.S);
    __shared__ uint32_t masked[4], first_valid[4]; // whether a segment of 32 keys has masked ones; whether its first key is not
    uint32_t own_first_valid = 0; // the same as bits, where thread 0 has the four segments' first keys
    if (threadIdx.x < 4) {
      masked[threadIdx.x] = 0u;
      if (STEPS != 4)
        first_valid[threadIdx.x] = 0u;
    }
    __syncthreads();
    float *t = p.table + (((uint64_t)b * p.KV + kvh) * tiles + tile) * (2u * kTile);
    float most = 0.0f;
#pragma unroll
    for (int step = 0; step < STEPS; ++step) {
      const uint32_t j = key_of(step);
      const bool exists = j < p.S;
      const uint64_t row = row_of(step);
      uint4 codes;
      float scale;
      quantise(step, codes, scale);
      int n2 = __dp4a((int)codes.x, (int)codes.x, 0);
      n2 = __dp4a((int)codes.y, (int)codes.y, n2);
      n2 = __dp4a((int)codes.z, (int)codes.z, n2);
      n2 = __dp4a((int)codes.w, (int)codes.w, n2);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
        n2 += __shfl_xor_sync(0xffffffffu, n2, o);
      float k22 = 0.0f, mask = -INFINITY, bound = 0.0f;
      if (exists) {
        reinterpret_cast<uint4 *>(p.k8 + row * kTile)[part] = codes;
        if (part == 0)
          p.ks[row] = scale;
        if (p.key_valid == nullptr || p.key_valid[(uint64_t)b * p.S + j] != 0) {
          key_entry(scale, n2, k22, bound);
          mask = 0.0f;
        }
      }
      most = fmaxf(most, bound);
      if (part == 0) {
        t[j % kTile] = k22;
        t[kTile + j % kTile] = mask;
        if (mask != 0.0f)
          masked[STEPS == 4 ? step : j % kTile / 32u] = 1u;
        else if (STEPS == 4)
          own_first_valid |= 1u << step;
        else if (j % 32u == 0u)
          first_valid[j % kTile / 32u] = 1u;
      }
    }
    __shared__ float warp_max[32 / STEPS];
    most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most))); // non-negative
    if (lane == 0)
      warp_max[warp] = most;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 32 / STEPS; ++w)
        most = fmaxf(most, warp_max[w]);
      p.tile_bound[((uint64_t)b * p.KV + kvh) * tiles + tile] = most;
      for (int segment = 0; segment < 4; ++segment)
        if (masked[segment] != 0u && (STEPS == 4 ? own_first_valid >> segment & 1u : first_valid[segment]) != 0u)
          t[kTile + 32 * segment] = -0.0f;
    }
  } else {
    auto row_of = [&](int step) { return (uint64_t)(blockIdx.x - p.key_blocks) * 128u + step * kStepRows + warp * 4u + (lane >> 3); };
#pragma unroll
    for (int step = 0; step < STEPS; ++step)
      request(step, p.q + after + (row_of(step) < p.q_rows ? row_of(step) : 0) * 16, row_of(step) < p.q_rows);
#pragma unroll
    for (int step = 0; step < STEPS; ++step) {
      const uint64_t row = row_of(step);
      const bool exists = row < p.q_rows;
      uint4 codes;
      float scale;
      quantise(step, codes, scale);
      if (exists) {
        reinterpret_cast<uint4 *>(p.q8 + row * kTile)[part] = codes;
        if (part == 0)
          p.qs[row] = scale;
      }
    }
  }
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t packed;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(hi), "f"(lo));
  return packed;
}

// 32 outputs bf16(o / l) from RN(1 / l) and one Markstein step (the product corrected by its residual, one rounding);
// where that has no finite value (o infinite) the product stands. A row without valid keys has l = 0 and gives 0. Both
// show as a NaN among the results, which a maximum over them carries to one test. (With a test and a choice per result, 64
// results of each thread and their staging took 3000 of the 13200 clocks of a CTA with one key tile, so 1900.)
__device__ __forceinline__ void normalise(const uint32_t (&o)[32], float l, uint32_t (&w)[16]) {
  const float y = __frcp_rn(l);
  const uint64_t y2 = pack2(y, y), negl2 = pack2(-l, -l);
  uint32_t most = 0;
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const uint64_t o2 = pack2(__uint_as_float(o[j]), __uint_as_float(o[j + 1]));
    const uint64_t q2 = mul2(o2, y2);
    float x0, x1;
    unpack2(fma2(fma2(q2, negl2, o2), y2, q2), x0, x1);
    w[j >> 1] = pack_bf16(x0, x1);
    asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(most) : "r"(w[j >> 1]));
  }
  if ((most & 0x7fffu) <= 0x7f80u && (most >> 16 & 0x7fffu) <= 0x7f80u)
    return;
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const uint64_t o2 = pack2(__uint_as_float(o[j]), __uint_as_float(o[j + 1]));
    const uint64_t q2 = mul2(o2, y2);
    float y0, y1, x0, x1;
    unpack2(q2, y0, y1);
    unpack2(fma2(fma2(q2, negl2, o2), y2, q2), x0, x1);
    w[j >> 1] = l > 0.0f ? pack_bf16(x0 == x0 ? x0 : y0, x1 == x1 ? x1 : y1) : 0u;
  }
}

// SPLIT: the launch whose items are shared by clusters (an instance of its own: run-time branches for it cost the
// plain one 2 %).
template <bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
attn_i8_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw_addr);
  const uint32_t stage_addr = base;                   // kStages x (K | V | ksmb)
  const uint32_t bar = stage_addr + kStages * kStageBytes;
  // barriers (8 bytes each)
  const uint32_t q_tma = bar;                         // Q codes are in shared memory
  const uint32_t q_full = bar + 8;                    // [2 tiles] they stand in tensor memory
  const uint32_t kv_full = q_full + 16, kv_empty = kv_full + 8 * kStages;
  const uint32_t s_full = kv_empty + 8 * kStages;     // [2] phase g: Q.K^T of step g is done, and P.V of step g - 2
  const uint32_t p_full = s_full + 16;                // [2] phase 0: scores of step 0 read; phase g + 1: P of step g stored, scores of g + 1 read
  const uint32_t pair_bar = p_full + 16;              // [2][4] the two warps of 32 rows have exchanged a word per row
  const uint32_t tmem_slot = pair_bar + 64;
  const uint32_t pair_mem = bar + 256;
  volatile uint32_t *slot_ptr = reinterpret_cast<volatile uint32_t *>(base_ptr + (tmem_slot - base));
  volatile uint32_t *abort_ptr = slot_ptr + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long wait_ns = p.wait_ns;
  const uint32_t split = SPLIT ? p.split : 1u, rank = SPLIT ? ptx::cluster_ctarank() : 0u;
  const uint32_t item = SPLIT ? p.item0 + blockIdx.x / split : blockIdx.x;
  // (every warp needs them: with divisions by the parameters it took 1240 clocks to the wait for the operands, so 380)
  const uint32_t batch_head = p.q_blocks.quotient(item), qb = item - batch_head * p.q_blocks.by;
  const uint32_t batch = p.heads.quotient(batch_head), head = batch_head - batch * p.H;
  const uint32_t kvh = p.group.quotient(head);
  const uint32_t q0 = qb * 256u;
  const uint32_t tiles = p.tile_count[0] + p.tile_count[1], first = SPLIT ? tiles * rank / split : 0u;
  const uint32_t n_kv = SPLIT ? tiles * (rank + 1u) / split - first : tiles; // of this CTA (at least one: split <= tiles)
  const uint32_t n_steps = 2u * n_kv;               // 64-key steps
  auto key_tile = [&](uint32_t i) {                 // i-th key tile of this CTA -> tile of the key axis
    if (SPLIT)
      i += first;
    return i < p.tile_count[0] ? p.tile_begin[0] + i : p.tile_begin[1] + (i - p.tile_count[0]);
  };

  auto load_tile = [&](uint32_t i, uint32_t s) { // K, V and the key table of this CTA's i-th tile into stage s
    const uint32_t k_dst = stage_addr + s * kStageBytes, v_dst = k_dst + kKBytes, t_dst = v_dst + kVBytes;
    const uint32_t tile = key_tile(i);
    const int32_t key0 = (int32_t)(tile * kTile);
    const float *table = p.table + ((uint64_t)batch * p.KV + kvh) * p.S_pad * 2u;
    ptx::mbar_expect_tx(kv_full + 8 * s, kKBytes + kVBytes + kKsBytes);
    ptx::tma_load_4d(k_dst, &map_k, kv_full + 8 * s, 0, (int32_t)kvh, key0, (int32_t)batch);
    ptx::tma_load_4d(v_dst, &map_v, kv_full + 8 * s, 0, (int32_t)kvh, key0, (int32_t)batch);
    ptx::tma_load_4d(v_dst + kVBytes / 2, &map_v, kv_full + 8 * s, 64, (int32_t)kvh, key0, (int32_t)batch);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
                     "r"(t_dst), "l"(reinterpret_cast<uint64_t>(table + (uint64_t)tile * (2u * kTile))),
                 "r"(kKsBytes), "r"(kv_full + 8 * s)
                 : "memory");
  };
  if (threadIdx.x == 0) {
    ptx::mbar_init(q_full, 8);
    ptx::mbar_init(q_full + 8, 8);
    ptx::mbar_init(q_tma, 1);
    for (int i = 0; i < 8; ++i)
      ptx::mbar_init(pair_bar + 8 * i, 2);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(kv_full + 8 * s, 1);
      ptx::mbar_init(kv_empty + 8 * s, 2);
    }
    for (int t = 0; t < 2; ++t) {
      ptx::mbar_init(s_full + 8 * t, 1);
      ptx::mbar_init(p_full + 8 * t, 8);
    }
    *abort_ptr = 0;
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  // The kernel in front makes the codes and the key table and may run up to here. A split launch behind the unsplit items
  // is independent of them: it fills the SMs as they become free, and only its end waits for them. It reads the operands
  // without a wait of its own. Every CTA of the unsplit launch lets it start only behind its own wait, when the operands'
  // kernel is complete and its writes are performed, and hands them on with a fence; the reader has the other half.
  if (!SPLIT || !p.behind_whole)
    grid_dependency_wait();
  else
    ptx::fence_device_and_tma();
  if (!SPLIT && warp == 3 && p.split_follows) { // (the idle one)
    ptx::fence_device_and_tma();
    grid_dependents_launch();
  }
  // Only Q is requested in front of the barrier. The first two tiles are 8 copies more, 700 to 1000 clocks of this one thread
  // for which all others waited, and the first Q.K^T needs them 2000 clocks later. With this, and the divisions and the
  // normalisation as they are now, 4096 queries of 24 heads over 77 keys 25.5 -> 22.9 us, over 512 39.4 -> 36.2, B1 S1101
  // H24 KV8 24.8 -> 24.3, B1 S4608 H24 188.2 -> 187.3.
  if (threadIdx.x == 0) {
    ptx::mbar_expect_tx(q_tma, 2 * kKBytes); // Q codes: staged where the ring is still free
    for (uint32_t t = 0; t < 2; ++t)
      ptx::tma_load_4d(stage_addr + (2u + t) * kStageBytes, &map_q, q_tma, 0, (int32_t)head, (int32_t)(q0 + t * 128u), (int32_t)batch);
  }
  // What the softmax warps need first, requested here and used behind the barrier: the row's scale, the bounds of the
  // first 128 key tiles.
  const float *bounds = p.tile_bound + ((uint64_t)batch * p.KV + kvh) * (p.S_pad / kTile);
  float A = 0.0f, near[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (warp >= 4) {
    const uint32_t qr = q0 + (uint32_t)((warp - 4) >> 3) * 128u + (warp & 3) * 32u + lane;
    A = load_produced(p.qs + ((uint64_t)batch * p.Sq + (qr < p.Sq ? qr : 0u)) * p.H + head);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (lane + 32u * u < n_kv)
        near[u] = load_produced(bounds + key_tile(lane + 32u * u));
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    // The producer and the MMA warps run their loops with all 32 lanes and warp-uniform control
    // flow (every wait ends in a vote); one elected lane issues the asynchronous instructions.
    // Addresses, descriptors and loop state are then warp-uniform values. As single-lane
    // (divergent) loops every TMA / MMA operand was first moved between register files. One warp for both
    // query tiles was the bound of the whole kernel: its control instructions are a serial chain of about 1500 clocks
    // per 64-key step, in which the MMAs themselves execute for 770. With one thread per query row, B2 S4608 H24 took
    // 443 us with one warp in the shortest loop (one wait, one commit per step) and 404 with two.
    auto give_up = [&](uint32_t role, uint32_t detail) {
      if (lane == 0) {
        if (!*abort_ptr)
          report(p.status, role, detail);
        *abort_ptr = 1;
      }
    };
    if (warp == 0) {
      // ---------------- TMA producer ----------------
      uint32_t s = 0, phase = 0;
      for (uint32_t i = 0; i < n_kv; ++i) {
        if (!ptx::mbar_wait_uniform(kv_empty + 8 * s, phase ^ 1u, abort_ptr, wait_ns) ||
            ((i == 2u || i == 3u) && !ptx::mbar_wait_uniform(q_full + 8 * (i - 2u), 0, abort_ptr, wait_ns))) {
          give_up(0, i);
          break;
        }
        if (ptx::elect_one())
          load_tile(i, s);
        if (++s == kStages) {
          s = 0;
          phase ^= 1u;
        }
      }
    } else if (warp < 3) {
      // ---------------- MMA issuers, one per query tile ----------------
      const uint32_t t = __shfl_sync(0xffffffffu, (uint32_t)warp - 1u, 0);
      constexpr uint32_t idesc_qk = ptx::make_idesc(2 /*S32*/, 1 /*S8*/, 1 /*S8*/, 0, 0, 128, 64);
      constexpr uint32_t idesc_pv = ptx::make_idesc(1 /*F32*/, 1 /*BF16*/, 1 /*BF16*/, 0, 1 /*V is N-major*/, 128, 128);
      const uint64_t k_desc0 = ptx::smem_desc_sw128(stage_addr, 16, 1024);
      // V tile, N-major: 64-wide halves 16 KB apart (leading offset), 8-key groups 1 KB apart.
      const uint64_t v_desc0 = ptx::smem_desc_sw128(stage_addr + kKBytes, kVBytes / 2, 1024);
      // Step g covers keys 64 g .. 64 g + 63, i.e. half g & 1 of the 128-key stage (g / 2) % kStages.
      // (called inside the elected lane's branch) Q.K^T of a step, keys from descriptor address b
      const uint32_t d_s = tmem + t * 256u, d_o = d_s + 128u, a_p = d_s + 64u, a_q = d_s + 96u;
      const uint32_t s_bar = s_full + 8 * t, p_bar = p_full + 8 * t;
      auto issue_qk = [&](uint32_t b) {
        const uint64_t kd = k_desc0 + b;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ptx::mma_i8_ts(d_s, a_q + 8u * k, kd + (uint64_t)(2 * k), idesc_qk, k != 0);
        ptx::mma_commit(s_bar);
      };
      bool ok = ptx::mbar_wait_uniform(kv_full, 0, abort_ptr, wait_ns) && ptx::mbar_wait_uniform(q_full + 8 * t, 0, abort_ptr, wait_ns);
      if (!ok)
        give_up(2, 0);
      if (ok) {
        ptx::tc_fence_after();
        if (ptx::elect_one())
          issue_qk(0);
        ok = ptx::mbar_wait_uniform(p_bar, 0, abort_ptr, wait_ns);
        if (!ok)
          give_up(2, 1);
        ptx::tc_fence_after();
        if (ok && ptx::elect_one())
          issue_qk(512u);
      }
      uint32_t st = 0, st_n = 1, phase_n = 0, acc = p.carry_in; // stages of the P.V and Q.K^T that come next
      for (uint32_t i = 0; i < n_steps && ok; ++i) {
        const uint32_t h = i & 1u;
        const bool more = i + 2u < n_steps;
        if (h == 0u && more && !ptx::mbar_wait_uniform(kv_full + 8 * st_n, phase_n, abort_ptr, wait_ns)) {
          give_up(2, 5);
          break;
        }
        if (!ptx::mbar_wait_uniform(p_bar, h ^ 1u, abort_ptr, wait_ns)) { // phase i + 1
          give_up(2, 3 + t);
          break;
        }
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          const uint64_t b = v_desc0 + (uint64_t)(st * (kStageBytes >> 4) + h * 512u);
          // A = P in tensor memory (32 columns of bf16 pairs);
          // B = the 64 keys of the V stage: 16 keys per MMA = 8 TMEM columns, 2048 bytes of V
          ptx::mma_f16_ts(d_o, a_p, b, idesc_pv, acc);
#pragma unroll
          for (int k = 1; k < 4; ++k)
            ptx::mma_f16_ts(d_o, a_p + 8u * k, b + (uint64_t)(128 * k), idesc_pv, 1);
          if (more)
            issue_qk(st_n * (kStageBytes >> 4) + h * 512u);
          else
            ptx::mma_commit(s_bar);
          if (h != 0u)
            ptx::mma_commit(kv_empty + 8 * st);
        }
        acc = 1u;
        if (h != 0u) {
          st = st_n;
          if (++st_n == kStages) {
            st_n = 0;
            phase_n ^= 1u;
          }
        }
      }
    }
    if (SPLIT) { // the three barriers of the outputs' exchange count every thread of the cluster
      __syncwarp();
      ptx::cluster_sync();
      ptx::cluster_sync();
      ptx::cluster_sync();
    }
  } else {
    // ---------------- softmax + epilogue, two threads per query row ----------------
    // Four warps per scheduler: the ld / st / barrier time of one is covered by the others. B2 S4608 H24 398 us with one
    // thread per row (two warps per scheduler, 64 columns each) and 367 with two. 32 x 128 + 112 x 512 registers are what
    // the launch has (96 x 640); without spills, which the smaller share had, it went from 363 to 352.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const uint32_t t = (uint32_t)(warp - 4) >> 3, hf = ((uint32_t)(warp - 4) >> 2) & 1u; // query tile 0 / 1; half of the columns
    const uint32_t quarter = (uint32_t)warp & 3u;
    const uint32_t row_in_tile = quarter * 32u + lane;
    const uint32_t qrow = q0 + t * 128u + row_in_tile;
    const bool row_ok = qrow < p.Sq;
    // of an existing row: its place in the carried state, that of its outputs, and the rows these share a place with
    auto state_row = [&]() { return ((uint64_t)batch * p.H + head) * p.Sq + qrow; };
    auto state_outputs = [&]() { return (state_row() - lane) * (kTile / 4) + lane; };
    auto state_pitch = [&]() { return min(32u, p.Sq - (qrow - lane)); };
    A = (row_ok ? A : 1.0f) * p.scale_log2e;
    const uint32_t lane_base = (quarter * 32u) << 16;
    const uint32_t s_tmem = tmem + lane_base + t * 256u, p_tmem = s_tmem + 64u, o_tmem = s_tmem + 128u;
    float m_run = -INFINITY, l = 0.0f;
    // Whether the warp goes on. Only waits that end in a vote decide it, so that the warp goes one way: lanes that gave
    // up alone would leave the others in a warp-wide instruction.
    bool alive = true;
    // A bound on every score of this row: |q8_i| * max_j(|k8_j| * ks'_j) * A. When it is small
    // for the whole warp, its ceiling is the fixed maximum m of the row and a key tile needs one
    // pass (no maximum, no rescaling); otherwise the warp keeps a running maximum.
    bool fixed_max = false;
    {
      float kmax = fmaxf(fmaxf(near[0], near[1]), fmaxf(near[2], near[3]));
      for (uint32_t i = lane + 128u; i < n_kv; i += 32u)
        kmax = fmaxf(kmax, load_produced(bounds + key_tile(i)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        kmax = fmaxf(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
      // the row's 128 codes: A operand of Q.K^T, 32 columns of which each of the row's threads brings half
      if (!ptx::mbar_wait_uniform(q_tma, 0, abort_ptr, wait_ns)) {
        if (lane == 0)
          report(p.status, 9 + t, 0);
        *abort_ptr = 1;
        alive = false;
      }
      const uint8_t *codes = base_ptr + (stage_addr - base) + (2u + t) * kStageBytes + row_in_tile * 128u;
      int n2 = 0;
      {
        uint32_t mine[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 w = *reinterpret_cast<const uint4 *>(codes + (((hf * 4u + c) ^ (lane & 7u)) << 4));
          mine[4 * c] = w.x;
          mine[4 * c + 1] = w.y;
          mine[4 * c + 2] = w.z;
          mine[4 * c + 3] = w.w;
        }
        ptx::tmem_st_32x16(s_tmem + 96u + 16u * hf, mine);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 w = *reinterpret_cast<const uint4 *>(codes + ((((hf ^ 1u) * 4u + c) ^ (lane & 7u)) << 4));
          n2 = __dp4a((int)w.x, (int)w.x, n2);
          n2 = __dp4a((int)w.y, (int)w.y, n2);
          n2 = __dp4a((int)w.z, (int)w.z, n2);
          n2 = __dp4a((int)w.w, (int)w.w, n2);
        }
#pragma unroll
        for (int c = 0; c < 16; ++c)
          n2 = __dp4a((int)mine[c], (int)mine[c], n2);
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before();
      ptx::fence_proxy_async();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(q_full + 8 * t);
      const float bound = __fmul_rn(__fmul_rn(A, __fsqrt_rn((float)n2)), kmax);
      const float m_fixed = ceilf(__fadd_rn(bound, 0.001f));
      // State carried in from the launch over the previous key ranges. m only ever grows, and
      // the fixed form may use any integer that is at least its bound: the larger of the carried m
      // and this launch's bound serves both, the carried l and O move to it by an exact power of
      // two, and the running form simply goes on from the carried m.
      float m_prev = -INFINITY;
      if (p.carry_in && row_ok) {
        const float2 ml = load_global(p.ml_state + state_row());
        m_prev = ml.x;
        l = hf == 0u ? ml.y : load_global(p.l2_state + state_row());
      }
      const float m_both = fmaxf(m_prev, m_fixed);
      // (a bound far above what the carried state holds would push that state towards underflow)
      fixed_max = __all_sync(0xffffffffu, m_both <= 60.0f && (m_prev == -INFINITY || m_both - m_prev <= 60.0f));
      m_run = fixed_max ? m_both : m_prev;
      if (p.carry_in) {
        const float factor = (fixed_max && m_prev != -INFINITY) ? ex2(m_prev - m_run) : (fixed_max ? 0.0f : 1.0f);
        l *= factor;
        const float4 *src = reinterpret_cast<const float4 *>(p.o_state) + state_outputs();
        const uint32_t pitch = state_pitch();
#pragma unroll 1
        for (int c = 2 * hf; c < 2 * hf + 2; ++c) {
          uint32_t o[32];
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const float4 x = row_ok ? load_global(src + (8 * c + v) * pitch) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            o[4 * v] = __float_as_uint(x.x * factor);
            o[4 * v + 1] = __float_as_uint(x.y * factor);
            o[4 * v + 2] = __float_as_uint(x.z * factor);
            o[4 * v + 3] = __float_as_uint(x.w * factor);
          }
          ptx::tmem_st_32x32(o_tmem + 32u * c, o);
        }
        ptx::tmem_st_wait(); // published to the MMA warp with the arrive behind the first P
      }
    }
    const uint64_t A2 = pack2(A, A);
    uint32_t r[32];
    uint32_t masked = 0; // the first mask entry of this thread's segment of the step whose scores are in r
    // the key scales of this thread's 32 columns of a step; the mask entries stand kTile floats behind
    auto segment = [&](uint32_t g) {
      return reinterpret_cast<const float *>(base_ptr + (stage_addr - base) + ((g >> 1) % kStages) * kStageBytes + kKBytes +
                                             kVBytes) + (g & 1u) * 64u + hf * 32u;
    };
    uint32_t pair_phase = 0;
    float *pair_slot = reinterpret_cast<float *>(base_ptr + (pair_mem - base)) + t * 256u + row_in_tile;
    // A word of each of the row's two threads to the other (bounded like every wait).
    auto exchange = [&](float x) {
      float *slot = pair_slot + (pair_phase & 1u) * 512u;
      slot[hf * 128u] = x;
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(pair_bar + 8u * (t * 4u + quarter));
      if (!ptx::mbar_wait_uniform(pair_bar + 8u * (t * 4u + quarter), pair_phase & 1u, abort_ptr, wait_ns)) {
        if (!*abort_ptr && lane == 0)
          report(p.status, 11 + t, 0);
        *abort_ptr = 1;
        alive = false;
      }
      ++pair_phase;
      return slot[(hf ^ 1u) * 128u];
    };
    // The scores of step g, when its Q.K^T is done. The stage's key table needs no wait of its own: it arrives on
    // the barrier of the V tile, which the MMA warp has seen complete before it issued the
    // Q.K^T whose completion is awaited here.
    auto await_scores = [&](uint32_t g) {
      if (!ptx::mbar_wait_uniform(s_full + 8 * t, g & 1u, abort_ptr, wait_ns)) {
        if (!*abort_ptr && lane == 0)
          report(p.status, 3 + t, g);
        *abort_ptr = 1;
        alive = false;
      }
      return alive;
    };
    if (n_steps != 0u && alive && await_scores(0)) {
      ptx::tc_fence_after();
      ptx::tmem_ld_32x32(s_tmem + 32u * hf, r);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(p_full + 8 * t);
      masked = __float_as_uint(segment(0)[kTile]);
    }
    // A loop for each way to the maximum: with both in one the registers are shared out worse (B2 S4608 H24 with q 4 times
    // larger, whose maximum runs, 588 us; 535 with a loop of its own).
    if (fixed_max) {
      for (uint32_t g = 0; g < n_steps && alive; ++g) {
        const float4 *tab = reinterpret_cast<const float4 *>(segment(g));
        // u of four neighbouring keys: float(acc) * ks', plus the mask entries where the segment has masked keys
        auto scores4 = [&](int j, bool with_mask, uint64_t &u01, uint64_t &u23) {
          const float4 ks = tab[j >> 2];
          u01 = pack2((float)(int32_t)r[j], (float)(int32_t)r[j + 1]);
          u23 = pack2((float)(int32_t)r[j + 2], (float)(int32_t)r[j + 3]);
          if (with_mask) { // (a product of 0 and the entry -0 is the sum +0, as without an entry)
            const float4 mask = tab[(kTile + j) >> 2];
            u01 = fma2(u01, pack2(ks.x, ks.y), pack2(mask.x, mask.y));
            u23 = fma2(u23, pack2(ks.z, ks.w), pack2(mask.z, mask.w));
          } else {
            u01 = mul2(u01, pack2(ks.x, ks.y));
            u23 = mul2(u23, pack2(ks.z, ks.w));
          }
        };
        uint32_t pk[16];
        uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull}; // 8 partial row sums as packed fp32 pairs
        auto weights = [&](int j, uint64_t e2) {
          float p0, p1;
          unpack2(e2, p0, p1);
          p0 = ex2(p0);
          p1 = ex2(p1);
          pk[j >> 1] = pack_bf16(p0, p1);
          sum2[(j >> 1) & 3] = add2(sum2[(j >> 1) & 3], pack2(p0, p1));
        };
        const uint64_t negm2 = pack2(-m_run, -m_run);
        if (masked == 0u) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            uint64_t u01, u23;
            scores4(j, false, u01, u23);
            weights(j, fma2(u01, A2, negm2));
            weights(j + 2, fma2(u23, A2, negm2));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            uint64_t u01, u23;
            scores4(j, true, u01, u23);
            weights(j, fma2(u01, A2, negm2));
            weights(j + 2, fma2(u23, A2, negm2));
          }
        }
        {
          float a0, a1, b0, b1;
          unpack2(add2(sum2[0], sum2[1]), a0, a1);
          unpack2(add2(sum2[2], sum2[3]), b0, b1);
          l += (a0 + a1) + (b0 + b1);
        }
        // P of this step takes the place of the last one's when that one's P.V is done: the Q.K^T of step g + 1 was issued
        // behind it, so its completion says so.
        if (!await_scores(g + 1u))
          break;
        if (g + 1u < n_steps) {
          ptx::tc_fence_after();
          ptx::tmem_ld_32x32(s_tmem + 32u * hf, r);
          masked = __float_as_uint(segment(g + 1u)[kTile]);
        }
        ptx::tmem_st_32x16(p_tmem + 16u * hf, pk);
        ptx::tmem_ld_wait();
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(p_full + 8 * t);
      }
    } else {
      for (uint32_t g = 0; g < n_steps && alive; ++g) {
        const float4 *tab = reinterpret_cast<const float4 *>(segment(g));
        uint32_t pk[16];
        uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull}; // 8 partial row sums as packed fp32 pairs
        auto weights = [&](int j, uint64_t e2) {
          float p0, p1;
          unpack2(e2, p0, p1);
          p0 = ex2(p0);
          p1 = ex2(p1);
          sum2[(j >> 1) & 3] = add2(sum2[(j >> 1) & 3], pack2(p0, p1));
          pk[j >> 1] = pack_bf16(p0, p1);
        };
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 ks = tab[j >> 2];
          float u[4];
          unpack2(mul2(pack2((float)(int32_t)r[j], (float)(int32_t)r[j + 1]), pack2(ks.x, ks.y)), u[0], u[1]);
          unpack2(mul2(pack2((float)(int32_t)r[j + 2], (float)(int32_t)r[j + 3]), pack2(ks.z, ks.w)), u[2], u[3]);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            r[j + i] = __float_as_uint(u[i]);
        }
        if (masked != 0u)
#pragma unroll
          for (int j = 0; j < 32; ++j)
            r[j] = __float_as_uint(__uint_as_float(r[j]) + reinterpret_cast<const float *>(tab)[kTile + j]);
#pragma unroll
        for (int j = 0; j < 32; j += 2)
          asm("max.f32 %0, %0, %1, %2;" : "+f"(mx4[(j >> 1) & 3]) : "f"(__uint_as_float(r[j])), "f"(__uint_as_float(r[j + 1])));
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        // power-of-two running maximum, of the whole row
        mx = fmaxf(mx, exchange(mx));
        if (!alive)
          break;
        float m_new = m_run;
        if (mx != -INFINITY)
          m_new = ceilf(mx * A);
        // Where it moves it goes kHeadroom beyond the ceiling, so that most steps move nothing (a move scales 128 output
        // columns, and without a headroom most warps had a row that moved in most steps) and no P exceeds 1: an output sum
        // stays within l max |V|. B2 S4608 H24 with q 4, 8 and 30 times larger: 704, 716 and 725 us without one, 586, 630 and 682
        // with 8, 566, 588 and 656 with 16, 566, 565 and 639 with 24, 566, 565 and 628 with 32. The rounding of the exponent's
        // fma (2^-20) does not show in the error against 64 bits; products below 2^-149 are lost, which for |V| above
        // 2^-115 is less than the rounding of the output (a maximum fixed at its bound may lie 60 above the scores).
        m_new = m_new > m_run ? m_new + kHeadroom : m_run;
        const bool grow = m_new > m_run && m_run != -INFINITY;
        if (__any_sync(0xffffffffu, grow)) {
          // rescale O (and l) by an exact power of two; needs P.V of the previous step finished
          // (grow implies an earlier step with a valid key, so g > 0)
          if (!ptx::mbar_wait(s_full + 8 * t, (g + 1u) & 1u, wait_ns)) { // a later wait of the warp ends the loop
            if (lane == 0)
              report(p.status, 5 + t, g);
            *abort_ptr = 1;
          }
          ptx::tc_fence_after();
          const float factor = grow ? ex2(m_run - m_new) : 1.0f;
          l *= factor;
#pragma unroll 1
          for (uint32_t c = 2u * hf; c < 2u * hf + 2u; ++c) {
            uint32_t o[32];
            ptx::tmem_ld_32x32(o_tmem + 32u * c, o);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j)
              o[j] = __float_as_uint(__uint_as_float(o[j]) * factor);
            ptx::tmem_st_32x32(o_tmem + 32u * c, o);
          }
          ptx::tmem_st_wait();
        }
        m_run = m_new;
        const float neg_m = (m_run == -INFINITY) ? 0.0f : -m_run;
        const uint64_t negm2 = pack2(neg_m, neg_m);
#pragma unroll
        for (int j = 0; j < 32; j += 2)
          weights(j, fma2(pack2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), A2, negm2));
        {
          float a0, a1, b0, b1;
          unpack2(add2(sum2[0], sum2[1]), a0, a1);
          unpack2(add2(sum2[2], sum2[3]), b0, b1);
          l += (a0 + a1) + (b0 + b1);
        }
        // P of this step takes the place of the last one's when that one's P.V is done: the Q.K^T of step g + 1 was issued
        // behind it, so its completion says so.
        if (!await_scores(g + 1u))
          break;
        if (g + 1u < n_steps) {
          ptx::tc_fence_after();
          ptx::tmem_ld_32x32(s_tmem + 32u * hf, r);
          masked = __float_as_uint(segment(g + 1u)[kTile]);
        }
        ptx::tmem_st_32x16(p_tmem + 16u * hf, pk);
        ptx::tmem_ld_wait();
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(p_full + 8 * t);
      }
    }
    const float l_own = l;
    if (alive)
      l += exchange(l);
    const uint32_t done_bar = s_full + 8 * t, done_parity = (n_steps + 1u) & 1u;
    // A row that other keys still join, in this cluster or in a later launch, is handed on as what its own keys
    // gave: no valid key counts as no maximum at all, and an m fixed at a bound so far above the scores that l is
    // smaller than a running maximum leaves it (2^-25 at least, which stays as it is: the next launch continues the
    // very same sums) comes down by the power of two that brings l to [1/2, 1). So every joined l is at least 2^-25, and
    // what a factor flushes (2^-127 and less) is too small to reach the sum. Gives the power of two.
    auto hand_on = [&](float &m_out) {
      float up = 1.0f;
      m_out = m_run;
      if (l == 0.0f) {
        m_out = -INFINITY;
      } else if (l < kLeastSum) {
        const int e = (int)(__float_as_uint(l) >> 23) - 126;
        m_out = m_run + (float)e;
        up = __uint_as_float((uint32_t)(127 - e) << 23);
        l *= up;
      }
      return up;
    };
    if (SPLIT) {
      // The CTAs of the cluster hold the unnormalised outputs of the same queries over parts of the keys. Every m
      // is an integer, so all move to the largest one by exact powers of two. Unit u = (query tile, 32 columns) is
      // finished by CTA u % split: the others send it their scaled fp32 sums through distributed shared memory.
      // Three cluster barriers, passed by every thread on every path.
      if (alive && !ptx::mbar_wait_warp(done_bar, done_parity, abort_ptr, wait_ns)) {
        if (!*abort_ptr && lane == 0)
          report(p.status, 7 + t, 0);
        *abort_ptr = 1;
        alive = false;
      }
      __syncwarp();
      ptx::cluster_sync(); // all MMAs of all CTAs are done: Q and the stage ring are free
      ptx::tc_fence_after();
      const uint32_t row = t * 128u + row_in_tile;
      float m_out;
      hand_on(m_out);
      for (uint32_t r = hf; r < split; r += 2u) // (m, l) of every CTA and row, behind the slots
        ptx::st_cluster_v2(ptx::mapa(stage_addr + 36u * kPartialBytes + (rank * 256u + row) * 8u, r), __float_as_uint(m_out), __float_as_uint(l));
      __syncwarp();
      ptx::cluster_sync();
      const float2 *mls = reinterpret_cast<const float2 *>(base_ptr + (stage_addr - base) + 36u * kPartialBytes) + row;
      float m_all = -INFINITY, l_all = 0.0f;
      for (uint32_t r = 0; r < split; ++r)
        m_all = fmaxf(m_all, mls[r * 256u].x);
      for (uint32_t r = 0; r < split; ++r)
        l_all += mls[r * 256u].x == -INFINITY ? 0.0f : mls[r * 256u].y * ex2(mls[r * 256u].x - m_all);
      const float factor = m_out == -INFINITY ? 0.0f : ex2(m_run - m_all);
      auto scaled = [&](uint32_t c, uint32_t(&o)[32]) {
        ptx::tmem_ld_32x32(o_tmem + 32u * c, o);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j)
          o[j] = __float_as_uint(__uint_as_float(o[j]) * factor);
      };
      // slot of (unit, sending CTA, lane quarter) in the ring of the unit's owner: at most 9 x 4 of 4 KB
      auto slot = [&](uint32_t u, uint32_t from) {
        return stage_addr + ((u / split * split + from) * 4u + quarter) * kPartialBytes + lane * 16u;
      };
#pragma unroll 1
      for (uint32_t c = 2u * hf; c < 2u * hf + 2u; ++c) {
        const uint32_t u = t * 4u + c, owner = u % split;
        if (owner == rank)
          continue;
        uint32_t o[32];
        scaled(c, o);
        const uint32_t dst = ptx::mapa(slot(u, rank), owner);
#pragma unroll
        for (int v = 0; v < 8; ++v)
          ptx::st_cluster_v4(dst + v * 512u, o[4 * v], o[4 * v + 1], o[4 * v + 2], o[4 * v + 3]);
      }
      __syncwarp();
      ptx::cluster_sync();
#pragma unroll 1
      for (uint32_t c = 2u * hf; c < 2u * hf + 2u; ++c) {
        const uint32_t u = t * 4u + c;
        if (u % split != rank)
          continue;
        uint32_t o[32];
        scaled(c, o);
        for (uint32_t from = 0; from < split; ++from) {
          if (from == rank)
            continue;
          const uint4 *part = reinterpret_cast<const uint4 *>(base_ptr + (slot(u, from) - base));
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const uint4 x = part[v * 32];
            o[4 * v] = __float_as_uint(__uint_as_float(o[4 * v]) + __uint_as_float(x.x));
            o[4 * v + 1] = __float_as_uint(__uint_as_float(o[4 * v + 1]) + __uint_as_float(x.y));
            o[4 * v + 2] = __float_as_uint(__uint_as_float(o[4 * v + 2]) + __uint_as_float(x.z));
            o[4 * v + 3] = __float_as_uint(__uint_as_float(o[4 * v + 3]) + __uint_as_float(x.w));
          }
        }
        uint32_t w[16];
        normalise(o, l_all, w);
        if (alive && row_ok) { // one launch's tail only: plain stores of 64 bytes per row
          uint4 *dst = reinterpret_cast<uint4 *>(p.out + (((uint64_t)batch * p.Sq + qrow) * p.H + head) * kTile + 32u * c);
#pragma unroll
          for (int v = 0; v < 4; ++v)
            dst[v] = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
        }
      }
    } else if (alive && n_kv > 0) {
      // Outputs are staged in a ring stage: tile 0 in the one after the last one used, tile 1 in the one after that. The
      // other query tile runs on its own and may still need what the stage held last (key tile n_kv - 4 + t, or Q codes).
      const uint32_t stage = (n_kv + t) % kStages;
      const bool free = n_kv + t >= (uint32_t)kStages
                            ? ptx::mbar_wait_uniform(kv_empty + 8 * stage, ((n_kv + t - kStages) / kStages) & 1u, abort_ptr, wait_ns)
                            : ptx::mbar_wait_uniform(q_full, 0, abort_ptr, wait_ns) &&
                                  ptx::mbar_wait_uniform(q_full + 8, 0, abort_ptr, wait_ns);
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(done_bar, done_parity, wait_ns)) || !free) {
        if (!*abort_ptr && lane == 0)
          report(p.status, 7 + t, 0);
        *abort_ptr = 1;
      } else {
        ptx::tc_fence_after();
        if (p.carry_out) {
          float m_out;
          const float up = hand_on(m_out);
          if (row_ok && hf == 0u)
            p.ml_state[state_row()] = make_float2(m_out, l_own * up);
          else if (row_ok)
            p.l2_state[state_row()] = l_own * up;
          float4 *carry = reinterpret_cast<float4 *>(p.o_state) + state_outputs();
          const uint32_t pitch = state_pitch();
#pragma unroll 1
          for (int c = 2 * (int)hf; c < 2 * (int)hf + 2; ++c) {
            uint32_t o[32];
            ptx::tmem_ld_32x32(o_tmem + 32u * c, o);
            ptx::tmem_ld_wait();
            if (row_ok) {
#pragma unroll
              for (int v = 0; v < 8; ++v)
                carry[(8 * c + v) * pitch] = make_float4(__uint_as_float(o[4 * v]) * up, __uint_as_float(o[4 * v + 1]) * up,
                                               __uint_as_float(o[4 * v + 2]) * up, __uint_as_float(o[4 * v + 3]) * up);
            }
          }
        } else {
          // Rows leave through shared memory, a warp's [32 rows x 64 columns] as four whole lines per store; a thread's
          // own stores touched 32 lines per instruction. (Tensor stores take the same time: until they have read the staging
          // the CTA waits 1200 clocks at its end.)
          uint8_t *box = base_ptr + (stage_addr - base) + stage * kStageBytes + (quarter * 2u + hf) * kOutBoxBytes;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t o[32];
            ptx::tmem_ld_32x32(o_tmem + 64u * hf + 32u * c, o);
            ptx::tmem_ld_wait();
            uint32_t w[16];
            normalise(o, l, w);
#pragma unroll
            for (int v = 0; v < 4; ++v)
              *reinterpret_cast<uint4 *>(box + lane * 128 + (((c * 4 + v) ^ (lane & 7)) << 4)) =
                  make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
          }
          __syncwarp();
          const uint32_t row0 = qrow - lane + (lane >> 3), part = lane & 7;
          uint4 *dst = reinterpret_cast<uint4 *>(p.out + (((uint64_t)batch * p.Sq + row0) * p.H + head) * kTile + 64u * hf) + part;
#pragma unroll
          for (uint32_t v = 0; v < 8; ++v) {
            const uint32_t row = 4u * v + (lane >> 3);
            if (row0 + 4u * v < p.Sq)
              dst[(uint64_t)(4u * v) * p.H * (kTile / 8)] = *reinterpret_cast<const uint4 *>(box + row * 128u + ((part ^ (row & 7u)) << 4));
          }
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (SPLIT && p.behind_whole)
    grid_dependency_wait();
}

void split_config(cudaLaunchConfig_t &config, cudaLaunchAttribute (&attrs)[2], uint32_t split) {
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kSmemBytes;
  attrs[0] = dependent_launch();
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = split;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  config.attrs = attrs;
  config.numAttrs = split > 1 ? 2 : 1;
}

// Clusters of `split` CTAs that fit on the device at once (one CTA per SM, clusters inside a GPC).
int resident_clusters(uint32_t split, int &count) {
  static const char keys[9] = {};
  return current_device_once(&keys[split], [](void *arg, int *value) -> int {
    cudaLaunchConfig_t config{};
    cudaLaunchAttribute attrs[2]{};
    const uint32_t ctas = *static_cast<uint32_t *>(arg);
    split_config(config, attrs, ctas);
    config.gridDim = dim3((unsigned)sm_count() / ctas * ctas); // the grid has to be a multiple of the cluster
    return check_cuda(cudaOccupancyMaxActiveClusters(value, attn_i8_kernel<true>, &config), "cudaOccupancyMaxActiveClusters");
  }, &split, &count);
}

// Items (batch, head, 256 queries) that run as one CTA each, and the split over the keys of the others. A last wave
// that is nearly empty costs as much as a full one: 3120 items of the 33272-token block are 21.08 waves of 148 SMs.
// Its items (or those of the last two waves) are split 2, 3, 4 or 8 ways over the key tiles by clusters. Modelled
// times in ns, measured on B200: 1480 per 128-key tile of a CTA, 6000 around them, 8000 more for a second launch
// and the exchange (an upper figure: the second launch fills the SMs as they become free), at least four tiles per CTA; a
// split has to give 3 %. H24, without -> with: 1 x 1700 tokens (1.14 waves) 56.0 -> 48.8 us, 1 x 2048 (1.30) 62.2 -> 56.8,
// 1 x 2304 (1.46) 68.0 -> 61.9, 2 x 2500 (3.24) 144.6 -> 134.4, 1 x 3300 (2.11) 131.6 -> 113.5; where the rule takes none,
// a split costs: 1 x 2560 (1.62) 74.6 -> 90.3, 1 x 2816 (1.78) 80.2 -> 96.9, 1 x 4608 (2.92) 182 -> 198.
int plan_split(uint64_t items, uint64_t tiles, uint64_t &whole, uint32_t &split) {
  constexpr uint64_t kTileNs = 1480, kItemNs = 6000, kExchangeNs = 8000;
  const uint64_t sms = (uint64_t)sm_count(), item_ns = kItemNs + tiles * kTileNs;
  whole = items;
  split = 1;
  uint64_t least = (items + sms - 1) / sms * item_ns * 97 / 100;
  for (uint64_t back = 0; back < 2; ++back) {
    if (items / sms < back)
      break;
    const uint64_t waves = items / sms - back, rest = items - waves * sms;
    if (rest == 0)
      continue;
    for (uint32_t s : {2u, 3u, 4u, 8u}) {
      if (tiles < 4ull * s)
        break;
      int resident = (int)(sms / s); // at most; asked for only where that would do
      auto time = [&]() {
        return waves * item_ns +
               (rest + resident - 1) / resident * (kItemNs + kExchangeNs + (tiles + s - 1) / s * kTileNs);
      };
      if (time() >= least)
        continue;
      if (int rc = resident_clusters(s, resident))
        return rc;
      if (resident > 0 && time() < least) {
        least = time();
        whole = waves * sms;
        split = s;
      }
    }
  }
  return kOk;
}

} // namespace

// Scratch: the key table (8 bytes per padded key and kv head) followed by one bound per key tile.
size_t attention_int8_scratch_bytes(uint64_t B, uint64_t S, uint64_t KV) {
  const uint64_t s_pad = (S + kTile - 1) / kTile * kTile;
  return (size_t)(B * KV * s_pad * sizeof(float2) + ((B * KV * (s_pad / kTile) * sizeof(float) + 15) & ~15ull));
}

size_t attention_int8_state_bytes(uint64_t B, uint64_t Sq, uint64_t H) {
  return (size_t)(B * Sq * H * (kTile * sizeof(float) + sizeof(float2) + sizeof(float)));
}

int attention_int8(const int8_t *q8, const float *qs, const int8_t *k8, const float *ks, const void *v_bf16,
                   const uint8_t *key_valid, uint64_t B, uint64_t Sq, uint64_t S, uint64_t H, uint64_t KV,
                   uint64_t D, float scale, void *scratch, size_t scratch_bytes, void *out_bf16,
                   cudaStream_t stream, const AttentionChunk *chunk, const AttentionSource *source) {
  // S is the number of key/value tokens from here on; Sq the number of query tokens.
  if (!q8 || !qs || !k8 || !ks || !v_bf16 || !out_bf16 || !scratch)
    return fail(kInvalidArgument, "Attention(INT8): null pointer");
  if (D != 128)
    return fail(kUnsupported, "Attention(INT8): head dimension must be 128");
  if (B == 0 || Sq == 0 || H == 0)
    return kOk;
  if (S == 0)
    return fail(kInvalidArgument, "Attention(INT8): no keys");
  if (KV == 0 || H % KV != 0)
    return fail(kInvalidArgument, "Attention(INT8): KvHeads must divide the head count");
  if (B * H * ((Sq + 255) / 256) > 0x7fffffffull || S > 0x7fffff00ull || Sq > 0x7fffff00ull)
    return fail(kUnsupported, "Attention(INT8): problem too large");
  if (scratch_bytes < attention_int8_scratch_bytes(B, S, KV))
    return fail(kInvalidArgument, "Attention(INT8): scratch buffer too small");
  if ((reinterpret_cast<uintptr_t>(q8) | reinterpret_cast<uintptr_t>(k8) |
       reinterpret_cast<uintptr_t>(v_bf16) | reinterpret_cast<uintptr_t>(out_bf16) |
       reinterpret_cast<uintptr_t>(scratch)) & 15)
    return fail(kUnsupported, "Attention(INT8): pointers must be 16-byte aligned");
  DeviceStatus *status = device_status_words();
  if (!status)
    return fail(kOutOfMemory, "Attention(INT8): device status words are unavailable");
  const uint32_t s_pad = (uint32_t)((S + kTile - 1) / kTile * kTile);
  const uint32_t all_tiles = s_pad / kTile;
  uint32_t begin[2] = {0, 0}, count[2] = {all_tiles, 0};
  if (chunk) {
    for (int i = 0; i < 2; ++i) {
      begin[i] = chunk->tile_begin[i];
      count[i] = chunk->tile_count[i];
      if ((uint64_t)begin[i] + count[i] > all_tiles)
        return fail(kInvalidArgument, "Attention(INT8): key tile range beyond the key axis");
    }
    if (count[0] + count[1] == 0)
      return fail(kInvalidArgument, "Attention(INT8): a launch needs at least one key tile");
    if ((chunk->carry_in || chunk->carry_out) && (!chunk->state || (reinterpret_cast<uintptr_t>(chunk->state) & 15)))
      return fail(kInvalidArgument, "Attention(INT8): carried state needs a 16-byte aligned state buffer");
  }

  CUtensorMap map_q, map_k, map_v;
  {
    const uint64_t dims[4] = {128, H, Sq, B};
    const uint64_t strides[3] = {128, H * 128, Sq * H * 128};
    const uint32_t box[4] = {128, 1, 128, 1};
    if (int rc = encode_tensor_map(&map_q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, q8, dims, strides, box,
                                   CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  }
  {
    const uint64_t dims[4] = {128, KV, S, B};
    const uint64_t strides[3] = {128, KV * 128, S * KV * 128};
    const uint32_t box[4] = {128, 1, 128, 1};
    if (int rc = encode_tensor_map(&map_k, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, k8, dims, strides, box,
                                   CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  }
  {
    const uint64_t dims[4] = {128, KV, S, B};
    const uint64_t strides[3] = {256, KV * 256, S * KV * 256};
    const uint32_t box[4] = {64, 1, 128, 1};
    if (int rc = encode_tensor_map(&map_v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, v_bf16, dims, strides, box,
                                   CU_TENSOR_MAP_SWIZZLE_128B))
      return rc;
  }
  static const char attr_key = 0; // the opt-in belongs to the function in one context: once per device
  if (int rc = current_device_once(&attr_key, [](void *, int *) -> int {
        for (auto *kernel : {attn_i8_kernel<false>, attn_i8_kernel<true>})
          if (int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)kSmemBytes),
                                  "cudaFuncSetAttribute(attn_i8_kernel)"))
            return rc;
        return kOk;
      }, nullptr, nullptr))
    return rc;

  float *table = static_cast<float *>(scratch);
  float *tile_bound = table + B * KV * s_pad * 2;
  // q / k still in bf16: one launch quantises them and, with k, also builds the key table
  if (source && (source->q || source->k)) {
    if (chunk || (reinterpret_cast<uintptr_t>(source->q) | reinterpret_cast<uintptr_t>(source->k)) & 15)
      return fail(kUnsupported, "Attention(INT8): pointers must be 16-byte aligned");
    OperandParams o{};
    o.q = static_cast<const uint4 *>(source->q);
    o.k = static_cast<const uint4 *>(source->k);
    o.q8 = const_cast<int8_t *>(q8);
    o.k8 = const_cast<int8_t *>(k8);
    o.qs = const_cast<float *>(qs);
    o.ks = const_cast<float *>(ks);
    o.key_valid = key_valid;
    o.table = table;
    o.tile_bound = tile_bound;
    o.q_rows = source->q ? B * Sq * H : 0;
    o.S = (uint32_t)S;
    o.KV = (uint32_t)KV;
    o.S_pad = s_pad;
    const uint64_t key_blocks = source->k ? B * KV * all_tiles : 0, blocks = key_blocks + (o.q_rows + 127) / 128;
    if (blocks > 0x7fffffffull)
      return fail(kUnsupported, "Attention(INT8): problem too large");
    o.key_blocks = (uint32_t)key_blocks;
    const bool one_round = blocks <= 2ull * (uint64_t)sm_count();
    if (int rc = launch_ahead("attention_operands_kernel launch", one_round ? attention_operands_kernel<2> : attention_operands_kernel<4>,
                              blocks, one_round ? 512 : 256, 0, stream, o))
      return rc;
  }
  if (!(source && source->k)) {
    const uint64_t blocks = B * KV * (count[0] + count[1]);
    if (blocks > 0x7fffffffull)
      return fail(kUnsupported, "Attention(INT8): problem too large");
    if (int rc = launch_ahead("key_table_kernel launch", key_table_kernel, blocks, 128, 0, stream, k8, ks, key_valid, table, tile_bound,
                              (uint32_t)S, (uint32_t)KV, s_pad, begin[0], count[0], begin[1], count[1]))
      return rc;
  }
  AttnParams p{};
  p.q8 = q8;
  p.qs = qs;
  p.table = table;
  p.tile_bound = tile_bound;
  p.out = static_cast<uint16_t *>(out_bf16);
  p.B = (uint32_t)B;
  p.Sq = (uint32_t)Sq;
  p.Sk = (uint32_t)S;
  p.H = (uint32_t)H;
  p.KV = (uint32_t)KV;
  p.q_blocks = divisor((Sq + 255) / 256);
  p.heads = divisor(H);
  p.group = divisor(H / KV);
  p.S_pad = s_pad;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.wait_ns = wait_limit_ns();
  p.status = status;
  for (int i = 0; i < 2; ++i) {
    p.tile_begin[i] = begin[i];
    p.tile_count[i] = count[i];
  }
  if (chunk && (chunk->carry_in || chunk->carry_out)) {
    // state buffer: fp32 outputs [B,Sq,H,128], then (m, l) and the other half's l per row
    p.o_state = static_cast<float *>(chunk->state);
    p.ml_state = reinterpret_cast<float2 *>(p.o_state + B * Sq * H * kTile);
    p.l2_state = reinterpret_cast<float *>(p.ml_state + B * Sq * H);
    p.carry_in = chunk->carry_in ? 1u : 0u;
    p.carry_out = chunk->carry_out ? 1u : 0u;
  }
  const uint64_t items = B * H * ((Sq + 255) / 256);
  uint64_t whole = items;
  uint32_t split = 1;
  if (!chunk)
    if (int rc = plan_split(items, all_tiles, whole, split))
      return rc;
  auto launch = [&](uint64_t first, uint64_t count, uint32_t ctas) {
    p.item0 = (uint32_t)first;
    // Items that start one by one, as SMs become free behind the unsplit ones, are 3 to 5 % of a call faster than all
    // together behind them, except where nearly all clusters of three that fit (45) are needed: started one by one they
    // leave gaps in the GPCs, and the last ones wait for a second round. 148 + n items of 16 tiles, one by one / together:
    // n = 40 69.5 / 72.3 us, 42 70.7 / 73.1, 43 74.7 / 73.5, 44 79.7 / 73.6, 45 81.7 / 73.6; of 32 tiles n = 42 116 / 118,
    // 43 120 / 117. Clusters of two, four and eight leave none: 74 of two 76.5 / 78.1, 33 of four 69.5 / 72.3, 15 of eight
    // (32 tiles) 104 / 107.
    bool together = false;
    if (first != 0 && ctas == 3) {
      int resident = 0;
      if (int rc = resident_clusters(ctas, resident))
        return rc;
      together = count + 2 >= (uint64_t)resident;
    }
    p.behind_whole = first != 0 && !together ? 1u : 0u;
    p.split_follows = first == 0 && count < items ? 1u : 0u;
    p.split = ctas;
    cudaLaunchConfig_t config{};
    cudaLaunchAttribute attrs[2]{};
    split_config(config, attrs, ctas);
    config.gridDim = dim3((unsigned)(count * ctas));
    config.stream = stream;
    if (together) {
      config.attrs = attrs + 1;
      config.numAttrs = 1;
    }
    return launched(cudaLaunchKernelEx(&config, ctas > 1 ? attn_i8_kernel<true> : attn_i8_kernel<false>, map_q, map_k, map_v, p),
                    "attn_i8_kernel launch");
  };
  if (whole)
    if (int rc = launch(0, whole, 1))
      return rc;
  return whole < items ? launch(whole, items - whole, split) : kOk;
}

} // namespace difb200
