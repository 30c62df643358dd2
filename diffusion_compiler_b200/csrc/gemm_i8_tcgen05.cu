// LinearInt8Scaled for sm_100a: Y[M,N] = bf16((float(X[M,K] . W[N,K]^T) * xs[m]) * ws[n]),
// optionally followed by the BiasAdd and tanh-Gelu ops that the W8A8 rewrite puts after it.
// Semantics: reference src/runtime/cpu_executor.cpp:309-335 (multiplication order row scale
// first, then column scale), BiasAdd :1288-1296, Gelu :93-113; it replaces the reference's
// Sm80 mma.sync CUTLASS kernel (src/runtime/cutlass_gemm.cu:185-303).
//
// Structure: persistent CTAs, one per SM. Both operands are K-major INT8, brought in by TMA as
// 128-byte-swizzled [rows x 128 B] boxes into a shared-memory ring. One thread issues
// tcgen05.mma kind::i8 into one of two BN-column INT32 accumulators in tensor memory, so the
// epilogue of tile i overlaps the MMAs of tile i+1. Warp roles: 0 = TMA producer, 1 = TMEM owner
// + MMA issuer, 2..9 = epilogue: two warps per TMEM lane quarter (warp_id % 4), one for each
// column half of the tile (four epilogue warps could not keep up with the K = 3072 main
// loop once bias and GELU are fused in).
//
// Forms of the same kernel (template parameters CTAS and BN, the tile's columns; choose_form has the rule):
//   CTAS = 1: 128 x BN tile per CTA, cta_group::1, 4 stages of 48 KB (BN 256) or 5 of 32 KB (BN 128). A tile
//             may be split over the k-blocks: the CTAs of a cluster each sum their share, then every CTA
//             finishes the 32-column chunks it owns (chunk % split) from its own accumulator and the others'
//             partial sums, which arrive in its freed stage ring through distributed shared memory. INT32
//             sums are exact, so the bits do not depend on the split.
//   CTAS = 2: a CTA pair (cluster of 2) computes a 256 x BN tile with cta_group::2 MMAs: each CTA
//             stages its 128 rows of A and only its BN / 2 rows (half) of the B tile, 5 stages of
//             32 KB (BN 256), 6 of 28 KB (BN 192) or 7 of 24 KB (BN 128). This halves the B bytes every SM moves through
//             shared memory per MAC -- at 8192 INT8 MACs/clk/SM the 128x256 single-CTA tile needs
//             48 KB written plus 48 KB read per 512 clocks, which is what bounds the CTAS = 1 form.
//             The leader CTA (cluster rank 0) issues the MMAs; both CTAs load, and both run the
//             epilogue on their own 128 rows.
//             TMA loads never use multicast. The bytes of both CTAs are counted on the leader's
//             mbarrier (the peer issues the cta_group::2 form of the load, whose completion may
//             target the peer CTA's barrier); the leader releases stages and publishes
//             accumulators to both CTAs with one tcgen05.commit that signals the mbarrier of both
//             CTAs. The only remaining software signal across the pair is the epilogue's arrive
//             on the leader's accumulator-empty barrier, with CTA-scope release: a cluster-scope
//             release arrive per k-block costs microseconds while TMA traffic is in flight.
// Problems of few rows have kernels of their own (linear_few_rows.cu).
#include "gemm_common.cuh"
#include "ptx.cuh"

#include <cstdio>
#include <cstdlib>
#include <mutex>

namespace difb200 {

int encode_tensor_map(CUtensorMap *out, CUtensorMapDataType type, uint32_t rank, const void *base,
                      const uint64_t *dims, const uint64_t *strides_bytes, const uint32_t *box,
                      CUtensorMapSwizzle swizzle) {
  typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                               const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                               const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn encode = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult query;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &query) ==
            cudaSuccess &&
        query == cudaDriverEntryPointSuccess)
      encode = reinterpret_cast<EncodeFn>(fn);
  });
  if (!encode)
    return fail(kInternalError, "cuTensorMapEncodeTiled is unavailable in this driver");
  cuuint32_t elem_strides[5] = {1, 1, 1, 1, 1};
  cuuint64_t gdims[5];
  cuuint64_t gstrides[5];
  cuuint32_t gbox[5];
  for (uint32_t i = 0; i < rank; ++i) {
    gdims[i] = dims[i];
    gbox[i] = box[i];
    if (i + 1 < rank)
      gstrides[i] = strides_bytes[i];
  }
  const CUresult rc = encode(out, type, rank, const_cast<void *>(base), gdims, gstrides, gbox,
                             elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS)
    return fail(kInvalidArgument, "cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)rc));
  return kOk;
}

namespace {

constexpr int kBM = 128, kBK = 128; // per-CTA rows, BK in bytes == INT8 elements
constexpr int kUmmaK = 32;
constexpr uint32_t kABytes = kBM * kBK;
constexpr int kThreads = 320;
constexpr int kEpilogueWarps = 8;
template <int CTAS, int BN>
struct Cfg {
  static constexpr uint32_t kBRows = BN / CTAS;                  // rows of the B tile this CTA stages
  static constexpr uint32_t kBBytes = kBRows * kBK;
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = kStageBytes <= 24 * 1024 ? 7 : kStageBytes <= 28 * 1024 ? 6 : kStageBytes <= 32 * 1024 ? 5 : 4; // 160-192 KB
  // staging boxes per epilogue warp (two let a TMA store drain while the next box is filled;
  // the 128x256 form has room for one)
  static constexpr uint32_t kBoxes = kStageBytes <= 32 * 1024 ? 2 : 1;
  static constexpr uint32_t kStagingBytes = kEpilogueWarps * kBoxes * 32 * 64;
  static constexpr uint32_t kScaleBytes = kEpilogueWarps * BN * 4; // per warp: scales and biases of its BN / 2 columns
  static constexpr uint32_t kTileM = kBM * CTAS;                 // rows of the (pair's) output tile
  static constexpr uint32_t kTmemCols = BN == 192 ? 512 : 2 * BN; // two accumulators; a power of two
};
// Epilogue staging: per epilogue warp one or two [32 rows x 32 bf16] boxes (64-byte rows, 64B TMA swizzle).
constexpr uint32_t kStoreBoxBytes = 32 * 64;
// Split form: a partial [32 rows x 32 columns] of INT32 on its way to the CTA that finishes it.
constexpr uint32_t kPartialBytes = 32 * 32 * 4;
template <int CTAS, int BN>
constexpr size_t smem_bytes() {
  return 1024 /*alignment slack*/ + (size_t)Cfg<CTAS, BN>::kStages * Cfg<CTAS, BN>::kStageBytes +
         Cfg<CTAS, BN>::kStagingBytes + Cfg<CTAS, BN>::kScaleBytes + 256;
}

__device__ __forceinline__ void report_timeout(DeviceStatus *status, uint32_t role, uint32_t detail) {
  if (atomicExch(&status->flag, 1u) == 0u) {
    status->kernel = 2u;
    status->role = role;
    status->detail = detail;
  }
}

template <int CTAS, int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_i8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_c, const GemmParams p) {
  constexpr int kStages = Cfg<CTAS, BN>::kStages;
  constexpr uint32_t kStageBytes = Cfg<CTAS, BN>::kStageBytes;
  constexpr uint32_t kTileM = Cfg<CTAS, BN>::kTileM;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t cta_rank = CTAS == 2 ? ptx::cluster_ctarank() : 0u;  // 0 = leader of the pair
  const uint32_t split = CTAS == 2 ? 1u : p.split, split_rank = split > 1 ? ptx::cluster_ctarank() : 0u;
  const uint32_t unit = CTAS == 2 ? blockIdx.x >> 1 : blockIdx.x / split; // tile-scheduling unit
  const uint32_t units = CTAS == 2 ? gridDim.x >> 1 : gridDim.x / split;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t staging_base = smem_base + kStages * kStageBytes;
  const uint32_t scale_base = staging_base + Cfg<CTAS, BN>::kStagingBytes;
  const uint32_t bar_base = scale_base + Cfg<CTAS, BN>::kScaleBytes;
  // barrier layout (8 bytes each): full[kStages], empty[kStages], tmem_full[2], tmem_empty[2]; then a word
  // for the TMEM base address and a word for the abort flag.
  const uint32_t full_bar = bar_base, empty_bar = bar_base + 8 * kStages;
  const uint32_t tfull_bar = bar_base + 16 * kStages, tempty_bar = tfull_bar + 16;
  const uint32_t tmem_slot = tempty_bar + 16;
  volatile uint32_t *slot_ptr =
      reinterpret_cast<volatile uint32_t *>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  volatile uint32_t *abort_ptr = slot_ptr + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long wait_ns = p.wait_ns;
  const uint32_t tiles_m = (p.M + kTileM - 1) / kTileM, tiles_n = (p.N + BN - 1) / BN;
  const uint32_t num_tiles = tiles_m * tiles_n;
  const uint32_t k_blocks = (p.K + kBK - 1) / kBK;
  // this CTA's k-blocks of every tile (all of them unless the tile is split; never empty: split <= k_blocks)
  const uint32_t kb_first = k_blocks * split_rank / split, kb_end = k_blocks * (split_rank + 1u) / split;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(full_bar + 8 * s, 1);
      ptx::mbar_init(empty_bar + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(tfull_bar + 8 * b, 1);
      ptx::mbar_init(tempty_bar + 8 * b, kEpilogueWarps * CTAS);    // epilogue warps of every CTA of the pair
    }
    *abort_ptr = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
  }
  if (warp == 1) {
    if (CTAS == 2) {
      ptx::tmem_alloc_pair(tmem_slot, Cfg<CTAS, BN>::kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_slot, Cfg<CTAS, BN>::kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (CTAS == 2)
    ptx::cluster_sync(); // the peer's barriers are initialised before anything arrives on them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *slot_ptr;

  // The producer warp and the MMA warp run their loops with all 32 lanes and warp-uniform
  // control flow (every wait ends in a vote) and let one elected lane issue the asynchronous
  // instructions. Loop state, addresses and descriptors are then warp-uniform values; with a
  // single-lane loop (divergent code) every operand of every TMA / MMA instruction is first
  // moved between register files, and that loop needed 640-680 cycles per k-block against the
  // 512 cycles the four MMAs of a k-block take.
  auto give_up = [&](uint32_t role, uint32_t detail) {
    if (lane == 0) {
      if (!*abort_ptr)
        report_timeout(p.status, role, detail);
      *abort_ptr = 1;
    }
  };
  // The kernel in front (the quantiser, as a rule) may still run up to here.
  if (warp != 0)
    grid_dependency_wait();
  if (warp == 0) {
    const uint32_t stage_tx = CTAS == 2 ? 2 * kStageBytes : Cfg<CTAS, BN>::kBBytes + p.a_rows * kBK; // bytes of a stage's loads
    auto rows_of = [&](uint32_t tile) { return (int32_t)((tile / tiles_n) * kTileM + cta_rank * kBM); };
    auto columns_of = [&](uint32_t tile) { return (int32_t)((tile % tiles_n) * BN + cta_rank * Cfg<CTAS, BN>::kBRows); };
    // One operand's part of k-block kb. A pair counts the bytes of both CTAs on the leader's barrier: the leader
    // expects them all, the peer's loads complete their bytes there (cta_group::2 form of the load) and the peer
    // itself never arrives.
    auto load = [&](const CUtensorMap *map, uint32_t dst, uint32_t bar, uint32_t kb, int32_t first) {
      if (CTAS == 2 && cta_rank != 0)
        ptx::tma_load_2d_pair(dst, map, ptx::mapa(bar, 0), (int32_t)(kb * kBK), first);
      else
        ptx::tma_load_2d(dst, map, bar, (int32_t)(kb * kBK), first);
    };
    // The first k-blocks of the first tile, as many as the ring holds, whose weights are requested before the wait and
    // whose rows behind it: a loop of its own, since a test for them in every k-block of the loop below cost the
    // 256 x 128 pairs 18 % (2048 x 12288 x 3072: 61 -> 72 us; a k-block of theirs takes 210 ns).
    const uint32_t early = p.weights_first && unit < num_tiles ? min(kb_end - kb_first, (uint32_t)kStages) : 0u;
    if (early != 0u && ptx::elect_one())
      for (uint32_t i = 0; i < early; ++i) {
        if (cta_rank == 0)
          ptx::mbar_expect_tx(full_bar + 8 * i, stage_tx);
        load(&map_b, smem_base + i * kStageBytes + kABytes, full_bar + 8 * i, kb_first + i, columns_of(unit));
      }
    grid_dependency_wait();
    if (early != 0u && ptx::elect_one())
      for (uint32_t i = 0; i < early; ++i)
        load(&map_a, smem_base + i * kStageBytes, full_bar + 8 * i, kb_first + i, rows_of(unit));
    uint32_t stage = early == (uint32_t)kStages ? 0u : early, phase = early == (uint32_t)kStages ? 1u : 0u;
    uint32_t kb = kb_first + early;
    bool ok = true;
    for (uint32_t tile = unit; tile < num_tiles && ok; tile += units) {
      const int32_t m0 = rows_of(tile), n0 = columns_of(tile);
      for (; kb < kb_end; ++kb) {
        if (!ptx::mbar_wait_warp(empty_bar + 8 * stage, phase ^ 1u, abort_ptr, wait_ns)) {
          give_up(0, kb);
          ok = false;
          break;
        }
        const uint32_t a_dst = smem_base + stage * kStageBytes, b_dst = a_dst + kABytes;
        const uint32_t bar = full_bar + 8 * stage;
        const int32_t k0 = (int32_t)(kb * kBK);
        if (kb == p.withhold_kb) {
          // test aid: the bytes are announced but never loaded, so the consumer's wait on this
          // stage runs out and the kernel leaves through its give-up path
          if (cta_rank == 0 && ptx::elect_one())
            ptx::mbar_expect_tx(bar, stage_tx);
        } else if (ptx::elect_one()) {
          if (CTAS == 2) {
            if (cta_rank == 0) {
              ptx::mbar_expect_tx(bar, stage_tx);
              ptx::tma_load_2d(a_dst, &map_a, bar, k0, m0);
              ptx::tma_load_2d(b_dst, &map_b, bar, k0, n0);
            } else {
              const uint32_t leader_bar = ptx::mapa(bar, 0);
              ptx::tma_load_2d_pair(a_dst, &map_a, leader_bar, k0, m0);
              ptx::tma_load_2d_pair(b_dst, &map_b, leader_bar, k0, n0);
            }
          } else {
            ptx::mbar_expect_tx(bar, stage_tx);
            ptx::tma_load_2d(a_dst, &map_a, bar, k0, m0);
            ptx::tma_load_2d(b_dst, &map_b, bar, k0, n0);
          }
        }
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      kb = kb_first;
    }
  } else if (warp == 1) {
    if (cta_rank == 0) {
      constexpr uint32_t idesc = ptx::make_idesc(2 /*S32*/, 1 /*S8*/, 1 /*S8*/, 0, 0, kTileM, BN);
      const uint64_t desc0 = ptx::smem_desc_sw128(smem_base, 16, 1024);
      uint32_t stage = 0, phase = 0, local = 0;
      bool ok = true;
      auto commit = [&](uint32_t bar) { // arrives on `bar` of every CTA of the pair
        if (CTAS == 2)
          ptx::mma_commit_pair_both(bar, (uint16_t)3);
        else
          ptx::mma_commit(bar);
      };
      for (uint32_t tile = unit; tile < num_tiles && ok; tile += units, ++local) {
        const uint32_t acc = local & 1u, acc_phase = (local >> 1) & 1u;
        if (!ptx::mbar_wait_warp(tempty_bar + 8 * acc, acc_phase ^ 1u, abort_ptr, wait_ns)) {
          give_up(1, 0xffffu);
          break;
        }
        ptx::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (uint32_t kb = kb_first; kb < kb_end; ++kb) {
          if (!ptx::mbar_wait_warp(full_bar + 8 * stage, phase, abort_ptr, wait_ns)) {
            give_up(1, kb);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          // descriptors of this stage: only the 14-bit address field (16-byte units) moves
          const uint64_t a_desc = desc0 + (uint64_t)((stage * kStageBytes) >> 4);
          const uint64_t b_desc = a_desc + (uint64_t)(kABytes >> 4);
          if (ptx::elect_one()) {
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; ++k) {
              const uint32_t accumulate = k != 0 ? 1u : (kb != kb_first ? 1u : 0u);
              if (CTAS == 2)
                ptx::mma_i8_ss_pair(d_tmem, a_desc + (uint64_t)(k * kUmmaK >> 4), b_desc + (uint64_t)(k * kUmmaK >> 4),
                                    idesc, accumulate);
              else
                ptx::mma_i8_ss(d_tmem, a_desc + (uint64_t)(k * kUmmaK >> 4), b_desc + (uint64_t)(k * kUmmaK >> 4),
                               idesc, accumulate);
            }
            commit(empty_bar + 8 * stage); // frees the smem stage when these MMAs retire
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok && ptx::elect_one())
          commit(tfull_bar + 8 * acc); // accumulator complete
      }
    }
  } else {
    const uint32_t quarter = (uint32_t)warp & 3u;        // TMEM lane quarter of this warp
    const uint32_t ewarp = (uint32_t)warp - 2u;          // 0..7
    const uint32_t col_half = ewarp >> 2;                // columns [BN/2 col_half, BN/2 col_half + BN/2)
    uint32_t local = 0, store_buf = 0;
    uint8_t *generic_base = smem_raw + (smem_base - smem_u32(smem_raw));
    float *scale_smem = reinterpret_cast<float *>(generic_base + (scale_base - smem_base));
    const uint32_t my_staging = staging_base + ewarp * Cfg<CTAS, BN>::kBoxes * kStoreBoxBytes;
    uint8_t *my_staging_ptr = generic_base + (my_staging - smem_base);
    for (uint32_t tile = unit; tile < num_tiles; tile += units, ++local) {
      const uint32_t acc = local & 1u, acc_phase = (local >> 1) & 1u;
      const uint32_t m0 = (tile / tiles_n) * kTileM + cta_rank * kBM, n0 = (tile % tiles_n) * BN;
      // column scales and biases of this tile -> this warp's private shared-memory copy
      // (warp-private so that no cross-warp barrier is needed)
      float *cs = scale_smem + ewarp * BN, *bs = cs + BN / 2; // this warp's BN / 2 columns
      __syncwarp();
#pragma unroll
      for (int i = 0; i < BN / 64; ++i) {
        const uint32_t c = lane + 32u * i, n = n0 + col_half * (BN / 2) + c;
        cs[c] = n < p.N ? load_produced(p.col_scales + n) : 0.0f;
        bs[c] = ((p.epilogue & kEpiBias) && n < p.N) ? bf16_bits_to_f32(load_produced(p.bias + n)) : 0.0f;
      }
      __syncwarp();
      const bool complete = ptx::mbar_wait_warp(tfull_bar + 8 * acc, acc_phase, abort_ptr, wait_ns);
      if (!complete) {
        if (!*abort_ptr && lane == 0)
          report_timeout(p.status, 2, tile);
        *abort_ptr = 1;
      }
      if (split > 1) { // a split launch has one tile per cluster: every thread passes here once
        __syncwarp();
        ptx::cluster_sync(); // every CTA's MMAs are complete: the stage rings are free to receive partial sums
        ptx::tc_fence_after();
#pragma unroll 1
        for (uint32_t sub = 0; sub < BN / 64; ++sub) {
          const uint32_t chunk = col_half * (BN / 64) + sub, owner = chunk % split;
          if (owner == split_rank)
            continue;
          uint32_t r[32];
          ptx::tmem_ld_32x32(tmem_base + ((quarter * 32u) << 16) + acc * BN + chunk * 32u, r);
          ptx::tmem_ld_wait();
          const uint32_t slot = (chunk / split * split + split_rank) * 4u + quarter;
          const uint32_t dst = ptx::mapa(smem_base + slot * kPartialBytes + lane * 16u, owner);
#pragma unroll
          for (int v = 0; v < 8; ++v)
            ptx::st_cluster_v4(dst + v * 512u, r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
        }
        __syncwarp();
        ptx::cluster_sync(); // all partial sums have arrived
      }
      if (!complete)
        break;
      ptx::tc_fence_after();
      const uint32_t row = m0 + quarter * 32u + lane;
      const bool row_ok = row < p.M;
      const float rs = row_ok ? load_produced(p.row_scales + row) : 0.0f;
      // A warp whose 32 rows lie behind the last one has nothing to convert. Nor may it fill a box: the wait for a box counts
      // the groups committed behind its last store, so that a fill without a store and commit of its own would let the next
      // fill overwrite a box that an earlier tile's store still reads.
      const uint32_t subs = m0 + quarter * 32u < p.M ? BN / 64 : 0u;
#pragma unroll 1
      for (uint32_t sub = 0; sub < subs; ++sub) {
        const uint32_t chunk = col_half * (BN / 64) + sub; // 32-column chunk of the tile
        uint32_t r[32];
        ptx::tmem_ld_32x32(tmem_base + ((quarter * 32u) << 16) + acc * BN + chunk * 32u, r);
        ptx::tmem_ld_wait();
        if (split > 1) {
          if (chunk % split != split_rank)
            continue; // finished by another CTA of the cluster
          for (uint32_t from = 0; from < split; ++from) { // INT32 sums: exact in any order
            if (from == split_rank)
              continue;
            const uint4 *part = reinterpret_cast<const uint4 *>(
                generic_base + ((chunk / split * split + from) * 4u + quarter) * kPartialBytes) + lane;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
              const uint4 x = part[v * 32];
              r[4 * v] += x.x;
              r[4 * v + 1] += x.y;
              r[4 * v + 2] += x.z;
              r[4 * v + 3] += x.w;
            }
          }
        }
        const uint32_t n_base = n0 + chunk * 32u;
        if (n_base >= p.N)
          continue; // (warp-uniform) whole chunk past the N edge
        if (p.acc_out && row_ok) {
          for (int i = 0; i < 32; ++i)
            if (n_base + i < p.N)
              p.acc_out[(size_t)row * p.N + n_base + i] = (int32_t)r[i];
        }
        uint32_t packed[16];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const float4 c4 = *reinterpret_cast<const float4 *>(cs + sub * 32 + 4 * g);
          const float4 b4 = *reinterpret_cast<const float4 *>(bs + sub * 32 + 4 * g);
          const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, bb[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = 4 * g + 2 * h;
            float y0 = __fmul_rn(__fmul_rn((float)(int32_t)r[i], rs), cc[2 * h]);
            float y1 = __fmul_rn(__fmul_rn((float)(int32_t)r[i + 1], rs), cc[2 * h + 1]);
            uint32_t pk = pack_bf16x2(y0, y1);
            if (p.epilogue & kEpiBias) {
              y0 = __fadd_rn(__uint_as_float(pk << 16), bb[2 * h]);
              y1 = __fadd_rn(__uint_as_float(pk & 0xffff0000u), bb[2 * h + 1]);
              pk = pack_bf16x2(y0, y1);
            }
            if (p.epilogue & kEpiGeluTanh) {
              y0 = gelu_tanh(__uint_as_float(pk << 16));
              y1 = gelu_tanh(__uint_as_float(pk & 0xffff0000u));
              pk = pack_bf16x2(y0, y1);
            }
            packed[i >> 1] = pk;
          }
        }
        if (p.tma_store) {
          // stage this warp's [32 x 32] box (64-byte rows, 16-byte chunk c of row r stored at
          // c ^ ((r >> 1) & 3): the 64B TMA swizzle, conflict-free), then one TMA store.
          if (lane == 0) { // the box about to be filled must have been read by its last store
            if (Cfg<CTAS, BN>::kBoxes == 2)
              asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            else
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          }
          __syncwarp();
          uint8_t *box = my_staging_ptr + store_buf * kStoreBoxBytes;
#pragma unroll
          for (int v = 0; v < 4; ++v)
            *reinterpret_cast<uint4 *>(box + lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4)) =
                make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
          ptx::fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                             reinterpret_cast<uint64_t>(&map_c)),
                         "r"(my_staging + store_buf * kStoreBoxBytes), "r"((int32_t)n_base),
                         "r"((int32_t)(m0 + quarter * 32u))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
          store_buf = Cfg<CTAS, BN>::kBoxes == 2 ? store_buf ^ 1u : 0u;
        } else if (row_ok) {
          uint16_t *dst = p.out + (size_t)row * p.N + n_base;
          for (int i = 0; i < 32; ++i)
            if (n_base + i < p.N)
              dst[i] = (uint16_t)((packed[i >> 1] >> (16 * (i & 1))) & 0xffffu);
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTAS == 2)
          ptx::mbar_arrive_remote(ptx::mapa(tempty_bar + 8 * acc, 0)); // the leader issues the MMAs
        else
          ptx::mbar_arrive(tempty_bar + 8 * acc);
      }
    }
    if (lane == 0)
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  if (split > 1 && warp < 2) { // the two barriers of the epilogue's exchange count every thread
    __syncwarp();
    ptx::cluster_sync();
    ptx::cluster_sync();
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (CTAS == 2)
    ptx::cluster_sync(); // neither CTA leaves (or frees TMEM) while the peer may still touch it
  if (warp == 1) {
    ptx::tc_fence_after();
    if (CTAS == 2)
      ptx::tmem_dealloc_pair(tmem_base, Cfg<CTAS, BN>::kTmemCols);
    else
      ptx::tmem_dealloc(tmem_base, Cfg<CTAS, BN>::kTmemCols);
  }
}

// Tile form of a problem: CTAs per tile, tile columns, and the CTAs that share the k-blocks of a tile.
struct Form {
  int ctas, tile_n, split;
};
// The form with the least modelled time: waves of tiles x k-blocks per CTA x time of a k-block, plus what a
// launch pays once (first loads, the last tile's epilogue, the exchange of a split). The figures, in ns, are
// fitted to event times of every form at N 3072 / 9216 / 12288 / 16384, K 3072 / 8192 / 12288 and 17 to 12000 rows; over 160
// such problems the form chosen is within 5 % of the best one, and within 2 % of it for all but 20. Large problems go to the
// 256 x 256 pair (fewest bytes per MAC). The narrower tiles and the splits are for problems that leave SMs idle, where time is
// one CTA's serial chain of k-blocks: 64 rows, K 12288, N 3072 take 37.7 us with 128 x 256 tiles (12 CTAs of 96 k-blocks), 26.0
// with 128 x 128, 17.3 shared by two CTAs and 13.9 by four (96 of 24), K 3072 13.7, 9.8, 8.6, 8.7; 512 rows, K 12288 37.3, 26.9
// and 23.2 with pairs of 256 x 128. A split costs more than it gives once its clusters need a second wave (512 rows, N 3072,
// K 3072: by four 25.4 us, not split 10.4), hence `resident`. Pairs of 192 columns
// fill waves that the others leave half empty (the GEMM alone, best of the others -> 192: 512 rows, N 12288, K 3072
// 21.9 -> 19.8 us; 900 rows, K 8192 26 -> 21; 1024 rows, K 12288 36 -> 29; 2048 rows, K 8192 41 -> 35).
Form choose_form(uint64_t M, uint64_t N, uint64_t K) {
  struct Cost {
    Form form;
    uint64_t block_ns, launch_ns;
  };
  static const Cost costs[] = {{{2, 256, 1}, 320, 6000}, {{2, 192, 1}, 265, 5200}, {{2, 128, 1}, 208, 4500}, {{1, 256, 1}, 363, 5100},
                               {{1, 128, 1}, 258, 3200}, {{1, 128, 2}, 320, 3500}, {{1, 128, 4}, 450, 4600}};
  const uint64_t sms = (uint64_t)sm_count(), k_blocks = (K + kBK - 1) / kBK;
  // DIFB200_GEMM_FORM=ctas,columns,split forces one of the forms, DIFB200_GEMM_CTAS=1|2 a 256-column one
  // (all give identical bits).
  Form want{0, 0, 0}, best{1, 256, 1};
  if (const char *force = std::getenv("DIFB200_GEMM_FORM"))
    std::sscanf(force, "%d,%d,%d", &want.ctas, &want.tile_n, &want.split);
  if (const char *force = std::getenv("DIFB200_GEMM_CTAS"))
    if (force[0] == '1' || force[0] == '2')
      want = Form{force[0] - '0', 256, 1};
  uint64_t least = ~0ull;
  for (const Cost &c : costs) {
    const Form &f = c.form;
    if ((uint64_t)f.split > k_blocks)
      continue;
    if (f.ctas == want.ctas && f.tile_n == want.tile_n && f.split == want.split)
      return f;
    const uint64_t tiles = ((M + kBM * f.ctas - 1) / (kBM * f.ctas)) * ((N + f.tile_n - 1) / f.tile_n);
    const uint64_t resident = f.split > 2 ? sms * 7 / 8 / f.split : sms / (f.ctas * f.split); // wide clusters leave gaps
    if ((f.ctas == 2 && M <= (uint64_t)kBM) || (f.split > 1 && tiles > resident))
      continue;
    const uint64_t waves = (tiles + resident - 1) / resident;
    const uint64_t time = waves * ((k_blocks + f.split - 1) / f.split) * c.block_ns + c.launch_ns;
    if (time < least) {
      least = time;
      best = f;
    }
  }
  return best;
}

template <int CTAS, int BN>
int launch_form(const CUtensorMap &map_a, const CUtensorMap &map_b, const CUtensorMap &map_c, const GemmParams &p,
                cudaStream_t stream) {
  // The dynamic shared-memory opt-in is an attribute of the function in one context, so it is
  // made once per device (a process may hold plugin contexts on several GPUs).
  static const char attr_key = 0;
  if (int rc = current_device_once(&attr_key, [](void *, int *) -> int {
        return check_cuda(cudaFuncSetAttribute(gemm_i8_kernel<CTAS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem_bytes<CTAS, BN>()),
                          "cudaFuncSetAttribute(gemm_i8_kernel)");
      }, nullptr, nullptr))
    return rc;
  const uint64_t tiles = (((uint64_t)p.M + Cfg<CTAS, BN>::kTileM - 1) / Cfg<CTAS, BN>::kTileM) *
                         (((uint64_t)p.N + BN - 1) / BN);
  cudaLaunchConfig_t config{};
  config.gridDim = dim3((unsigned)sm_count());
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem_bytes<CTAS, BN>();
  config.stream = stream;
  cudaLaunchAttribute attrs[2]{dependent_launch(), {}};
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = CTAS == 2 ? 2u : p.split;
  attrs[1].val.clusterDim.y = 1;
  attrs[1].val.clusterDim.z = 1;
  uint64_t units = (uint64_t)sm_count();
  config.attrs = attrs;
  config.numAttrs = CTAS == 2 || p.split > 1 ? 2 : 1;
  if (CTAS == 2) {
    // The kernel is persistent: launch exactly as many CTA pairs as can be resident at once
    // (SM pairs are formed inside a GPC, so this can be fewer than SMs / 2); a per-device figure.
    static const char pairs_key = 0;
    int resident_pairs = 0;
    if (int rc = current_device_once(&pairs_key, [](void *arg, int *value) -> int {
          int n = 0;
          if (int rc = check_cuda(cudaOccupancyMaxActiveClusters(&n, gemm_i8_kernel<CTAS, BN>,
                                                                 static_cast<cudaLaunchConfig_t *>(arg)),
                                  "cudaOccupancyMaxActiveClusters"))
            return rc;
          *value = n > 0 ? n : 1;
          return kOk;
        }, &config, &resident_pairs))
      return rc;
    units = (uint64_t)resident_pairs;
  }
  if (CTAS == 1 && p.split > 1) {
    // one cluster per tile: clusters do not wait for one another, so they need not all be resident
    if (tiles * p.split > 0x7fffffffull)
      return fail(kUnsupported, "LinearInt8Scaled: problem too large");
    config.gridDim = dim3((unsigned)(tiles * p.split));
  } else {
    config.gridDim = dim3((unsigned)(CTAS * (units < tiles ? units : tiles)));
  }
  return launched(cudaLaunchKernelEx(&config, gemm_i8_kernel<CTAS, BN>, map_a, map_b, map_c, p),
                  "gemm_i8_kernel launch");
}

} // namespace

int linear_int8_scaled(const int8_t *x, const int8_t *w, const float *row_scales,
                       const float *col_scales, const void *bias_bf16, uint32_t epilogue, uint64_t M,
                       uint64_t N, uint64_t K, void *out_bf16, int32_t *acc_out, cudaStream_t stream,
                       DeviceStatus *status_words, bool weights_ready) {
  if (!x || !w || !row_scales || !col_scales || !out_bf16)
    return fail(kInvalidArgument, "LinearInt8Scaled: null pointer");
  if ((epilogue & kEpiBias) && !bias_bf16)
    return fail(kInvalidArgument, "LinearInt8Scaled: bias epilogue without a bias pointer");
  if (epilogue & ~(kEpiBias | kEpiGeluTanh))
    return fail(kInvalidArgument, "LinearInt8Scaled: unknown epilogue flags");
  if (M == 0 || N == 0)
    return kOk;
  if (K == 0 || K % 16 != 0)
    return fail(kUnsupported, "LinearInt8Scaled: K must be a positive multiple of 16 (TMA row pitch)");
  if (M > 0x7fffffffull || N > 0x7fffffffull || K > 0x7fffffffull)
    return fail(kUnsupported, "LinearInt8Scaled: dimension too large");
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15))
    return fail(kUnsupported, "LinearInt8Scaled: operands must be 16-byte aligned");
  DeviceStatus *status = status_words ? status_words : device_status_words();
  if (!status)
    return fail(kOutOfMemory, "LinearInt8Scaled: device status words are unavailable");

  GemmParams p{};
  p.row_scales = row_scales;
  p.col_scales = col_scales;
  p.bias = static_cast<const uint16_t *>(bias_bf16);
  p.out = static_cast<uint16_t *>(out_bf16);
  p.acc_out = acc_out;
  p.M = (uint32_t)M;
  p.N = (uint32_t)N;
  p.K = (uint32_t)K;
  p.epilogue = epilogue;
  p.withhold_kb = take_withheld_gemm_load();
  p.weights_first = weights_ready && p.withhold_kb == 0xffffffffu ? 1u : 0u;
  p.wait_ns = wait_limit_ns();
  p.status = status;
  if (p.withhold_kb == 0xffffffffu && few_rows(M, N, K, p.weights_first != 0u))
    return launch_few_rows(x, w, p, stream);

  const Form form = choose_form(M, N, K);
  CUtensorMap map_a, map_b;
  const uint64_t dims_a[2] = {K, M}, dims_b[2] = {K, N};
  const uint64_t strides[1] = {K};
  // Where all rows are one tile of a CTA, loads end with them (a multiple of 8 rows, the swizzle's period): rows beyond
  // the tensor are not free, 17 x 3072 x 16384 took 15.3 us with boxes of 128 rows and takes 9.4 with boxes of 24. What stands in the
  // others' place meets only rows of the accumulator that are never read.
  p.a_rows = form.ctas == 1 && M < (uint64_t)kBM ? (uint32_t)(M + 7) / 8 * 8 : (uint32_t)kBM;
  const uint32_t box_a[2] = {(uint32_t)kBK, p.a_rows}, box_b[2] = {(uint32_t)kBK, (uint32_t)(form.tile_n / form.ctas)};
  if (int rc = encode_tensor_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, x, dims_a, strides, box_a,
                                 CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;
  if (int rc = encode_tensor_map(&map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, w, dims_b, strides, box_b,
                                 CU_TENSOR_MAP_SWIZZLE_128B))
    return rc;

  const bool tma_store = (N % 8 == 0) && ((reinterpret_cast<uintptr_t>(out_bf16) & 15) == 0);
  CUtensorMap map_c = map_a; // placeholder when stores go out directly
  if (tma_store) {
    const uint64_t dims_c[2] = {N, M};
    const uint64_t strides_c[1] = {N * 2};
    const uint32_t box_c[2] = {32, 32};
    if (int rc = encode_tensor_map(&map_c, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, out_bf16, dims_c,
                                   strides_c, box_c, CU_TENSOR_MAP_SWIZZLE_64B))
      return rc;
  }

  p.split = (uint32_t)form.split;
  p.tma_store = tma_store ? 1u : 0u;
  if (form.ctas == 2)
    return form.tile_n == 256   ? launch_form<2, 256>(map_a, map_b, map_c, p, stream)
           : form.tile_n == 192 ? launch_form<2, 192>(map_a, map_b, map_c, p, stream)
                                : launch_form<2, 128>(map_a, map_b, map_c, p, stream);
  return form.tile_n == 256 ? launch_form<1, 256>(map_a, map_b, map_c, p, stream)
                            : launch_form<1, 128>(map_a, map_b, map_c, p, stream);
}

} // namespace difb200
