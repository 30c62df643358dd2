// Weight packing with the 256-wide ConvRot variants for sm_100a: convrot256.cuh with the scale search and / or input equalisation.
// A translation unit of its own: its kernels are loaded by those who pack weights (the first quantiser call of a process 22 ms as one
// unit, 8 so).
#include "convrot256.cuh"

namespace difb200 {
namespace {

template <bool SIGNED>
int launch_pack(const QuantParams &p, bool f32, cudaStream_t stream) {
  if (p.rcodes)
    return fail(kUnsupported, "QuantizeInt8Rows: weight packing (MSE scale, input equalisation) exists for "
                              "the 256-wide variants without residual outputs");
  if (!p.mse)
    return f32 ? launch_single<SIGNED, true, false, kEqualise>(p, stream) : launch_single<SIGNED, false, false, kEqualise>(p, stream);
  // The scale search is arithmetic per row as well as per element: three blocks per warp where they divide the row and
  // the rows are more than the machine holds at once, 16 warps per SM (12288 x 3072 one block and 24 warps 65.1 us, three with a
  // prefetch and 12 warps 61.0, this without a prefetch 56.3; 3072 x 8192, whose last warp would be a third empty, 51.5 / 53.6 / 56.2).
  const uint32_t blocks = ((p.columns >> 8) + 3u) / 4u;
  const bool three = blocks % 3u == 0u && p.rows * blocks > (uint64_t)sm_count() * 24u;
  if (p.equalise) {
    // With input equalisation one CTA per SM, whose rows share the table: 16 warps of three blocks with a prefetch, or 24 of one. The
    // table takes 1.5 us, so from three rounds of 24 warps per SM on, and not where rows of more than 8 blocks leave warps idle. From a
    // graph, every row its own reciprocals / table: 16384 x 3072 91.0 / 77.4, 12288 x 3072 70.0 / 63.1, 3072 x 12288 70.4 / 67.7, 3072 x
    // 8192 51.2 / 52.2, fp32 107.5 / 93.4, 80.3 / 73.1, 86.9 / 84.1, 55.6 / 54.3; but 1500 x 10240 34.9 / 39.2, 3000 x 2304 20.4 / 21.9,
    // 3000 x 512 9.0 / 10.7.
    if (p.rows * blocks >= (uint64_t)sm_count() * 72u && (blocks % 3u == 0u || blocks <= 8u))
      return f32     ? launch_form<SIGNED, true, false, kPackTable, 1, false, 768, 1>(p, stream)
             : three ? launch_form<SIGNED, false, false, kPackTable, 3, true, 512, 1>(p, stream)
                     : launch_form<SIGNED, false, false, kPackTable, 1, false, 768, 1>(p, stream);
    return f32     ? launch_single<SIGNED, true, false, kPackEqualise>(p, stream)
           : three ? launch_form<SIGNED, false, false, kPackEqualise, 3, false, 256, 2>(p, stream)
                   : launch_single<SIGNED, false, false, kPackEqualise>(p, stream);
  }
  return f32     ? launch_single<SIGNED, true, false, kPack>(p, stream)
         : three ? launch_form<SIGNED, false, false, kPack, 3, false, 256, 2>(p, stream)
                 : launch_single<SIGNED, false, false, kPack>(p, stream);
}

} // namespace

int launch_convrot256_pack(const QuantParams &p, bool is_signed, bool f32, cudaStream_t stream) {
  return is_signed ? launch_pack<true>(p, f32, stream) : launch_pack<false>(p, f32, stream);
}

} // namespace difb200
