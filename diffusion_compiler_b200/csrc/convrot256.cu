// QuantizeInt8Rows of activations with the 256-wide ConvRot variants for sm_100a (convrot256.cuh): plain, with residual outputs, behind a norm.
#include "convrot256.cuh"

namespace difb200 {
namespace {

template <bool SIGNED, bool F32>
int launch_variant(const QuantParams &p, cudaStream_t stream) {
  if (p.rcodes)
    return launch_single<SIGNED, F32, true, kPlain>(p, stream);
  if (p.norm_scale)
    return p.norm_bias ? launch_single<SIGNED, F32, false, kLayer>(p, stream) : launch_single<SIGNED, F32, false, kNorm>(p, stream);
  return launch_single<SIGNED, F32, false, kPlain>(p, stream);
}

} // namespace

// Rows of at most 16384 columns.
int launch_convrot256(const QuantParams &p, int implementation, cudaStream_t stream) {
  const bool is_signed = implementation == 3 || implementation == 6, f32 = implementation >= 5;
  if (p.mse || p.equalise)
    return launch_convrot256_pack(p, is_signed, f32, stream);
  if (f32)
    return is_signed ? launch_variant<true, true>(p, stream) : launch_variant<false, true>(p, stream);
  return is_signed ? launch_variant<true, false>(p, stream) : launch_variant<false, false>(p, stream);
}

} // namespace difb200
