// fp32 instances of the one-block-per-lane kernels (frsz2_laneblock.cuh), bits 4..32.
#include "frsz2_laneblock.cuh"

namespace frsz2b {

cudaError_t launch_laneblock_f32(int bits, bool compress, const Job& j, cudaStream_t s)
{
  static constexpr auto table = make_laneblock_table<float, 4>(std::make_integer_sequence<int, 29>{});
  if (bits < 4 || bits > 32) return cudaErrorNotSupported;
  return table[bits - 4](compress, j, s);
}

} // namespace frsz2b
