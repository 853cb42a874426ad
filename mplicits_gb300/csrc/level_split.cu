// FP32 level kernels on split FP16 operands: dispatch by padded width.
#include "level_split.cuh"

namespace mpl {
int launch_level_split(const LevelArgs& a, cudaStream_t s) {
  switch (a.lay.WP) {
    case 64: return split::launch_wp<64>(a, s);
    case 128: return split::launch_wp<128>(a, s);
    case 256: return split::launch_wp<256>(a, s);
    default: return MPL_ERR_UNSUPPORTED;
  }
}
}  // namespace mpl
