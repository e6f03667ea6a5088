// Running-median detrend of an [n, nq] image by groups of windows.
#include "gfilter_groups.cuh"

namespace gtrap {

// A row group's lanes: a whole warp of curves (coalesced rows; some lanes idle below 32 curves),
// or, where under a third of the lanes would work, one curve a block.
int gfilter_groups_image(const float *in, float *out, uint32_t n, uint32_t nq, uint32_t r, cudaStream_t stream) {
  if (nq < 12) return gfilter_groups_columns(in, out, n, nq, r, stream);
  return launch_groups<32>(in, out, nullptr, nullptr, nq, n, r, stream);
}

}  // namespace gtrap
