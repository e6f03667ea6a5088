// Running-median detrend of packed curves, and of images of a few curves, by groups of windows.
#include "gfilter_groups.cuh"

namespace gtrap {

int gfilter_groups_packed(const float *in, float *out, const unsigned long long *off, const uint32_t *n,
                          uint32_t ncurves, uint32_t max_n, uint32_t r, cudaStream_t stream) {
  return launch_groups<1>(in, out, off, n, ncurves, max_n, r, stream);
}

int gfilter_groups_columns(const float *in, float *out, uint32_t n, uint32_t nq, uint32_t r, cudaStream_t stream) {
  return launch_groups<1>(in, out, nullptr, nullptr, nq, n, r, stream);
}

}  // namespace gtrap
