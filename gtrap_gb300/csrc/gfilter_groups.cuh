// The running-median detrend by groups of windows (medgroup.cuh): the kernel and its launcher,
// instantiated for images in gfilter_image.cu and for packed curves in gfilter_packed.cu (two
// files because the unrolled networks are slow to compile).
#pragma once

#include "common.cuh"
#include "medgroup.cuh"

namespace {

// Where row j of a block, from a whole number of groups on, lies: one word of padding a group of T rows.
template <int T>
__device__ __forceinline__ int group_slot(int j) {
  static_assert(T == 4 || T == 8 || T == 16, "groups of 4, 8 or 16 rows");
  return j + (j >> (T == 16 ? 4 : T == 8 ? 3 : 2));
}

// Groups of T windows (medgroup.cuh).  A group that holds a value that is not finite takes the same
// networks over integer keys, which put NaN in a place of its own.  65,536 x 128, without / with such a value
// in most groups: r = 5 46 / 69 us, r = 24 81 / 156, r = 63 151 / 290 (by an insertion sort and slides in
// thread-local memory, which this replaces: 278, 1705, 15,660 us).  A function of its own, taking the
// pointer: inlined, or with the row accessor passed on, it takes registers from the common path.
template <int T, int A, int LC>
__device__ __noinline__ void group_medians_by_keys(const float *mine, int B, float (&med)[T]) {
  int key[T];
  float unused = 0.0f;
  gtrap::group_medians<T, A>(B, [mine](int k) { return gtrap::median_key(mine[group_slot<T>(k) * LC]); }, key, unused);
#pragma unroll
  for (int k = 0; k < T; ++k) med[k] = gtrap::median_value(key[k]);
}

// The medians of the group whose row k lies at mine[group_slot(k) LC].
template <int T, int A, int LC>
__device__ __forceinline__ void medians_of_group(const float *mine, int r, float (&med)[T]) {
  float bad = 0.0f;
  gtrap::group_medians<T, A>(r - T * A, [mine](int k) { return mine[group_slot<T>(k) * LC]; }, med, bad);
  if (bad != 0.0f) {  // NaN: some value is not finite
    float m[T];
    group_medians_by_keys<T, A, LC>(mine, r - T * A, m);
#pragma unroll
    for (int k = 0; k < T; ++k) med[k] = m[k];
  }
}

constexpr int kGroupThreads = 256;

// One block: the rows [row0, row0 + rows) of LC curves (lane = curve within a row group), staged
// in shared memory as [row + row / T][curve]: the padding of one row a group spreads the row
// groups of a warp over the banks for LC < 32, and a group's rows lie at constant distances.
// Image (offs null): curves blockIdx.y * LC + lane of an [n, nq] image; packed: curve
// blockIdx.y, LC = 1, samples [offs, offs + lens) of a flat array (stride 1).
template <int T, int A, int LC>
__global__ void __launch_bounds__(kGroupThreads, T == 16 && A > 1 ? 2 : 3) gfilter_group_kernel(
    const float *__restrict__ in, float *__restrict__ out, const unsigned long long *__restrict__ offs,
    const uint32_t *__restrict__ lens, unsigned ncurves, unsigned n_all, int r) {
  extern __shared__ float stage[];
  constexpr int kHalo = T * (A + 1);   // > r, a whole number of groups
  auto slot = [](int j) { return group_slot<T>(j); };
  const int lane = (int)threadIdx.x % LC, group = (int)threadIdx.x / LC, step = (int)blockDim.x / LC;
  const int rows = step * T;
  for (unsigned long long c0 = (unsigned long long)blockIdx.y * LC; c0 < ncurves;
       c0 += (unsigned long long)gridDim.y * LC) {
    const unsigned long long q = c0 + lane;
    const bool live = q < ncurves;
    const long long n = offs ? (long long)lens[c0] : (long long)n_all;
    const size_t stride = offs ? 1 : ncurves;
    const size_t base = offs ? (size_t)offs[c0] : (size_t)q;
    const long long row0 = (long long)blockIdx.x * rows;
    if (row0 >= n) continue;  // the whole block
    const float *x = in + base;
    __syncthreads();          // the previous curves' stage is no longer read
    // asynchronous copies: every row of the block in flight at once (a missing row is filled with
    // zero: nothing is read)
    for (int j = kHalo - r + group; j < kHalo + rows + r; j += step) {
      const long long i = row0 - kHalo + j;
      const bool there = live && i >= 0 && i < n;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(stage + slot(j) * LC + lane);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst),
                   "l"(there ? x + (size_t)i * stride : in), "r"(there ? 4 : 0) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // row k of this thread's group: the group starts at a whole number of groups, so slot() of
    // the sum is the sum of the slots and a constant k costs nothing
    float *mine = stage + (size_t)(group + kHalo / T) * (T + 1) * LC + lane;
    const long long i0 = row0 + (long long)group * T;
    float res[T];
#pragma unroll
    for (int k = 0; k < T; ++k) res[k] = 0.0f;
    if (live && i0 < n) {
      medians_of_group<T, A, LC>(mine, r, res);
#pragma unroll
      for (int k = 0; k < T; ++k) res[k] = __fsub_rn(mine[slot(k) * LC], res[k]);
    }
    if constexpr (LC == 32) {
      if (live) {
        float *y = out + base + (size_t)i0 * stride;
#pragma unroll
        for (int k = 0; k < T; ++k)
          if (i0 + k < n) y[(size_t)k * stride] = res[k];
      }
    } else {
      __syncthreads();
#pragma unroll
      for (int k = 0; k < T; ++k) mine[k * LC] = res[k];
      __syncthreads();
      for (int j = group; j < rows; j += step)
        if (live && row0 + j < n)
          out[base + (size_t)(row0 + j) * stride] = stage[slot(j + kHalo) * LC + lane];
    }
  }
}

// Blocks of up to kGroupThreads threads, smaller ones for a few short curves, so that their
// groups spread over the SMs.
template <int T, int A, int LC>
int launch_group(const float *in, float *out, const unsigned long long *off, const uint32_t *lens, uint32_t ncurves,
                 uint32_t n, uint32_t r, cudaStream_t stream) {
  const size_t lanes = ((size_t)ncurves + LC - 1) / LC * LC;
  int threads = kGroupThreads;
  while (threads > 32 && lanes * n < (size_t)gtrap::sm_count() * 2 * threads * T) threads /= 2;
  const size_t rows = (size_t)(threads / LC) * T;
  const size_t smem = (rows + 2 * T * (A + 1)) / T * (T + 1) * LC * sizeof(float);
  const size_t gx = (n + rows - 1) / rows, gy = lanes / LC;
  if (gx >= (1ull << 31)) return gtrap::fail(GTRAP_ERR_INVALID_ARG, "gfilter: n too large");
  GTRAP_TRY(gtrap::ensure_smem((const void *)gfilter_group_kernel<T, A, LC>, smem, "gfilter"));
  gfilter_group_kernel<T, A, LC><<<dim3((unsigned)gx, (unsigned)(gy < 65535 ? gy : 65535)), threads, smem, stream>>>(
      in, out, off, lens, ncurves, n, (int)r);
  return gtrap::check_launch("gfilter_group_kernel");
}

template <int LC>
int launch_groups(const float *in, float *out, const unsigned long long *off, const uint32_t *lens, uint32_t ncurves,
                  uint32_t n, uint32_t r, cudaStream_t stream) {
  if (r < 8) return launch_group<4, 1, LC>(in, out, off, lens, ncurves, n, r, stream);
  if (r < 16) return launch_group<8, 1, LC>(in, out, off, lens, ncurves, n, r, stream);
  if (r < 32) return launch_group<16, 1, LC>(in, out, off, lens, ncurves, n, r, stream);
  if (r < 48) return launch_group<16, 2, LC>(in, out, off, lens, ncurves, n, r, stream);
  return launch_group<16, 3, LC>(in, out, off, lens, ncurves, n, r, stream);
}

}  // namespace
