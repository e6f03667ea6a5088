// Running-median detrend for radii of 64 and more: a sorted core that moves by merging.
//
// Groups of T = 16 windows as in medgroup.cuh, whose common core (2r + 2 - T rows) is too large for a
// thread's registers: each lane keeps its core sorted in shared memory ([rank][lane]: no bank
// conflicts), and takes the medians of a group from the core's T middle values and the rows before
// and behind it.  From one group to the next 16 rows leave the core and 16 enter.  Both are sorted by
// a network, and one pass over the core copies it, leaving out the former and putting in the
// latter: 2r + 2 steps for 16 rows, each one element per lane, with the next elements already loaded.
// The pass writes 16 slots below (ascending) or above (descending, the next time) where it reads, so
// that the core moves within 16 spare slots.  Values are integer keys in the order of the floats
// (median_key), so that every element that leaves is found, whatever it is.
//
// Bound by the latency of the pass's steps at the few warps an SM has room for (five at r = 128), and
// then by issue.  The first core of a run costs about r / 17 passes, so each lane's run is as long
// as leaves one wave of blocks.  Sliding a sorted window by one row at a time, as the other radii do,
// costs a chain of moves a row; before / now, normal noise: 65,536 x 128 r = 64 2500 / 140 us,
// r = 128 10,513 / 274, r = 256 56,631 / 773, r = 800 1,296,579 / 6348; 65,536 x 8 r = 128 3548 / 99;
// 3001 x 1 r = 128 954 / 61 (the first core: few lanes, each its 15 blocks); 160 packed curves of
// 3.5 M samples r = 128 1359 / 408, one of 19,254 378 / 60.  A smooth curve (short moves): 65,536 x 128
// r = 128 6193 / 272.
#include "common.cuh"
#include "medgroup.cuh"

namespace {

constexpr int kT = 16;
// rows of 32 words: a spare one, E between guards, L, the core with its spare slots, a guard, a spare one
constexpr int kE = 2, kL = kE + kT + 1, kS = kL + kT + 1;
constexpr int kExtraRows = kS + kT + 2;

using gtrap::median_key;
using gtrap::median_value;

// One pass: the lane's array at s, in the direction's order, without the kT keys of L (kLeave) and with
// the kT keys of E, to o.  steps: elements at s + kT.  A step takes the next of E, copies the next
// of s, or drops it.
template <bool kUp, bool kLeave>
__device__ __forceinline__ void merge_pass(int *lane, int s, int o, int steps) {
  constexpr int kStep = kUp ? 32 : -32;
  const int *ps = lane + 32 * s, *pe = lane + 32 * (kUp ? kE : kE + kT - 1), *pl = lane + 32 * (kUp ? kL : kL + kT - 1);
  int *po = lane + 32 * o;
  int v = ps[0], vn = ps[kStep], e = pe[0], en = pe[kStep];
  int l = kLeave ? pl[0] : 0, ln = kLeave ? pl[kStep] : 0;
  ps += 2 * kStep;
  pe += 2 * kStep;
  pl += 2 * kStep;
#pragma unroll 4
  for (int k = 0; k < steps; ++k) {
    const bool take = kUp ? e < v : e > v;
    const bool drop = kLeave && !take && v == l;
    if (!drop) {
      *po = take ? e : v;
      po += kStep;
    }
    if (take) {
      e = en;
      en = *pe;
      pe += kStep;
    } else {
      v = vn;
      vn = *ps;
      ps += kStep;
    }
    if (drop) {
      l = ln;
      ln = *pl;
      pl += kStep;
    }
  }
}

// Image (offs null): lane = curve 32 blockIdx.x + lane of an [n, ncurves] image, blockIdx.y = run of
// `run` rows.  Otherwise curve blockIdx.y (packed, or a column of an image with lens null) and lane =
// run 32 blockIdx.x + lane of it.
template <bool kColumns>
__global__ void __launch_bounds__(32) gfilter_merge_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                           const unsigned long long *__restrict__ offs,
                                                           const uint32_t *__restrict__ lens, unsigned ncurves,
                                                           unsigned n_all, int r, int run) {
  extern __shared__ int sorted_cores[];
  int *lane = sorted_cores + threadIdx.x;
  auto at = [&](int row) -> int & { return lane[32 * row]; };
  const int C = 2 * r + 2 - kT;
  const int top = kS + kT + C;   // the row behind the core's slots: its upper guard
  for (unsigned q0 = blockIdx.y; q0 < (kColumns ? ncurves : blockIdx.y + 1); q0 += gridDim.y) {
    const unsigned q = kColumns ? q0 : blockIdx.x * 32 + threadIdx.x;
    const bool live = q < ncurves;
    const long long n = !live ? 0 : lens ? (long long)lens[q] : (long long)n_all;
    const size_t stride = lens ? 1 : ncurves;
    const size_t base = !live ? 0 : offs ? (size_t)offs[q] : (size_t)q;
    const long long first = (kColumns ? (long long)blockIdx.x * 32 : (long long)q0) * run;   // the warp's first row
    if (first >= (kColumns ? n : (long long)n_all)) continue;
    const long long row0 = first + (kColumns ? (long long)threadIdx.x * run : 0);
    const float *x = in + base;
    auto row = [&](long long i) -> float { return i >= 0 && i < n ? __ldg(x + (size_t)i * stride) : 0.0f; };
    auto keys = [&](long long i, int (&k)[kT]) {
      float v[kT];
#pragma unroll
      for (int j = 0; j < kT; ++j) v[j] = row(i + j);
      __syncwarp();   // the loads in flight together
#pragma unroll
      for (int j = 0; j < kT; ++j) k[j] = median_key(v[j]);
    };
    auto put_sorted = [&](int to, const int (&k)[kT]) {
      int s[kT];
#pragma unroll
      for (int j = 0; j < kT; ++j) s[j] = k[j];
      gtrap::net_sort(s);
#pragma unroll
      for (int j = 0; j < kT; ++j) at(to + j) = s[j];
    };
    // ---- the first group's core, rows row0 + 15 - r .. row0 + r: C mod 16 rows, then 16 at a time
    at(kE - 1) = INT_MIN;
    at(kL - 1) = INT_MAX;
    at(top) = INT_MAX;
    long long next = row0 + kT - 1 - r;
    int size = C & (kT - 1);
    {
      int k[kT];
      keys(next, k);
#pragma unroll
      for (int j = 0; j < kT; ++j) k[j] = j < size ? k[j] : INT_MAX;
      gtrap::net_sort(k);
#pragma unroll
      for (int j = 0; j < kT; ++j)
        if (j < size) at(top - size + j) = k[j];
      next += size;
    }
    for (; size < C; size += kT, next += kT) {
      int k[kT];
      keys(next, k);
      put_sorted(kE, k);
      merge_pass<true, false>(lane, top - size, top - size - kT, size + kT);
    }
    int left[kT];
    keys(row0 - r - 1, left);
    bool high = true;   // the core lies in [kS + kT, top), or in [kS, kS + C)
    const long long count = kColumns ? (n - first < run ? n - first : run) : (n_all - first < run ? n_all - first : run);
    const int groups = (int)((count + kT - 1) / kT);
    for (int g = 0;; ++g) {
      const long long i0 = row0 + (long long)g * kT;
      int enter[kT], core[kT], med[kT];
      keys(i0 + r + 1, enter);
      const int c0 = (high ? kS + kT : kS) + r - kT + 1;
#pragma unroll
      for (int j = 0; j < kT; ++j) core[j] = at(c0 + j);
      gtrap::median_halves<kT, kT, 0>(core, left, enter, med);
#pragma unroll
      for (int j = 0; j < kT; ++j) {
        const long long i = i0 + j;
        if (i < n) out[base + (size_t)i * stride] = __fsub_rn(__ldg(x + (size_t)i * stride), median_value(med[j]));
      }
      if (g + 1 == groups) break;
      keys(i0 + kT - 1 - r, left);
      put_sorted(kE, enter);
      put_sorted(kL, left);
      at(kL - 1) = at(kS - 1) = high ? INT_MAX : INT_MIN;
      if (high)
        merge_pass<true, true>(lane, kS + kT, kS, C + kT);
      else
        merge_pass<false, true>(lane, kS + C - 1, top - 1, C + kT);
      high = !high;
    }
  }
}

}  // namespace

namespace gtrap {

size_t gfilter_merge_smem(uint32_t r) { return (2 * (size_t)r + 2 - kT + kExtraRows) * 32 * sizeof(int); }

int gfilter_merge(const float *in, float *out, const unsigned long long *off, const uint32_t *lens, uint32_t ncurves,
                  uint32_t n, uint32_t r, cudaStream_t stream) {
  const bool columns = lens || ncurves < 12;
  const size_t smem = gfilter_merge_smem(r);
  // runs that fill the SMs' room for blocks once (a run's first core costs r / 17 of its groups)
  size_t per_sm = (size_t)(max_smem_optin() + 1024) / (smem + 1024);
  if (per_sm > 32) per_sm = 32;
  const size_t lanes = (size_t)sm_count() * per_sm * 32;
  const size_t width = columns ? ncurves : ((size_t)ncurves + 31) / 32 * 32;
  size_t run = ((size_t)n * width + lanes - 1) / lanes;
  run = (run + kT - 1) / kT * kT;
  const void *kernel = columns ? (const void *)gfilter_merge_kernel<true> : (const void *)gfilter_merge_kernel<false>;
  GTRAP_TRY(ensure_smem(kernel, smem, "gfilter"));
  if (columns) {
    const dim3 grid((unsigned)((n + run * 32 - 1) / (run * 32)), ncurves < 65535 ? ncurves : 65535);
    gfilter_merge_kernel<true><<<grid, 32, smem, stream>>>(in, out, off, lens, ncurves, n, (int)r, (int)run);
  } else {
    const size_t runs = (n + run - 1) / run;
    if (runs > 65535) run = ((n + 65534) / 65535 + kT - 1) / kT * kT;
    const dim3 grid((unsigned)(width / 32), (unsigned)((n + run - 1) / run));
    gfilter_merge_kernel<false><<<grid, 32, smem, stream>>>(in, out, off, lens, ncurves, n, (int)r, (int)run);
  }
  return check_launch("gfilter_merge_kernel");
}

}  // namespace gtrap
