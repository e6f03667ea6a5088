// Trapezoid grid fit of the reference's CPU TLS path (gtrap/tls.py:2-110) on the device, in
// FP64 like the reference: gen_trapzoid (:2-15), get_chi2Hmax (:44-79; get_Hmax :17-42 is its
// H without the mean subtraction) and the grid search of tlsfit (:82-110).
//
// The reference masks the whole series per template (about 15 passes over n samples).  Here
// the samples are sorted by time once, so a template's samples are the index window whose
// t - t0 lies in [-W/2, W/2] (wider when L/2 > W/4), and each region is an index range:
// seven binary searches on the monotone predicate fl(t - t0) >= a (rounding is monotone) find
// them, and one thread per template makes three passes over the ranges, with no comparisons of
// times and no cross-lane reductions (both would issue on the narrow FP64 pipe): the mean
// over |t - t0| <= W/2 (divx), the region sums, and the residual with the fitted depth.  The
// region masks, the boundary expressions (-W/4 - L/2 evaluated as (-W/4) - L/2 ...), the
// nansum semantics (counts over all samples, sums over finite flux) and the formulas of denA,
// numB, Hmax and the residual follow the reference's.  Two things differ in rounding alone: a thread adds
// its samples in time order (numpy adds pairwise), and takes each product into its sum by one FMA, so
// that a term is rounded once and not twice.
//
// Bound by the FP64 pipe, which takes a warp's instruction 16 cycles here: a sample is tested for NaN
// and infinity on its bits, and products go into their sums by one FMA (7 FP64 instructions a window
// sample, 12 before); the searches compare integers, and the widest templates run first (269,504
// templates on 17,000 samples: 1037 -> 900 us).
#include "common.cuh"

#include <cooperative_groups.h>
#include <math.h>

namespace {

using gtrap::fail;

constexpr int kFitThreads = 256;

struct Bounds {  // region boundaries of a template, as the reference forms them
  double a1, a2, a3, a4, a5, a6;  // -W/2, -W/4-L/2, -W/4+L/2, W/4-L/2, W/4+L/2, W/2
};

__device__ __forceinline__ Bounds bounds_of(double W, double L) {
  const double mW4 = __ddiv_rn(-W, 4.0), W4 = __ddiv_rn(W, 4.0), L2 = __ddiv_rn(L, 2.0);
  return Bounds{__ddiv_rn(-W, 2.0), __dsub_rn(mW4, L2), __dadd_rn(mW4, L2), __dsub_rn(W4, L2),
                __dadd_rn(W4, L2), __ddiv_rn(W, 2.0)};
}

__device__ __forceinline__ int high_of(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ bool is_nan(double v) {
  const int h = high_of(v);
  return h > 0x7ff00000 || (h == 0x7ff00000 && __double2loint(v) != 0);
}
__device__ __forceinline__ bool is_finite(double v) { return high_of(v) < 0x7ff00000; }

// integers in the order of the doubles, +0 and -0 alike (NaN: see the caller)
__device__ __forceinline__ long long key_of(double v) {
  const long long b = __double_as_longlong(v);
  return (b & 0x7fffffffffffffffll) == 0 ? 0 : b < 0 ? b ^ 0x7fffffffffffffffll : b;
}

// first i in [0, n) with fl(t[i] - t0) >= a (strict: > a), n when none (a or t0 NaN: none)
__device__ __forceinline__ uint32_t first_at_least(const double *t, uint32_t n, double t0, double a, bool strict) {
  if (is_nan(a) || is_nan(t0)) return n;
  const long long ka = key_of(a) + (strict ? 1 : 0);
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    const double tn = __dsub_rn(t[mid], t0);
    if (!is_nan(tn) && key_of(tn) >= ka) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// One thread per template k = (iW * nL + iL) * nT + iT: consecutive threads take consecutive
// epochs of one (W, L), whose windows overlap, so a warp's loads stay within a few cache lines
// and its loops have nearly equal trip counts.  t sorted ascending over [0, n) (finite times;
// non-finite times belong to no region and are left out by the caller).
__global__ void __launch_bounds__(kFitThreads) tlsfit_kernel(
    const double *__restrict__ t, const double *__restrict__ xx, uint32_t n,
    const double *__restrict__ Wl, uint32_t nW, const double *__restrict__ Ll, uint32_t nL,
    const double *__restrict__ tl, uint32_t nT, double sigma, int divx, double *Hout,
    double *res_out, int32_t *n_out, double *xsum_out, double *sn_out) {
  // the widest templates, whose windows hold the most samples, first: the last blocks are short ones
  const uint64_t block = Wl[nW - 1] > Wl[0] ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const uint64_t k = block * kFitThreads + threadIdx.x;
  const uint64_t total = (uint64_t)nW * nL * nT;
  if (k >= total) return;
  const uint32_t iT = (uint32_t)(k % nT), iL = (uint32_t)((k / nT) % nL), iW = (uint32_t)(k / ((uint64_t)nT * nL));
  const double W = Wl[iW], L = Ll[iL], t0 = tl[iT];
  const Bounds b = bounds_of(W, L);
  // Every region is an interval of fl(t - t0), so on the sorted series an index range:
  // A = [i1, i2), B = [i2, i3), C = [i3, i4), D = [i4, i5), E = [i5, i6) with i(a) the first
  // index where fl(t - t0) >= a (empty or overlapping as the boundaries fall when L/2 > W/4,
  // like the reference's masks); the mean's closed interval [a1, a6] is [i1, j6).
  const uint32_t i1 = first_at_least(t, n, t0, b.a1, false), i6 = first_at_least(t, n, t0, b.a6, false);
  const uint32_t j6 = first_at_least(t, n, t0, b.a6, true);
  const uint32_t i2 = first_at_least(t, n, t0, b.a2, false), i3 = first_at_least(t, n, t0, b.a3, false);
  const uint32_t i4 = first_at_least(t, n, t0, b.a4, false), i5 = first_at_least(t, n, t0, b.a5, false);
  auto cnt = [](uint32_t a, uint32_t e) { return e > a ? (int)(e - a) : 0; };
  const int nA = cnt(i1, i2), nB = cnt(i2, i3), nC = cnt(i3, i4), nD = cnt(i4, i5), nE = cnt(i5, i6);

  double xsum = 0.0;
  if (divx) {  // np.nanmean(xx[(tn >= -W/2) * (tn <= W/2)])
    double s = 0.0;
    int c = 0;
    for (uint32_t i = i1; i < j6; ++i) {
      const double v = xx[i];
      if (!is_nan(v)) { s = __dadd_rn(s, v); ++c; }
    }
    xsum = __ddiv_rn(s, (double)c);  // 0/0 = NaN as numpy's mean of nothing
  }
  const bool mean_ok = is_finite(xsum);   // else every difference from it is looked at itself
  // region sums (np.nansum: NaN terms are skipped; the counts take every sample)
  auto flux_sum = [&](uint32_t a, uint32_t e) {
    double acc = 0.0;
    for (uint32_t i = a; i < e; ++i) {
      const double v = xx[i];
      const double x = __dsub_rn(v, xsum);
      if (mean_ok ? !is_nan(v) : !isnan(x)) acc = __dadd_rn(acc, x);
    }
    return acc;
  };
  struct Ramp { double s, xt, tsum, t2; };
  auto ramp_sums = [&](uint32_t a, uint32_t e) {
    Ramp m{0.0, 0.0, 0.0, 0.0};
    for (uint32_t i = a; i < e; ++i) {
      const double tn = __dsub_rn(t[i], t0), v = xx[i];
      m.tsum = __dadd_rn(m.tsum, tn);
      m.t2 = __fma_rn(tn, tn, m.t2);
      if (is_finite(v) && mean_ok) {
        const double x = __dsub_rn(v, xsum);
        m.s = __dadd_rn(m.s, x);
        m.xt = __fma_rn(x, tn, m.xt);
      } else {
        const double x = __dsub_rn(v, xsum);
        if (!isnan(x)) m.s = __dadd_rn(m.s, x);
        const double xt = __dmul_rn(x, tn);  // NaN for a NaN flux, or an infinite one at tn = 0
        if (!isnan(xt)) m.xt = __dadd_rn(m.xt, xt);
      }
    }
    return m;
  };
  const double sA = flux_sum(i1, i2), sC = flux_sum(i3, i4), sE = flux_sum(i5, i6);
  const Ramp mB = ramp_sums(i2, i3), mD = ramp_sums(i4, i5);
  const double xAEC = __dadd_rn(__dadd_rn(sA, sE), sC);
  const double xBD = __dadd_rn(mB.s, mD.s);
  const double t2BD = __dadd_rn(mB.t2, mD.t2);
  // denA = 4*L*L*(nA-nC+nE) + W*W*(nB+nD) + 8*W*(tB-tD) + 16*t2BD, left to right
  const double denA = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(__dmul_rn(4.0, L), L), (double)(nA - nC + nE)),
                                                    __dmul_rn(__dmul_rn(W, W), (double)(nB + nD))),
                                          __dmul_rn(__dmul_rn(8.0, W), __dsub_rn(mB.tsum, mD.tsum))),
                                __dmul_rn(16.0, t2BD));
  // numB = 8*L*L*xAEC - 4*W*L*xBD + 16*L*(xtD-xtB)
  const double numB = __dadd_rn(__dsub_rn(__dmul_rn(__dmul_rn(__dmul_rn(8.0, L), L), xAEC),
                                          __dmul_rn(__dmul_rn(__dmul_rn(4.0, W), L), xBD)),
                                __dmul_rn(__dmul_rn(16.0, L), __dsub_rn(mD.xt, mB.xt)));
  const double H = __ddiv_rn(-numB, denA);
  const double Hh = __ddiv_rn(H, 2.0), HL = __ddiv_rn(H, L), W4 = __ddiv_rn(W, 4.0);
  // residual with the fitted depth: np.nansum of the squared differences per region, which
  // skips every NaN term (a NaN flux, or every term when the depth itself is NaN)
  auto nadd = [](double acc, double d) { const double q = __dmul_rn(d, d); return isnan(q) ? acc : __dadd_rn(acc, q); };
  const bool all_ok = mean_ok && is_finite(H) && is_finite(HL);
  auto flat_res = [&](uint32_t a, uint32_t e, double level) {  // sum (x - level)^2
    double acc = 0.0;
    for (uint32_t i = a; i < e; ++i) {
      const double v = xx[i];
      const double d = __dsub_rn(__dsub_rn(v, xsum), level);
      if (all_ok && is_finite(v)) acc = __fma_rn(d, d, acc);
      else acc = nadd(acc, d);
    }
    return acc;
  };
  const double rA = flat_res(i1, i2, -Hh), rC = flat_res(i3, i4, Hh), rE = flat_res(i5, i6, -Hh);
  auto ramp_res = [&](uint32_t a, uint32_t e, double slope, double centre) {  // sum (x - slope (tn + centre))^2
    double acc = 0.0;
    for (uint32_t i = a; i < e; ++i) {
      const double u = __dadd_rn(__dsub_rn(t[i], t0), centre), v = xx[i];
      const double x = __dsub_rn(v, xsum);
      if (all_ok && is_finite(v)) {
        const double d = __fma_rn(-slope, u, x);
        acc = __fma_rn(d, d, acc);
      } else {
        acc = nadd(acc, __dsub_rn(x, __dmul_rn(slope, u)));
      }
    }
    return acc;
  };
  const double rB = ramp_res(i2, i3, HL, W4), rD = ramp_res(i4, i5, -HL, -W4);
  double res = __dadd_rn(__dadd_rn(rA, rC), rE);
  res = __dadd_rn(res, rB);
  res = __dadd_rn(res, rD);
  res = __ddiv_rn(res, __dmul_rn(sigma, sigma));
  const int npt = nA + nB + nC + nD + nE;
  Hout[k] = H;
  res_out[k] = res;
  n_out[k] = npt;
  xsum_out[k] = xsum;
  // tlsfit: sn = -H / sqrt(res / (n - 3))
  sn_out[k] = __ddiv_rn(-H, sqrt(__ddiv_rn(res, (double)(npt - 3))));
}

// First index of the largest non-NaN value (np.nanargmax); -1 when every value is NaN.  One cluster
// of eight blocks, the values as integer keys in their order (+0 and -0 alike) with eight loads in
// flight a thread: bound by the loads' latency (269,504 values: 164 us in one block, now 11).
constexpr int kArgThreads = 1024;
constexpr int kArgRanks = 8;

__global__ void __cluster_dims__(kArgRanks, 1, 1) __launch_bounds__(kArgThreads, 1)
nanargmax_kernel(const double *__restrict__ v, uint64_t count, int64_t *out) {
  namespace cg = cooperative_groups;
  constexpr int kU = 8;
  __shared__ long long bk[kArgThreads / 32], bi[kArgThreads / 32];
  __shared__ long long rk[kArgRanks], ri[kArgRanks];   // rank 0: every block's best
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)blockIdx.x;
  cluster.sync();   // every block has started: rank 0's shared memory may be written
  long long k = INT64_MIN, ki = -1;   // (no value's key is the smallest integer)
  auto better = [](long long a, long long ai, long long b, long long bj) {  // (a, ai) beats (b, bj)
    return ai >= 0 && (bj < 0 || a > b || (a == b && ai < bj));
  };
  for (uint64_t i0 = 0; i0 < count; i0 += (uint64_t)kArgRanks * kArgThreads * kU) {
    long long x[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t i = i0 + (uint64_t)(u * kArgRanks + rank) * kArgThreads + tid;
      x[u] = i < count ? __ldg(reinterpret_cast<const long long *>(v) + i) : 0x7fffffffffffffffll;   // a NaN
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const long long mag = x[u] & 0x7fffffffffffffffll;
      if (mag > 0x7ff0000000000000ll) continue;
      const long long key = mag == 0 ? 0 : x[u] < 0 ? x[u] ^ 0x7fffffffffffffffll : x[u];
      const long long i = (long long)(i0 + (uint64_t)(u * kArgRanks + rank) * kArgThreads + tid);
      if (ki < 0 || key > k) { k = key; ki = i; }  // ascending: the first of equal values per thread
    }
  }
  auto over_warp = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long ok = __shfl_xor_sync(0xffffffffu, k, o), oi = __shfl_xor_sync(0xffffffffu, ki, o);
      if (better(ok, oi, k, ki)) { k = ok; ki = oi; }
    }
  };
  over_warp();
  if (lane == 0) { bk[warp] = k; bi[warp] = ki; }
  __syncthreads();
  if (warp == 0) {
    k = bk[lane];
    ki = bi[lane];
    over_warp();
    if (lane == 0) { *cluster.map_shared_rank(rk + rank, 0) = k; *cluster.map_shared_rank(ri + rank, 0) = ki; }
  }
  cluster.sync();
  if (rank == 0 && tid == 0) {
    for (int r = 1; r < kArgRanks; ++r)
      if (better(rk[r], ri[r], rk[0], ri[0])) { rk[0] = rk[r]; ri[0] = ri[r]; }
    *out = ri[0];
  }
}

// gen_trapzoid (gtrap/tls.py:2-15) plus an offset, with the reference's assignment order:
// later masks overwrite earlier ones where they overlap.
__global__ void __launch_bounds__(256) trapezoid_kernel(double *out, const double *__restrict__ t, uint32_t n,
                                                        double H, double W, double L, double t0, double offset) {
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const Bounds b = bounds_of(W, L);
  const double tn = __dsub_rn(t[i], t0);
  const double mH2 = __ddiv_rn(-H, 2.0), W4 = __ddiv_rn(W, 4.0);
  double x = 0.0;
  if (tn <= b.a2) x = mH2;                                             // maskAx
  if (tn >= b.a5) x = mH2;                                             // maskEx
  if (tn < b.a4 && tn >= b.a3) x = __ddiv_rn(H, 2.0);                  // maskC
  if (tn > b.a2 && tn <= b.a3) x = __dmul_rn(__ddiv_rn(H, L), __dadd_rn(tn, W4));    // maskB
  if (tn < b.a5 && tn >= b.a4) x = __dmul_rn(__ddiv_rn(-H, L), __dsub_rn(tn, W4));   // maskD
  out[i] = __dadd_rn(x, offset);
}

}  // namespace

extern "C" {

int gtrap_tlsfit_grid(const double *t, const double *x, uint32_t n, const double *W, uint32_t nW,
                      const double *L, uint32_t nL, const double *t0, uint32_t nT, double sigma,
                      int32_t divx, double *H, double *res, int32_t *npts, double *xsum, double *sn,
                      gtrap_stream_t stream) {
  using namespace gtrap;
  const uint64_t total = (uint64_t)nW * nL * nT;
  if (total == 0) return GTRAP_OK;
  if (!t || !x || !W || !L || !t0 || !H || !res || !npts || !xsum || !sn)
    return fail(GTRAP_ERR_INVALID_ARG, "tlsfit_grid: null pointer");
  if (total > (uint64_t)0x7fffffff * kFitThreads)
    return fail(GTRAP_ERR_INVALID_ARG, "tlsfit_grid: too many templates (%llu)", (unsigned long long)total);
  const uint64_t blocks = (total + kFitThreads - 1) / kFitThreads;
  tlsfit_kernel<<<(unsigned)blocks, kFitThreads, 0, stream>>>(t, x, n, W, nW, L, nL, t0, nT, sigma, divx, H, res,
                                                              npts, xsum, sn);
  return check_launch("tlsfit_kernel");
}

int gtrap_nanargmax(const double *v, uint64_t count, int64_t *index, gtrap_stream_t stream) {
  using namespace gtrap;
  if (!v || !index) return fail(GTRAP_ERR_INVALID_ARG, "nanargmax: null pointer");
  nanargmax_kernel<<<kArgRanks, kArgThreads, 0, stream>>>(v, count, index);
  return check_launch("nanargmax_kernel");
}

int gtrap_gen_trapezoid(double *out, const double *t, uint32_t n, double H, double W, double L, double t0,
                        double offset, gtrap_stream_t stream) {
  using namespace gtrap;
  if (n == 0) return GTRAP_OK;
  if (!out || !t) return fail(GTRAP_ERR_INVALID_ARG, "gen_trapezoid: null pointer");
  trapezoid_kernel<<<(n + 255) / 256, 256, 0, stream>>>(out, t, n, H, W, L, t0, offset);
  return check_launch("trapezoid_kernel");
}

}  // extern "C"
