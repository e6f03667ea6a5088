// Per-curve peak statistics of a GTLS S/N series on the device (the host epilogue of
// gtrap/gtls.py:245-273 with detect_peaks, gtrap/detect_peaks.py:104-143).
//
// One block per curve.  For the series x[0..n) of a curve:
//  * max (first index on ties), median (numpy convention: mean of the two middle values for
//    even n), population std of the positive values, far = (max - median) / std, and the
//    count of positive values;
//  * peaks as detect_peaks(x, mpd, edge='rising') finds them: i in [1, n-2] with
//    x[i] > x[i-1] and x[i+1] <= x[i] (no NaN at i-1, i, i+1), then, in order of decreasing
//    height, every kept peak deletes the others within +-mpd.  That greedy set is computed
//    in rounds: an undecided candidate is deleted when a kept peak lies in its window and
//    kept when no undecided candidate of higher priority (height, then lower index) does.
//    Each round decides at least the highest-priority undecided candidate, and the result
//    does not depend on the order in which threads see each other's decisions;
//  * the k highest peaks (height desc, index asc), and with ntop: pssn = (top - medc) / stdc
//    over the peaks after the ntop highest (nanmedian / nanstd), diff = (ntop-th peak -
//    median) / std; pssn = inf and diff = 0 when there are at most ntop peaks.
// Medians are exact order statistics found by radix selection over the float bit patterns.
#include "common.cuh"
#include "peakstate.cuh"

#include <math.h>

namespace {

using gtrap::fail;

constexpr int kPkThreads = 512;
constexpr unsigned char kNone = 0, kUndecided = 1, kKept = 2, kDeleted = 3;

// Order-preserving key of a float.  NaN with the sign bit set ranks below all, without it as -0: one rule
// for every order statistic here, whichever kernel a series runs on.  (Written out: with the sign bit put
// into a float's bits by an or, the compiler's code gave that very key for such a NaN.)
__device__ __forceinline__ unsigned okey(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : b > 0x7f800000u ? 0x7fffffffu : (b | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
// priority of peak (v, i) over (w, j): higher value, then lower index
__device__ __forceinline__ bool prio_gt(float v, int i, float w, int j) {
  return v > w || (v == w && i < j);
}

struct Series {
  const float *x;
  size_t stride;
  int n;
  __device__ __forceinline__ float operator[](int e) const { return __ldg(x + (size_t)e * stride); }
};

// block-wide sums (double) and counts; every thread gets the result
__device__ double block_sum(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int k = 0; k < kPkThreads / 32; ++k) t += red[k];  // fixed order: deterministic
  return t;
}

// k-th smallest (0-based) of the selected values by radix selection over 8-bit digits
template <typename Sel>
__device__ float select_kth(const Series &s, Sel sel, unsigned k, unsigned *hist) {
  unsigned prefix = 0, mask = 0;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int b = threadIdx.x; b < 256; b += kPkThreads) hist[b] = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < s.n; e += kPkThreads) {
      if (!sel(e)) continue;
      const unsigned u = okey(s[e]);
      if ((u & mask) == prefix) atomicAdd(hist + ((u >> shift) & 255u), 1u);
    }
    __syncthreads();
    __shared__ unsigned s_digit, s_below;
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0) { s_digit = 255; s_below = 0; }  // (k beyond the count: unused)
      __syncwarp();
      // lane l owns bins 8l .. 8l+7
      unsigned c[8], tot = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) { c[q] = hist[8 * threadIdx.x + q]; tot += c[q]; }
      unsigned incl = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += u;
      }
      const unsigned excl = incl - tot;
      if (k >= excl && k < incl) {
        unsigned run = excl;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (k >= run && k < run + c[q]) { s_digit = 8 * threadIdx.x + q; s_below = run; }
          run += c[q];
        }
      }
    }
    __syncthreads();
    prefix |= s_digit << shift;
    mask |= 255u << shift;
    k -= s_below;
    __syncthreads();
  }
  return okey_inv(prefix);
}

__global__ void __launch_bounds__(kPkThreads) peakstat_kernel(
    const float *__restrict__ x, const unsigned long long *__restrict__ off,
    const uint32_t *__restrict__ len, size_t stride, uint32_t mpd, uint32_t ntop, uint32_t k,
    gtrap_peak_stats *out, uint32_t *peak_idx, float *peak_val) {
  extern __shared__ unsigned char state[];  // [n] candidate states
  __shared__ double red[kPkThreads / 32];
  __shared__ unsigned hist[256];
  __shared__ unsigned long long s_best;
  const int q = blockIdx.x;
  const Series s{x + off[q], stride, (int)len[q]};
  const int n = s.n;
  const int tid = threadIdx.x;
  gtrap_peak_stats r;
  r.argmax = 0; r.lent = 0; r.npeaks = 0;
  r.maxsn = 0.0f; r.median = 0.0; r.std = 0.0; r.far = 0.0; r.pssn = INFINITY; r.diff = 0.0;
  r.medc = 0.0; r.stdc = 0.0;

  // ---- pass 1: max / argmax, positive count and sum, candidates
  float vmax = -INFINITY;
  int imax = INT_MAX;
  double psum = 0.0;
  unsigned pcnt = 0;
  for (int e = tid; e < n; e += kPkThreads) {
    const float v = s[e];
    if (v > vmax || (v == vmax && e < imax) || (isnan(v) && !isnan(vmax))) { vmax = v; imax = e; }
    if (v > 0.0f) { psum += (double)v; ++pcnt; }
    unsigned char st = kNone;
    if (e >= 1 && e + 1 < n) {
      const float a = s[e - 1], c = s[e + 1];
      if (!isnan(a) && !isnan(v) && !isnan(c) && v > a && !(c > v)) st = kUndecided;
    }
    state[e] = st;
  }
  // block argmax (NaN wins, as np.max propagates it; then the larger value, then lower index)
  {
    unsigned long long key = 0ull;
    if (imax != INT_MAX) {
      const unsigned kv = isnan(vmax) ? 0xffffffffu : okey(vmax);
      key = ((unsigned long long)kv << 32) | (0xffffffffu - (unsigned)imax);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      key = ok > key ? ok : key;
    }
    if (tid == 0) s_best = 0ull;
    __syncthreads();
    if ((tid & 31) == 0 && key) atomicMax(&s_best, key);
    __syncthreads();
    if (s_best) {
      r.argmax = 0xffffffffu - (unsigned)(s_best & 0xffffffffull);
      r.maxsn = s[(int)r.argmax];
    }
  }
  const double tsum = block_sum(psum, red);
  const double tcnt = block_sum((double)pcnt, red);
  r.lent = (uint32_t)tcnt;
  // population std of the positive values (two passes)
  if (r.lent > 0) {
    const double mean = tsum / tcnt;
    double ss = 0.0;
    for (int e = tid; e < n; e += kPkThreads) {
      const float v = s[e];
      if (v > 0.0f) { const double d = (double)v - mean; ss += d * d; }
    }
    r.std = sqrt(block_sum(ss, red) / tcnt);
  } else {
    r.std = NAN;
  }
  // median of all values
  if (n > 0) {
    auto all = [&](int) { return true; };
    const float m1 = select_kth(s, all, (unsigned)(n - 1) / 2, hist);
    const float m2 = (n % 2) ? m1 : select_kth(s, all, (unsigned)n / 2, hist);
    r.median = 0.5 * ((double)m1 + (double)m2);
  }
  r.far = ((double)r.maxsn - r.median) / r.std;
  __syncthreads();

  // ---- greedy suppression within +-mpd, in rounds
  const int w = (int)mpd;
  if (w > 0) {
    for (int round = 0; round <= n; ++round) {
      int busy = 0;
      for (int e = tid; e < n; e += kPkThreads) {
        if (state[e] != kUndecided) continue;
        const float v = s[e];
        bool blocked = false, del = false;
        const int lo = max(0, e - w), hi = min(n - 1, e + w);
        for (int j = lo; j <= hi && !del; ++j) {
          if (j == e) continue;
          const unsigned char sj = ((volatile unsigned char *)state)[j];
          if (sj == kKept) del = true;
          else if (sj == kUndecided && prio_gt(s[j], j, v, e)) blocked = true;
        }
        if (del) state[e] = kDeleted;
        else if (!blocked) state[e] = kKept;
        else busy = 1;
      }
      if (!__syncthreads_or(busy)) break;
    }
  } else {
    for (int e = tid; e < n; e += kPkThreads)
      if (state[e] == kUndecided) state[e] = kKept;
  }
  __syncthreads();
  unsigned pk = 0;
  for (int e = tid; e < n; e += kPkThreads) pk += state[e] == kKept;
  r.npeaks = (uint32_t)block_sum((double)pk, red);

  // ---- the highest peaks in priority order
  const uint32_t kk = max(k, ntop);
  float lv = INFINITY;  // last selected peak (value, index): the next one ranks below it
  int li = -1;
  float top0 = 0.0f, topn = 0.0f;
  int topn_i = -1;
  for (uint32_t t = 0; t < kk && t < r.npeaks; ++t) {
    unsigned long long key = 0ull;
    for (int e = tid; e < n; e += kPkThreads) {
      if (state[e] != kKept) continue;
      const float v = s[e];
      if (!prio_gt(lv, li, v, e)) continue;  // already selected
      const unsigned long long kv = ((unsigned long long)okey(v) << 32) | (0xffffffffu - (unsigned)e);
      key = kv > key ? kv : key;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      key = ok > key ? ok : key;
    }
    if (tid == 0) s_best = 0ull;
    __syncthreads();
    if ((tid & 31) == 0 && key) atomicMax(&s_best, key);
    __syncthreads();
    const unsigned long long b = s_best;
    li = (int)(0xffffffffu - (unsigned)(b & 0xffffffffull));
    lv = okey_inv((unsigned)(b >> 32));
    if (t == 0) top0 = lv;
    if (t + 1 == ntop) { topn = lv; topn_i = li; }
    if (tid == 0 && t < k) {
      peak_idx[(size_t)q * k + t] = (uint32_t)li;
      peak_val[(size_t)q * k + t] = lv;
    }
    __syncthreads();
  }
  if (tid == 0)
    for (uint32_t t = min(r.npeaks, k); t < k; ++t) {
      peak_idx[(size_t)q * k + t] = 0xffffffffu;
      peak_val[(size_t)q * k + t] = 0.0f;
    }

  // ---- statistics of the peaks after the ntop highest
  if (ntop > 0 && r.npeaks > ntop) {
    const uint32_t m = r.npeaks - ntop;
    auto rest = [&](int e) { return state[e] == kKept && prio_gt(topn, topn_i, s[e], e); };
    double rs = 0.0;
    for (int e = tid; e < n; e += kPkThreads)
      if (rest(e)) rs += (double)s[e];
    const double mean = block_sum(rs, red) / (double)m;
    double ss = 0.0;
    for (int e = tid; e < n; e += kPkThreads)
      if (rest(e)) { const double d = (double)s[e] - mean; ss += d * d; }
    r.stdc = sqrt(block_sum(ss, red) / (double)m);
    const float c1 = select_kth(s, rest, (m - 1) / 2, hist);
    const float c2 = (m % 2) ? c1 : select_kth(s, rest, m / 2, hist);
    r.medc = 0.5 * ((double)c1 + (double)c2);
    r.pssn = ((double)top0 - r.medc) / r.stdc;
    r.diff = ((double)topn - r.median) / r.std;
  }
  if (tid == 0) out[q] = r;
}

// ---- series that fit in shared memory

constexpr int kStThreads = 1024;
constexpr int kStBins = 2048;   // digits of 11 + 11 + 10 bits

struct StScratch {
  float part[3][kStThreads / 32];
  float m0;
  unsigned wsum[kStThreads / 32];
  unsigned wkey[2][kStThreads / 32], widx[2][kStThreads / 32];
  unsigned digit, below, count, vmin;
};

// A sum of floats as three floats (error-free transformations; about 70 bits).  The FP64 pipe of
// this part takes a warp's 32 additions in 16 cycles or more, so the long sums run on FP32 and only
// their totals are joined in FP64.
struct Sum3 {
  float a = 0.0f, b = 0.0f, c = 0.0f;
  static __device__ __forceinline__ float two_sum(float x, float y, float &e) {
    const float s = __fadd_rn(x, y), t = __fsub_rn(s, x);
    e = __fadd_rn(__fsub_rn(x, __fsub_rn(s, t)), __fsub_rn(y, t));
    return s;
  }
  __device__ __forceinline__ void add(float v) {
    float e1, e2;
    a = two_sum(a, v, e1);
    b = two_sum(b, e1, e2);
    c = __fadd_rn(c, e2);
  }
  __device__ __forceinline__ void add(const Sum3 &o) { add(o.a); add(o.b); add(o.c); }
  __device__ __forceinline__ void add_product(float x, float y) {   // x y exactly
    const float p = __fmul_rn(x, y);
    add(p);
    add(__fmaf_rn(x, y, -p));
  }
  __device__ __forceinline__ void over_warp() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      Sum3 u;
      u.a = __shfl_xor_sync(0xffffffffu, a, o);
      u.b = __shfl_xor_sync(0xffffffffu, b, o);
      u.c = __shfl_xor_sync(0xffffffffu, c, o);
      // the same order on both sides of an exchange: every lane gets the same total
      Sum3 lo = threadIdx.x & o ? u : *this;
      lo.add(threadIdx.x & o ? *this : u);
      *this = lo;
    }
  }
};

// the block's total, on warp 0 (all its lanes)
__device__ __forceinline__ Sum3 st_total(Sum3 v, StScratch &sc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v.over_warp();
  __syncthreads();
  if (lane == 0) { sc.part[0][warp] = v.a; sc.part[1][warp] = v.b; sc.part[2][warp] = v.c; }
  __syncthreads();
  Sum3 w;
  if (warp == 0) {
    w.a = sc.part[0][lane]; w.b = sc.part[1][lane]; w.c = sc.part[2][lane];
    w.over_warp();
  }
  return w;
}

// Population standard deviation of the val(e), e < n, with use(e) (count of them, at least one),
// from the deviations about the mean's float; on thread 0.
template <typename Val, typename Use>
__device__ __forceinline__ double st_std(Val val, Use use, unsigned n, unsigned count, StScratch &sc) {
  const int tid = threadIdx.x;
  // a power of two out of the squares' way: the largest magnitude times 2^-ex is below 4
  __syncthreads();
  if (tid == 0) sc.vmin = 0u;
  __syncthreads();
  unsigned big = 0u;
  for (unsigned e = tid; e < n; e += kStThreads)
    if (use(e)) big = max(big, __float_as_uint(fabsf(val(e))));
  big = __reduce_max_sync(0xffffffffu, big);
  if ((tid & 31) == 0) atomicMax(&sc.vmin, big);
  __syncthreads();
  const float vbig = __uint_as_float(sc.vmin);
  const int ex = isfinite(vbig) && vbig > 0.0f ? min(max(ilogbf(vbig), -126), 126) : 0;
  const float down = ldexpf(1.0f, -ex);
  Sum3 s;
  for (unsigned e = tid; e < n; e += kStThreads)
    if (use(e)) s.add(__fmul_rn(val(e), down));
  const Sum3 all = st_total(s, sc);
  double total = 0.0;
  if (tid == 0) {   // (FP64 on one warp only: a division takes a warp hundreds of cycles here)
    total = (double)all.a + ((double)all.b + (double)all.c);
    sc.m0 = (float)(total / (double)count);
  }
  __syncthreads();
  const float m0 = sc.m0;
  Sum3 ss;
  for (unsigned e = tid; e < n; e += kStThreads) {
    if (!use(e)) continue;
    float lo;
    const float d = Sum3::two_sum(__fmul_rn(val(e), down), -m0, lo);   // value - m0 = d + lo exactly
    ss.add_product(d, d);
    ss.add_product(d, __fadd_rn(lo, lo));
    ss.add(__fmul_rn(lo, lo));
  }
  const Sum3 sq = st_total(ss, sc);
  double std = 0.0;
  if (tid == 0) {
    const double dev = total - (double)count * (double)m0;   // sum of the deviations from m0
    const double var = ((double)sq.a + ((double)sq.b + (double)sq.c) - dev * dev / (double)count) / (double)count;
    std = ldexp(sqrt(var <= 0.0 ? 0.0 : var), ex);
  }
  return std;
}

// exclusive prefix over the block's threads; the total in sc.count
__device__ __forceinline__ unsigned st_scan(unsigned c, StScratch &sc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  __syncthreads();
  if (lane == 31) sc.wsum[warp] = incl;
  __syncthreads();
  const unsigned w = sc.wsum[lane];
  const unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
  const unsigned all = __reduce_add_sync(0xffffffffu, w);
  if (threadIdx.x == 0) sc.count = all;
  return before + incl - c;
}

// the k-th and (k + step)-th smallest (0-based, step 0 or 1) of val(0 .. n): radix selection over
// three digits of the order-preserving keys; the next larger value by one more pass if it is not
// the same one
template <typename Val>
__device__ __forceinline__ void st_select(Val val, unsigned n, unsigned k, unsigned step, unsigned *hist,
                                          StScratch &sc, float &a, float &b) {
  const int tid = threadIdx.x;
  unsigned prefix = 0, mask = 0, left = k, same = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int shift = d == 0 ? 21 : d == 1 ? 10 : 0;
    const unsigned bins = d == 2 ? 1024u : 2048u;
    __syncthreads();
    hist[tid] = 0;
    hist[tid + kStThreads] = 0;
    __syncthreads();
    for (unsigned e = tid; e < n; e += kStThreads) {
      const unsigned u = okey(val(e));
      if ((u & mask) == prefix) atomicAdd(hist + ((u >> shift) & (bins - 1)), 1u);
    }
    __syncthreads();
    const unsigned c0 = hist[2 * tid], c1 = hist[2 * tid + 1];
    const unsigned before = st_scan(c0 + c1, sc);
    if (left >= before && left < before + c0) { sc.digit = 2 * tid; sc.below = before; sc.vmin = c0; }
    if (left >= before + c0 && left < before + c0 + c1) { sc.digit = 2 * tid + 1; sc.below = before + c0; sc.vmin = c1; }
    __syncthreads();
    prefix |= sc.digit << shift;
    mask |= (bins - 1) << shift;
    left -= sc.below;
    same = sc.vmin;
  }
  a = okey_inv(prefix);
  b = a;
  if (left + step >= same) {   // the next value is a larger one (uniform)
    __syncthreads();
    if (tid == 0) sc.vmin = 0xffffffffu;
    __syncthreads();
    unsigned m = 0xffffffffu;
    for (unsigned e = tid; e < n; e += kStThreads) {
      const unsigned u = okey(val(e));
      if (u > prefix) m = min(m, u);
    }
    m = __reduce_min_sync(0xffffffffu, m);
    if ((tid & 31) == 0) atomicMin(&sc.vmin, m);
    __syncthreads();
    b = okey_inv(sc.vmin);
  }
}

// peakstat_kernel for series that fit (staged_max(): about 35,000 samples): the series is copied
// to shared memory once (a column of an [n, nq] image touches a sector a sample, so each of the
// passes below cost 32 bytes a sample out of L2 before), candidates become a list in index order
// and the suppression, the highest peaks and the statistics of the rest run over lists.  Latency
// bound (block-wide steps over a few samples a thread): 96 series of 18,000 samples 815 -> 81 us,
// of which the copy takes 10, the suppression's 8 rounds 10 and the two deviations 20.
__global__ void __launch_bounds__(kStThreads, 1) peakstat_staged_kernel(
    const float *__restrict__ x, const unsigned long long *__restrict__ off,
    const uint32_t *__restrict__ len, size_t stride, uint32_t max_n, uint32_t mpd, uint32_t ntop, uint32_t k,
    gtrap_peak_stats *out, uint32_t *peak_idx, float *peak_val) {
  extern __shared__ __align__(16) float sv[];     // [max_n] the series
  // candidates' states (peakstate.cuh; a zero word on either side), their positions, and the kept
  // peaks' positions (while the suppression runs: the masks of higher candidates)
  volatile uint64_t *state = reinterpret_cast<uint64_t *>(sv + ((max_n + 1) & ~1u)) + 1;   // [-1 .. max_n / 64 + 1]
  unsigned short *list = reinterpret_cast<unsigned short *>(sv + ((max_n + 1) & ~1u)) + 4 * (max_n / 64 + 3);
  unsigned short *kept = list + max_n / 2 + 1;   // both [max_n / 2 + 1]
  __shared__ unsigned hist[kStBins];
  __shared__ StScratch sc;
  const int q = blockIdx.x, tid = threadIdx.x;
  const int n = (int)len[q];
  {
    const float *src = x + off[q];
    for (int e = tid; e < n; e += kStThreads) {
      const unsigned dst = (unsigned)__cvta_generic_to_shared(sv + e);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src + (size_t)e * stride) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  gtrap_peak_stats r;
  r.argmax = 0; r.lent = 0; r.npeaks = 0;
  r.maxsn = 0.0f; r.median = 0.0; r.std = 0.0; r.far = 0.0; r.pssn = INFINITY; r.diff = 0.0;
  r.medc = 0.0; r.stdc = 0.0;

  // ---- max / argmax (NaN wins, as np.max propagates it; then the larger value, then the lower
  // index), positive count and sum; candidates, counted and then listed in index order: a thread
  // takes a run of samples (an odd number: no bank conflicts)
  const int run = ((n + kStThreads - 1) / kStThreads) | 1;
  const int e0 = min(n, tid * run), e1 = min(n, e0 + run);
  auto candidate = [&](int e) {
    if (e < 1 || e + 1 >= n) return false;
    const float a = sv[e - 1], v = sv[e], c = sv[e + 1];
    return !isnan(a) && !isnan(v) && !isnan(c) && v > a && !(c > v);
  };
  // the highest key, then the lowest index (largest complement) of it, over the block; buffer `w`
  auto block_best = [&](unsigned key, unsigned idx, int w) -> uint2 {
    const unsigned m = __reduce_max_sync(0xffffffffu, key);
    const unsigned i = __reduce_max_sync(0xffffffffu, key == m ? idx : 0u);
    if ((tid & 31) == 0) { sc.wkey[w][tid >> 5] = m; sc.widx[w][tid >> 5] = i; }
    __syncthreads();
    const unsigned km = sc.wkey[w][tid & 31], ki = sc.widx[w][tid & 31];
    const unsigned bm = __reduce_max_sync(0xffffffffu, km);
    return make_uint2(bm, __reduce_max_sync(0xffffffffu, km == bm ? ki : 0u));
  };
  unsigned pcnt = 0, ncand = 0;
  uint2 top;
  {
    float vmax = -INFINITY;
    int imax = INT_MAX;
    for (int e = e0; e < e1; ++e) {
      const float v = sv[e];
      if (v > vmax || (v == vmax && e < imax) || (isnan(v) && !isnan(vmax))) { vmax = v; imax = e; }
      pcnt += v > 0.0f ? 1u : 0u;
      ncand += candidate(e) ? 1u : 0u;
    }
    const bool any = imax != INT_MAX;
    top = block_best(!any ? 0u : isnan(vmax) ? 0xffffffffu : okey(vmax), any ? 0xffffffffu - (unsigned)imax : 0u, 0);
  }
  unsigned at = st_scan(ncand, sc);
  for (int e = e0; e < e1; ++e)
    if (candidate(e)) list[at++] = (unsigned short)e;
  __syncthreads();
  const int M = (int)sc.count;
  if (top.y) {
    r.argmax = 0xffffffffu - top.y;
    r.maxsn = sv[r.argmax];
  }
  __syncthreads();
  st_scan(pcnt, sc);
  __syncthreads();
  r.lent = sc.count;
  r.std = NAN;
  // population std of the positive values, median of all; r's FP64 members are thread 0's alone
  if (r.lent > 0)
    r.std = st_std([&](unsigned e) { return sv[e]; }, [&](unsigned e) { return sv[e] > 0.0f; }, (unsigned)n, r.lent, sc);
  if (n > 0) {
    float m1, m2;
    st_select([&](unsigned e) { return sv[e]; }, (unsigned)n, (unsigned)(n - 1) / 2, n % 2 ? 0u : 1u, hist, sc, m1, m2);
    if (tid == 0) r.median = 0.5 * ((double)m1 + (double)m2);
  }
  if (tid == 0) r.far = ((double)r.maxsn - r.median) / r.std;

  // ---- greedy suppression within +-mpd, in rounds over the list, a warp taking 32 candidates, one
  // word of each state, at a time.  Only a candidate of higher priority can delete or hold up
  // another, and candidates are never adjacent: for windows of up to 16 samples the higher ones among
  // the eight entries on either side are found once, as a mask, and a round compares it with the
  // states' bits there; wider windows look at their entries one by one
  const int w = (int)mpd, lane = tid & 31;
  const int nword = (M + 31) >> 5;
  const bool masks = w > 0 && w <= 16;
  unsigned short *higher = kept;   // bit j: entry c - 8 + j (j < 8) or c - 7 + j
  if (tid < 2) state[tid ? nword : -1] = 0u;
  for (int i = tid >> 5; i < nword; i += kStThreads / 32) {
    const int c = 32 * i + lane;
    unsigned m = w > 0 ? 1u : 0u;
    if (masks && c < M) {
      const int e = list[c];
      const float v = sv[e];
      m = 0u;
      for (int d = 1; d <= w / 2; ++d) {   // the d-th entry on either side is 2d samples away at least
        const int p = c >= d ? (int)list[c - d] : -70000, s2 = c + d < M ? (int)list[c + d] : 200000;
        if (e - p <= w && prio_gt(sv[p], p, v, e)) m |= 1u << (8 - d);
        if (s2 - e <= w && prio_gt(sv[s2], s2, v, e)) m |= 1u << (7 + d);
      }
      higher[c] = (unsigned short)m;
    }
    const unsigned u = __ballot_sync(0xffffffffu, c < M && m), k0 = __ballot_sync(0xffffffffu, c < M && !m);
    if (lane == 0) state[i] = gtrap::peak_word(u, k0);
  }
  __syncthreads();
  if (w > 0) {
    for (int round = 0; round <= M; ++round) {
      int busy = 0;
      for (int i = tid >> 5; i < nword; i += kStThreads / 32) {
        const uint64_t own = state[i];   // (this warp alone writes it)
        const unsigned U = gtrap::undecided_of(own);
        if (!U) continue;
        const bool mine = (U >> lane) & 1u;
        bool del = false, blocked = false;
        const int c = 32 * i + lane;
        if (masks) {
          const uint64_t before = state[i - 1], behind = state[i + 1];
          gtrap::peak_decide<8>(before, own, behind, mine ? higher[c] : 0u, lane, del, blocked);
        } else if (mine) {
          const int e = list[c];
          const float v = sv[e];
          auto look = [&](int j) {   // false: past the window
            const int p = list[j];
            if (abs(p - e) > w) return false;
            const unsigned bit = 1u << (j & 31);
            const uint64_t s = state[j >> 5];
            if (gtrap::undecided_of(s) & bit) blocked |= prio_gt(sv[p], p, v, e);
            else if (gtrap::kept_of(s) & bit) del = true;
            return true;
          };
          for (int j = c - 1; j >= 0 && !del && look(j); --j) {}
          for (int j = c + 1; j < M && !del && look(j); ++j) {}
        }
        const unsigned kb = __ballot_sync(0xffffffffu, mine && !del && !blocked);
        const unsigned db = __ballot_sync(0xffffffffu, mine && del);
        if (lane == 0) state[i] = gtrap::peak_word(U & ~(kb | db), gtrap::kept_of(own) | kb);
        busy |= (U & ~(kb | db)) != 0u;
      }
      if (!__syncthreads_or(busy)) break;
    }
  }
  __syncthreads();
  // the kept peaks as a list of their own, in index order
  {
    unsigned cnt = 0;
    for (int i = tid; i < nword; i += kStThreads) cnt += __popc(gtrap::kept_of(state[i]));   // (nword <= threads)
    unsigned to = st_scan(cnt, sc);
    for (int i = tid; i < nword; i += kStThreads)
      for (unsigned m = gtrap::kept_of(state[i]); m; m &= m - 1) kept[to++] = list[32 * i + __ffs(m) - 1];
  }
  __syncthreads();
  const unsigned K = sc.count;
  r.npeaks = K;
  __syncthreads();

  // ---- the highest peaks in priority order
  const uint32_t kk = max(k, ntop);
  float lv = INFINITY;  // last selected peak (value, index): the next one ranks below it
  int li = -1;
  float top0 = 0.0f, topn = 0.0f;
  int topn_i = -1;
  for (uint32_t t = 0; t < kk && t < K; ++t) {
    unsigned key = 0u, idx = 0u;
    for (unsigned c = tid; c < K; c += kStThreads) {
      const int e = kept[c];
      const float v = sv[e];
      if (!prio_gt(lv, li, v, e)) continue;  // already selected
      const unsigned kv = okey(v), ki = 0xffffffffu - (unsigned)e;
      if (kv > key || (kv == key && ki > idx)) { key = kv; idx = ki; }
    }
    const uint2 b = block_best(key, idx, t & 1);   // (the other buffer's reads ended a barrier ago)
    li = (int)(0xffffffffu - b.y);
    lv = okey_inv(b.x);
    if (t == 0) top0 = lv;
    if (t + 1 == ntop) { topn = lv; topn_i = li; }
    if (tid == 0 && t < k) {
      peak_idx[(size_t)q * k + t] = (uint32_t)li;
      peak_val[(size_t)q * k + t] = lv;
    }
  }
  if (tid == 0)
    for (uint32_t t = min(K, k); t < k; ++t) {
      peak_idx[(size_t)q * k + t] = 0xffffffffu;
      peak_val[(size_t)q * k + t] = 0.0f;
    }

  // ---- statistics of the peaks after the ntop highest
  if (ntop > 0 && K > ntop) {
    const uint32_t m = K - ntop;
    auto rest = [&](int e) { return prio_gt(topn, topn_i, sv[e], e); };
    r.stdc = st_std([&](unsigned c) { return sv[kept[c]]; }, [&](unsigned c) { return rest(kept[c]); }, K, m, sc);
    // the rest are the K - ntop lowest of the kept: ranks of the rest are ranks of them all
    float c1, c2;
    st_select([&](unsigned c) { return sv[kept[c]]; }, K, (m - 1) / 2, m % 2 ? 0u : 1u, hist, sc, c1, c2);
    if (tid == 0) {
      r.medc = 0.5 * ((double)c1 + (double)c2);
      r.pssn = ((double)top0 - r.medc) / r.stdc;
      r.diff = ((double)topn - r.median) / r.std;
    }
  }
  if (tid == 0) out[q] = r;
}

// Shared memory of a staged series: values, states and two lists of positions (candidates are
// never adjacent, so at most half as many as samples).
size_t staged_bytes(size_t max_n) { return 4 * ((max_n + 1) & ~size_t(1)) + 8 * (max_n / 64 + 3) + 4 * (max_n / 2 + 1); }

size_t staged_max() {
  const size_t room = (size_t)gtrap::max_smem_optin() - sizeof(StScratch) - kStBins * sizeof(unsigned) - 256;
  size_t n = room / 6;
  // positions are 16-bit, and a thread lists the kept of one word of states
  if (n > 64 * kStThreads - 64) n = 64 * kStThreads - 64;
  while (n && staged_bytes(n) > room) --n;
  return n;
}

}  // namespace

extern "C" {

size_t gtrap_peakstat_max_samples(void) {
  return (size_t)gtrap::max_smem_optin() - 4096;
}

int gtrap_peakstat(const float *sn, const uint64_t *off, const uint32_t *n, uint64_t stride,
                   uint32_t ncurves, uint32_t max_n, uint32_t mpd, uint32_t ntop, uint32_t k,
                   gtrap_peak_stats *stats, uint32_t *peak_idx, float *peak_val,
                   gtrap_stream_t stream) {
  using namespace gtrap;
  if (ncurves == 0) return GTRAP_OK;
  if (!sn || !off || !n || !stats || (k && (!peak_idx || !peak_val)))
    return fail(GTRAP_ERR_INVALID_ARG, "peakstat: null pointer");
  if (stride == 0) return fail(GTRAP_ERR_INVALID_ARG, "peakstat: stride must be positive");
  if (k > 1024 || ntop > 1024) return fail(GTRAP_ERR_INVALID_ARG, "peakstat: k and ntop must be at most 1024");
  const size_t smem = max_n ? (size_t)max_n : 1;
  if (smem > gtrap_peakstat_max_samples())
    return fail(GTRAP_ERR_UNSUPPORTED, "peakstat: series of %u samples exceed the %zu that fit in shared memory",
                max_n, gtrap_peakstat_max_samples());
  // Short series with wide windows, many of them: the staged kernel's walks over a list that one window spans leave
  // most of its 1024 threads idle, and it runs one block an SM.  Staged / the other, 5000 series: mpd 100, 200
  // samples 1783 / 1216 us, 500 2297 / 1934, 700 2732 / 2783; mpd 17, 200 samples 1264 / 1189; 100 series
  // of 200 with mpd 100 87 / 131; mpd 16, the masks' reach, 5000 of 200 891 / 1176.
  const bool wide_short = mpd > 16 && smem <= 512 && ncurves > 4u * (uint32_t)sm_count();
  if (smem <= staged_max() && !wide_short) {
    const size_t bytes = staged_bytes(smem);
    GTRAP_TRY(ensure_smem((const void *)peakstat_staged_kernel, bytes, "peakstat"));
    peakstat_staged_kernel<<<ncurves, kStThreads, bytes, stream>>>(sn, (const unsigned long long *)off, n, (size_t)stride,
                                                                  (uint32_t)smem, mpd, ntop, k, stats, peak_idx, peak_val);
    return check_launch("peakstat_staged_kernel");
  }
  GTRAP_TRY(ensure_smem((const void *)peakstat_kernel, smem, "peakstat"));
  peakstat_kernel<<<ncurves, kPkThreads, smem, stream>>>(sn, (const unsigned long long *)off, n,
                                                         (size_t)stride, mpd, ntop, k, stats,
                                                         peak_idx, peak_val);
  return check_launch("peakstat_kernel");
}

}  // extern "C"
