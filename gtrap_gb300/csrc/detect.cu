// detect_peaks (gtrap/detect_peaks.py:13-143) on the device, every option but the plot.
//
// A cluster of eight blocks per call (one block for the shortest series).  As the reference, in
// float64: x = -x for valleys; NaN values become
// +inf for the height tests, and a difference involving a NaN becomes +inf when the series
// holds a NaN (inf - inf stays NaN otherwise, as numpy leaves it); candidates by edge rule
// (None: dx[i] < 0 < dx[i-1]; rising: dx[i] <= 0 < dx[i-1]; falling: dx[i] < 0 <= dx[i-1];
// both: rising or falling), none within one sample of a NaN, neither end; then height >= mph,
// then min(x[i] - x[i-1], x[i] - x[i+1]) >= threshold (when threshold > 0); then, when
// mpd > 1, the greedy suppression in order of decreasing height: a kept peak deletes the
// candidates within +-mpd (only the strictly lower ones with kpsh).  The greedy set is
// computed in rounds as in peakstat_kernel: an undecided candidate is deleted when a kept
// peak that may delete it lies in its window, and kept when no undecided candidate that may
// delete it and ranks above it does.  Equal heights rank by index (lower first): the
// reference's unstable argsort leaves their order open.  The survivors are written in
// increasing index order.
#include "common.cuh"
#include "peakstate.cuh"

#include <cooperative_groups.h>
#include <math.h>

namespace {

using gtrap::fail;

constexpr int kDpThreads = 1024;
constexpr unsigned char kNone = 0, kUndecided = 1, kKept = 2, kDeleted = 3;

struct DpArgs {
  const double *x;
  uint64_t n;
  double mph, threshold;
  uint32_t mpd;
  int has_mph, edge, kpsh, valley;  // edge: 0 none, 1 rising, 2 falling, 3 both
  unsigned char *state;
  int64_t *out;
  uint64_t *count;
};

__device__ __forceinline__ double xv(const DpArgs &a, int64_t i) {  // height used by the tests
  double v = a.x[i];
  if (a.valley) v = -v;
  return isnan(v) ? INFINITY : v;
}

__global__ void __launch_bounds__(kDpThreads) detect_peaks_kernel(const DpArgs a) {
  __shared__ unsigned long long warp_tot[kDpThreads / 32];
  __shared__ unsigned long long s_base;
  const int64_t n = (int64_t)a.n;
  const int tid = threadIdx.x;
  int any_nan = 0;
  for (int64_t i = tid; i < n; i += kDpThreads) any_nan |= isnan(a.x[i]) ? 1 : 0;
  const bool has_nan = __syncthreads_or(any_nan);
  // difference x[i+1] - x[i] of the (negated) values, NaN -> +inf when the series holds a NaN
  auto dx = [&](int64_t i) {
    double u = a.x[i], w = a.x[i + 1];
    if (a.valley) { u = -u; w = -w; }
    const double d = w - u;
    return (isnan(d) && has_nan) ? INFINITY : d;
  };
  for (int64_t i = tid; i < n; i += kDpThreads) {
    unsigned char st = kNone;
    if (i >= 1 && i + 1 < n && !isnan(a.x[i - 1]) && !isnan(a.x[i]) && !isnan(a.x[i + 1])) {
      const double dl = dx(i - 1), dr = dx(i);
      bool c;
      if (a.edge == 0) {
        c = dr < 0.0 && dl > 0.0;
      } else {
        const bool rise = dr <= 0.0 && dl > 0.0, fall = dr < 0.0 && dl >= 0.0;
        c = (a.edge & 1 && rise) || (a.edge & 2 && fall);
      }
      const double v = xv(a, i);
      if (c && a.has_mph && !(v >= a.mph)) c = false;
      if (c && a.threshold > 0.0) {  // np.min propagates a NaN (inf - inf), which is kept
        const double d1 = v - xv(a, i - 1), d2 = v - xv(a, i + 1);
        if (!isnan(d1) && !isnan(d2) && fmin(d1, d2) < a.threshold) c = false;
      }
      if (c) st = kUndecided;
    }
    a.state[i] = st;
  }
  __syncthreads();
  // greedy suppression within +-mpd, in rounds (mpd > 1 only, as the reference)
  const int64_t w = (int64_t)a.mpd;
  if (w > 1) {
    for (int64_t round = 0; round <= n; ++round) {
      int busy = 0;
      for (int64_t e = tid; e < n; e += kDpThreads) {
        if (a.state[e] != kUndecided) continue;
        const double v = xv(a, e);
        bool blocked = false, del = false;
        const int64_t lo = e - w > 0 ? e - w : 0, hi = e + w < n - 1 ? e + w : n - 1;
        for (int64_t j = lo; j <= hi && !del; ++j) {
          if (j == e) continue;
          const unsigned char sj = ((volatile unsigned char *)a.state)[j];
          if (sj != kKept && sj != kUndecided) continue;
          const double u = xv(a, j);
          // may j delete e?  always, or only when strictly higher with kpsh
          const bool may = a.kpsh ? u > v : true;
          if (!may) continue;
          if (sj == kKept) del = true;
          else if (u > v || (u == v && j < e)) blocked = true;  // j ranks above e
        }
        if (del) a.state[e] = kDeleted;
        else if (!blocked) a.state[e] = kKept;
        else busy = 1;
      }
      if (!__syncthreads_or(busy)) break;
    }
  } else {
    for (int64_t e = tid; e < n; e += kDpThreads)
      if (a.state[e] == kUndecided) a.state[e] = kKept;
  }
  __syncthreads();
  // compaction in index order: chunks of kDpThreads elements, a block scan per chunk
  if (tid == 0) s_base = 0;
  __syncthreads();
  for (int64_t c0 = 0; c0 < n; c0 += kDpThreads) {
    const int64_t i = c0 + tid;
    const unsigned keep = (i < n && a.state[i] == kKept) ? 1u : 0u;
    const unsigned ball = __ballot_sync(0xffffffffu, keep);
    const int lane = tid & 31, warp = tid >> 5;
    if (lane == 0) warp_tot[warp] = __popc(ball);
    __syncthreads();
    unsigned long long before = s_base;
    for (int k = 0; k < warp; ++k) before += warp_tot[k];
    if (keep) a.out[before + __popc(ball & ((1u << lane) - 1u))] = i;
    __syncthreads();
    if (tid == 0) {
      unsigned long long tot = 0;
      for (int k = 0; k < kDpThreads / 32; ++k) tot += warp_tot[k];
      s_base += tot;
    }
    __syncthreads();
  }
  if (tid == 0) *a.count = s_base;
}

// ---- the same over a cluster of blocks

constexpr int kDcRanks = 8;
constexpr int kDcAhead = 8;          // words of states a warp compacts at once
constexpr uint64_t kDcMinN = 64;     // 7 bytes of alignment and n / 32 + 3 words fit the caller's byte a sample
constexpr uint64_t kDcMaxN = 0x7fffffff;

// Doubles are compared as integers (an FP64 instruction takes a warp 16 cycles or more here): keys
// in the order of the values, +0 and -0 alike.  A difference of two values that are not NaN has the
// sign of their comparison, except that of equal infinities, which is NaN.
__device__ __forceinline__ long long dp_bits(const DpArgs &a, int64_t i) {
  const long long b = __ldg(reinterpret_cast<const long long *>(a.x) + i);
  return a.valley ? b ^ (long long)0x8000000000000000ull : b;
}
__device__ __forceinline__ bool dp_nan(long long b) {
  return (b & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ long long dp_key(long long b) {
  if ((b & 0x7fffffffffffffffll) == 0) return 0;
  return b < 0 ? b ^ 0x7fffffffffffffffll : b;
}

// A word of states is read by warps of every block while its own warp writes it: one access each, at L2.
__device__ __forceinline__ uint64_t load_word(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_word(uint64_t *p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Blocks 0 .. kDcRanks - 1 of one cluster.  Candidates are listed in index order (each block a
// run of samples), their states kept as bits (peakstate.cuh), and a round of the suppression compares
// the mask of a candidate's higher neighbours with the states' bits around it, a warp taking 32
// candidates: a candidate is decided by candidates that rank above it alone.  Scratch: positions in
// the upper half of the index output (peak k is written only when the positions up to the k-th
// candidate have been read, which lie past it), masks in the lower half, states in `state`.  Bound by
// the latency of the rounds and of the list steps.  One block, walking samples / the cluster, mpd 10:
// 20,011 samples 779 / 28 us, 2^20 samples 40.2 / 0.63 ms; mpd 100: 3.9 / 0.23 ms, 135 / 4.6 ms.
__global__ void __cluster_dims__(kDcRanks, 1, 1) __launch_bounds__(kDpThreads, 1)
detect_peaks_cluster_kernel(const DpArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ unsigned flags[2][kDcRanks];   // one word of every block, which each posts to all
  __shared__ unsigned warp_cnt[kDpThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)blockIdx.x;
  const int64_t n = (int64_t)a.n;
  auto post = [&](int slot, unsigned v) {
    if (tid < kDcRanks) *cluster.map_shared_rank(&flags[slot][rank], tid) = v;
  };
  auto sum_over = [&](int slot, int ranks) {
    unsigned s = 0;
    for (int r = 0; r < ranks; ++r) s += flags[slot][r];
    return s;
  };
  unsigned *const list = reinterpret_cast<unsigned *>(a.out) + n;          // positions of the candidates
  unsigned *const higher = reinterpret_cast<unsigned *>(a.out);             // masks (bits 0-15 before, 16-31 behind)
  // states of 32 candidates a word, a zero word on either side
  uint64_t *const state = reinterpret_cast<uint64_t *>(((uintptr_t)a.state + 7) & ~uintptr_t(7)) + 1;

  cluster.sync();   // every block has started: its shared memory may be written

  // ---- any NaN
  int any_nan = 0;
  for (int64_t i = (int64_t)rank * kDpThreads + tid; i < n; i += (int64_t)kDcRanks * kDpThreads)
    any_nan |= dp_nan(dp_bits(a, i)) ? 1 : 0;
  any_nan = __syncthreads_or(any_nan);
  post(0, any_nan ? 1u : 0u);
  cluster.sync();
  const bool has_nan = sum_over(0, kDcRanks) != 0u;

  // ---- candidates of this block's run of samples: counted, then listed
  const long long inf = 0x7ff0000000000000ll, mph = dp_key(__double_as_longlong(a.mph));
  const bool mph_nan = dp_nan(__double_as_longlong(a.mph));
  auto candidate = [&](int64_t i) -> bool {
    if (i < 1 || i + 1 >= n) return false;
    const long long bl = dp_bits(a, i - 1), b = dp_bits(a, i), br = dp_bits(a, i + 1);
    if (dp_nan(bl) || dp_nan(b) || dp_nan(br)) return false;
    const long long kl = dp_key(bl), k = dp_key(b), kr = dp_key(br);
    const bool infk = (k == inf) || (k == dp_key((long long)0xfff0000000000000ull));
    // the signs of the differences to the left (value - left) and right (right - value); of equal
    // infinities +inf when the series holds a NaN, else NaN (no comparison holds)
    const bool xl = infk && kl == k, xr = infk && kr == k;
    const bool l_pos = xl ? has_nan : k > kl, l_ge = xl ? has_nan : k >= kl;
    const bool r_neg = !xr && kr < k, r_le = !xr && kr <= k;
    bool c;
    if (a.edge == 0) c = r_neg && l_pos;
    else c = (a.edge & 1 && r_le && l_pos) || (a.edge & 2 && r_neg && l_ge);
    if (c && a.has_mph && (mph_nan || k < mph)) c = false;
    if (c && a.threshold > 0.0) {  // np.min propagates a NaN (inf - inf), which is kept
      const double v = __longlong_as_double(b);
      const double d1 = v - __longlong_as_double(bl), d2 = v - __longlong_as_double(br);
      if (!isnan(d1) && !isnan(d2) && fmin(d1, d2) < a.threshold) c = false;
    }
    return c;
  };
  const int64_t run = (n + kDcRanks - 1) / kDcRanks;
  const int64_t i0 = min(n, rank * run), i1 = min(n, i0 + run);
  {
    unsigned cnt = 0;
    for (int64_t i = i0 + tid; i < i1; i += kDpThreads) cnt += candidate(i) ? 1u : 0u;
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) warp_cnt[warp] = cnt;
    __syncthreads();
    const unsigned all = __reduce_add_sync(0xffffffffu, warp_cnt[lane]);
    post(1, all);
  }
  cluster.sync();
  const int64_t M = sum_over(1, kDcRanks);
  {
    unsigned base = sum_over(1, rank);
    for (int64_t c0 = i0; c0 < i1; c0 += kDpThreads) {   // the same count of steps for every thread
      const int64_t i = c0 + tid;
      const bool f = i < i1 && candidate(i);
      const unsigned ball = __ballot_sync(0xffffffffu, f);
      __syncthreads();
      if (lane == 0) warp_cnt[warp] = __popc(ball);
      __syncthreads();
      const unsigned w = warp_cnt[lane];
      const unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
      if (f) __stcg(list + base + before + __popc(ball & ((1u << lane) - 1u)), (unsigned)i);
      base += __reduce_add_sync(0xffffffffu, w);
    }
  }
  cluster.sync();

  // ---- masks of higher candidates and the first states
  const int64_t nword = (M + 31) / 32;
  const int64_t w = (int64_t)a.mpd;
  auto value = [&](unsigned p) { return dp_key(dp_bits(a, p)); };
  // whether the candidate at position p (value u) may delete, and so ranks above, that at e (value v)
  auto above = [&](long long u, unsigned p, long long v, unsigned e) { return u > v || (!a.kpsh && u == v && p < e); };
  // rising and falling edges together can mark neighbouring samples, one rule alone cannot
  const int near = a.edge == 3 ? (int)min(w, (int64_t)17) : (int)(min(w, (int64_t)34) / 2);
  const bool masks = near <= 16;   // the entries within the window are among the 16 on either side
  const int64_t gwarp = (int64_t)rank * (kDpThreads / 32) + warp, nwarp = kDcRanks * (kDpThreads / 32);
  if (gwarp == 0 && lane < 2) store_word(state + (lane ? nword : -1), 0u);
  for (int64_t i = gwarp; i < nword; i += nwarp) {
    const int64_t c = 32 * i + lane;
    unsigned m = w > 1 ? 1u : 0u;
    if (w > 1 && masks && c < M) {
      const unsigned e = __ldcg(list + c);
      const long long v = value(e);
      m = 0u;
      for (int d = 1; d <= near; ++d) {
        if (c >= d) {
          const unsigned p = __ldcg(list + c - d);
          if ((int64_t)e - p <= w && above(value(p), p, v, e)) m |= 1u << (16 - d);
        }
        if (c + d < M) {
          const unsigned p = __ldcg(list + c + d);
          if ((int64_t)p - e <= w && above(value(p), p, v, e)) m |= 1u << (15 + d);
        }
      }
      __stcg(higher + c, m);
    }
    const unsigned u = __ballot_sync(0xffffffffu, c < M && m), k0 = __ballot_sync(0xffffffffu, c < M && !m);
    if (lane == 0) store_word(state + i, gtrap::peak_word(u, k0));
  }
  cluster.sync();
  // ---- rounds; each decides at least the highest undecided candidate
  if (w > 1) {
    for (int64_t round = 0; round <= M; ++round) {
      int busy = 0;
      for (int64_t i = gwarp; i < nword; i += nwarp) {
        const uint64_t own = load_word(state + i);   // (this warp alone writes it)
        const unsigned U = gtrap::undecided_of(own);
        if (!U) continue;
        const bool mine = (U >> lane) & 1u;
        bool del = false, blocked = false;
        const int64_t c = 32 * i + lane;
        if (masks) {
          const uint64_t before = load_word(state + i - 1), behind = load_word(state + i + 1);
          gtrap::peak_decide<16>(before, own, behind, mine ? __ldcg(higher + c) : 0u, lane, del, blocked);
        } else if (mine) {
          const unsigned e = __ldcg(list + c);
          const long long v = value(e);
          auto look = [&](int64_t j) {   // false: past the window
            const unsigned p = __ldcg(list + j);
            if ((p > e ? p - e : e - p) > w) return false;
            const unsigned bit = 1u << (j & 31);
            const uint64_t s = load_word(state + (j >> 5));
            const bool isu = gtrap::undecided_of(s) & bit, isk = gtrap::kept_of(s) & bit;
            if ((isu || isk) && above(value(p), p, v, e)) {
              if (isk) del = true;
              else blocked = true;
            }
            return true;
          };
          for (int64_t j = c - 1; j >= 0 && !del && look(j); --j) {}
          for (int64_t j = c + 1; j < M && !del && look(j); ++j) {}
        }
        const unsigned kb = __ballot_sync(0xffffffffu, mine && !del && !blocked);
        const unsigned db = __ballot_sync(0xffffffffu, mine && del);
        if (lane == 0 && (kb | db)) store_word(state + i, gtrap::peak_word(U & ~(kb | db), gtrap::kept_of(own) | kb));
        busy |= (U & ~(kb | db)) != 0u;
      }
      busy = __syncthreads_or(busy);
      post(round & 1, busy ? 1u : 0u);   // (the slots of two rounds take turns: read before they are posted again)
      cluster.sync();
      if (!sum_over(round & 1, kDcRanks)) break;
    }
  }
  // ---- rank 0 writes the kept in index order
  cluster.sync();
  if (rank != 0) return;
  uint64_t base = 0;
  for (int64_t w0 = 0; w0 < nword; w0 += (kDpThreads / 32) * kDcAhead) {
    unsigned bits[kDcAhead], pos[kDcAhead], before[kDcAhead], mine = 0;
#pragma unroll
    for (int u = 0; u < kDcAhead; ++u) {
      const int64_t i = w0 + (int64_t)warp * kDcAhead + u;
      bits[u] = i < nword ? gtrap::kept_of(load_word(state + i)) : 0u;
      pos[u] = (bits[u] >> lane) & 1u ? __ldcg(list + 32 * i + lane) : 0u;
      before[u] = mine;
      mine += __popc(bits[u]);
    }
    __syncthreads();   // (also: every position of this step has been read)
    if (lane == 0) warp_cnt[warp] = mine;
    __syncthreads();
    const unsigned wc = warp_cnt[lane];
    const uint64_t first = base + __reduce_add_sync(0xffffffffu, lane < warp ? wc : 0u);
#pragma unroll
    for (int u = 0; u < kDcAhead; ++u)
      if ((bits[u] >> lane) & 1u) a.out[first + before[u] + __popc(bits[u] & ((1u << lane) - 1u))] = (int64_t)pos[u];
    base += __reduce_add_sync(0xffffffffu, wc);
    __syncthreads();
  }
  if (tid == 0) *a.count = base;
}

}  // namespace

extern "C" {

int gtrap_detect_peaks(const double *x, uint64_t n, int32_t has_mph, double mph, uint32_t mpd,
                       double threshold, int32_t edge, int32_t kpsh, int32_t valley, unsigned char *state,
                       int64_t *indices, uint64_t *count, gtrap_stream_t stream) {
  using namespace gtrap;
  if (!count) return fail(GTRAP_ERR_INVALID_ARG, "detect_peaks: null pointer");
  if (n > 0 && (!x || !state || !indices)) return fail(GTRAP_ERR_INVALID_ARG, "detect_peaks: null pointer");
  if (edge < 0 || edge > 3) return fail(GTRAP_ERR_INVALID_ARG, "detect_peaks: edge=%d must be in [0, 3]", edge);
  DpArgs a;
  a.x = x; a.n = n < 3 ? 0 : n;  // fewer than three values: no peak
  a.mph = mph; a.threshold = threshold; a.mpd = mpd;
  a.has_mph = has_mph; a.edge = edge; a.kpsh = kpsh; a.valley = valley;
  a.state = state; a.out = indices; a.count = count;
  // a cluster of blocks from the length on where its states fit the caller's scratch; without a
  // suppression (mpd <= 1) one block is as fast on a short series (300 samples: 15 against 20 us;
  // 2000: 20 against 15)
  if (a.n >= (mpd > 1 ? kDcMinN : 1024) && a.n <= kDcMaxN && !((uintptr_t)indices & 7)) {
    detect_peaks_cluster_kernel<<<kDcRanks, kDpThreads, 0, stream>>>(a);
    return check_launch("detect_peaks_cluster_kernel");
  }
  detect_peaks_kernel<<<1, kDpThreads, 0, stream>>>(a);
  return check_launch("detect_peaks_kernel");
}

}  // extern "C"
