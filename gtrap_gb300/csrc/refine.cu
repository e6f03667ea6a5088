// Refinement of each curve's best BLS peak on a fine frequency / phase neighbourhood.
//
// The reference stops at the grid maximum: getmax + combine_stat (gtrap/getstat.py:14-57,
// 100-123) report the period of the best grid frequency and its start / end bins.  With the
// usual grids (nf ~ 8 per day of baseline) neighbouring frequencies shift the phases of the
// last samples by about a quarter cycle, so a box of a few per cent of the period peaks
// between grid points.  Here, for each curve:
//   * the grid peak j (first maximum of the spectrum) and its window [p1, p2] (end bin
//     inclusive, possibly past nb) are read from the search's outputs;
//   * 2K+1 trial frequencies f_k = f_j + (k - K) df / K, k = 0 .. 2K, cover [f_j - df, f_j + df];
//   * at each, the samples whose phase falls within M bins of the grid window are binned on a
//     grid S times finer than the search's; every window of whole bins inside that
//     neighbourhood (width in (kmi, kma] bins), then every window with fine edges within one bin
//     of the best one's edges, holding more than max(kkmi, 5) samples, is evaluated:
//     power = s^2 / (kk (N - kk)) in FP64, the statistic of the search (include/geebls.h:123)
//     at the finer resolution.
// Phases are exact 64-bit fixed-point fractions of the float32 times and frequencies (as in
// the search), referred at each trial frequency to the middle t_ref of the curve's valid time
// span, so a transit train keeps its phase while the frequency moves; bin sums are exact
// 64-bit integers of the flux quantised to 2^-40 of its range, so the result does not depend
// on the order of the additions and is the same alone or batched.  At k = K the grid window is among the
// candidates, so the refined power is never below the grid one (up to the quantisation).
#include "common.cuh"

#include <climits>

namespace {

using gtrap::fail;
using gtrap::frac64;

constexpr int kThreads = 384;
constexpr int kMaxFine = 4096;        // fine bins of one neighbourhood, (p2 - p1 + 1 + 2M) * S
constexpr double kXqMax = 1099511627776.0;  // |quantised flux| < 2^40
constexpr int kMaxGroup = 33;               // trials per block at most
constexpr int kFineMax = 2047;              // samples a fine bin's 32-bit words hold
constexpr size_t kSmemBudget = 96 * 1024;   // fine histograms of one block (two blocks per SM)

// One trial frequency's best window (and the curve's constants every block recomputes).
struct Part {
  double pw;            // power (-1: no window accepted)
  long long s;          // quantised flux sum of the window
  long long stot;       // quantised flux sum of every valid sample
  uint32_t a, b, kk;    // window [a, b) in fine bins, samples in it
  uint32_t nv;          // valid samples
  uint32_t j, p1;       // grid peak and its start bin
  int32_t sx;           // flux scale exponent
  float tref;           // middle of the valid time span (float32)
};

// What every trial of a curve shares, from one block a curve: the grid peak, its neighbourhood, the
// flux scale and the reference time.  (Every block of trials found them again before, from the whole
// spectrum and the whole curve.)
struct Head {
  uint32_t j, p1, L, M;   // grid peak, its start bin, coarse bins and margin of the neighbourhood
  uint32_t nv;            // valid samples
  int32_t sx;             // flux scale exponent
  float tref;             // middle of the valid time span (float32)
  int32_t ok;             // 0: no refinement
};

struct RefCurve {
  uint64_t off, stride, out;  // sample i at [off + i*stride]; spectrum at [out, out + nf)
  uint32_t n, nf, ntrue, kkmi;
  float fmin, df, offset;
};

struct RefArgs {
  const float *blsp;
  const uint32_t *ph1, *ph2;
  const float *t, *x;
  const gtrap_bls_curve *curves;  // packed form, or null for an [n, nq] image
  const uint32_t *sel;            // packed: curve of output c (c when null)
  const float *offset;            // image form
  const uint32_t *ntrue;
  uint32_t n, nq, nf, kkmi;
  float fmin, df;
  uint32_t nb, kma, kmi, K, S, M;
  uint32_t smem, min_groups;      // a block's dynamic shared memory, groups of trials a curve at least
  int lognb, logK;
  Part *part;                     // [count, 2K + 1]
  Head *head;                     // [count]
  gtrap_bls_refined *out;
};

__device__ RefCurve curve_of(const RefArgs &a, uint32_t c) {
  RefCurve r;
  if (a.curves) {
    const gtrap_bls_curve g = a.curves[a.sel ? a.sel[c] : c];
    r.off = g.off; r.stride = 1; r.out = g.out;
    r.n = g.n; r.nf = g.nf; r.ntrue = g.ntrue; r.kkmi = g.kkmi;
    r.fmin = g.fmin; r.df = g.df; r.offset = g.offset;
  } else {
    r.off = c; r.stride = a.nq; r.out = (uint64_t)c * a.nf;
    r.n = a.n; r.nf = a.nf; r.ntrue = a.ntrue[c]; r.kkmi = a.kkmi;
    r.fmin = a.fmin; r.df = a.df; r.offset = a.offset[c];
  }
  return r;
}

// (x - offset is finite in double whenever both are finite floats; a non-finite offset is
// checked once per curve)
__device__ __forceinline__ bool valid(float t, float x) {
  return t >= 0.0f && isfinite(t) && isfinite(x);
}

// rint((x - off) * 2^sx) for finite floats with |x - off| * 2^sx < 2^40 (at most one unit off
// the exact rounding), in FP32 and integer instructions: x - off = s + e exactly (TwoSum),
// s * 2^sx split into 20-bit halves.  2^sx comes as two factors (either may be out of the float
// range as one); scaling up is exact, and what scaling down rounds is below one unit.
struct Scale {
  float a, b;
  __device__ explicit Scale(int sx) : a(ldexpf(1.0f, sx / 2)), b(ldexpf(1.0f, sx - sx / 2)) {}
};

__device__ __forceinline__ long long quantise(float x, float off, const Scale &sc) {
  const float s = __fsub_rn(x, off);
  const float bv = __fsub_rn(s, x);
  const float e = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bv)), __fsub_rn(-off, bv));
  const float S = __fmul_rn(__fmul_rn(s, sc.a), sc.b), Es = __fmul_rn(__fmul_rn(e, sc.a), sc.b);
  const float hi = truncf(__fmul_rn(S, 0x1p-20f));
  const float lo = __fsub_rn(S, __fmul_rn(hi, 0x1p20f));  // exact: S with its top bits removed
  return ((long long)__float2int_rz(hi) << 20) + (long long)__float2int_rn(lo) + (long long)__float2int_rn(Es);
}

// Block reduction (kThreads threads); every thread gets the result.
template <typename T>
__device__ T block_sum(T v, T *sh) {  // fixed order: lanes by shuffle tree, warps in order
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = sh[0];
  for (int w = 1; w < kThreads / 32; ++w) v += sh[w];
  return v;
}

// better window: higher power, then lower start, then lower end
__device__ __forceinline__ bool better(double p, uint32_t a, uint32_t b, double bp, uint32_t ba, uint32_t bb) {
  return p > bp || (p == bp && (a < ba || (a == ba && b < bb)));
}

constexpr int kHeadThreads = 512;

__global__ void __launch_bounds__(kHeadThreads) refine_head_kernel(const RefArgs a) {
  constexpr int kW = kHeadThreads / 32, kU = 8;
  __shared__ float shf[4][kW];
  __shared__ uint32_t shn[kW], sj;
  const uint32_t c = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const RefCurve cv = curve_of(a, c);
  // grid peak: first maximum of the spectrum
  float best = -INFINITY;
  uint32_t bj = UINT_MAX;
  for (uint32_t j0 = 0; j0 < cv.nf; j0 += kHeadThreads * kU) {   // kU loads ahead of their uses
    float v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t j = j0 + u * kHeadThreads + tid;
      v[u] = j < cv.nf ? __ldg(a.blsp + cv.out + j) : -INFINITY;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (v[u] > best) { best = v[u]; bj = j0 + u * kHeadThreads + tid; }  // ascending: this thread's first maximum
  }
  // scale, reference time, valid count (a non-finite offset leaves no valid sample)
  const bool off_ok = isfinite(cv.offset);
  float amax = 0.0f, tlo = INFINITY, thi = -INFINITY;
  uint32_t cnt = 0;
  for (uint32_t i0 = 0; i0 < cv.n; i0 += kHeadThreads * kU) {
    float tv[kU], xv[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t i = i0 + u * kHeadThreads + tid;
      const size_t idx = cv.off + (size_t)i * cv.stride;
      tv[u] = i < cv.n ? __ldg(a.t + idx) : -1.0f;
      xv[u] = i < cv.n ? __ldg(a.x + idx) : 0.0f;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (off_ok && valid(tv[u], xv[u])) {
        amax = fmaxf(amax, fabsf(__fsub_rz(xv[u], cv.offset)));
        tlo = fminf(tlo, tv[u]);
        thi = fmaxf(thi, tv[u]);
        ++cnt;
      }
    }
  }
  float gmax = best;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    tlo = fminf(tlo, __shfl_xor_sync(0xffffffffu, tlo, o));
    thi = fmaxf(thi, __shfl_xor_sync(0xffffffffu, thi, o));
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if (tid == 0) sj = UINT_MAX;
  if (lane == 0) { shf[0][warp] = gmax; shf[1][warp] = amax; shf[2][warp] = tlo; shf[3][warp] = thi; shn[warp] = cnt; }
  __syncthreads();
  gmax = shf[0][0]; amax = shf[1][0]; tlo = shf[2][0]; thi = shf[3][0]; cnt = shn[0];
  for (int w = 1; w < kW; ++w) {
    gmax = fmaxf(gmax, shf[0][w]); amax = fmaxf(amax, shf[1][w]);
    tlo = fminf(tlo, shf[2][w]); thi = fmaxf(thi, shf[3][w]); cnt += shn[w];
  }
  if (best == gmax && bj != UINT_MAX) atomicMin(&sj, bj);
  __syncthreads();
  if (tid != 0) return;
  const uint32_t j = sj, nb = a.nb;
  Head h;
  h.j = j == UINT_MAX ? 0u : j;
  h.p1 = j == UINT_MAX ? 0u : a.ph1[cv.out + j];
  const uint32_t p2 = j == UINT_MAX ? 0u : a.ph2[cv.out + j];
  // no positive peak, or a window the search cannot have produced (start past nb, end before
  // start, wider than kma): no refinement (the neighbourhood must fit the host-sized bins)
  h.ok = gmax > 0.0f && j != UINT_MAX && h.p1 < nb && p2 >= h.p1 && p2 - h.p1 + 1 <= a.kma;
  // neighbourhood: grid window widened by M bins on each side, at most one cycle
  uint32_t M = a.M;
  const uint32_t w0 = p2 - h.p1 + 1;
  while (M > 0 && w0 + 2 * M > nb) --M;
  h.M = M;
  h.L = w0 + 2 * M;
  h.nv = cnt;
  h.sx = amax > 0.0f ? ilogb(kXqMax) - ilogbf(amax) - 1 : 0;
  // reference time: the middle of the valid time span, in float32 (order-independent)
  h.tref = cnt ? __fmul_rn(__fadd_rn(tlo, thi), 0.5f) : 0.0f;
  a.head[c] = h;
}

// Shared memory of a trial with L coarse and LS fine bins: exact prefix of the flux and the counts a
// fine entry, float prefix and row maxima a coarse entry.
__host__ __device__ inline uint32_t trial_bytes(uint32_t L, uint32_t LS) { return (LS + 1) * 12 + 4 + (L + 1) * 12; }

// |v| in floats, off by less than 2^-23 of itself, without the FP64 pipe's conversion
__device__ __forceinline__ float ll_mag(long long v) {
  const int l = (int)(unsigned)(v & 0xffffffffll);
  const int h = (int)((v - (long long)l) >> 32);
  return fabsf(__fmaf_rn((float)h, 4294967296.0f, (float)l));
}

// One block per (curve, group of G consecutive trials): the samples are read and their exact
// phase pairs formed once for the group, and each trial gets its own fine histogram; a warp then
// takes a trial at a time.  G is what the neighbourhood leaves room for (wider ones take more
// shared memory), less where there are too few curves to fill the SMs.  Bound by the phase and
// histogram work of the samples; the FP64 powers are kept to the windows that FP32 bounds leave
// (64 curves of 18,000 samples, 65 trials each: 893 us with three trials a block, every block
// finding peak and scale again, every window twice and 64-bit compare-and-swap atomics; 303 us with
// those gone; 230 us with a shift for the fine bin where S is a power of two, windows screened
// by a product and no quotient, and 12 warps a block for 8: 256 threads take 243 us, 512 (fewer
// registers each) 275 us).  Where a block has under seven trials its warps share them as teams: a lone
// curve of 9000 samples, nb = 2048, kma = 205 in 42-53 us a call (a warp a trial, the block's
// others idle: 104 for one of 500 samples, 490 with 64 fine bins a bin; now 39 and 111).
__global__ void __launch_bounds__(kThreads, 2) refine_trial_kernel(const RefArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ long long shl[kThreads / 32];
  const uint32_t c = blockIdx.x;
  const Head hd = a.head[c];
  const uint32_t nk_all = 2 * a.K + 1;
  const uint32_t L = hd.L, S = a.S, LS = L * S;   // coarse and fine bins (host check: LS <= kMaxFine)
  const uint32_t E = LS + 1;                      // prefix entries per trial
  uint32_t G = 1;
  if (hd.ok) {
    const uint32_t fit = min((uint32_t)kMaxGroup, a.smem / trial_bytes(L, LS));
    const uint32_t groups = max((nk_all + fit - 1) / fit, a.min_groups);
    G = (nk_all + groups - 1) / groups;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Part *pt = a.part + (size_t)c * nk_all;
  if (!hd.ok) {
    if (blockIdx.y == 0)
      for (uint32_t k = tid; k < nk_all; k += kThreads) { pt[k].pw = -1.0; pt[k].j = hd.j; }
    return;
  }
  const uint32_t k0 = blockIdx.y * G;
  if (k0 >= nk_all) return;
  const uint32_t nk = min(G, nk_all - k0);
  pt += k0;
  const RefCurve cv = curve_of(a, c);
  const bool off_ok = isfinite(cv.offset);
  const uint32_t nb = a.nb, j = hd.j, p1 = hd.p1, M = hd.M;
  const int sx = hd.sx;

  // ---- exact phases: trial k is A + J_k B' - (k - K) R' with B' = frac(t df/K), R' = frac(tref
  // df/K) and J_k = j K + k - K; consecutive trials differ by B' - R'
  const float dfK = ldexpf(cv.df, -a.logK);
  const unsigned long long Rp = frac64(hd.tref, dfK);
  const long long J0 = (long long)j * a.K + ((long long)k0 - (long long)a.K);
  const unsigned long long shift0 = (unsigned long long)((long long)k0 - (long long)a.K) * Rp;
  const unsigned long long lo =
      (unsigned long long)((p1 + nb - M) & (nb - 1)) << (64 - a.lognb);  // neighbourhood start
  // flux sums: two 32-bit words while folding (a 64-bit shared atomic is a loop of
  // compare-and-swaps), the signed high part of xq = hi 2^20 + lo in the second; exact while a fine
  // bin holds at most kFineMax samples, checked afterwards
  long long *hs = reinterpret_cast<long long *>(dyn);                 // [nk][E]
  int *hc = reinterpret_cast<int *>(hs + (size_t)nk * E);             // [nk][E] counts
  float2 *cp = reinterpret_cast<float2 *>(hc + (((size_t)nk * E + 1) & ~size_t(1)));   // [nk][L + 1] flux, count
  float *rm = reinterpret_cast<float *>(cp + (size_t)nk * (L + 1));   // [nk][L + 1] a start's largest bound
  for (uint32_t b = tid; b < nk * E; b += kThreads) { hs[b] = 0; hc[b] = 0; }
  __syncthreads();
  const double unscale = ldexp(1.0, -sx);
  const uint32_t nbS = a.nb * S;
  const bool pow2 = (S & (S - 1)) == 0;
  const int fine_shift = 1 + __clz(nbS);   // 32 - log2(nb S)
  const Scale sc(sx);
  long long stot = 0;
  float tn, xn;
  auto load = [&](uint32_t i) {   // a sample ahead of its use
    const size_t idx = cv.off + (size_t)i * cv.stride;
    tn = i < cv.n ? __ldg(a.t + idx) : -1.0f;
    xn = i < cv.n ? __ldg(a.x + idx) : 0.0f;
  };
  load(tid);
  for (uint32_t i = tid; i < cv.n; i += kThreads) {
    const float tv = tn, xv = xn;
    load(i + kThreads);
    if (!off_ok || !valid(tv, xv)) continue;
    const long long xq = quantise(xv, cv.offset, sc);
    stot += xq;
    const unsigned xlo = (unsigned)xq & 0xfffffu, xhi = (unsigned)(xq >> 20);
    const unsigned long long bp = frac64(tv, dfK);
    unsigned long long ph = frac64(tv, cv.fmin) + (unsigned long long)J0 * bp - shift0 - lo;
    const unsigned long long step = bp - Rp;
    // fine bin from the neighbourhood start: floor(ph nb S / 2^64), nb S < 2^20 (S a power of two: a shift)
    auto trials = [&](auto bin) {
      uint32_t row = 0;
#pragma unroll 4
      for (uint32_t g = 0; g < nk; ++g, ph += step, row += E) {
        const uint32_t fb = bin(ph);
        if (fb < LS) {
          unsigned *h = reinterpret_cast<unsigned *>(hs + row + fb);
          atomicAdd(h, xlo);
          atomicAdd(h + 1, xhi);
          atomicAdd(hc + row + fb, 1);
        }
      }
    };
    if (pow2)
      trials([&](unsigned long long p) { return (uint32_t)(p >> 32) >> fine_shift; });
    else
      trials([&](unsigned long long p) {
        return (uint32_t)(((p >> 32) * nbS + (((p & 0xffffffffull) * nbS) >> 32)) >> 32);
      });
  }
  stot = block_sum<long long>(stot, shl);
  __syncthreads();

  // ---- a warp per trial, or a team of warps where the block has fewer trials than half its warps (a few
  // curves, or neighbourhoods that leave room for little), from here on: exclusive prefix sums, then stage 1, every window of whole
  // bins in the neighbourhood (width in (kmi, kma] bins), then stage 2, fine edges within one bin of
  // the stage-1 window's edges (width in (kmi S, kma S] fine bins).  Both stages screen in FP32 with
  // error bounds: windows whose upper bound reaches a lower bound of the largest power are compared
  // exactly in FP64.
  const double N = (double)cv.ntrue;
  const float Nf = (float)cv.ntrue;
  const int kkmi = (int)(cv.kkmi < 5u ? 5u : cv.kkmi);
  const float kkmi_f = (float)kkmi;
  const int kma = (int)a.kma, kmi = (int)a.kmi, iL = (int)L;
  auto warp_max = [](float v) {   // non-negative values
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
  };
  __shared__ float team_pm[kThreads / 32], team_thr[kThreads / 32], team_top[kThreads / 32];
  __shared__ double best_p[kThreads / 32];
  __shared__ uint32_t best_a[kThreads / 32], best_b[kThreads / 32];
  const int W = max(1, kThreads / 32 / (int)nk), team = warp / W, member = warp - team * W;
  auto team_sync = [&]() {
    if (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(32 * W) : "memory");
  };
  auto team_max = [&](float v, float *sh) {   // of warp-uniform values
    if (W == 1) return v;
    if (lane == 0) sh[warp] = v;
    team_sync();
    for (int m = 0; m < W; ++m) v = fmaxf(v, sh[team * W + m]);
    return v;
  };
  for (uint32_t g = team; g < nk; g += kThreads / 32 / W) {   // (a team: one trial)
    long long *H = hs + (size_t)g * E;
    int *C = hc + (size_t)g * E;
    float2 *P = cp + (size_t)g * (L + 1);
    float *R = rm + (size_t)g * (L + 1);
    if (member == 0) {
      // each lane a run of entries (an odd number: fewer bank conflicts), a warp scan of the totals
      const uint32_t run = ((E + 31) / 32) | 1u;
      const uint32_t b0 = min(E, lane * run), b1 = min(E, b0 + run);
      long long ls = 0;
      int lc = 0, cmax = 0;
      for (uint32_t b = b0; b < b1; ++b) {
        const uint2 v = reinterpret_cast<const uint2 *>(H)[b];
        H[b] = ((long long)(int)v.y << 20) + (long long)v.x;
        ls += H[b];
        lc += C[b];
        cmax = max(cmax, C[b]);
      }
      if (__any_sync(0xffffffffu, cmax > kFineMax)) {   // rare: this trial's sums again, 64 bits at a time
        __syncwarp();   // (a vote orders no memory: every lane's run has been read and written)
        for (uint32_t b = lane; b < E; b += 32) H[b] = 0;
        __syncwarp();
        for (uint32_t i = lane; i < cv.n; i += 32) {
          const size_t idx = cv.off + (size_t)i * cv.stride;
          const float t = a.t[idx], x = a.x[idx];
          if (!off_ok || !valid(t, x)) continue;
          const unsigned long long bp = frac64(t, dfK);
          const unsigned long long ph = frac64(t, cv.fmin) + (unsigned long long)J0 * bp - shift0 - lo + g * (bp - Rp);
          const uint64_t fb = __umul64hi(ph, (uint64_t)nbS);
          if (fb < LS)
            atomicAdd(reinterpret_cast<unsigned long long *>(H + fb), (unsigned long long)quantise(x, cv.offset, sc));
        }
        __syncwarp();
        ls = 0;
        for (uint32_t b = b0; b < b1; ++b) ls += H[b];
      }
      long long es = ls;
      int ec = lc;
      for (int o = 1; o < 32; o <<= 1) {
        const long long us = __shfl_up_sync(0xffffffffu, es, o);
        const int uc = __shfl_up_sync(0xffffffffu, ec, o);
        if (lane >= o) { es += us; ec += uc; }
      }
      es -= ls;
      ec -= lc;
      for (uint32_t b = b0; b < b1; ++b) {
        const long long vs = H[b];
        const int vc = C[b];
        H[b] = es;
        C[b] = ec;
        es += vs;
        ec += vc;
      }
    }
    team_sync();
    // the coarse entries as floats and their largest magnitude.  Quantised units: |H| < 2^63 whole numbers,
    // so a square stays below 2^126, and a power that is not zero above 2^-62: nothing leaves the normal
    // range (in real units the threshold of a long curve of 2^-50 flux is subnormal, and a bound
    // multiplied out of it passes over the best window)
    float pm = 0.0f;
    for (int e = 32 * member + lane; e <= iL; e += 32 * W) {
      const float v = __ll2float_rn(H[e * S]);
      P[e] = make_float2(v, (float)C[e * S]);
      pm = fmaxf(pm, fabsf(v));
    }
    pm = team_max(warp_max(pm), team_pm);
    __syncwarp();   // (a team's entries: its barrier)
    // |P - exact| <= 2^-24 |exact| per entry, so a difference is off by at most 2^-23 pmax
    // plus 2^-24 of itself (both taken twice here); den is exact to 2^-24 and the quotient
    // from __fdividef within 2 ulp, inside the 2^-20 factors
    const float e0 = pm * (1.0f / 4194304.0f);
    auto power = [&](int ws, int we, double &pw) -> bool {
      const int kk = C[we] - C[ws];
      if (kk <= kkmi) return false;
      const double den = (double)kk * (N - (double)kk);
      if (!(den > 0.0)) return false;
      const double sv = (double)(H[we] - H[ws]) * unscale;
      pw = sv * sv / den;
      return true;
    };
    auto upper = [&](float2 A, float2 B) -> float {   // 0 where the window does not count
      const float kk = B.y - A.y, den = kk * (Nf - kk);
      const float sv = fabsf(B.x - A.x), hi = sv + (e0 + sv * (1.0f / 4194304.0f));
      return kk > kkmi_f && den > 0.0f ? __fdividef(hi * hi, den) * (1.0f + 1.0f / 1048576.0f) : 0.0f;
    };
    float thr = 0.0f;
    {
      // a lower bound of the largest power: first from the windows around the grid's, then raised by every
      // window whose upper bound reaches it; the rows with such a window are the only ones compared
      // exactly.  One product compared a window instead of a quotient: this stage of 64 curves x 65
      // trials, windows of up to 205 bins, took 150 and takes 90 us.
      auto lower = [&](float2 A, float2 B) -> float {   // 0 where the window does not count
        const float kk = B.y - A.y, den = kk * (Nf - kk);
        const float sv = fabsf(B.x - A.x), low = fmaxf(sv - (e0 + sv * (1.0f / 4194304.0f)), 0.0f);
        return kk > kkmi_f && den > 0.0f ? __fdividef(low * low, den) * (1.0f - 1.0f / 1048576.0f) : 0.0f;
      };
      const int g0 = (int)M, g1 = iL - (int)M;   // the grid's window
      for (int q = lane; q < 9 * 9; q += 32) {
        const int ws = g0 + q / 9 - 4, we = g1 + q % 9 - 4;
        if (ws >= 0 && we <= iL && we - ws > kmi && we - ws <= kma) thr = fmaxf(thr, lower(P[ws], P[we]));
      }
      thr = warp_max(thr);
      for (int s = member; s < iL; s += W) {
        const float2 A = P[s];
        const int wmax = min(kma, iL - s);
        bool hit = false;
#pragma unroll 2
        for (int w = kmi + 1 + lane; w <= wmax; w += 32) {
          const float2 B = P[s + w];
          const float kk = B.y - A.y, den = kk * (Nf - kk);
          const float sv = fabsf(B.x - A.x), hi = sv + (e0 + sv * (1.0f / 4194304.0f));
          if (kk > kkmi_f && den > 0.0f && hi * hi * (1.0f + 1.0f / 524288.0f) >= thr * den) {
            hit = true;
            thr = fmaxf(thr, lower(A, B));
          }
        }
        const bool any = __any_sync(0xffffffffu, hit);
        if (any) thr = warp_max(thr);
        if (lane == 0) R[s] = any ? 1.0f : 0.0f;
      }
      thr = team_max(thr, team_thr);
    }
    __syncwarp();   // (a warp reads its own rows of R)
    double bp = -1.0;
    uint32_t ba = UINT_MAX, bb = UINT_MAX;
    auto trial_best = [&]() {   // fixed-order argmax
      for (int o = 16; o > 0; o >>= 1) {
        const double op = __shfl_xor_sync(0xffffffffu, bp, o);
        const uint32_t oa = __shfl_xor_sync(0xffffffffu, ba, o);
        const uint32_t ob = __shfl_xor_sync(0xffffffffu, bb, o);
        if (better(op, oa, ob, bp, ba, bb)) { bp = op; ba = oa; bb = ob; }
      }
      if (W == 1) return;
      if (lane == 0) { best_p[warp] = bp; best_a[warp] = ba; best_b[warp] = bb; }
      team_sync();
      for (int m = team * W; m < team * W + W; ++m)
        if (better(best_p[m], best_a[m], best_b[m], bp, ba, bb)) { bp = best_p[m]; ba = best_a[m]; bb = best_b[m]; }
    };
    for (int s0 = 0; s0 < iL; s0 += 32) {
      const bool in = s0 + lane < iL && (W == 1 || (s0 + lane) % W == member) && R[s0 + lane] > 0.0f;
      for (unsigned rows = __ballot_sync(0xffffffffu, in); rows; rows &= rows - 1) {
        const int s = s0 + __ffs(rows) - 1;
        const float2 A = P[s];
        const int wmax = min(kma, iL - s);
        for (int w = kmi + 1 + lane; w <= wmax; w += 32) {
          if (upper(A, P[s + w]) < thr) continue;
          const uint32_t ws = s * S, we = (s + w) * S;
          double pw;
          if (power((int)ws, (int)we, pw) && better(pw, ws, we, bp, ba, bb)) { bp = pw; ba = ws; bb = we; }
        }
      }
    }
    trial_best();
    if (ba != UINT_MAX) {
      const uint32_t a0 = ba > S ? ba - S : 0u, a1 = ba + S < LS ? ba + S : LS;
      const uint32_t b0 = bb > S ? bb - S : 0u, b1 = bb + S < LS ? bb + S : LS;
      const uint32_t na = a1 - a0 + 1, nbw = b1 - b0 + 1;
      const uint32_t wmin = a.kmi * S, wmax = a.kma * S;
      // the power in quantised units, within 2^-20 of itself (0 where the window does not count)
      auto approx = [&](uint32_t ws, uint32_t we) -> float {
        if (we <= ws || we - ws <= wmin || we - ws > wmax) return 0.0f;
        const float kk = (float)(C[we] - C[ws]), den = kk * (Nf - kk);
        const float sv = ll_mag(H[we] - H[ws]);
        return kk > kkmi_f && den > 0.0f ? __fdividef(sv * sv, den) : 0.0f;
      };
      float top = 0.0f;
      const uint32_t q0 = 32 * member + lane, dq = 32 * W;
      for (uint32_t q = q0; q < na * nbw; q += dq) top = fmaxf(top, approx(a0 + q / nbw, b0 + q % nbw));
      const float low = team_max(warp_max(top), team_top) * (1.0f - 1.0f / 262144.0f);
      for (uint32_t q = q0; q < na * nbw; q += dq) {
        const uint32_t ws = a0 + q / nbw, we = b0 + q % nbw;
        if (we <= ws || we - ws <= wmin || we - ws > wmax) continue;
        if (approx(ws, we) < low) continue;
        double pw;
        if (power((int)ws, (int)we, pw) && better(pw, ws, we, bp, ba, bb)) { bp = pw; ba = ws; bb = we; }
      }
      trial_best();
    }
    if (lane == 0 && member == 0) {
      Part &o = pt[g];
      o.pw = ba == UINT_MAX ? -1.0 : bp;
      o.s = ba == UINT_MAX ? 0 : H[bb] - H[ba];
      o.kk = ba == UINT_MAX ? 0u : (uint32_t)(C[bb] - C[ba]);
      o.a = ba;
      o.b = bb;
      o.stot = stot;
      o.nv = hd.nv;
      o.j = j;
      o.p1 = (p1 + nb - M) & (nb - 1);  // neighbourhood start bin
      o.sx = sx;
      o.tref = hd.tref;
    }
  }
}

// One warp per curve: the best trial (higher power, then lower k), then the record.
__global__ void __launch_bounds__(128) refine_pick_kernel(const RefArgs a, uint32_t count) {
  const uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= count) return;
  const uint32_t nk = 2 * a.K + 1;
  const Part *pc = a.part + (size_t)c * nk;
  double bp = -1.0;
  uint32_t bk = UINT_MAX;
  for (uint32_t k = lane; k < nk; k += 32) {
    const double p = pc[k].pw;
    if (p > bp) { bp = p; bk = k; }  // ascending k: first maximum of this lane
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double op = __shfl_xor_sync(0xffffffffu, bp, o);
    const uint32_t ok = __shfl_xor_sync(0xffffffffu, bk, o);
    if (op > bp || (op == bp && ok < bk)) { bp = op; bk = ok; }
  }
  if (lane != 0) return;
  const RefCurve cv = curve_of(a, c);
  gtrap_bls_refined r;
  r.jgrid = pc[0].j;
  r.sr_grid = cv.nf ? a.blsp[cv.out + pc[0].j] : 0.0f;
  if (!(bp >= 0.0) || bk == UINT_MAX) {
    r.freq = r.period = r.phase = r.duration = r.t0 = r.depth = r.sr = 0.0;
    r.dk = 0;
    r.kk = 0;
    a.out[c] = r;
    return;
  }
  const Part p = pc[bk];
  const double K = (double)a.K;
  const double dfr = (double)cv.df / K;
  const long long J = (long long)p.j * a.K + ((long long)bk - (long long)a.K);
  const double f = (double)cv.fmin + (double)J * dfr;
  const double dfk = ((double)bk - K) * dfr;                    // trial offset from the grid
  const double nbS = (double)a.nb * (double)a.S;
  // window start in the phase of frac(t f): the neighbourhood's phase plus the t_ref shift
  double ph = (double)p.p1 / (double)a.nb + (double)p.a / nbS + (double)p.tref * dfk;
  ph -= floor(ph);
  const double dur = (double)(p.b - p.a) / nbS;
  double mid = ph + 0.5 * dur;
  const double m = rint((double)p.tref * f - mid);
  const double scale = ldexp(1.0, -p.sx);
  const double s = (double)p.s * scale;
  const double in_mean = p.kk ? s / (double)p.kk : 0.0;
  const double out_mean = p.nv > p.kk ? ((double)(p.stot - p.s) * scale) / (double)(p.nv - p.kk) : 0.0;
  r.freq = f;
  r.period = 1.0 / f;
  r.phase = ph;
  r.duration = dur;
  r.t0 = (m + mid) / f;
  r.depth = out_mean - in_mean;
  r.sr = sqrt(bp);
  r.dk = (int32_t)bk - (int32_t)a.K;
  r.kk = p.kk;
  a.out[c] = r;
}

int refine_common(RefArgs &a, uint32_t count, void *workspace, size_t workspace_bytes,
                  cudaStream_t stream, const char *name) {
  if (count == 0) return GTRAP_OK;
  if (!a.blsp || !a.ph1 || !a.ph2 || !a.t || !a.x || !a.out)
    return fail(GTRAP_ERR_INVALID_ARG, "%s: null pointer", name);
  if (!gtrap::is_pow2(a.nb) || a.nb < 2 || a.nb > 8192)
    return fail(GTRAP_ERR_INVALID_ARG, "%s: nb=%u must be a power of two in [2, 8192]", name, a.nb);
  if (a.kma == 0 || a.kma > a.nb) return fail(GTRAP_ERR_INVALID_ARG, "%s: kma=%u must be in [1, nb]", name, a.kma);
  if (!gtrap::is_pow2(a.K) || a.K > 1024) return fail(GTRAP_ERR_INVALID_ARG, "%s: K=%u must be a power of two <= 1024", name, a.K);
  if (a.S == 0 || a.S > 64) return fail(GTRAP_ERR_INVALID_ARG, "%s: S=%u must be in [1, 64]", name, a.S);
  if (a.M > 64) return fail(GTRAP_ERR_INVALID_ARG, "%s: M=%u must be at most 64", name, a.M);
  if ((uint64_t)(a.kma + 2 * a.M) * a.S > (uint64_t)kMaxFine)
    return fail(GTRAP_ERR_INVALID_ARG, "%s: (kma + 2M) * S = %u exceeds %d fine bins", name,
                (a.kma + 2 * a.M) * a.S, kMaxFine);
  const size_t parts = gtrap::align256((size_t)count * (2 * (size_t)a.K + 1) * sizeof(Part));
  const size_t need = parts + (size_t)count * sizeof(Head);
  if (!workspace || ((uintptr_t)workspace & 255) || workspace_bytes < need)
    return fail(GTRAP_ERR_WORKSPACE, "%s: workspace of %zu bytes (256-byte aligned) needed", name, need);
  if (count > 65535u * 4u) return fail(GTRAP_ERR_INVALID_ARG, "%s: at most %u curves per call", name, 65535u * 4u);
  // more than kmi bins and at most kma: no window from kma on, and the kernels index from kmi as an int
  a.kmi = a.kmi < 1 ? 1 : a.kmi < a.kma ? a.kmi : a.kma;
  a.lognb = gtrap::ilog2u(a.nb);
  a.logK = gtrap::ilog2u(a.K);
  a.part = reinterpret_cast<Part *>(workspace);
  a.head = reinterpret_cast<Head *>((char *)workspace + parts);
  // trials per block: chosen on the device by the neighbourhood's size, within a block's budget; two
  // blocks an SM's worth of groups where there are few curves
  const uint32_t nk = 2 * a.K + 1, widest = a.kma + 2 * a.M;
  const size_t worst = trial_bytes(widest, widest * a.S);
  const size_t smem = worst > kSmemBudget ? worst : kSmemBudget;
  a.smem = (uint32_t)smem;
  const uint32_t want = ((uint32_t)gtrap::sm_count() * 2 + count - 1) / count;
  a.min_groups = want > nk ? nk : want;
  uint32_t fit = (uint32_t)(smem / worst);
  if (fit > (uint32_t)kMaxGroup) fit = kMaxGroup;
  const uint32_t groups = (nk + fit - 1) / fit > a.min_groups ? (nk + fit - 1) / fit : a.min_groups;
  GTRAP_TRY(gtrap::ensure_smem((const void *)refine_trial_kernel, smem, name));
  refine_head_kernel<<<count, kHeadThreads, 0, stream>>>(a);
  GTRAP_TRY(gtrap::check_launch("refine_head_kernel"));
  refine_trial_kernel<<<dim3(count, groups), kThreads, smem, stream>>>(a);
  GTRAP_TRY(gtrap::check_launch("refine_trial_kernel"));
  refine_pick_kernel<<<(count + 3) / 4, 128, 0, stream>>>(a, count);
  return gtrap::check_launch("refine_pick_kernel");
}

}  // namespace

extern "C" {

size_t gtrap_bls_refine_workspace_size(uint32_t ncurves, uint32_t K) {
  return gtrap::align256((size_t)ncurves * (2 * (size_t)K + 1) * sizeof(Part)) +
         gtrap::align256((size_t)ncurves * sizeof(Head)) + 256;
}

int gtrap_bls_refine(const float *blsp, const uint32_t *phase1, const uint32_t *phase2, const float *lc,
                     const float *tu, const float *offset, const uint32_t *ntrue, uint32_t n, uint32_t nq,
                     uint32_t nf, uint32_t nb, uint32_t kma, uint32_t kmi, uint32_t kkmi, float fmin,
                     float df, uint32_t K, uint32_t S, uint32_t M, gtrap_bls_refined *out, void *workspace,
                     size_t workspace_bytes, gtrap_stream_t stream) {
  if (nq == 0 || nf == 0) return GTRAP_OK;
  if (!offset || !ntrue) return fail(GTRAP_ERR_INVALID_ARG, "bls_refine: offset and ntrue are required");
  if (n == 0 || n >= (1u << 23)) return fail(GTRAP_ERR_INVALID_ARG, "bls_refine: n=%u must be in [1, 2^23)", n);
  RefArgs a = {};
  a.blsp = blsp; a.ph1 = phase1; a.ph2 = phase2; a.t = tu; a.x = lc;
  a.offset = offset; a.ntrue = ntrue;
  a.n = n; a.nq = nq; a.nf = nf; a.kkmi = kkmi; a.fmin = fmin; a.df = df;
  a.nb = nb; a.kma = kma; a.kmi = kmi; a.K = K; a.S = S; a.M = M;
  a.out = out;
  return refine_common(a, nq, workspace, workspace_bytes, stream, "bls_refine");
}

int gtrap_bls_refine_packed(const float *blsp, const uint32_t *phase1, const uint32_t *phase2,
                            const gtrap_bls_curve *curves, const uint32_t *sel, uint32_t count,
                            const float *t, const float *x, uint32_t nb, uint32_t kma, uint32_t kmi,
                            uint32_t K, uint32_t S, uint32_t M, gtrap_bls_refined *out, void *workspace,
                            size_t workspace_bytes, gtrap_stream_t stream) {
  if (count == 0) return GTRAP_OK;
  if (!curves) return fail(GTRAP_ERR_INVALID_ARG, "bls_refine_packed: null pointer");
  RefArgs a = {};
  a.blsp = blsp; a.ph1 = phase1; a.ph2 = phase2; a.t = t; a.x = x;
  a.curves = curves; a.sel = sel;
  a.nb = nb; a.kma = kma; a.kmi = kmi; a.K = K; a.S = S; a.M = M;
  a.out = out;
  return refine_common(a, count, workspace, workspace_bytes, stream, "bls_refine_packed");
}

}  // extern "C"
