// Median-filter detrend (gfilter) and per-curve offset (get_offset).
//
// Reference behaviour: gtrap/gfilter.py:13-86 computes, for every sample, the exact
// (r+1)-th order statistic of the zero-padded window x[i-r .. i+r] by bisection over
// the window values and writes x[i] - median.
//
// Radii 4 .. 63 (every survey detrend): one thread takes a group of 4, 8 or 16 consecutive rows
// of a curve and finds their medians in registers (medgroup.cuh).  Image: consecutive threads
// take consecutive curves of a row group, so a row's loads are coalesced whatever nq.  Packed
// curves: a block stages its rows in shared memory (padded by one word a group: no conflicts)
// and writes its residuals back through it.  About 72 min / max instructions a sample at r = 24
// (issued at half rate) and as many others, whatever the values; before, each lane of a warp slid
// a sorted window of its own by dependent shared-memory moves.  Before / now, r = 24:
// 65,536 x 128 479 / 81 us, 65,536 x 8 207 / 16 us, 3001 x 1 98 / 17 us (launch rate), 160 packed
// curves of 3.5 M samples 462 / 47 us, one of 19,254 69 / 10 us; r = 5 119 / 47, r = 63 2421 / 153
// us on 65,536 x 128.
//
// Radii of 64 and more, as far as their cores fit in shared memory (r <= 888 with 227 KB): groups of
// 16 rows whose common core is kept sorted in shared memory and moves by merging (gfilter_merge.cu).
//
// Other radii: every warp owns 32 adjacent curves (one per lane, so each row it touches is one
// coalesced 128-byte line of the [n, nq] image) and a run of consecutive rows.  Each lane keeps
// its window sorted in shared memory, laid out [rank][lane] so that every access is
// bank-conflict free, and slides it one row at a time: the leaving value is located by binary
// search and the entering value is moved into place by shifting the values between the two.
// The median is then the element of rank r.  Work per output is O(displacement) instead of
// O(window * bisection steps), but each step waits on the one before.
//
// Either way the result is the same order statistic, so the residual is bit-identical to the
// reference's and to scipy.signal.medfilt.
#include "common.cuh"

#include <cooperative_groups.h>

#include "medwindow.cuh"

namespace {

using gtrap::window_slide;
using gtrap::window_sort;

__device__ __forceinline__ float load_padded(const float *__restrict__ in, long long i, long long n,
                                             size_t nq, int q, bool qok) {
  return (qok && i >= 0 && i < n) ? __ldg(in + (size_t)i * nq + q) : 0.0f;
}

__global__ void __launch_bounds__(256) gfilter_kernel(const float *__restrict__ in,
                                                      float *__restrict__ out, int n, int nq,
                                                      int r, int rows_per_warp) {
  extern __shared__ float sorted_windows[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int w = 2 * r + 1;
  float *S = sorted_windows + (size_t)warp * w * 32 + lane;  // rank k lives at S[32 * k]
  const int q = blockIdx.x * 32 + lane;
  const bool qok = q < nq;
  const long long row0 = ((long long)blockIdx.y * (blockDim.x >> 5) + warp) * rows_per_warp;
  if (row0 >= n) return;
  const long long row1 = min((long long)n, row0 + rows_per_warp);
  const size_t stride = (size_t)nq;

  // Sorted window of the first output row (insertion sort; amortised over the run).  The
  // window's values are loaded first, all loads in flight together, then sorted in place.
  for (int k = 0; k < w; ++k) S[32 * k] = load_padded(in, row0 - r + k, n, stride, q, qok);
  window_sort(S, w, true);

  // each row's three loads are issued one row ahead, under the previous row's window update
  float xi = qok ? __ldg(in + (size_t)row0 * stride + q) : 0.0f;
  float vold = load_padded(in, row0 - r, n, stride, q, qok);
  float vnew = load_padded(in, row0 + r + 1, n, stride, q, qok);
  for (long long i = row0; i < row1; ++i) {
    const bool more = i + 1 < row1;
    const float xn = (qok && more) ? __ldg(in + (size_t)(i + 1) * stride + q) : 0.0f;
    const float von = more ? load_padded(in, i + 1 - r, n, stride, q, qok) : 0.0f;
    const float vnn = more ? load_padded(in, i + r + 2, n, stride, q, qok) : 0.0f;
    const float med = S[32 * r];
    if (qok) out[(size_t)i * stride + q] = __fsub_rn(xi, med);
    if (!more) break;
    const float vo = vold, vn = vnew;
    xi = xn; vold = von; vnew = vnn;
    if (vn == vo) continue;
    window_slide(S, w, vo, vn, true);
  }
}

// Packed curves (curve q = samples [off[q], off[q] + len[q]) of a flat array): each lane
// filters a run of `run` consecutive rows of one curve with its own sorted window, as above.
__global__ void __launch_bounds__(256) gfilter_packed_kernel(const float *__restrict__ in,
                                                             float *__restrict__ out,
                                                             const unsigned long long *__restrict__ offs,
                                                             const uint32_t *__restrict__ lens,
                                                             unsigned ncurves, int r, int run) {
  extern __shared__ float sorted_windows[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int w = 2 * r + 1;
  float *S = sorted_windows + (size_t)warp * w * 32 + lane;
  for (unsigned q = blockIdx.y; q < ncurves; q += gridDim.y) {
    const unsigned long long off = offs[q];
    const long long n = (long long)lens[q];
    const float *x = in + off;
    float *y = out + off;
    const long long row0 = ((long long)(blockIdx.x * (blockDim.x >> 5) + warp) * 32 + lane) * run;
    if (row0 >= n) continue;
    const long long row1 = min(n, row0 + run);
    auto ld = [&](long long i) -> float { return (i >= 0 && i < n) ? __ldg(x + i) : 0.0f; };
    // the window's values loaded first (all in flight together), then sorted in place
    bool nan_seen = false;
    for (int k = 0; k < w; ++k) {
      const float v = ld(row0 - r + k);
      nan_seen |= isnan(v);
      S[32 * k] = v;
    }
    window_sort(S, w, nan_seen);
    // each row's three loads are issued one row ahead, under the previous row's update
    float xi = __ldg(x + row0), vold = ld(row0 - r), vnew = ld(row0 + r + 1);
    for (long long i = row0; i < row1; ++i) {
      const bool more = i + 1 < row1;
      const float xn = more ? __ldg(x + i + 1) : 0.0f;
      const float von = more ? ld(i + 1 - r) : 0.0f;
      const float vnn = more ? ld(i + r + 2) : 0.0f;
      y[i] = __fsub_rn(xi, S[32 * r]);
      if (!more) break;
      const float vo = vold, vn = vnew;
      xi = xn; vold = von; vnew = vnn;
      if (vn == vo) continue;
      nan_seen |= isnan(vn);
      window_slide(S, w, vo, vn, nan_seen);
    }
  }
}

// offset[q] = sum of resid over samples whose time is not negative, divided by n.
// The summation order (shared with the packed batches' bls_ragged_offset_kernel, so a curve
// gets the same offset to the bit in an image and in a packed batch): kOffParts = 256
// partials, partial p summing the samples i = p mod 256 in order with Neumaier compensation;
// each partial rounded to double as sum + compensation; s_r = the partials r, r + 32, ...,
// r + 224 added in that order, and the offset = s_0 + s_1 + ... + s_31 in that order, divided
// by n.  A partial is a chain of dependent additions behind strided loads, so the kernel is
// bound by latency, not by bandwidth: what counts is how many chains run at once and how many
// loads each has in flight.  A cluster of kOffRanks = 8 blocks takes blockDim.x curves (up to
// 16: full sectors of a row, and twice the blocks of 32): thread (row, lane) of block u owns the
// one partial row + 32u with kOffAhead loads in flight, and block 0 adds the partials out of
// the cluster's shared memory in the order above.  The form before, one block of 32 lanes a
// group with eight partials a thread, left most SMs idle and all but nq lanes of a small image.
// Before / now (n x nq): 65,536 x 128 396 / 28 us, 65,536 x 1 269 / 22 us, 18,000 x 1024
// 194 / 45 us, 3001 x 1 26.5 / 17.7 us (launches back to back).
constexpr int kOffParts = 256;
constexpr int kOffRanks = kOffParts / 32;
constexpr int kOffLanes = 16;
constexpr int kOffAhead = 16;

__global__ void __cluster_dims__(1, kOffRanks, 1) __launch_bounds__(32 * kOffLanes)
offset_kernel(const float *__restrict__ resid, const float *__restrict__ tu,
              float *__restrict__ offset, int n, int nq) {
  namespace cg = cooperative_groups;
  __shared__ double part[32][kOffLanes + 1];
  __shared__ double acc[32][kOffLanes + 1];
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x, row = threadIdx.y;
  const int q = blockIdx.x * blockDim.x + lane;
  part[row][lane] = gtrap::offset_partial<kOffAhead>(tu + q, resid + q, row + 32 * (int)blockIdx.y, kOffParts, n, nq,
                                                     q < nq);
  cluster.sync();
  if (blockIdx.y == 0) {  // the cluster's rank 0: the grid has kOffRanks blocks along y
    double sr = 0.0;
#pragma unroll
    for (int u = 0; u < kOffRanks; ++u) sr += cluster.map_shared_rank(&part[0][0], u)[row * (kOffLanes + 1) + lane];
    acc[row][lane] = sr;
    __syncthreads();
    if (row == 0 && q < nq) {
      double s = 0.0;
      for (int k = 0; k < 32; ++k) s += acc[k][lane];
      offset[q] = (float)(s / (double)n);
    }
  }
  cluster.sync();  // the other blocks' shared memory stays until rank 0 has read it
}

// The same sums of many short curves, where the threads of a cluster would have a few samples each and the
// clusters' start is what takes the time: one block a group of curves, thread (row, lane) taking the partials row,
// row + 32, ... one after the other.  For more clusters than two blocks an SM and up to kOffShort samples;
// cluster / this (n x nq): 100 x 10,000 95 / 21 us, 1000 x 1000 17 / 11, 4000 x 1000 17 / 17, 4000 x 10,000
// 119 / 76; past it 10,000 x 10,000 196 / 213, and with fewer curves 1000 x 300 8 / 11.
constexpr int kOffShort = 4096;

__global__ void __launch_bounds__(32 * kOffLanes)
offset_short_kernel(const float *__restrict__ resid, const float *__restrict__ tu,
                    float *__restrict__ offset, int n, int nq) {
  __shared__ double acc[32][kOffLanes + 1];
  const int lane = threadIdx.x, row = threadIdx.y;
  const int q = blockIdx.x * blockDim.x + lane;
  double sr = 0.0;   // (a partial without samples is zero: left out)
  for (int p = 0; p < kOffParts && p < n; p += 32)
    sr += gtrap::offset_partial<2>(tu + q, resid + q, p + row, kOffParts, n, nq, q < nq);
  acc[row][lane] = sr;
  __syncthreads();
  if (row == 0 && q < nq) {
    double s = 0.0;
    for (int k = 0; k < 32; ++k) s += acc[k][lane];
    offset[q] = (float)(s / (double)n);
  }
}

}  // namespace

extern "C" {

int gtrap_gfilter(const float *in, float *out, uint32_t n, uint32_t nq, uint32_t r,
                  gtrap_stream_t stream) {
  using namespace gtrap;
  if (n == 0 || nq == 0) return GTRAP_OK;
  if (!in || !out) return fail(GTRAP_ERR_INVALID_ARG, "gfilter: null pointer");
  if (in == out) return fail(GTRAP_ERR_INVALID_ARG, "gfilter: in and out must not alias");
  if (n > 0x7fffffffu || nq > 0x7fffffffu)
    return fail(GTRAP_ERR_INVALID_ARG, "gfilter: n and nq must be below 2^31");
  if (r >= kGroupMinR && r <= kGroupMaxR) return gfilter_groups_image(in, out, n, nq, r, stream);
  if (r > kGroupMaxR && gfilter_merge_smem(r) <= (size_t)max_smem_optin())
    return gfilter_merge(in, out, nullptr, nullptr, nq, n, r, stream);
  const size_t w = 2 * (size_t)r + 1;
  const size_t per_warp = w * 32 * sizeof(float);
  const size_t budget = (size_t)max_smem_optin();
  if (per_warp > budget)
    return fail(GTRAP_ERR_INVALID_ARG, "gfilter: r=%u needs %zu bytes of shared memory per warp",
                r, per_warp);
  int warps = (int)(budget / per_warp);
  if (warps > 8) warps = 8;
  // Smaller windows afford more resident blocks: keep a block's share near 1/4 SM.
  while (warps > 1 && per_warp * warps > 56 * 1024) --warps;
  long long rows_per_warp = 8 * (long long)w;
  if (rows_per_warp < 256) rows_per_warp = 256;
  if (rows_per_warp > 4096) rows_per_warp = 4096;
  // Keep enough warps for the GPU when there are few curve groups.
  const long long groups = (nq + 31) / 32;
  const long long want_warps = 8LL * sm_count() * 8;
  while (rows_per_warp > 64 && groups * ((n + rows_per_warp - 1) / rows_per_warp) < want_warps)
    rows_per_warp /= 2;
  const long long rows_per_block = rows_per_warp * warps;
  const long long gy = (n + rows_per_block - 1) / rows_per_block;
  if (gy > 65535) rows_per_warp = (n + 65535LL * warps - 1) / (65535LL * warps);
  const long long gy2 = (n + rows_per_warp * warps - 1) / (rows_per_warp * warps);
  const size_t smem = per_warp * warps;
  GTRAP_TRY(ensure_smem((const void *)gfilter_kernel, smem, "gfilter"));
  dim3 grid((unsigned)groups, (unsigned)gy2);
  gfilter_kernel<<<grid, 32 * warps, smem, stream>>>(in, out, (int)n, (int)nq, (int)r,
                                                     (int)rows_per_warp);
  return check_launch("gfilter_kernel");
}

int gtrap_gfilter_packed(const float *in, float *out, const uint64_t *off, const uint32_t *n,
                         uint32_t ncurves, uint32_t max_n, uint32_t r, gtrap_stream_t stream) {
  using namespace gtrap;
  if (ncurves == 0 || max_n == 0) return GTRAP_OK;
  if (!in || !out || !off || !n) return fail(GTRAP_ERR_INVALID_ARG, "gfilter_packed: null pointer");
  if (in == out) return fail(GTRAP_ERR_INVALID_ARG, "gfilter_packed: in and out must not alias");
  if (r >= kGroupMinR && r <= kGroupMaxR)
    return gfilter_groups_packed(in, out, (const unsigned long long *)off, n, ncurves, max_n, r, stream);
  if (r > kGroupMaxR && gfilter_merge_smem(r) <= (size_t)max_smem_optin())
    return gfilter_merge(in, out, (const unsigned long long *)off, n, ncurves, max_n, r, stream);
  const size_t w = 2 * (size_t)r + 1;
  const size_t per_warp = w * 32 * sizeof(float);
  const size_t budget = (size_t)max_smem_optin();
  if (per_warp > budget)
    return fail(GTRAP_ERR_INVALID_ARG, "gfilter_packed: r=%u needs %zu bytes of shared memory per warp", r, per_warp);
  int warps = (int)(budget / per_warp);
  if (warps > 8) warps = 8;
  while (warps > 1 && per_warp * warps > 56 * 1024) --warps;
  // rows per lane: long runs amortise each lane's initial sort (about w^2 / 4 steps) over a
  // big batch; a few curves (a served step) get short runs so that their rows still spread
  // over many lanes (a run costs about its length in dependent row updates)
  const size_t rows = (size_t)max_n * ncurves;  // upper bound of the batch's rows
  // rows is an upper bound (the longest curve times the count), so aim at 512 lanes an SM
  const size_t lanes_wanted = (size_t)sm_count() * 512;
  size_t run_fill = (rows + lanes_wanted - 1) / lanes_wanted;
  int run = (int)(8 * w);
  if (run < 64) run = 64;
  if (run > 1024) run = 1024;
  if (run_fill < (size_t)run) run = run_fill < 16 ? 16 : (int)run_fill;
  const size_t rows_per_block = (size_t)run * 32 * warps;
  const unsigned gx = (unsigned)((max_n + rows_per_block - 1) / rows_per_block);
  const unsigned gy = ncurves < 65535 ? ncurves : 65535;
  const size_t smem = per_warp * warps;
  GTRAP_TRY(ensure_smem((const void *)gfilter_packed_kernel, smem, "gfilter_packed"));
  gfilter_packed_kernel<<<dim3(gx, gy), 32 * warps, smem, stream>>>(
      in, out, (const unsigned long long *)off, n, ncurves, (int)r, run);
  return check_launch("gfilter_packed_kernel");
}

int gtrap_offset(const float *resid, const float *tu, float *offset, uint32_t n, uint32_t nq,
                 gtrap_stream_t stream) {
  using namespace gtrap;
  if (nq == 0) return GTRAP_OK;
  if (!resid || !tu || !offset) return fail(GTRAP_ERR_INVALID_ARG, "offset: null pointer");
  if (n == 0) return fail(GTRAP_ERR_INVALID_ARG, "offset: n must be positive");
  if (n > 0x7fffffffu || nq > 0x7fffffffu)
    return fail(GTRAP_ERR_INVALID_ARG, "offset: n and nq must be below 2^31");
  unsigned lanes = 1;
  while (lanes < (unsigned)kOffLanes && lanes < nq) lanes *= 2;
  const unsigned groups = (nq + lanes - 1) / lanes;
  if (n <= (uint32_t)kOffShort && groups * kOffRanks > 2u * sm_count()) {
    offset_short_kernel<<<groups, dim3(lanes, 32), 0, stream>>>(resid, tu, offset, (int)n, (int)nq);
    return check_launch("offset_short_kernel");
  }
  offset_kernel<<<dim3(groups, kOffRanks), dim3(lanes, 32), 0, stream>>>(resid, tu, offset, (int)n, (int)nq);
  return check_launch("offset_kernel");
}

}  // extern "C"
