// Running medians of a group of T consecutive windows by one thread, in registers.
//
// The windows of T consecutive rows (2r + 1 rows each, r = T A + B with 0 <= B < T) share a core
// of 2r + 2 - T rows; window k adds the last T - 1 - k of the T - 1 rows before the core (left
// extras) and the first k of the T - 1 rows behind it (right extras).  As T - 1 rows enter, the
// median of each window is one of the T middle values of the core (ranks r - T + 1 .. r).
//   * The core is 2A - 1 whole aligned blocks of T rows and B + 1 rows of the blocks on either
//     side (padded with -inf on the left and +inf on the right, equally many, which keeps the
//     middle where it is): each is sorted by a network and they are merged, keeping only the
//     values that can still be in the middle.
//   * Then the group is halved: each half's core takes T / 2 more rows (sorted), and the middle
//     T / 2 of the 3T / 2 values stay, until one value is left for each window: its median.
// Every step is a compare-exchange of registers, whatever the values: no shared memory, no
// divergence, no dependence on how far a value travels.  The result is the order statistic
// itself, so it equals a sorted window's to the bit.  Floats must not be NaN (the caller checks); keys may
// be anything.
#pragma once

#include <climits>
#include <type_traits>

namespace gtrap {

// The networks sort floats, or integer keys in the order of the floats: -0 below +0, NaN past the infinity
// of its sign.  INT_MAX and INT_MIN stay free for guards.
__device__ __forceinline__ int median_key(float v) {
  const int b = __float_as_int(v);
  return max(min(b ^ ((b >> 31) & 0x7fffffff), INT_MAX - 1), INT_MIN + 1);
}
__device__ __forceinline__ float median_value(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

__device__ __forceinline__ float lesser(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float greater(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ int lesser(int a, int b) { return min(a, b); }
__device__ __forceinline__ int greater(int a, int b) { return max(a, b); }

template <class V>
__device__ __forceinline__ void cx(V &a, V &b) {
  const V lo = lesser(a, b), hi = greater(a, b);
  a = lo;
  b = hi;
}

// Batcher's odd-even merge sort of v[0 .. N), N a power of two.
template <int N, class V>
__device__ __forceinline__ void net_sort(V (&v)[N]) {
#pragma unroll
  for (int p = 1; p < N; p *= 2) {
#pragma unroll
    for (int k = p; k >= 1; k /= 2) {
#pragma unroll
      for (int j = k % p; j + k < N; j += 2 * k) {
#pragma unroll
        for (int i = 0; i < k; ++i)
          if (i + j + k < N && (i + j) / (2 * p) == (i + j + k) / (2 * p)) cx(v[i + j], v[i + j + k]);
      }
    }
  }
}

// A bitonic sequence into ascending order.
template <int N, class V>
__device__ __forceinline__ void net_clean(V (&v)[N]) {
#pragma unroll
  for (int s = N / 2; s >= 1; s /= 2) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (!(i & s)) cx(v[i], v[i + s]);
  }
}

// Two ascending sequences of N into one of 2N.
template <int N, class V>
__device__ __forceinline__ void net_merge(const V (&a)[N], const V (&b)[N], V (&out)[2 * N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    out[i] = a[i];
    out[2 * N - 1 - i] = b[i];
  }
  net_clean(out);
}

// The middle H of the 3H values of a (2H, ascending) and b (H, ascending), ascending: the H
// smallest are among a's lower half and b, the H largest of the rest among what is left of those
// and a's upper half.
template <int H, class V>
__device__ __forceinline__ void net_middle(const V (&a)[2 * H], const V (&b)[H], V (&out)[H]) {
  V x[H];
#pragma unroll
  for (int i = 0; i < H; ++i) x[i] = greater(a[i], b[H - 1 - i]);
  net_clean(x);
#pragma unroll
  for (int i = 0; i < H; ++i) out[i] = lesser(x[i], a[2 * H - 1 - i]);
  net_clean(out);
}

// The middle N of two ascending sequences of N, ascending (the N / 2 smallest and the N / 2
// largest left out).
template <int N, class V>
__device__ __forceinline__ void net_middle_of_two(const V (&a)[N], const V (&b)[N], V (&out)[N]) {
  V lo[N], hi[N];   // the N smallest and the N largest, each bitonic
#pragma unroll
  for (int i = 0; i < N; ++i) {
    lo[i] = lesser(a[i], b[N - 1 - i]);
    hi[i] = greater(a[i], b[N - 1 - i]);
  }
  V u[N / 2], w[N / 2];   // the upper half of the low ones, the lower half of the high ones
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    u[i] = greater(lo[i], lo[i + N / 2]);
    w[i] = lesser(hi[i], hi[i + N / 2]);
  }
  net_clean(u);
  net_clean(w);
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    out[i] = u[i];
    out[i + N / 2] = w[i];
  }
}

// The medians of windows K0 .. K0 + T - 1 of a group of T0 from the T middle values of their
// common core.  left[j] (j = 1 .. T0 - 1): the row that windows 0 .. j - 1 hold; right[j]
// (j = 0 .. T0 - 2): the row that windows j + 1 .. T0 - 1 hold.
template <int T0, int T, int K0, class V>
__device__ __forceinline__ void median_halves(const V (&core)[T], const V (&left)[T0], const V (&right)[T0],
                                              V (&med)[T0]) {
  if constexpr (T == 1) {
    med[K0] = core[0];
  } else {
    constexpr int H = T / 2;
    V e[H], mid[H];
#pragma unroll
    for (int i = 0; i < H; ++i) e[i] = left[K0 + H + i];
    net_sort(e);
    net_middle<H>(core, e, mid);
    median_halves<T0, H, K0>(mid, left, right, med);
#pragma unroll
    for (int i = 0; i < H; ++i) e[i] = right[K0 + i];
    net_sort(e);
    net_middle<H>(core, e, mid);
    median_halves<T0, H, K0 + H>(mid, left, right, med);
  }
}

// Medians of the windows of rows 0 .. T - 1 (relative to the group), r = T A + B.
// row(k): the value (V float) or key (V int) of row k, -r <= k <= T - 1 + r.  `bad` becomes NaN if a float
// is not finite (with a NaN among them the medians are not to be used).
template <int T, int A, class V, class Row>
__device__ __forceinline__ void group_medians(int B, Row row, V (&med)[T], float &bad) {
  static_assert(A >= 1 && A <= 3, "cores of one to five whole blocks");
  constexpr bool kFloat = std::is_same<V, float>::value;
  V least, most;
  if constexpr (kFloat) { least = -INFINITY; most = INFINITY; }
  else { least = INT_MIN; most = INT_MAX; }
  auto check = [&](V v) {
    if constexpr (kFloat) bad = fmaf(v, 0.0f, bad);
  };
  auto block = [&](int at, V (&v)[T]) {
#pragma unroll
    for (int i = 0; i < T; ++i) {
      v[i] = row(at + i);
      check(v[i]);
    }
    net_sort(v);
  };
  V core[T];
  {
    V edge[2 * T];   // the rows on either side of the whole blocks
    {
      V s[T], p[T];
#pragma unroll
      for (int i = 0; i < T; ++i) {
        const bool in = i <= B;
        s[i] = in ? row(-T * A + T - 1 - i) : least;
        p[i] = in ? row(T * A + i) : most;
        check(in ? s[i] : V(0));
        check(in ? p[i] : V(0));
      }
      net_sort(s);
      net_sort(p);
      net_merge(s, p, edge);
    }
    V b0[T];
    if constexpr (A == 1) {
      block(0, b0);
      net_middle<T>(edge, b0, core);
    } else {
      V pair[2 * T], c[T];
      block(-T, b0);
      block(T, c);
      net_merge(b0, c, pair);
      if constexpr (A == 2) {   // edge + pair + one block: the middle 2T of the first 4T stay
        V m[2 * T];
        net_middle_of_two<2 * T>(edge, pair, m);
        block(0, b0);
        net_middle<T>(m, b0, core);
      } else {                  // edge + two pairs + one block
        V all[4 * T], m[2 * T];
        net_merge(edge, pair, all);
        block(-2 * T, b0);
        block(2 * T, c);
        net_merge(b0, c, pair);
        net_middle<2 * T>(all, pair, m);
        block(0, b0);
        net_middle<T>(m, b0, core);
      }
    }
  }
  V left[T], right[T];
  const int r = T * A + B;
  left[0] = right[T - 1] = V(0);   // not used
#pragma unroll
  for (int j = 1; j < T; ++j) {
    left[j] = row(j - 1 - r);
    right[j - 1] = row(r + j);
    check(left[j]);
    check(right[j - 1]);
  }
  median_halves<T, T, 0>(core, left, right, med);
}

}  // namespace gtrap
