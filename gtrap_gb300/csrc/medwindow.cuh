// A running median's window kept sorted, one element at a time: the insertion sort that fills it
// and the slide by one row.
#pragma once

#include <cuda_runtime.h>

namespace gtrap {

// The window S[ST * k], k < w, of one lane (ST = 32: [rank][lane] in shared memory; 1: a thread's
// own array).  Both functions give the
// element-by-element result of an insertion sort / slide, which keeps equal values in their
// order.  With `linear` false the window must be sorted (it has never held a NaN): each
// insertion point is then found by binary search and the elements between move as a block
// (loads before stores, not one dependent compare per element), which is faster where a lane
// waits on its own chain (the packed detrend: 5.2 -> 3.3 ms on 2000 uneven curves, a lone
// 10,069-sample curve 0.112 -> 0.075 ms).  With `linear` true the element-by-element loops
// run: their cost follows the displacement, which wins where many warps share an SM and the
// windows are nearly sorted (the image detrend of 128 Kepler-like curves: 0.53 ms against
// 0.89 ms with binary searches), and they are the order with NaN, which is what it is.

// Moves S[lo..hi) up by one slot (to S[lo+1..hi]).
template <int ST = 32>
__device__ __forceinline__ void window_move_up(float *S, int lo, int hi) {
  int j = hi;
  for (; j - 4 >= lo; j -= 4) {
    const float a0 = S[ST * (j - 1)], a1 = S[ST * (j - 2)], a2 = S[ST * (j - 3)], a3 = S[ST * (j - 4)];
    S[ST * j] = a0; S[ST * (j - 1)] = a1; S[ST * (j - 2)] = a2; S[ST * (j - 3)] = a3;
  }
  for (; j > lo; --j) S[ST * j] = S[ST * (j - 1)];
}

// Moves S(lo..hi] down by one slot (to S[lo..hi)).
template <int ST = 32>
__device__ __forceinline__ void window_move_down(float *S, int lo, int hi) {
  int j = lo;
  for (; j + 4 <= hi; j += 4) {
    const float a0 = S[ST * (j + 1)], a1 = S[ST * (j + 2)], a2 = S[ST * (j + 3)], a3 = S[ST * (j + 4)];
    S[ST * j] = a0; S[ST * (j + 1)] = a1; S[ST * (j + 2)] = a2; S[ST * (j + 3)] = a3;
  }
  for (; j < hi; ++j) S[ST * j] = S[ST * (j + 1)];
}

// Sorts the loaded window in place (stable insertion sort).
template <int ST = 32>
__device__ __forceinline__ void window_sort(float *S, int w, bool linear) {
  for (int k = 1; k < w; ++k) {
    const float v = S[ST * k];
    if (!linear) {
      int lo = 0, hi = k;  // the insertion point: the number of elements <= v
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (S[ST * mid] <= v) lo = mid + 1; else hi = mid;
      }
      window_move_up<ST>(S, lo, k);
      S[ST * lo] = v;
    } else {
      int j = k;
      while (j > 0) {
        const float u = S[ST * (j - 1)];
        if (u <= v) break;
        S[ST * j] = u;
        --j;
      }
      S[ST * j] = v;
    }
  }
}

// Slides the window by one row: vold leaves, vnew (!= vold) enters.
template <int ST = 32>
__device__ __forceinline__ void window_slide(float *S, int w, float vold, float vnew, bool linear) {
  // lowest rank holding the leaving value (present in the window by construction)
  int lo = 0, hi = w - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (S[ST * mid] < vold) lo = mid + 1; else hi = mid;
  }
  int j = lo;
  if (!linear) {
    if (vnew > vold) {  // vnew lands before the first element >= vnew above the freed slot
      int a = j + 1, b = w;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (S[ST * mid] < vnew) a = mid + 1; else b = mid;
      }
      window_move_down<ST>(S, j, a - 1);
      S[ST * (a - 1)] = vnew;
    } else {            // vnew lands after the last element <= vnew below the freed slot
      int a = 0, b = j;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (S[ST * mid] <= vnew) a = mid + 1; else b = mid;
      }
      window_move_up<ST>(S, a, j);
      S[ST * a] = vnew;
    }
    return;
  }
  if (vnew > vold) {
    while (j + 1 < w) {
      const float u = S[ST * (j + 1)];
      if (!(u < vnew)) break;
      S[ST * j] = u;
      ++j;
    }
  } else {
    while (j > 0) {
      const float u = S[ST * (j - 1)];
      if (!(u > vnew)) break;
      S[ST * j] = u;
      --j;
    }
  }
  S[ST * j] = vnew;
}

}  // namespace gtrap
