// A running median's window kept sorted, one element at a time: the insertion sort that fills it
// and the slide by one row.
#pragma once

#include <cuda_runtime.h>

namespace gtrap {

// The window S[32 * k], k < w, of one lane ([rank][lane] in shared memory).  Both functions give the
// element-by-element result of an insertion sort / slide, which keeps equal values in their
// order.  With `linear` false the window must be sorted (it has never held a NaN): each
// insertion point is then found by binary search and the elements between move as a block
// (loads before stores, not one dependent compare per element), for the packed detrend, whose lanes
// wait on their own chains.  With `linear` true the element-by-element loops run: their cost follows
// the displacement (the image detrend, and windows that have held a NaN; the order with NaN is
// what they leave).  Only radii below 4 and past 888 come here; the others have kernels of their own.

// Moves S[lo..hi) up by one slot (to S[lo+1..hi]).
__device__ __forceinline__ void window_move_up(float *S, int lo, int hi) {
  int j = hi;
  for (; j - 4 >= lo; j -= 4) {
    const float a0 = S[32 * (j - 1)], a1 = S[32 * (j - 2)], a2 = S[32 * (j - 3)], a3 = S[32 * (j - 4)];
    S[32 * j] = a0; S[32 * (j - 1)] = a1; S[32 * (j - 2)] = a2; S[32 * (j - 3)] = a3;
  }
  for (; j > lo; --j) S[32 * j] = S[32 * (j - 1)];
}

// Moves S(lo..hi] down by one slot (to S[lo..hi)).
__device__ __forceinline__ void window_move_down(float *S, int lo, int hi) {
  int j = lo;
  for (; j + 4 <= hi; j += 4) {
    const float a0 = S[32 * (j + 1)], a1 = S[32 * (j + 2)], a2 = S[32 * (j + 3)], a3 = S[32 * (j + 4)];
    S[32 * j] = a0; S[32 * (j + 1)] = a1; S[32 * (j + 2)] = a2; S[32 * (j + 3)] = a3;
  }
  for (; j < hi; ++j) S[32 * j] = S[32 * (j + 1)];
}

// Sorts the loaded window in place (stable insertion sort).
__device__ __forceinline__ void window_sort(float *S, int w, bool linear) {
  for (int k = 1; k < w; ++k) {
    const float v = S[32 * k];
    if (!linear) {
      int lo = 0, hi = k;  // the insertion point: the number of elements <= v
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (S[32 * mid] <= v) lo = mid + 1; else hi = mid;
      }
      window_move_up(S, lo, k);
      S[32 * lo] = v;
    } else {
      int j = k;
      while (j > 0) {
        const float u = S[32 * (j - 1)];
        if (u <= v) break;
        S[32 * j] = u;
        --j;
      }
      S[32 * j] = v;
    }
  }
}

// Slides the window by one row: vold leaves, vnew (!= vold) enters.
__device__ __forceinline__ void window_slide(float *S, int w, float vold, float vnew, bool linear) {
  // lowest rank holding the leaving value (present in the window by construction)
  int lo = 0, hi = w - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (S[32 * mid] < vold) lo = mid + 1; else hi = mid;
  }
  int j = lo;
  if (!linear) {
    if (vnew > vold) {  // vnew lands before the first element >= vnew above the freed slot
      int a = j + 1, b = w;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (S[32 * mid] < vnew) a = mid + 1; else b = mid;
      }
      window_move_down(S, j, a - 1);
      S[32 * (a - 1)] = vnew;
    } else {            // vnew lands after the last element <= vnew below the freed slot
      int a = 0, b = j;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (S[32 * mid] <= vnew) a = mid + 1; else b = mid;
      }
      window_move_up(S, a, j);
      S[32 * a] = vnew;
    }
    return;
  }
  if (vnew > vold) {
    while (j + 1 < w) {
      const float u = S[32 * (j + 1)];
      if (!(u < vnew)) break;
      S[32 * j] = u;
      ++j;
    }
  } else {
    while (j > 0) {
      const float u = S[32 * (j - 1)];
      if (!(u > vnew)) break;
      S[32 * j] = u;
      --j;
    }
  }
  S[32 * j] = vnew;
}

}  // namespace gtrap
