// tn_order.h -- the decreasing order of a list of norms, as a rank per value.
//
// Ranks index shared memory, so they have to be a permutation whatever the
// values are: comparisons with NaN are all false, and counting them gives one
// rank to several values and leaves others without a holder (and a sort by
// exchange lets its padding in among the values).  Values that are not finite
// count as -1, below every norm; equal ones go by index.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define TN_ORDER_FN __device__ __forceinline__
namespace tn {
#else
#define TN_ORDER_FN inline
namespace tn {
using std::isfinite;
#endif

constexpr double kOrderPad = -2.0;  // key of a sort's padding, behind every order_key

template <typename R>
TN_ORDER_FN R order_key(R x) {
  return isfinite(x) ? x : R(-1);
}

// Square of a sorted key; not a number where its value was not finite, so that
// a sum of them tells.
TN_ORDER_FN double order_square(double key) { return key < 0.0 ? NAN : key * key; }

// Place of v[j] among v[0 .. n) in decreasing order.
template <typename R>
TN_ORDER_FN int order_rank(const R *v, int n, int j) {
  const R x = order_key(v[j]);
  int rank = 0;
  for (int i = 0; i < n; ++i) {
    const R y = order_key(v[i]);
    rank += (y > x || (y == x && i < j)) ? 1 : 0;
  }
  return rank;
}

}  // namespace tn
