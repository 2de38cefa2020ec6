// pm_bp.cuh -- the belief-propagation update shared by the pull (BP_F) and
// the count-driven kernel (k_bp).
#pragma once
#include "pm_common.cuh"

namespace pm {

template <class T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };
__device__ __forceinline__ float bp_exp(float x) { return expf(x); }
__device__ __forceinline__ double bp_exp(double x) { return exp(x); }
__device__ __forceinline__ float bp_log(float x) { return logf(x); }
__device__ __forceinline__ double bp_log(double x) { return log(x); }

// Edge potentials, one 2 x 2 matrix for every edge.
template <class T>
struct BpPsi {
  T p00, p01, p10, p11;
};

// k times the logarithm of the message of a vertex with prior pr and
// log-products l, normalised to sum 1: belief[i] = sum_j pr[j] psi[i][j]
// exp(l[j]).  The products are scaled by the larger one, whose own factor is
// exp(0) = 1 and is not computed.
template <class T>
__device__ __forceinline__ typename Vec2<T>::type bp_message(const BpPsi<T> &p, typename Vec2<T>::type pr,
                                                             typename Vec2<T>::type l, int k) {
  const bool first = l.x > l.y;
  const T lm = first ? l.x : l.y;
  const T low = bp_exp((first ? l.y : l.x) - lm);
  const T a0 = pr.x * (first ? T(1) : low), a1 = pr.y * (first ? low : T(1));
  const T b0 = p.p00 * a0 + p.p01 * a1, b1 = p.p10 * a0 + p.p11 * a1;
  const T lz = bp_log(b0 + b1);
  typename Vec2<T>::type out;
  out.x = (T)k * (bp_log(b0) - lz);
  out.y = (T)k * (bp_log(b1) - lz);
  return out;
}

}  // namespace pm
