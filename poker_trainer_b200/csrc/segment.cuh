// A decision node's arithmetic for one hand, shared by the segment passes
// (segment.cu) and the batch's (batch.cu): the reference's f32 operations in
// its order. Arrays have MAXA entries of which the first na count: the others
// are left out of every sum by selection, with no branch per action.
#pragma once

#include <type_traits>

#include "plan.hpp"
#include "row_items.cuh"

namespace dcfr {

// f(most, na): a node's work with arrays of `most` entries. The usual action
// counts are exact, so that their arrays have no entries to leave out.
template <int MAXA, typename F>
__device__ __forceinline__ void by_actions(int na, F&& f) {
  if (na == 2) f(std::integral_constant<int, 2>(), 2);
  else if (na == 3) f(std::integral_constant<int, 3>(), 3);
  else if (MAXA <= 4 || na == 4) f(std::integral_constant<int, 4>(), MAXA <= 4 ? na : 4);
  else f(std::integral_constant<int, MAXA>(), na);
}

// Strategy from regrets (regret_match_into, cfr.rs:161-192) or from strategy
// sums (normalize_in_place, cfr.rs:124-154), in place.
template <int MAXA, bool REGRETS>
__device__ __forceinline__ void to_strategy(float (&x)[MAXA], int na, float uniform) {
#pragma unroll
  for (int a = 0; a < MAXA; a++)
    if (REGRETS) x[a] = max0(x[a]);
  float s = x[0];
#pragma unroll
  for (int a = 1; a < MAXA; a++) s = a < na ? s + x[a] : s;
  const float inv = recipf(s);
#pragma unroll
  for (int a = 0; a < MAXA; a++) x[a] = inv == 0.0f ? uniform : x[a] * inv;
}

// Strategy sum after an iteration (cfr.rs:395-407).
__device__ __forceinline__ float next_sum(float s, float sigma, float r, const DiscountD& d) {
  const float add = d.reach_weighted ? sigma * r : sigma;
  return s * d.strat + add;
}

// Value of the traverser's node under its regrets' strategy (own_node_update,
// cfr.rs:315-382).
template <int MAXA>
__device__ __forceinline__ void own_value(const float (&r)[MAXA], const float (&v)[MAXA], int na, float uniform,
                                          float& out) {
  float s = max0(r[0]);
#pragma unroll
  for (int a = 1; a < MAXA; a++) s = a < na ? s + max0(r[a]) : s;
  const float iv = recipf(s);
  float o = 0.0f, m = -0.0f;
#pragma unroll
  for (int a = 0; a < MAXA; a++) {
    o = a < na ? o + max0(r[a]) * v[a] : o;
    m = a < na ? m + v[a] : m;
  }
  out = iv == 0.0f ? m * uniform : o * iv;
}

__device__ __forceinline__ float next_regret(float r, float v, float out, const DiscountD& d) {
  const float disc = r > 0.0f ? d.pos : d.neg;
  return r * disc + v - out;
}

}  // namespace dcfr
