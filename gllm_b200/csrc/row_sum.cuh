// The result of routed experts before it is added up: token t's row is the sum over its slots s, in slot order, of
// weights[t, s] (or 1) times row row_of_pair[t * top + s] (or t * top + s) of y, itself the sum of `n_parts` unsummed
// parts in ascending order.  All fp32.
#pragma once
#include "common.cuh"

struct RowSum {
  const float* y;                // null: there is none
  int n_parts;
  int64_t part_stride;
  const int* row_of_pair;
  const float* weights;
  int top;

  template <int VEC> static __device__ __forceinline__ void load(const float* p, float (&v)[VEC]) {
    static_assert(VEC == 4 || VEC == 1, "one load");
    if constexpr (VEC == 4) {
      const float4 x = __ldcg(reinterpret_cast<const float4*>(p));
      v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    } else {
      v[0] = __ldcg(p);
    }
  }

  // columns c .. c + VEC - 1 of token t (VEC 4: 16-byte aligned); AT_ONCE: slots whose rows are requested together (those that are
  // not there read the group's first one's once more: two and three slots are still faster so than one after the other)
  template <int VEC, int AT_ONCE = 4> __device__ __forceinline__ void sum(int64_t t, int c, int width, float (&acc)[VEC]) const {
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
    for (int s0 = 0; s0 < top; s0 += AT_ONCE) {
      // (rows and weights, then the first part of every slot: nothing waits for the slot before it)
      const float* p[AT_ONCE];
      float w[AT_ONCE], v[AT_ONCE][VEC];
#pragma unroll
      for (int q = 0; q < AT_ONCE; ++q) {
        const bool in = s0 + q < top;
        const int64_t slot = t * top + (in ? s0 + q : s0);
        p[q] = y + (row_of_pair ? (int64_t)row_of_pair[slot] : slot) * width + c;
        w[q] = weights ? weights[slot] : 1.f;
      }
#pragma unroll
      for (int q = 0; q < AT_ONCE; ++q) load<VEC>(p[q], v[q]);
      for (int k = 1; k < n_parts; ++k)
#pragma unroll
        for (int q = 0; q < AT_ONCE; ++q) {
          float x[VEC];
          load<VEC>(p[q] + k * part_stride, x);
#pragma unroll
          for (int e = 0; e < VEC; ++e) v[q][e] += x[e];
        }
#pragma unroll
      for (int q = 0; q < AT_ONCE; ++q) {
        if (s0 + q >= top) break;
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] = fmaf(w[q], v[q][e], acc[e]);
      }
    }
  }
};
