// The last inputs of a short causal convolution, for a thread that owns one 16-byte piece of the channels and walks a
// run of tokens of the flat batch.
#pragma once
#include "common.cuh"

template <typename T>
struct alignas(16) ConvPiece {
  static constexpr int N = 16 / sizeof(T);
  T v[N];
};

template <typename T, int TAPS>
struct ConvWindow {
  static constexpr int N = ConvPiece<T>::N;
  float wt[TAPS][N];                   // wt[j]: the weight of the input j tokens back
  float past[TAPS - 1][N];             // past[j]: the input j + 1 tokens back
  int row = -1, pos = 0;               // of the token before the one in hand

  // w [channels, TAPS], last column the current token; 16-byte aligned
  __device__ __forceinline__ void load_weights(const float* __restrict__ w, int c) {
    float flat[TAPS * N];
#pragma unroll
    for (int e = 0; e < TAPS * N; e += 4) {
      const float4 f = *reinterpret_cast<const float4*>(w + (int64_t)c * TAPS + e);
      flat[e] = f.x, flat[e + 1] = f.y, flat[e + 2] = f.z, flat[e + 3] = f.w;
    }
#pragma unroll
    for (int j = 0; j < TAPS; ++j)
#pragma unroll
      for (int e = 0; e < N; ++e) wt[j][e] = flat[e * TAPS + TAPS - 1 - j];
  }
  // To token i of the batch (row_i, pos_i), whose inputs of these channels lie at x_c[i * x_stride].  Where the request's
  // earlier tokens are not the ones just walked, they come from the batch (`first`: i starts the run) and, behind those
  // that the batch holds, from conv_state [slots, TAPS-1, channels], oldest first.
  __device__ __forceinline__ void move_to(int i, bool first, int row_i, int pos_i, const T* __restrict__ x_c,
                                          int64_t x_stride, const float* __restrict__ conv_state, int channels, int c,
                                          const int* __restrict__ positions, const int* __restrict__ token_row) {
    if (first || row_i != row || pos_i != pos + 1) {
      int here = 0;
      if (first)
        while (here < TAPS - 1 && i - here - 1 >= 0 && token_row[i - here - 1] == row_i && positions[i - here - 1] == pos_i - here - 1) ++here;
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) {
        if (j < here) {
          const ConvPiece<T> p = *reinterpret_cast<const ConvPiece<T>*>(x_c + (int64_t)(i - j - 1) * x_stride);
#pragma unroll
          for (int e = 0; e < N; ++e) past[j][e] = to_float(p.v[e]);
        } else {
          const float* p = conv_state + ((int64_t)row_i * (TAPS - 1) + TAPS - 2 - (j - here)) * channels + c;
#pragma unroll
          for (int e = 0; e < N; e += 4) {
            const float4 f = *reinterpret_cast<const float4*>(p + e);
            past[j][e] = f.x, past[j][e + 1] = f.y, past[j][e + 2] = f.z, past[j][e + 3] = f.w;
          }
        }
      }
    }
    row = row_i, pos = pos_i;
  }
  // The sum of channel e for the input v of the token in hand, which joins the window.
  __device__ __forceinline__ float step(int e, float v, float bias) {
    float acc = fmaf(wt[0][e], v, bias);
#pragma unroll
    for (int j = 1; j < TAPS; ++j) acc = fmaf(wt[j][e], past[j - 1][e], acc);
#pragma unroll
    for (int j = TAPS - 2; j > 0; --j) past[j][e] = past[j - 1][e];
    past[0][e] = v;
    return acc;
  }
};
