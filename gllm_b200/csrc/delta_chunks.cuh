// The gated delta rule in chunks of 64 tokens, for heads of 64 key channels; fp32 throughout.
//
// Within a chunk, with G_t the sum of the log decays up to and with token t (per key channel), S the state before the
// chunk and u_t = beta_t (v_t - S_t'^T k_t) the tokens' writes:
//     (I + A) U = diag(beta) (V - K~ S),   A_ts = beta_t sum_d k_t k_s exp(G_t - G_s)  (s < t),   K~_t = exp(G_t) k_t
//     O  = Q~ S + P U,                     P_ts = sum_d q_t k_s exp(G_t - G_s)  (s <= t),         Q~_t = exp(G_t) q_t
//     S <- diag(exp(G_64)) S + K^^T U,     K^_s = exp(G_64 - G_s) k_s
// Two kernels.  prepare_kernel, one block per (chunk, head), all in parallel: G, A, P, then W = (I + A)^-1 diag(beta) K~
// and U0 = (I + A)^-1 diag(beta) V, left in a record per (chunk, head).  walk_kernel, one block per (request, head, 16
// value columns), chunk after chunk: U = U0 - W S, O, S.
//
// No exponent is ever positive: sixteen tokens are a block; between blocks exp(G_t - G_s) is the product of exp(G_t - G_b)
// and exp(G_b - G_s) with b the start of t's block, inside a block it is formed for every pair and channel.  Decays are
// multiplied up, never exponentiated: a decay that has kept more than half as one minus its loss (the loss of a product
// rounds at its own size, so slow decays do not drift), any other as the product itself.
//
// What bounds it: prepare_kernel the instructions of a chunk (0.75 M multiply-adds and the decays of every pair, two
// blocks an SM); walk_kernel the chain of a chunk, 3.4 us of two products of 64 x 64 x 16 one after the other (four
// warps; four more make the outputs beside them), shared-memory loads and two barriers.  2,048 tokens of one request,
// 16 heads of 64 x 128: 71 + 110 us against 451 token by token (220 ns a token); 512: 62 us for both against 130.
// Relative error against 64 bits there: outputs 2.0e-7, state 2.0e-7 (1.7e-7 and 1.6e-7 token by token); decays a hundred
// times slower 2.8e-7 and 2.5e-7 (3.3e-7 and 3.3e-7).
#pragma once
#include "common.cuh"

namespace delta_chunks {
constexpr int L = 64, DK = 64, PITCH = DK + 4, SUB = 16, COLS = 16, UP = COLS + 4;
constexpr int MAT = L * PITCH;                        // floats of a 64 x 64 matrix with padded rows
constexpr int REC_HEAD = 4 * MAT + 2 * DK;            // W | Q~ | P | K^ transposed | exp(G_64) | 1 - exp(G_64)
constexpr int U0_BLOCK = L * UP;                      // U0 of 16 columns
constexpr int PREP_THREADS = 256, WALK_THREADS = 256;

__host__ __device__ inline int64_t record_floats(int dv) { return REC_HEAD + (int64_t)(dv / COLS) * U0_BLOCK; }
// Request r's first record: as many as its earlier requests can have chunks.
__host__ __device__ inline int64_t first_record(int cu, int r) { return cu / L + r; }

__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float both(unsigned long long v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

// A product of decays 1 - loss.
struct Decay {
  float lost = 0.f, product = 1.f;
  __device__ __forceinline__ void times(float loss) {
    lost = fmaf(loss, 1.f - lost, lost);
    product = fmaf(-loss, product, product);
  }
  __device__ __forceinline__ float kept() const { return lost < 0.5f ? 1.f - lost : product; }
};

struct PrepSmem {
  float k[L][PITCH];         // k, then exp(G_b - G_s) k for the next block b, at last K^
  float q[L][PITCH];         // q, then Q~; later a stretch of V
  float l[L][PITCH];         // losses, then K~
  float a[L][PITCH], p[L][PITCH];
  float x[4][SUB][SUB + 4];  // inverses of the diagonal blocks of I + A
  float block_loss[4][DK], block_decay[4][DK];
  float beta[L];
};

// R <- (I + A)^-1 diag(beta) R for N matrices of 64 columns, block row after block row.
template <int N>
__device__ __forceinline__ void solve(PrepSmem& s, float (*const (&R)[N])[PITCH]) {
  const int c = threadIdx.x & 63, rg = (threadIdx.x >> 6) * 4;
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const int t = i * SUB + rg;
    float acc[N][4];
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][e] = s.beta[t + e] * R[m][t + e][c];
#pragma unroll 2
    for (int j = 0; j < i * SUB; j += 4) {
      float4 a[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = *reinterpret_cast<const float4*>(&s.a[t + e][j]);
#pragma unroll
      for (int m = 0; m < N; ++m) {
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] = R[m][j + e][c];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          acc[m][e] = fmaf(-a[e].w, r[3], fmaf(-a[e].z, r[2], fmaf(-a[e].y, r[1], fmaf(-a[e].x, r[0], acc[m][e]))));
      }
    }
    // (a thread writes the elements that only it has read)
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) R[m][t + e][c] = acc[m][e];
    __syncthreads();
    float out[N][4];
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) out[m][e] = 0.f;
#pragma unroll
    for (int j = 0; j < SUB; j += 4) {
      float4 x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = *reinterpret_cast<const float4*>(&s.x[i][rg + e][j]);
#pragma unroll
      for (int m = 0; m < N; ++m) {
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] = R[m][i * SUB + j + e][c];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          out[m][e] = fmaf(x[e].x, r[0], fmaf(x[e].y, r[1], fmaf(x[e].z, r[2], fmaf(x[e].w, r[3], out[m][e]))));
      }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) R[m][t + e][c] = out[m][e];
    __syncthreads();
  }
}

template <bool HEAD>
__global__ void __launch_bounds__(PREP_THREADS, 2)
prepare_kernel(const float* __restrict__ qk, const float* __restrict__ v, const float* __restrict__ g,
               const float* __restrict__ beta, const int* __restrict__ cu_q, int requests, int heads, int kv_heads,
               int dv, int from, float* __restrict__ records) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PrepSmem& s = *reinterpret_cast<PrepSmem*>(smem_raw);
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, h = blockIdx.y, hg = h / (heads / kv_heads);
  // the request that owns this record
  int lo = 0, hi = requests - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first_record(cu_q[mid], mid) <= (int64_t)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const int start = cu_q[lo], end = cu_q[lo + 1];
  const int t0 = start + ((int)blockIdx.x - (int)first_record(start, lo)) * L;
  if (t0 >= end || end - start < from) return;
  const int nt = min(L, end - t0);
  float* rec = records + ((int64_t)blockIdx.x * heads + h) * record_floats(dv);

  const int qk_cols = 2 * kv_heads * DK;
  for (int idx = tid; idx < L * (DK / 4); idx += PREP_THREADS) {
    const int t = idx / (DK / 4), d = (idx % (DK / 4)) * 4;
    float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f), k4 = q4, g4 = q4;
    if (t < nt) {
      const float* row = qk + (int64_t)(t0 + t) * qk_cols + hg * DK + d;
      q4 = *reinterpret_cast<const float4*>(row);
      k4 = *reinterpret_cast<const float4*>(row + kv_heads * DK);
      if (HEAD) {
        const float x = g[(int64_t)(t0 + t) * heads + h];
        g4 = make_float4(x, x, x, x);
      } else {
        g4 = *reinterpret_cast<const float4*>(g + ((int64_t)(t0 + t) * heads + h) * DK + d);
      }
    }
    *reinterpret_cast<float4*>(&s.q[t][d]) = q4;
    *reinterpret_cast<float4*>(&s.k[t][d]) = k4;
    *reinterpret_cast<float4*>(&s.l[t][d]) = g4;
    *reinterpret_cast<float4*>(&s.a[t][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(&s.p[t][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tid < L) s.beta[tid] = tid < nt ? beta[(int64_t)(t0 + tid) * heads + h] : 0.f;
  __syncthreads();
  const int d_mine = tid & 63, b_mine = tid >> 6;
  {
    // pairs inside a block of sixteen: four threads a key s, each with sixteen channels (in fours, sixteen apart)
    const int key = (tid >> 2) & 15, part = (tid & 3) * 4, row0 = b_mine * SUB;
    Decay w[16];
    float ks[16];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 x = *reinterpret_cast<const float4*>(&s.k[row0 + key][c * 16 + part]);
      ks[4 * c] = x.x, ks[4 * c + 1] = x.y, ks[4 * c + 2] = x.z, ks[4 * c + 3] = x.w;
    }
#pragma unroll 1
    for (int t = 0; t < SUB; ++t) {
      float kk = 0.f, qk_ = 0.f;
      if (t >= key) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 loss = *reinterpret_cast<const float4*>(&s.l[row0 + t][c * 16 + part]);
          const float4 kt = *reinterpret_cast<const float4*>(&s.k[row0 + t][c * 16 + part]);
          const float4 qt = *reinterpret_cast<const float4*>(&s.q[row0 + t][c * 16 + part]);
          const float ls[4] = {loss.x, loss.y, loss.z, loss.w}, k4[4] = {kt.x, kt.y, kt.z, kt.w}, q4[4] = {qt.x, qt.y, qt.z, qt.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (t > key) w[4 * c + e].times(ls[e]);
            const float x = ks[4 * c + e] * w[4 * c + e].kept();
            kk = fmaf(k4[e], x, kk);
            qk_ = fmaf(q4[e], x, qk_);
          }
        }
      }
      kk += __shfl_xor_sync(0xffffffffu, kk, 1);
      qk_ += __shfl_xor_sync(0xffffffffu, qk_, 1);
      kk += __shfl_xor_sync(0xffffffffu, kk, 2);
      qk_ += __shfl_xor_sync(0xffffffffu, qk_, 2);
      if (part == 0 && t >= key) {
        if (t > key) s.a[row0 + t][row0 + key] = s.beta[row0 + t] * kk;
        s.p[row0 + t][row0 + key] = qk_;
      }
    }
  }
  __syncthreads();
  {
    float k_[SUB], loss[SUB];
#pragma unroll
    for (int i = 0; i < SUB; ++i) k_[i] = s.k[b_mine * SUB + i][d_mine], loss[i] = s.l[b_mine * SUB + i][d_mine];
    Decay from_start, to_end;
#pragma unroll
    for (int i = 0; i < SUB; ++i) {
      from_start.times(loss[i]);
      s.l[b_mine * SUB + i][d_mine] = k_[i] * from_start.kept();
      s.q[b_mine * SUB + i][d_mine] *= from_start.kept();
    }
#pragma unroll
    for (int i = SUB - 1; i >= 0; --i) {
      s.k[b_mine * SUB + i][d_mine] = k_[i] * to_end.kept();
      to_end.times(loss[i]);
    }
    s.block_loss[b_mine][d_mine] = from_start.lost;
    s.block_decay[b_mine][d_mine] = from_start.kept();
  }
  __syncthreads();
  // block row after block row: pairs with earlier blocks
  const int tx = tid & 15, ty = tid >> 4;
#pragma unroll 1
  for (int i = 1; i < 4; ++i) {
    const int row = i * SUB + ty;
    unsigned long long ka[3] = {0ull, 0ull, 0ull}, qa[3] = {0ull, 0ull, 0ull};
#pragma unroll 4
    for (int d = 0; d < DK; d += 4) {
      const ulonglong2 kt = *reinterpret_cast<const ulonglong2*>(&s.l[row][d]);
      const ulonglong2 qt = *reinterpret_cast<const ulonglong2*>(&s.q[row][d]);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j < i) {
          const ulonglong2 ks = *reinterpret_cast<const ulonglong2*>(&s.k[j * SUB + tx][d]);
          fma2(ka[j], kt.x, ks.x);
          fma2(ka[j], kt.y, ks.y);
          fma2(qa[j], qt.x, ks.x);
          fma2(qa[j], qt.y, ks.y);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (j < i) {
        s.a[row][j * SUB + tx] = s.beta[row] * both(ka[j]);
        s.p[row][j * SUB + tx] = both(qa[j]);
      }
    }
    __syncthreads();
    const float e = s.block_decay[i][d_mine];
    for (int t = b_mine; t < i * SUB; t += 4) s.k[t][d_mine] *= e;
    __syncthreads();
  }
  {
    float before = 1.f;
    for (int b = 0; b < b_mine; ++b) before *= s.block_decay[b][d_mine];
    for (int i = 0; i < SUB; ++i) {
      const int t = b_mine * SUB + i;
      s.l[t][d_mine] *= before;
      const float x = s.q[t][d_mine] * before;
      rec[MAT + t * PITCH + d_mine] = x;
    }
    if (b_mine == 3) {
      float lost = 0.f;
      for (int b = 0; b < 4; ++b) lost = fmaf(s.block_loss[b][d_mine], 1.f - lost, lost);
      rec[4 * MAT + d_mine] = before * s.block_decay[3][d_mine];
      rec[4 * MAT + DK + d_mine] = lost;
    }
    for (int idx = tid; idx < L * DK; idx += PREP_THREADS) rec[3 * MAT + (idx / L) * PITCH + idx % L] = s.k[idx % L][idx / L];
    for (int idx = tid; idx < L * (L / 4); idx += PREP_THREADS) {
      const int t = idx / (L / 4), c = (idx % (L / 4)) * 4;
      *reinterpret_cast<float4*>(rec + 2 * MAT + t * PITCH + c) = *reinterpret_cast<const float4*>(&s.p[t][c]);
    }
  }
  if (tid < 64) {                              // inverses of the diagonal blocks, a column a thread
    const int b = tid >> 4, c = tid & 15;
    float x[SUB];
#pragma unroll
    for (int t = 0; t < SUB; ++t) {
      float acc = t == c ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < t; ++j) acc = fmaf(-s.a[b * SUB + t][b * SUB + j], x[j], acc);
      x[t] = acc;
      s.x[b][t][c] = acc;
    }
  }
  __syncthreads();                             // (k and q are in the record by now: their places take stretches of V)
  auto load_v = [&](float (*dst)[PITCH], int c0) {
    for (int idx = tid; idx < L * 16; idx += PREP_THREADS) {
      const int t = idx >> 4, c = (idx & 15) * 4;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < nt && c0 + c < dv) x = *reinterpret_cast<const float4*>(v + ((int64_t)(t0 + t) * heads + h) * dv + c0 + c);
      *reinterpret_cast<float4*>(&dst[t][c]) = x;
    }
  };
  auto store_u0 = [&](float (*src)[PITCH], int c0) {
    for (int idx = tid; idx < L * 16; idx += PREP_THREADS) {
      const int t = idx >> 4, c = (idx & 15) * 4;
      if (c0 + c < dv)
        *reinterpret_cast<float4*>(rec + REC_HEAD + (int64_t)((c0 + c) / COLS) * U0_BLOCK + t * UP + c % COLS) =
            *reinterpret_cast<const float4*>(&src[t][c]);
    }
  };
  load_v(s.q, 0);
  if (dv > 64) load_v(s.k, 64);
  __syncthreads();
  if (dv > 64) {
    float (*const R[3])[PITCH] = {s.l, s.q, s.k};
    solve<3>(s, R);
    store_u0(s.k, 64);
  } else {
    float (*const R[2])[PITCH] = {s.l, s.q};
    solve<2>(s, R);
  }
  store_u0(s.q, 0);
  for (int idx = tid; idx < L * (DK / 4); idx += PREP_THREADS) {
    const int t = idx / (DK / 4), d = (idx % (DK / 4)) * 4;
    *reinterpret_cast<float4*>(rec + t * PITCH + d) = *reinterpret_cast<const float4*>(&s.l[t][d]);
  }
  for (int c0 = 128; c0 < dv; c0 += 128) {
    __syncthreads();
    load_v(s.q, c0);
    load_v(s.k, c0 + 64);
    __syncthreads();
    float (*const R[2])[PITCH] = {s.q, s.k};
    solve<2>(s, R);
    store_u0(s.q, c0);
    store_u0(s.k, c0 + 64);
  }
}

struct WalkSmem {
  float rec[2][REC_HEAD];
  float u0[2][U0_BLOCK];
  float s[2][COLS][PITCH];     // the state, a row per value column
  float u[COLS][PITCH];
};

// acc += M[rows][k0 .. k1) * B[cols][k0 .. k1)^T for this thread's 4 rows (16 apart) and 2 columns (8 apart); only the
// rows from I0 on.
template <int I0>
__device__ __forceinline__ void multiply(unsigned long long (&acc)[4][2], const float* m, const float* b, int k0, int k1) {
#pragma unroll 4
  for (int k = k0; k < k1; k += 4) {
    ulonglong2 x[4];
#pragma unroll
    for (int i = I0; i < 4; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(m + i * 16 * PITCH + k);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(b + j * 8 * PITCH + k);
#pragma unroll
      for (int i = I0; i < 4; ++i) fma2(acc[i][j], x[i].x, y.x);
#pragma unroll
      for (int i = I0; i < 4; ++i) fma2(acc[i][j], x[i].y, y.y);
    }
  }
}

__global__ void __launch_bounds__(WALK_THREADS, 1)
walk_kernel(const float* __restrict__ records, float* __restrict__ state, const int* __restrict__ cu_q,
            const int* __restrict__ state_slots, float* __restrict__ out, int heads, int dv, int from) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WalkSmem& s = *reinterpret_cast<WalkSmem*>(smem_raw);
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * COLS;
  const int start = cu_q[r], end = cu_q[r + 1];
  if (start >= end || end - start < from) return;
  const int64_t rec_floats = record_floats(dv), stride = rec_floats * heads;
  const float* rec = records + (first_record(start, r) * heads + h) * rec_floats;
  const float* u0 = rec + REC_HEAD + (int64_t)blockIdx.x * U0_BLOCK;
  auto request = [&](int chunk, int buf) {
    const float* src = rec + chunk * stride;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s.rec[buf]), dst_u = (uint32_t)__cvta_generic_to_shared(s.u0[buf]);
    for (int i = tid; i < REC_HEAD / 4; i += WALK_THREADS)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(src + i * 4) : "memory");
    const float* src_u = u0 + chunk * stride;
    for (int i = tid; i < U0_BLOCK / 4; i += WALK_THREADS)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_u + i * 16), "l"(src_u + i * 4) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  request(0, 0);
  float* sp = state + (((int64_t)state_slots[r] * heads + h) * dv + col0) * DK;
  for (int i = tid; i < COLS * (DK / 4); i += WALK_THREADS)
    *reinterpret_cast<float4*>(&s.s[0][i / (DK / 4)][(i % (DK / 4)) * 4]) = *reinterpret_cast<const float4*>(sp + i * 4);
  // four warps walk the chain, four make the outputs; a half warp is 4 x 4 threads
  const bool chain = warp < 4;
  const int ty = (warp & 3) * 4 + ((lane >> 2) & 3), tx = (lane & 3) + (lane >> 4) * 4;
  const int chunks = (end - start + L - 1) / L;
  int buf = 0;
  for (int c = 0; c < chunks; ++c, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                            // this chunk's record, the state after the last one
    if (c + 1 < chunks) request(c + 1, buf ^ 1);
    const float* m = s.rec[buf] + ty * PITCH;
    const float* st = &s.s[buf][tx][0];
    const float* us = &s.u[tx][0];
    unsigned long long acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[i][j] = 0ull;
    multiply<0>(acc, m + (chain ? 0 : MAT), st, 0, DK);        // W S, or Q~ S
    if (chain) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          s.u[tx + 8 * j][ty + 16 * i] = s.u0[buf][(ty + 16 * i) * UP + tx + 8 * j] - both(acc[i][j]);
          acc[i][j] = 0ull;
        }
    }
    __syncthreads();                            // U
    if (chain) {
      multiply<0>(acc, m + 3 * MAT, us, 0, L);
      const float* decay = s.rec[buf] + 4 * MAT;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int d = ty + 16 * i, col = tx + 8 * j;
          const float old = s.s[buf][col][d], add = both(acc[i][j]), lost = decay[DK + d];
          s.s[buf ^ 1][col][d] = lost < 0.5f ? old + fmaf(-lost, old, add) : fmaf(decay[d], old, add);
        }
    } else {
      multiply<0>(acc, m + 2 * MAT, us, 0, 16);                 // P is lower triangular
      multiply<1>(acc, m + 2 * MAT, us, 16, 32);
      multiply<2>(acc, m + 2 * MAT, us, 32, 48);
      multiply<3>(acc, m + 2 * MAT, us, 48, 64);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = start + c * L + ty + 16 * i;
        if (t < end)
#pragma unroll
          for (int j = 0; j < 2; ++j) out[((int64_t)t * heads + h) * dv + col0 + tx + 8 * j] = both(acc[i][j]);
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < COLS * (DK / 4); i += WALK_THREADS)
    *reinterpret_cast<float4*>(sp + i * 4) = *reinterpret_cast<const float4*>(&s.s[buf][i / (DK / 4)][(i % (DK / 4)) * 4]);
}

// Floats of records that a step of `tokens` tokens of `requests` requests takes.
inline int64_t workspace_floats(int tokens, int requests, int heads, int dv) {
  return (first_record(tokens, requests)) * heads * record_floats(dv);
}

inline int launch(const float* qk, const float* v, const float* g, const float* beta, float* state, const int* cu_q,
                  const int* state_slots, float* out, float* records, int tokens, int requests, int heads, int kv_heads,
                  int dv, bool per_head, int from, cudaStream_t stream) {
  auto prepare = per_head ? prepare_kernel<true> : prepare_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PrepSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WalkSmem));
  if (e != cudaSuccess) return (int)e;
  const int rc = gllm_launch(prepare, dim3((unsigned)first_record(tokens, requests), heads), dim3(PREP_THREADS),
                             sizeof(PrepSmem), stream, qk, v, g, beta, cu_q, requests, heads, kv_heads, dv, from, records);
  if (rc != 0) return rc;
  return gllm_launch(walk_kernel, dim3(dv / COLS, heads, requests), dim3(WALK_THREADS), sizeof(WalkSmem), stream, records,
                     state, cu_q, state_slots, out, heads, dv, from);
}
}  // namespace delta_chunks
