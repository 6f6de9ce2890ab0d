// The step-sized matrix recurrence (state-space duality) in chunks of 64 tokens on the tensor cores, for bfloat16
// operands.  With a_t = A dt_t, G_t the sum of a up to and with token t of the chunk, and S the state before the chunk:
//     y_t = exp(G_t) C_t S^T  +  sum_{s <= t} exp(G_t - G_s) dt_s (C_t . B_s) x_s
//     S  <- exp(G_64) S       +  sum_s exp(G_64 - G_s) dt_s x_s B_s^T
// so a chunk is four matrix products (C B^T, C S^T, M x, x^T B) and only the state goes from chunk to chunk.
//
// Precision.  C, B and x are bfloat16 and enter as they are.  What is held in 32 bits (S, M, the weighted x) enters a
// product as three bfloat16 parts, 24 bits and more, with fp32 accumulation; the state itself stays in fp32 registers.
// G is summed in 64 bits and split into a multiple of 2^-12 and a rest, so that the difference of two of them loses
// nothing; what the state loses over a chunk comes from expm1.  Relative error against 64 bits over 2,048 tokens, 64
// heads of 64 x 128: y 9.7e-8, state 1.1e-7 (1.3e-7 and 1.1e-7 token by token); decays a hundred times slower 8.7e-8 and
// 9.2e-8 (2.0e-7 and 6.4e-7).  With the tensor cores adding into long-lived accumulators they were 6.1e-7 and 2.5e-7.
//
// A block takes 32 value columns of one (request, head); eight warps.  Warp w owns rows 16 (w / 2) .. of the chunk
// (half of its causal tiles of C B^T, then 16 of the 32 columns of y) and DK / 8 columns of the state.  The next chunk's
// C, B and x are copied and its decays summed (by a ninth warp) while this one is computed.  What bounds it: the chain of a
// chunk, 4.4 us of two barriers and about 1,200 instructions a warp with two warps a scheduler (tensor pipe 22 % busy),
// times the chunks of the longest request; token by token a chunk is a chain of 64 steps, 23 us.  2,048 tokens of one
// request, 64 heads of 64 x 128: 142 us against 727; four of 512: 147 against 672; 64: 17 against 28.
#pragma once
#include "mma_utils.cuh"

namespace ssd {
constexpr int L = 64, COLS = 32, THREADS = 256;     // (and one warp more, for the decays)
constexpr int XP = COLS + 8, MP = L + 8;            // rows padded by 16 bytes: ldmatrix without bank conflicts

template <int DK> struct Smem {
  static constexpr int P = DK + 8;
  __nv_bfloat16 c[2][L][P], b[2][L][P], x[2][L][XP];
  __nv_bfloat16 xw[3][L][XP];                       // x times its weight in the new state, in three parts
  __nv_bfloat16 m[3][L][MP];
  __nv_bfloat16 s[3][COLS][P];                      // the state before the chunk
  float g_hi[2][L], g_lo[2][L], eg[2][L], dt[2][L], w[2][L];
  float loss[2], keep[2];
};

// d = a b from zero: the tensor cores add into an accumulator by cutting bits off, always towards zero; a product that
// starts from zero and is added with a rounding instruction keeps that error to the product's own size.
__device__ __forceinline__ void mma_bf16_new(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_add(float (&sum)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float d[4];
  mma_bf16_new(d, a, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; ++e) sum[e] += d[e];
}
__device__ __forceinline__ void block_barrier() { asm volatile("bar.sync 0, %0;" ::"n"(THREADS + 32) : "memory"); }

__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const float ra = a - __low2float(h), rb = b - __high2float(h);
  const __nv_bfloat162 m = __floats2bfloat162_rn(ra, rb);
  const __nv_bfloat162 l = __floats2bfloat162_rn(ra - __low2float(m), rb - __high2float(m));
  hi = *reinterpret_cast<const uint32_t*>(&h), mid = *reinterpret_cast<const uint32_t*>(&m),
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

template <int DK>
__global__ void __launch_bounds__(THREADS + 32, 1)
chunk_kernel(const __nv_bfloat16* __restrict__ q, int64_t q_stride, const __nv_bfloat16* __restrict__ k,
             int64_t k_stride, const __nv_bfloat16* __restrict__ v, int64_t v_stride, const float* __restrict__ gates,
             int64_t gates_stride, const float* __restrict__ gate_bias, const float* __restrict__ rate, float q_scale,
             float* __restrict__ state, const int* __restrict__ cu_q, const int* __restrict__ state_slots,
             float* __restrict__ out, int64_t out_stride, int heads, int dv, int kv_div, int from) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<DK>& sm = *reinterpret_cast<Smem<DK>*>(smem_raw);
  constexpr int KS = DK / 16, NT = DK / 64;         // k steps of a product over DK; tiles of 8 state columns a warp owns
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * COLS;
  const int start = cu_q[r], end = cu_q[r + 1];
  if (start >= end || end - start < from) return;   // (shorter requests are another kernel's)
  const int mt = warp >> 1, half = warp & 1, gr = lane >> 2, gc = (lane & 3) * 2;
  const float A = rate[h], bias = gate_bias[h];
  const __nv_bfloat16* q_src = q + (h / kv_div) * DK;
  const __nv_bfloat16* k_src = k + (h / kv_div) * DK;
  const __nv_bfloat16* v_src = v + (int64_t)h * dv + col0;

  auto request = [&](int t0, int buf) {
    const int nt = min(L, end - t0);
#pragma unroll
    for (int i = 0; i < L * (DK / 8) / THREADS; ++i) {
      const int idx = tid + i * THREADS, t = idx / (DK / 8), p = (idx % (DK / 8)) * 8;
      const int64_t tok = t0 + min(t, nt - 1);
      cp_async16(smem_u32(&sm.c[buf][t][p]), q_src + tok * q_stride + p, t < nt);
      cp_async16(smem_u32(&sm.b[buf][t][p]), k_src + tok * k_stride + p, t < nt);
    }
    {
      const int t = tid >> 2, p = (tid & 3) * 8;
      cp_async16(smem_u32(&sm.x[buf][t][p]), v_src + (int64_t)(t0 + min(t, nt - 1)) * v_stride + p, t < nt);
    }
    cp_async_commit();
  };
  auto put_state = [&](const float (&S)[2][NT][4]) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t part[3];
          split3(S[m][n][2 * e], S[m][n][2 * e + 1], part[0], part[1], part[2]);
#pragma unroll
          for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint32_t*>(&sm.s[p][m * 16 + gr + 8 * e][(warp * NT + n) * 8 + gc]) = part[p];
        }
  };

  if (warp == THREADS / 32) {
    // the decays of a chunk, made while the chunk before it is computed: two tokens a lane
    float raw0 = 0.f, raw1 = 0.f;
    auto fetch = [&](int t0) {
      const int t = t0 + lane * 2;
      raw0 = t < end ? gates[(int64_t)t * gates_stride + h] : 0.f;
      raw1 = t + 1 < end ? gates[(int64_t)(t + 1) * gates_stride + h] : 0.f;
    };
    auto scan = [&](int t0, int buf) {
      const int t = t0 + lane * 2;
      const float x0 = raw0 + bias, x1 = raw1 + bias;
      if (t0 + L < end) fetch(t0 + L);
      const float d0 = t < end ? fmaxf(x0, 0.f) + log1pf(expf(-fabsf(x0))) : 0.f;
      const float d1 = t + 1 < end ? fmaxf(x1, 0.f) + log1pf(expf(-fabsf(x1))) : 0.f;
      const double a0 = (double)A * d0, a1 = (double)A * d1;
      double g1 = a0 + a1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, g1, o);
        if (lane >= o) g1 += up;
      }
      const double g0 = g1 - a1, gl = __shfl_sync(0xffffffffu, g1, 31);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double g = e ? g1 : g0;
        const float d = e ? d1 : d0, hi = rintf((float)g * 4096.f) * (1.f / 4096.f);
        sm.g_hi[buf][lane * 2 + e] = hi;
        sm.g_lo[buf][lane * 2 + e] = (float)(g - hi);
        sm.eg[buf][lane * 2 + e] = expf((float)g);
        sm.dt[buf][lane * 2 + e] = d;
        sm.w[buf][lane * 2 + e] = expf((float)(gl - g)) * d;
      }
      if (lane == 0) sm.loss[buf] = -expm1f((float)gl), sm.keep[buf] = expf((float)gl);
    };
    fetch(start);
    scan(start, 0);
    for (int t0 = start, buf = 0; t0 < end; t0 += L, buf ^= 1) {
      block_barrier();
      if (t0 + L < end) scan(t0 + L, buf ^ 1);
      block_barrier();
    }
    return;
  }
  request(start, 0);
  float S[2][NT][4];
  float* sp = state + (((int64_t)state_slots[r] * heads + h) * dv + col0 + gr) * DK + warp * NT * 8 + gc;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float2 x = *reinterpret_cast<const float2*>(sp + (int64_t)(m * 16 + 8 * e) * DK + n * 8);
        S[m][n][2 * e] = x.x, S[m][n][2 * e + 1] = x.y;
      }
  put_state(S);

  int buf = 0;
  for (int t0 = start; t0 < end; t0 += L, buf ^= 1) {
    cp_async_wait<0>();
    block_barrier();                                // the chunk's operands and decays and the state's parts are there
    if (t0 + L < end) request(t0 + L, buf ^ 1);
    // C B^T of this warp's causal tiles, C S^T of its columns
    float cb[4][4], y[2][4], y_low[2][4];           // (y_low: the products of the state's lower parts)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) cb[n][e] = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) y[n][e] = y_low[n][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < KS; ks += 2) {
      uint32_t a0[4], a1[4];
      const __nv_bfloat16* a_row = &sm.c[buf][mt * 16 + (lane & 15)][(lane >> 4) * 8];
      ldmatrix_x4(a0, smem_u32(a_row + ks * 16));
      ldmatrix_x4(a1, smem_u32(a_row + ks * 16 + 16));
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (n <= mt) {
          uint32_t bb[4];
          ldmatrix_x4(bb, smem_u32(&sm.b[buf][(half * (mt + 1) + n) * 8 + (lane & 7)][ks * 16 + (lane >> 3) * 8]));
          mma_add(cb[n], a0, bb[0], bb[1]);
          mma_add(cb[n], a1, bb[2], bb[3]);
        }
      }
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          uint32_t bb[4];
          ldmatrix_x4(bb, smem_u32(&sm.s[p][half * 16 + n * 8 + (lane & 7)][ks * 16 + (lane >> 3) * 8]));
          if (p == 0) {
            mma_add(y[n], a0, bb[0], bb[1]);
            mma_add(y[n], a1, bb[2], bb[3]);
          } else {
            mma_bf16(y_low[n], a0, bb[0], bb[1]);
            mma_bf16(y_low[n], a1, bb[2], bb[3]);
          }
        }
    }
    const int row = mt * 16 + gr;
    {
      const float e0 = sm.eg[buf][row], e1 = sm.eg[buf][row + 8];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          y[n][e] = (y[n][e] + y_low[n][e]) * (e < 2 ? e0 : e1);
          y_low[n][e] = 0.f;
        }
      const float h0 = sm.g_hi[buf][row], l0 = sm.g_lo[buf][row], h1 = sm.g_hi[buf][row + 8], l1 = sm.g_lo[buf][row + 8];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (n <= mt) {
          const int c = (half * (mt + 1) + n) * 8 + gc;
          float val[4];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float ch = sm.g_hi[buf][c + e], cl = sm.g_lo[buf][c + e], d = sm.dt[buf][c + e];
            val[e] = c + e <= row ? cb[n][e] * expf((h0 - ch) + (l0 - cl)) * d : 0.f;
            val[2 + e] = c + e <= row + 8 ? cb[n][2 + e] * expf((h1 - ch) + (l1 - cl)) * d : 0.f;
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t part[3];
            split3(val[2 * e], val[2 * e + 1], part[0], part[1], part[2]);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(&sm.m[p][row + 8 * e][c]) = part[p];
          }
        }
      }
      const int t = tid >> 2, p0 = (tid & 3) * 8;
      const float w = sm.w[buf][t];
      uint4 raw = *reinterpret_cast<const uint4*>(&sm.x[buf][t][p0]);
      const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
      uint32_t parts[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 two = *reinterpret_cast<const __nv_bfloat162*>(&in[i]);
        split3(__low2float(two) * w, __high2float(two) * w, parts[0][i], parts[1][i], parts[2][i]);
      }
#pragma unroll
      for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(&sm.xw[p][t][p0]) = make_uint4(parts[p][0], parts[p][1], parts[p][2], parts[p][3]);
    }
    const float loss = sm.loss[buf], keep = sm.keep[buf];
    block_barrier();                                // M and the weighted x are there; nobody reads the state's parts any more
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      if (ks <= mt) {
        uint32_t bb[4];
        ldmatrix_x4_trans(bb, smem_u32(&sm.x[buf][ks * 16 + (lane & 15)][half * 16 + (lane >> 4) * 8]));
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          uint32_t a[4];
          ldmatrix_x4(a, smem_u32(&sm.m[p][mt * 16 + (lane & 15)][ks * 16 + (lane >> 4) * 8]));
          if (p == 0) {
            mma_add(y[0], a, bb[0], bb[1]);
            mma_add(y[1], a, bb[2], bb[3]);
          } else {
            mma_bf16(y_low[0], a, bb[0], bb[1]);
            mma_bf16(y_low[1], a, bb[2], bb[3]);
          }
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = t0 + row + 8 * e;
      if (t < end) {
        float* dst = out + (int64_t)t * out_stride + (int64_t)h * dv + col0 + half * 16 + gc;
#pragma unroll
        for (int n = 0; n < 2; ++n)
          *reinterpret_cast<float2*>(dst + n * 8) = make_float2((y[n][2 * e] + y_low[n][2 * e]) * q_scale, (y[n][2 * e + 1] + y_low[n][2 * e + 1]) * q_scale);
      }
    }
    float add[2][NT][4], add_low[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) add[m][n][e] = add_low[m][n][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ks += 2) {
      uint32_t bb[2][4];                            // tiles of B: [k step][tile 0: two, tile 1: two]
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (NT == 2) {
          ldmatrix_x4_trans(bb[j], smem_u32(&sm.b[buf][(ks + j) * 16 + (lane & 15)][warp * 16 + (lane >> 4) * 8]));
        } else if (j == 0) {
          uint32_t both[4];
          ldmatrix_x4_trans(both, smem_u32(&sm.b[buf][ks * 16 + lane][warp * 8]));
          bb[0][0] = both[0], bb[0][1] = both[1], bb[1][0] = both[2], bb[1][1] = both[3];
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            uint32_t a[4];
            ldmatrix_x4_trans(a, smem_u32(&sm.xw[p][(ks + j) * 16 + (lane >> 4) * 8 + (lane & 7)][m * 16 + ((lane >> 3) & 1) * 8]));
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              if (p == 0) mma_add(add[m][n], a, bb[j][2 * n], bb[j][2 * n + 1]);
              else mma_bf16(add_low[m][n], a, bb[j][2 * n], bb[j][2 * n + 1]);
            }
          }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float sum = add[m][n][e] + add_low[m][n][e];
          // (a slow state loses little and is changed by that little; a fast one is mostly replaced)
          S[m][n][e] = loss < 0.5f ? S[m][n][e] + fmaf(-loss, S[m][n][e], sum) : fmaf(keep, S[m][n][e], sum);
        }
    if (t0 + L < end) put_state(S);
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<float2*>(sp + (int64_t)(m * 16 + 8 * e) * DK + n * 8) = make_float2(S[m][n][2 * e], S[m][n][2 * e + 1]);
}

// Whether chunk_kernel takes these operands: bfloat16 rows on 16-byte boundaries, 64 or 128 key channels, value columns
// in blocks of 32, the state on 8-byte boundaries.  (Whether it is the quicker one is the caller's rule.)
inline bool takes(const void* q, int64_t q_stride, const void* k, int64_t k_stride, const void* v, int64_t v_stride,
                  const float* state, const float* out, int64_t out_stride, int dk, int dv) {
  const uintptr_t p = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v);
  return (dk == 64 || dk == 128) && dv % COLS == 0 && (p & 15) == 0 && ((q_stride | k_stride | v_stride) & 7) == 0 &&
         (reinterpret_cast<uintptr_t>(state) & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0 && out_stride % 2 == 0;
}

inline int launch(const __nv_bfloat16* q, int64_t q_stride, const __nv_bfloat16* k, int64_t k_stride,
                  const __nv_bfloat16* v, int64_t v_stride, const float* gates, int64_t gates_stride,
                  const float* gate_bias, const float* rate, float q_scale, float* state, const int* cu_q,
                  const int* state_slots, float* out, int64_t out_stride, int requests, int heads, int dk, int dv,
                  int kv_div, int from, cudaStream_t stream) {
  auto kernel = dk == 64 ? chunk_kernel<64> : chunk_kernel<128>;
  const size_t smem = dk == 64 ? sizeof(Smem<64>) : sizeof(Smem<128>);
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return gllm_launch(kernel, dim3(dv / COLS, heads, requests), dim3(THREADS + 32), smem, stream, q, q_stride, k, k_stride, v,
                     v_stride, gates, gates_stride, gate_bias, rate, q_scale, state, cu_q, state_slots, out, out_stride,
                     heads, dv, kv_div, from);
}
}  // namespace ssd
