// Attention of the 32-bit path over the paged cache, for head sizes 32, 64 and 128: a tiled kernel for portions of
// prompts and a split-KV kernel (with its merge) for single tokens.  No tensor-core mode: packed 32-bit multiply-adds,
// `expf`, fp32 everything.  A token at position p sees the keys first_visible_key(p, window) .. p.  Keys are taken in
// tiles (portions) or chunks (single tokens) aligned to absolute positions, so the order of a token's sums depends on its
// position and on whether it came in a portion or as a single token (a portion of one is one), and on nothing else of the
// cut or of the batch.
// Head sizes other than these run attention_simt.cu (a warp per token and head).
#include "common.cuh"

namespace {
__device__ __forceinline__ unsigned long long twice(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}

// ---- portions.  A block takes 64 rows (tokens x the query heads of one kv head) of one request and walks its keys in
// tiles of 64: S = Q K^T and O += P V, each thread 4 rows x 8 keys and 4 rows x D/8 columns.
// What bounds it: the latency of the shared-memory loads that feed the multiply-adds (12 sixteen-byte loads per 64 packed
// ones in S, as many and 16 register pairs in P V) with three warps a scheduler (head size 64; two took 3 us more); a half warp is 4 x 4 threads, so a load takes
// no more than two passes over the banks.  The warp-per-token kernel read every key row once per token and head, 32 rows
// side by side: 2,515 us for 512 and 200 (over 300) tokens beside 8 single ones (about 1,000 keys), 32 heads of 64 over 8;
// this kernel takes 105 us for the portions (10 of them for the look at broken values below), the split one 19 and its
// merge 5 for the single tokens.
constexpr int ROWS = 64, KEYS = 64, PF_THREADS = 128, P_PITCH = KEYS + 4;

template <int D> struct PortionSmem {
  float q[ROWS][D + 4];
  float k[KEYS][D + 4];
  float v[KEYS][D + 4];
  float p[ROWS][P_PITCH];
  int key_ok[2][KEYS];
};

// PER_SM: blocks an SM has to hold (0: the compiler's choice)
template <int D, int PER_SM>
__global__ void __launch_bounds__(PF_THREADS, PER_SM)
attention_f32_portion_kernel(const float* __restrict__ q, int64_t q_stride, float* __restrict__ out, int64_t out_stride,
                             const float* __restrict__ cache, const int* __restrict__ block_table, int bt_stride,
                             const int* __restrict__ cu_q, const int* __restrict__ ctx_lens,
                             const int* __restrict__ slots, int requests, int hq, int hkv, int block_size, int num_pages,
                             float scale, int window, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PortionSmem<D>& s = *reinterpret_cast<PortionSmem<D>*>(smem_raw);
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // 8 threads (tx) share a row of S, in two groups of four lanes; 16 of them (ty) lie below one another
  const int tx = (lane & 3) + (lane >> 4) * 4, ty = warp * 4 + ((lane >> 2) & 3);
  const int g = hq / hkv, tokens = ROWS / g;
  // The last tokens see the most keys: a request's tiles are taken from its end, the kv heads and the requests side by side, so
  // that the blocks that share an SM are a long one, a middling one and a short one.  (Tile after tile of a kv head, three
  // long ones could meet.)
  const int kvh = (int)blockIdx.x % hkv, rest = (int)blockIdx.x / hkv, r = rest % requests;
  const int t0 = cu_q[r], len = cu_q[r + 1] - t0;
  const int first = ((len + tokens - 1) / tokens - 1 - rest / requests) * tokens;
  if (first < 0) return;
  const int count = min(tokens, len - first), rows = count * g;
  const int ctx = ctx_lens[r];
  const int* bt = block_table + (int64_t)slots[r] * bt_stride;
  const int pos0 = ctx + first, pos_last = pos0 + count - 1;
  const size_t head_elems = (size_t)block_size * D, page_elems = (size_t)2 * hkv * head_elems;
  const int j_low = first_visible_key(pos0, window);     // (pages below it may have been given back)
  const int j_first = j_low & ~(KEYS - 1);

  // the copies of a tile: two threads a key, pieces of 16 bytes in turn
  const int my_key = tid >> 1, my_piece = tid & 1;
  const uint32_t k_dst = (uint32_t)__cvta_generic_to_shared(&s.k[my_key][my_piece * 4]);
  const uint32_t v_dst = (uint32_t)__cvta_generic_to_shared(&s.v[my_key][my_piece * 4]);
  auto page_of = [&](int j0) {                 // page of this thread's key of the tile at j0; -1: none
    const int j = j0 + my_key;
    if (j > pos_last || j < j_low) return -1;
    const int page = bt[j / block_size];
    if (page < 0 || page >= num_pages) {
      atomicOr(status, GLLM_STATUS_PAGE_RANGE);
      return -1;
    }
    return page;
  };
  auto copy = [&](uint32_t dst, int j0, int page, size_t half) {
    const float* src = cache;
    if (page >= 0) src += (size_t)page * page_elems + half + (size_t)kvh * head_elems + (size_t)((j0 + my_key) % block_size) * D + my_piece * 4;
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 32),
                   "l"(page >= 0 ? src + i * 8 : cache), "r"(page >= 0 ? 16 : 0) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const size_t v_half = (size_t)hkv * head_elems;

  int page = page_of(j_first);
  if (my_piece == 0) s.key_ok[0][my_key] = page >= 0;
  copy(k_dst, j_first, page, 0);
  copy(v_dst, j_first, page, v_half);
  for (int idx = tid; idx < ROWS * (D / 4); idx += PF_THREADS) {
    const int row = idx / (D / 4), c = (idx % (D / 4)) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows)
      x = *reinterpret_cast<const float4*>(q + (int64_t)(t0 + first + row / g) * q_stride + (int64_t)(kvh * g + row % g) * D + c);
    *reinterpret_cast<float4*>(&s.q[row][c]) = x;
  }
  constexpr int CP = D / 16;                     // pairs of output columns a thread keeps: D / 8 columns
  unsigned long long o[4][CP];
  float m[4], l[4];
  int row_pos[4], row_first[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = ty + 16 * i;
    row_pos[i] = row < rows ? pos0 + row / g : -1;
    row_first[i] = row < rows ? first_visible_key(row_pos[i], window) : 0;
    m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < CP; ++c) o[i][c] = 0ull;
  }
  int turn = 0;
  for (int j0 = j_first; j0 <= pos_last; j0 += KEYS, turn ^= 1) {
    const bool more = j0 + KEYS <= pos_last;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                                 // the keys (and the first time the queries) are there
    const int next_page = more ? page_of(j0 + KEYS) : -1;
    unsigned long long acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
#pragma unroll 4
    for (int c = 0; c < D; c += 4) {
      ulonglong2 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(&s.q[ty + 16 * i][c]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&s.k[tx + 8 * j][c]);
#pragma unroll
        for (int i = 0; i < 4; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < 4; ++i) fma2(acc[i][j], a[i].y, b.y);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float x[8], top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int key = tx + 8 * j, at = j0 + key;
        const bool sees = at <= row_pos[i] && at >= row_first[i] && s.key_ok[turn][key];
        x[j] = sees ? (pair_low(acc[i][j]) + pair_high(acc[i][j])) * scale : -INFINITY;
        top = fmaxf(top, x[j]);
      }
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
      const float m_new = fmaxf(m[i], top);
      const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float p = x[j] == -INFINITY ? 0.f : expf(x[j] - m_new);
        sum += p;
        s.p[ty + 16 * i][tx + 8 * j] = p;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      l[i] = l[i] * corr + sum;
      m[i] = m_new;
      const unsigned long long c2 = twice(corr);
#pragma unroll
      for (int c = 0; c < CP; ++c) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(o[i][c]) : "l"(c2));
    }
    __syncthreads();                                                 // everybody is done with the keys
    if (my_piece == 0) s.key_ok[turn ^ 1][my_key] = next_page >= 0;
    if (more) copy(k_dst, j0 + KEYS, next_page, 0);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    // A weight of zero must not meet an infinity or a NaN among the values of a key that its row does not see: where some
    // row does not see all of the tile, this thread looks at the values that it copied.
    bool broken = false;
    if (j0 + KEYS - 1 > pos0 || j0 < first_visible_key(pos_last, window)) {
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(&s.v[my_key][my_piece * 4 + i * 8]);
        broken = broken || !isfinite(x.x) || !isfinite(x.y) || !isfinite(x.z) || !isfinite(x.w);
      }
    }
    if (__syncthreads_or(broken)) {                                  // the values are there, and everybody's P
#pragma unroll 1
      for (int c = 0; c < KEYS; ++c) {
        ulonglong2 b[(CP + 1) / 2];
#pragma unroll
        for (int h = 0; h < (CP + 1) / 2; ++h) b[h] = *reinterpret_cast<const ulonglong2*>(&s.v[c][h * 32 + tx * 4]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (j0 + c > row_pos[i] || j0 + c < row_first[i]) continue;
          const unsigned long long p2 = twice(s.p[ty + 16 * i][c]);
#pragma unroll
          for (int c2 = 0; c2 < CP; ++c2) fma2(o[i][c2], p2, c2 % 2 ? b[c2 / 2].y : b[c2 / 2].x);
        }
      }
    } else
#pragma unroll 2
    for (int c = 0; c < KEYS; c += 4) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(&s.p[ty + 16 * i][c]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        ulonglong2 b[(CP + 1) / 2];
#pragma unroll
        for (int h = 0; h < (CP + 1) / 2; ++h) b[h] = *reinterpret_cast<const ulonglong2*>(&s.v[c + e][h * 32 + tx * 4]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned long long p2 = twice(e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w);
#pragma unroll
          for (int c2 = 0; c2 < CP; ++c2) fma2(o[i][c2], p2, c2 % 2 ? b[c2 / 2].y : b[c2 / 2].x);
        }
      }
    }
    __syncthreads();                                                 // everybody is done with the values and with P
    if (more) copy(v_dst, j0 + KEYS, next_page, v_half);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = ty + 16 * i;
    if (row >= rows) continue;
    const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
    float* dst = out + (int64_t)(t0 + first + row / g) * out_stride + (int64_t)(kvh * g + row % g) * D;
#pragma unroll
    for (int h = 0; h < (CP + 1) / 2; ++h)
      *reinterpret_cast<float4*>(dst + h * 32 + tx * 4) =
          make_float4(pair_low(o[i][2 * h]) * inv, pair_high(o[i][2 * h]) * inv, pair_low(o[i][2 * h + 1]) * inv, pair_high(o[i][2 * h + 1]) * inv);
  }
}

// ---- single tokens.  One block per (chunk of 128 keys, kv head, token), for up to eight query heads of the kv head at
// a time: a thread scores one key, then adds the values of its columns.  Bound by the cache's bytes once there are a few
// blocks an SM; chunks of 128 keys give a single token over 2,048 keys of 8 kv heads 128 blocks.
constexpr int CHUNK = 128, DEC_HEADS = 8;

template <int D>
__global__ void __launch_bounds__(CHUNK)
attention_f32_single_kernel(const float* __restrict__ q, int64_t q_stride, const float* __restrict__ cache,
                            const int* __restrict__ block_table, int bt_stride, const int* __restrict__ positions,
                            const int* __restrict__ token_row, float* __restrict__ part_o, float* __restrict__ part_ml,
                            int hq, int hkv, int block_size, int num_pages, int chunks, float scale, int window,
                            int* __restrict__ status) {
  __shared__ __align__(16) float q_s[DEC_HEADS][D];
  __shared__ float p_s[DEC_HEADS][CHUNK];
  __shared__ float red[DEC_HEADS][4], red_sum[DEC_HEADS][4];
  __shared__ int64_t base_s[CHUNK];
  __shared__ float o_s[DEC_HEADS][CHUNK];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = blockIdx.x, kvh = blockIdx.y % hkv, n = blockIdx.z, g = hq / hkv;
  const int h0 = kvh * g + (blockIdx.y / hkv) * DEC_HEADS, nh = min(DEC_HEADS, (kvh + 1) * g - h0);
  const int pos = positions[n], start = first_visible_key(pos, window);
  const int j0 = (start / CHUNK + chunk) * CHUNK;
  if (j0 > pos) return;                                  // the merge knows
  const int j = j0 + tid;
  const size_t head_elems = (size_t)block_size * D, page_elems = (size_t)2 * hkv * head_elems;
  int64_t base = -1;
  if (j <= pos && j >= start) {
    const int page = block_table[(int64_t)token_row[n] * bt_stride + j / block_size];
    if (page < 0 || page >= num_pages) atomicOr(status, GLLM_STATUS_PAGE_RANGE);
    else base = (int64_t)((size_t)page * page_elems + (size_t)kvh * head_elems + (size_t)(j % block_size) * D);
  }
  base_s[tid] = base;
  for (int i = tid; i < nh * D; i += CHUNK) q_s[i / D][i % D] = q[(int64_t)n * q_stride + (int64_t)h0 * D + i];
  __syncthreads();
  float dot[DEC_HEADS];
#pragma unroll
  for (int h = 0; h < DEC_HEADS; ++h) dot[h] = 0.f;
  if (base >= 0) {
    const float4* kp = reinterpret_cast<const float4*>(cache + base);
#pragma unroll 8
    for (int c = 0; c < D / 4; ++c) {
      const float4 k = kp[c];
#pragma unroll
      for (int h = 0; h < DEC_HEADS; ++h) {
        if (h < nh) {
          const float4 x = *reinterpret_cast<const float4*>(&q_s[h][c * 4]);
          dot[h] = fmaf(x.x, k.x, fmaf(x.y, k.y, fmaf(x.z, k.z, fmaf(x.w, k.w, dot[h]))));
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < DEC_HEADS; ++h) {
    if (h < nh) {
      dot[h] = base >= 0 ? dot[h] * scale : -INFINITY;
      const float top = warp_max(dot[h]);
      if (lane == 0) red[h][warp] = top;
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < DEC_HEADS; ++h) {
    if (h < nh) {
      const float top = fmaxf(fmaxf(red[h][0], red[h][1]), fmaxf(red[h][2], red[h][3]));
      const float p = dot[h] == -INFINITY ? 0.f : expf(dot[h] - top);
      p_s[h][tid] = p;
      const float sum = warp_sum(p);
      if (lane == 0) red_sum[h][warp] = sum;
    }
  }
  __syncthreads();
  // a thread adds column tid % D over every (CHUNK / D)-th key
  constexpr int SETS = CHUNK / D;
  const int col = tid % D, set = tid / D;
  float acc[DEC_HEADS];
#pragma unroll
  for (int h = 0; h < DEC_HEADS; ++h) acc[h] = 0.f;
  const float* vp = cache + (size_t)hkv * head_elems + col;
  const int last = min(CHUNK, pos - j0 + 1);
#pragma unroll 8
  for (int key = set; key < last; key += SETS) {
    const int64_t b = base_s[key];
    const float v = b >= 0 ? vp[b] : 0.f;
#pragma unroll
    for (int h = 0; h < DEC_HEADS; ++h)
      if (h < nh) acc[h] = fmaf(p_s[h][key], v, acc[h]);
  }
#pragma unroll
  for (int h = 0; h < DEC_HEADS; ++h)
    if (h < nh) o_s[h][tid] = acc[h];
  __syncthreads();
  for (int i = tid; i < nh * D; i += CHUNK) {
    const int h = i / D, c = i % D;
    float v = 0.f;
#pragma unroll
    for (int x = 0; x < SETS; ++x) v += o_s[h][x * D + c];
    part_o[(((int64_t)n * hq + h0 + h) * chunks + chunk) * D + c] = v;
  }
  if (tid < nh) {
    float* ml = part_ml + (((int64_t)n * hq + h0 + tid) * chunks + chunk) * 2;
    ml[0] = fmaxf(fmaxf(red[tid][0], red[tid][1]), fmaxf(red[tid][2], red[tid][3]));
    ml[1] = (red_sum[tid][0] + red_sum[tid][1]) + (red_sum[tid][2] + red_sum[tid][3]);
  }
}

// One warp per (token, query head) puts the chunks' results together, in ascending order.
template <int D>
__global__ void __launch_bounds__(128)
attention_f32_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                           const int* __restrict__ positions, float* __restrict__ out, int64_t out_stride, int n_tokens,
                           int hq, int chunks, int window) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= (int64_t)n_tokens * hq) return;
  const int n = (int)(item / hq);
  const int pos = positions[n], c0 = first_visible_key(pos, window) / CHUNK;
  const int used = min(chunks, pos / CHUNK - c0 + 1);
  const float* ml = part_ml + item * chunks * 2;
  float top = -INFINITY;
  for (int c = lane; c < used; c += 32) top = fmaxf(top, __ldcg(ml + 2 * c));
  top = warp_max(top);
  float l = 0.f, acc[D / 32];
#pragma unroll
  for (int i = 0; i < D / 32; ++i) acc[i] = 0.f;
#pragma unroll 4
  for (int c = 0; c < used; ++c) {
    const float m = __ldcg(ml + 2 * c);
    const float w = m == -INFINITY ? 0.f : expf(m - top);
    l = fmaf(w, __ldcg(ml + 2 * c + 1), l);
#pragma unroll
    for (int i = 0; i < D / 32; ++i) acc[i] = fmaf(w, __ldcg(part_o + (item * chunks + c) * D + lane + 32 * i), acc[i]);
  }
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  float* dst = out + (int64_t)n * out_stride + (int64_t)(item - (int64_t)n * hq) * D;
#pragma unroll
  for (int i = 0; i < D / 32; ++i) dst[lane + 32 * i] = acc[i] * inv;
}

template <int D>
int portions_launch(const float* q, int64_t q_stride, float* out, int64_t out_stride, const float* cache,
                    const int* block_table, int bt_stride, const int* cu_q, const int* ctx_lens, const int* slots,
                    int requests, int max_q_len, int hq, int hkv, int block_size, int num_pages, float scale,
                    int window, int* status, cudaStream_t stream) {
  const int tokens = ROWS / (hq / hkv);
  const int64_t blocks = (int64_t)((max_q_len + tokens - 1) / tokens) * hkv * requests;
  if (blocks > 0x7fffffff) return (int)cudaErrorInvalidValue;
  // Head size 64: a third block on an SM is paid for in registers, which only a grid that has it is to pay: 16 prompts of 16 tokens
  // (128 blocks) 14.9 us with two, 17.1 with three, 4 of 130 (288) 31.9 and 31.4; 16 of 100 (896) 64 and 57, 2,000 tokens (1,000) 627
  // and 569.  The other sizes are left to the compiler (asked for one block, head size 32 took 188 registers for 167 and lost its
  // third one: 3 of 200 tokens behind 300 111 us for 86).
  auto kernel = D != 64 ? attention_f32_portion_kernel<D, 0>
                        : blocks > 2 * gllm_sm_count() ? attention_f32_portion_kernel<D, D == 64 ? 3 : 0>
                                                       : attention_f32_portion_kernel<D, D == 64 ? 1 : 0>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PortionSmem<D>));
  if (e != cudaSuccess) return (int)e;
  // Blocks of unequal length that share SMs do not start early (gllm_launch_in_order): behind another kernel, head size 64, 300 tokens
  // 64 us early and 49 in order, 3 of 200 behind 300 153 and 134, 4 of 130 45 and 35; but 8 of 128 39 and 43, 16 of 100 59 and 61.
  // (With head size 128 a block has an SM to itself: 8 of 128 100 and 102, 1,024 tokens 394 and 396.)
  const bool in_order = D < 128 && max_q_len > 2 * KEYS && blocks > gllm_sm_count();
  auto start = [&](auto launch) {
    return launch(kernel, dim3((unsigned)blocks), dim3(PF_THREADS), sizeof(PortionSmem<D>), stream, q, q_stride, out, out_stride,
                  cache, block_table, bt_stride, cu_q, ctx_lens, slots, requests, hq, hkv, block_size, num_pages, scale, window,
                  status);
  };
  if (in_order) return start([](auto... a) { return gllm_launch_in_order(a...); });
  return start([](auto... a) { return gllm_launch(a...); });
}

template <int D>
int singles_launch(const float* q, int64_t q_stride, float* out, int64_t out_stride, const float* cache,
                   const int* block_table, int bt_stride, const int* positions, const int* token_row, int n_tokens,
                   float* part_o, float* part_ml, int hq, int hkv, int block_size, int num_pages, int chunks,
                   float scale, int window, int* status, cudaStream_t stream) {
  const int sets = (hq / hkv + DEC_HEADS - 1) / DEC_HEADS;
  int rc = gllm_launch(attention_f32_single_kernel<D>, dim3(chunks, hkv * sets, n_tokens), dim3(CHUNK), 0, stream, q,
                       q_stride, cache, block_table, bt_stride, positions, token_row, part_o, part_ml, hq, hkv,
                       block_size, num_pages, chunks, scale, window, status);
  if (rc != 0) return rc;
  return gllm_launch(attention_f32_merge_kernel<D>, dim3((unsigned)(((int64_t)n_tokens * hq + 3) / 4)), dim3(128), 0,
                     stream, part_o, part_ml, positions, out, out_stride, n_tokens, hq, chunks, window);
}
}  // namespace

// Portions of prompts: request r owns tokens cu_q[r] .. cu_q[r+1]-1 after ctx_lens[r] cached ones.
GLLM_API int gllm_attention_f32_portions(const float* q, int64_t q_stride, float* out, int64_t out_stride,
                                         const float* cache, const int* block_table, int bt_stride, const int* cu_q,
                                         const int* ctx_lens, const int* slots, int requests, int max_q_len, int hq,
                                         int hkv, int d, int block_size, int num_pages, float scale, int window,
                                         int* status, cudaStream_t stream) {
  if (requests <= 0 || max_q_len <= 0) return 0;
  if (hq <= 0 || hkv <= 0 || hq % hkv || hq / hkv > ROWS || hkv > 65535 || requests > 65535) return (int)cudaErrorInvalidValue;
#define GLLM_F32_PORTIONS(D)                                                                                          \
  if (d == D)                                                                                                         \
    return portions_launch<D>(q, q_stride, out, out_stride, cache, block_table, bt_stride, cu_q, ctx_lens, slots,      \
                              requests, max_q_len, hq, hkv, block_size, num_pages, scale, window, status, stream);
  GLLM_F32_PORTIONS(32) GLLM_F32_PORTIONS(64) GLLM_F32_PORTIONS(128)
#undef GLLM_F32_PORTIONS
  return (int)cudaErrorInvalidValue;
}

// Single tokens; `chunks` spans of gllm_attention_f32_chunk() keys cover what any of them sees.
GLLM_API int gllm_attention_f32_chunk() { return CHUNK; }
GLLM_API int gllm_attention_f32_singles(const float* q, int64_t q_stride, float* out, int64_t out_stride,
                                        const float* cache, const int* block_table, int bt_stride,
                                        const int* positions, const int* token_row, int n_tokens, float* part_o,
                                        float* part_ml, int hq, int hkv, int d, int block_size, int num_pages,
                                        int chunks, float scale, int window, int* status, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (hq <= 0 || hkv <= 0 || hq % hkv || chunks <= 0 || n_tokens > 65535 || (int64_t)hkv * ((hq / hkv + 7) / 8) > 65535)
    return (int)cudaErrorInvalidValue;
#define GLLM_F32_SINGLES(D)                                                                                           \
  if (d == D)                                                                                                         \
    return singles_launch<D>(q, q_stride, out, out_stride, cache, block_table, bt_stride, positions, token_row,       \
                             n_tokens, part_o, part_ml, hq, hkv, block_size, num_pages, chunks, scale, window, status, \
                             stream);
  GLLM_F32_SINGLES(32) GLLM_F32_SINGLES(64) GLLM_F32_SINGLES(128)
#undef GLLM_F32_SINGLES
  return (int)cudaErrorInvalidValue;
}
