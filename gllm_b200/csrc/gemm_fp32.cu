// True 32-bit matrix product C[M,N] = X[M,K] * W[N,K]^T, the `x @ W.T` of
// gllm/model/layers/linear.py:20 with W stored [out, in].  This is the path
// that shows faults bf16 hides: no operand is rounded.
//
// Three kernels.  Rows on 16-byte boundaries and K a multiple of 4 run, up to
// K = 512, on packed 32-bit multiply-adds (tiles of 16 x 16 to 64 x 64), and
// beyond on the tensor cores with every 32-bit number cut into three bfloat16
// whose sum it is (8 bits of its significand each, rounded to nearest; times
// 2^16 first, so that nothing is lost of the smallest numbers either):
//   x = x0 + x1 + x2,  w = w0 + w1 + w2,
//   x w = w0 x0 + (w0 x1 + w1 x0 + w0 x2 + w1 x1 + w2 x0) + terms of up to 2^-24 |x w|.
// Everything else runs a plain 64 x 64 tile of 32-bit multiply-adds.  In both
// multiply-add kernels an output is two sums, of even and odd k or of the first
// and second half.
//
// The tensor cores' own additions truncate.  The leading products' accumulator
// is therefore taken out of tensor memory every 128 .. 256 of K (chunk_of) and
// added to 32-bit sums in registers, rounded to nearest; the other five
// products are 2^-8 of it and stay in theirs for a whole range of K.
//
// K is cut into ranges that depend on (N, K) alone.  A work item is a tile of
// 128 weight rows x BT tokens times one range (few tokens: the blocks of a
// tile's ranges are a cluster and add up through shared memory) or all ranges
// one after the other; the ranges' sums are added in ascending order either
// way, so a token's result does not depend on the batch it is in.
//
// A result that is not finite is computed again with 32-bit multiply-adds from
// the operands themselves: the parts of an infinity are not its sum, and sums
// that are 2^32 times too large may end where the result does not (from 2^96 on,
// or with operands from 2^111 on).
//
// What bounds it: with many tokens the cutting (sixteen warps, about 400 issue
// cycles for a block of 32 k) and shared memory (110 KB, 860 cycles), where the
// products of 96 tokens take 583; with few the same chain at half of what
// DRAM gives.  700 x 16,384 x 2,048: 266 us = 177 TFLOP/s, 1,014 us with
// packed multiply-adds on the CUDA cores; 700 x 2,048 x 8,192: 148 for 627;
// 8 x 16,384 x 2,048: 28 for 79; 300 x 2,048 x 2,048: 42 for 108.  Relative
// error against 64 bits at K = 1,024, 2,048 and 8,192: 1.3e-7, 1.7e-7 and
// 2.4e-7 for 4.1e-7, 5.7e-7 and 1.1e-6; operands of one sign 1.7e-7, 2.8e-7 ..
// 3.3e-7 and 3.8e-7 for 2.5e-7, 3.5e-7 and 7.0e-7.
#include "umma_utils.cuh"

namespace {
// ------------------------------------------------------------------ plain tile
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;  // 256 threads

__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N,
                int K, int64_t lda, int64_t ldb, int64_t ldc) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // Two sums an output, of the first half of the k-tiles and of the rest: an addition's rounding is that of a sum half as long.
  // (Sums of even and of odd k, live side by side in the loop, took 364 us for 700 x 2,048 x 2,049, one sum and these 254.)
  float acc[TM][TN], first[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  // each thread loads 4 elements of A and 4 of B per k-tile
  const int lrow = tid / 4;        // 0..63
  const int lk = (tid % 4) * 4;    // 0,4,8,12
  const int half = (K + BK - 1) / BK / 2 * BK;
  for (int part = 0; part < 2; ++part) {
    for (int k0 = part == 0 ? 0 : half; k0 < (part == 0 ? half : K); k0 += BK) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = k0 + lk + e;
        const int am = m0 + lrow, bn = n0 + lrow;
        As[lk + e][lrow] = (am < M && k < K) ? A[(int64_t)am * lda + k] : 0.f;
        Bs[lk + e][lrow] = (bn < N && k < K) ? B[(int64_t)bn * ldb + k] : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        float a[TM], b[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx * TN + j];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
    }
    if (part == 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) first[i][j] = acc[i][j], acc[i][j] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n < N) C[(int64_t)m * ldc + n] = first[i][j] + acc[i][j];
    }
  }
}

// ------------------------------------------------------------------ packed multiply-adds
// Rows lie in shared memory as they do in memory, [row][k], filled by cp.async several k-tiles ahead.
// A thread owns TM x TN outputs (rows and columns TY and TX apart).  Four k at a time it reads 16 bytes of each of its
// rows and multiplies them as two packed pairs (fma.rn.f32x2), so an output is kept as two sums, of the products with
// even and with odd k, each in ascending order; they are added at the end.
constexpr int PK = 32, PITCH = PK + 4;   // (a pitch of 9 sixteen-byte pieces: eight neighbouring rows on eight bank groups)

template <int BM_, int BN_, int TM_, int TN_, int STAGES, int UNROLL>
__global__ void __launch_bounds__((BM_ / TM_) * (BN_ / TN_))
gemm_f32_pairs_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N,
                      int K, int64_t lda, int64_t ldb, int64_t ldc) {
  constexpr int TY = BM_ / TM_, TX = BN_ / TN_, THREADS = TX * TY, ROWS = BM_ + BN_;
  static_assert(TX % 8 == 0 && TY % 4 == 0, "a warp's threads lie 4 by 8");
  extern __shared__ __align__(16) float tiles[];          // [STAGES][BM_ + BN_][PITCH]
  pdl_trigger();
  // A warp's threads lie 4 rows by 8 columns, a half warp 4 by 4: a 16-byte load is served a half warp at a time when
  // its addresses fit one pass over the banks, so neither operand's load takes more than two.
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (warp % (TX / 8)) * 8 + (lane & 3) + (lane >> 4) * 4, ty = (warp / (TX / 8)) * 4 + ((lane >> 2) & 3);
  const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN_;
  // a thread copies piece `piece` of the rows row0, row0 + STEP, ...: of A's first, of B's behind them
  constexpr int PIECES = PK / 4, STEP = THREADS / PIECES, COPIES = ROWS / STEP;
  static_assert(THREADS % PIECES == 0 && BM_ % STEP == 0 && BN_ % STEP == 0, "whole rows per round of copies");
  const int piece = tid % PIECES, row0 = tid / PIECES;
  const float* a_src = A + (int64_t)(m0 + row0) * lda + piece * 4;
  const float* b_src = B + (int64_t)(n0 + row0) * ldb + piece * 4;
  const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(tiles) + (uint32_t)((row0 * PITCH + piece * 4) * sizeof(float));
  auto request = [&](int k0, int stage) {
    const bool k_in = k0 + piece * 4 < K;
    const uint32_t dst = dst0 + (uint32_t)(stage * ROWS * PITCH * sizeof(float));
#pragma unroll
    for (int c = 0; c < COPIES; ++c) {
      const bool is_a = c < BM_ / STEP;
      const int r = is_a ? c * STEP : c * STEP - BM_;
      const bool in = k_in && (is_a ? m0 + row0 + r < M : n0 + row0 + r < N);
      const float* src = is_a ? a_src + k0 + r * lda : b_src + k0 + r * ldb;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(c * STEP * PITCH * sizeof(float))),
                   "l"(in ? src : A), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned long long acc[TM_][TN_];
#pragma unroll
  for (int i = 0; i < TM_; ++i)
#pragma unroll
    for (int j = 0; j < TN_; ++j) acc[i][j] = 0ull;
  const int k_tiles = (K + PK - 1) / PK;
  pdl_wait();
#pragma unroll
  for (int t = 0; t < STAGES - 1; ++t) {
    if (t < k_tiles) request(t * PK, t);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int stage = 0;
  for (int t = 0; t < k_tiles; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                       // tile t is there, and nobody reads tile t - 1 any more
    const int ahead = t + STAGES - 1;
    if (ahead < k_tiles) request(ahead * PK, stage == 0 ? STAGES - 1 : stage - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const float* a_s = tiles + (stage * ROWS + ty) * PITCH;
    const float* b_s = tiles + (stage * ROWS + BM_ + tx) * PITCH;
#pragma unroll UNROLL
    for (int kk = 0; kk < PK; kk += 4) {
      ulonglong2 a[TM_];
#pragma unroll
      for (int i = 0; i < TM_; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a_s + i * TY * PITCH + kk);
#pragma unroll
      for (int j = 0; j < TN_; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(b_s + j * TX * PITCH + kk);
#pragma unroll
        for (int i = 0; i < TM_; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < TM_; ++i) fma2(acc[i][j], a[i].y, b.y);
      }
    }
    stage = stage + 1 == STAGES ? 0 : stage + 1;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int i = 0; i < TM_; ++i) {
    const int m = m0 + ty + i * TY;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN_; ++j) {
      const int n = n0 + tx + j * TX;
      if (n < N)
        C[(int64_t)m * ldc + n] = pair_sum(acc[i][j]);
    }
  }
}

template <int BM_, int BN_, int TM_, int TN_, int STAGES, int UNROLL>
int gemm_f32_pairs(const float* A, const float* B, float* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                   cudaStream_t stream) {
  constexpr size_t smem = sizeof(float) * STAGES * (BM_ + BN_) * PITCH;
  auto kernel = gemm_f32_pairs_kernel<BM_, BN_, TM_, TN_, STAGES, UNROLL>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return (int)e;
  // (tiles of rows lie along y, at most 65,535 a launch)
  for (int m0 = 0; m0 < M; m0 += 65535 * BM_) {
    const int rows = M - m0 < 65535 * BM_ ? M - m0 : 65535 * BM_;
    const dim3 grid((N + BN_ - 1) / BN_, (rows + BM_ - 1) / BM_);
    // Blocks that start while the kernel before them drains land wherever a place frees first.  Asking for a share of an
    // SM's shared memory that lets no SM take more than its even share of the blocks keeps them spread.
    const int64_t per_sm = ((int64_t)grid.x * grid.y + gllm_sm_count() - 1) / gllm_sm_count();
    const int64_t share = 228 * 1024 / per_sm - 1024;            // (1 KB of every block's share is the system's)
    const size_t ask = share > (int64_t)smem ? (size_t)(share < 227 * 1024 ? share : 227 * 1024) : smem;
    const int rc = gllm_launch(kernel, grid, dim3((BM_ / TM_) * (BN_ / TN_)), ask, stream, A + (int64_t)m0 * lda, B,
                               C + (int64_t)m0 * ldc, rows, N, K, lda, ldb, ldc);
    if (rc != 0) return rc;
  }
  return 0;
}
// Which tile: the one whose fullest SM ends first.  A tile's time per k is `chain` (ns) while it has an SM to itself and
// `work` times the tiles of the SM once they fill it; tiles of two warps count in pairs (an SM has four schedulers).
// Measured per tile at K = 8,192 and 148 SMs (one tile an SM; 10 and more): the larger a tile the less it reads per
// product, the smaller the better it spreads.  Steps of up to 16 tokens take the smallest tile, which streams the
// weight best (16,384 x 2,048: 64 us against 95 with 32 x 32).
int pairs_tile_of(int M, int N) {
  struct Tile { int m, n, pairs; float chain, work; };
  static const Tile tiles[] = {{16, 16, 1, 10.4f, 3.66f}, {32, 16, 1, 13.2f, 5.2f}, {32, 32, 1, 19.4f, 7.4f},
                               {64, 32, 1, 30.f, 13.8f}, {64, 64, 0, 33.7f, 26.4f}, {64, 64, 1, 56.4f, 25.f}};
  if (M <= 16) return 0;
  int best = 0;
  float best_time = 0.f;
  for (int i = 0; i < 6; ++i) {
    const Tile& t = tiles[i];
    int64_t per_sm = ((int64_t)((M + t.m - 1) / t.m) * ((N + t.n - 1) / t.n) + gllm_sm_count() - 1) / gllm_sm_count();
    if (t.pairs) per_sm = (per_sm + 1) & ~(int64_t)1;
    const float work = t.work * (float)per_sm, time = work > t.chain ? work : t.chain;
    if (i == 0 || time < best_time) best = i, best_time = time;
  }
  return best;
}

// ------------------------------------------------------------------ three parts a number, on the tensor cores
namespace parts3 {
constexpr int ROWS = 128;           // weight rows of a tile (MMA M)
constexpr int KB = 32;              // k per block: 32 floats = one 128-byte swizzle row, 32 bf16 = one of 64 bytes
constexpr int WORKERS = 16;         // warps that cut operands into parts and keep the sums
constexpr int GROUPS = 4;           // of workers, that take turns with the blocks
constexpr int THREADS = (WORKERS + 2) * 32;
constexpr int RANGE_BLOCKS = 64;    // longest range of K (2,048), as long as there are at most 16 of them
constexpr int MOST_RANGES = 16;     // (eight where they are a cluster's blocks)
constexpr int MOST_BLOCKS = 8;
constexpr int A_COLS = 3 * KB / 2;  // tensor-memory columns of one block of the weight's parts
constexpr float UP = 65536.f;       // operands are cut times 2^16: the last bit of the smallest number is then one bfloat16 has
constexpr float DOWN = 1.f / (UP * UP);

template <int BT>
struct Shape {
  static constexpr int RAW = (ROWS + BT) * KB * 4;
  // blocks of parts in flight: no fewer than GROUPS (a group waits for one phase of a stage), more where tensor memory has room,
  // so that the groups do not fall into step with the products
  static constexpr int CUT = BT <= 32 ? 8 : 4;
  static constexpr int PARTS = ((3 * BT * KB * 2 + 1023) / 1024) * 1024;
  static constexpr int STAGES_ = (224 * 1024 - CUT * PARTS) / RAW;
  static constexpr int STAGES = STAGES_ > 8 ? 8 : STAGES_;                 // raw blocks in flight
  static constexpr int CROSS = BT <= 80 ? 2 : 1;                           // accumulators of the five smaller products
  static constexpr int COLS = (2 + CROSS) * BT + CUT * A_COLS;
  static constexpr int TMEM_COLS = COLS <= 256 ? 256 : 512;
  static constexpr int SMEM = STAGES * RAW + CUT * PARTS + 1024;
  static_assert(COLS <= 512 && CUT >= GROUPS && STAGES >= CUT, "fits, and no wait is more than a phase behind");
};

// Shared-memory descriptor of a K-major tile with rows of 64 bytes, 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t desc64(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)4 << 61);
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(taddr));
}
// sum[i] += the accumulator's columns taddr + i of this thread's row
template <int C>
__device__ __forceinline__ void add_columns(uint32_t taddr, float (&sum)[C]) {
  constexpr int STEP = C % 8 == 0 ? 8 : 4;
#pragma unroll
  for (int c = 0; c < C; c += STEP) {
    float v[STEP];
    if constexpr (STEP == 8) tmem_ld8_nowait(taddr + (uint32_t)c, v);
    else tmem_ld4_nowait(taddr + (uint32_t)c, v);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < STEP; ++i) {
      asm volatile("" : "+f"(v[i])::"memory");             // (not read ahead of the wait)
      sum[c + i] += v[i];
    }
  }
}

__device__ __forceinline__ uint32_t pack2(float low, float high) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ unsigned long long pair_of(float low, float high) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(low), "f"(high));
  return v;
}
// Eight numbers, times 2^16, as three parts each, two to a word.
__device__ __forceinline__ void cut8(const float4& a, const float4& b, uint32_t (&p)[3][4]) {
  const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned long long left = pair_of(x[2 * i], x[2 * i + 1]);
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(left) : "l"(pair_of(UP, UP)));
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      const uint32_t w = pack2(pair_low(left), pair_high(left));
      p[part][i] = w;                                      // (exact: what is left has no more bits than the number had)
      asm("sub.rn.f32x2 %0, %0, %1;" : "+l"(left) : "l"(pair_of(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u))));
    }
  }
}

struct Cut {                        // how the work is laid out
  int tiles_n, tiles_m;             // tiles of weight rows, of tokens
  int ranges, range_blocks, blocks; // of K
  int chunk, extra;                 // blocks between two visits to the leading accumulator; more in a range's first
  int split;                        // 1: an item is one range of a tile, a block each, a cluster a tile; 0: all of them
};

// Item w: neighbouring CTAs share a tile of weight rows (or take the ranges of one).
template <int BT>
__device__ __forceinline__ void place(const Cut& cut, int w, int& n0, int& m0, int& kb_begin, int& kb_end, int& range) {
  range = 0;
  if (cut.split) {
    range = w % cut.ranges;
    w /= cut.ranges;
  }
  const int tn = w / cut.tiles_m, tm = w - tn * cut.tiles_m;
  n0 = tn * ROWS, m0 = tm * BT;
  kb_begin = cut.split ? range * cut.range_blocks : 0;
  kb_end = cut.split ? min(cut.blocks, kb_begin + cut.range_blocks) : cut.blocks;
}

__device__ __forceinline__ bool is_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool any_of_workers(bool mine) {          // (a barrier of theirs as well)
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"(mine ? 1u : 0u), "n"(WORKERS * 32)
      : "memory");
  return any != 0;
}
// The results that are not finite, of the weight rows n0 .. n0 + rows and the tokens m0 .. m0 + BT, once more with 32-bit
// multiply-adds (two sums each, of even and of odd k) by all workers, who are done with the stages: their memory holds the tiles.
// A thread takes rows 32 and columns 16 apart; a warp's threads lie 4 rows by 8 columns, a half warp 4 by 4.  What bounds it: the
// shared-memory loads.  700 x 16,384 x 2,048 with a NaN in one token 784 us, in every token 2,030; 669 and 34,400 when a thread
// walked a weight row for each result, 1,020 where all of it is multiply-adds.
template <int BT>
__device__ __noinline__ void once_more(const float* __restrict__ X, const float* __restrict__ W, float* out, int M, int N, int K,
                                       int64_t ldx, int64_t ldw, int64_t ldo, int n0, int rows, int m0) {
  extern __shared__ unsigned char smem_dyn[];
  constexpr int PITCH_ = KB + 4, COLS = BT / 16, LINES = ROWS + BT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ty = (warp >> 1) * 4 + ((lane >> 2) & 3), tx = (warp & 1) * 8 + (lane & 3) + (lane >> 4) * 4;
  const int count = min(rows, N - n0), tokens = min(BT, M - m0);
  auto at = [&](int i, int j) { return out + (int64_t)(m0 + tx + 16 * j) * ldo + n0 + ty + 32 * i; };
  uint32_t need = 0;                                       // the columns (of 16 apart) that this warp has to do
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < COLS; ++j)
      if (ty + 32 * i < count && tx + 16 * j < tokens && !is_finite(__ldcg(at(i, j)))) need |= 1u << j;
  need = __reduce_or_sync(0xffffffffu, need);
  if (!any_of_workers(need != 0)) return;
  const uint32_t base = (smem_addr(smem_dyn) + 15u) & ~15u;
  const float* const tiles = reinterpret_cast<const float*>(smem_dyn + (base - smem_addr(smem_dyn)));
  auto request = [&](int k0, int stage) {
    for (int p = threadIdx.x; p < LINES * (KB / 4); p += WORKERS * 32) {
      const int line = p / (KB / 4), k = k0 + p % (KB / 4) * 4;
      const bool of_w = line < ROWS, in = k < K && (of_w ? line < count : line - ROWS < tokens);
      const float* src = !in ? W : of_w ? W + (int64_t)(n0 + line) * ldw + k : X + (int64_t)(m0 + line - ROWS) * ldx + k;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (uint32_t)((stage * LINES + line) * PITCH_ + k - k0) * 4u),
                   "l"(src), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned long long sum[4][COLS];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[i][j] = 0ull;
  constexpr int AHEAD = 3;                                 // tiles in flight
  static_assert((AHEAD + 1) * LINES * PITCH_ * 4 <= Shape<BT>::STAGES * Shape<BT>::RAW, "the stages' memory");
  for (int t = 0; t < AHEAD; ++t) request(t * KB, t);
  for (int k0 = 0, stage = 0; k0 < K; k0 += KB, stage = (stage + 1) & AHEAD) {
    asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
    any_of_workers(false);                                 // the tile is there, and nobody reads the one before any more
    request(k0 + AHEAD * KB, (stage + AHEAD) & AHEAD);
    const float* w_s = tiles + (stage * LINES + ty) * PITCH_;
    const float* x_s = tiles + (stage * LINES + ROWS + tx) * PITCH_;
    if (!need) continue;
#pragma unroll 2
    for (int k = 0; k < KB; k += 4) {
      ulonglong2 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const ulonglong2*>(w_s + 32 * i * PITCH_ + k);
#pragma unroll
      for (int j = 0; j < COLS; ++j) {
        if (!(need >> j & 1)) continue;
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(x_s + 16 * j * PITCH_ + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) fma2(sum[i][j], w[i].x, x.x), fma2(sum[i][j], w[i].y, x.y);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < COLS; ++j)
      if (ty + 32 * i < count && tx + 16 * j < tokens && !is_finite(__ldcg(at(i, j)))) *at(i, j) = pair_sum(sum[i][j]);
  asm volatile("cp.async.wait_all;" ::: "memory");
  any_of_workers(false);                                   // (the next tile goes over this one)
}
// The sum of one range of several, out of the accumulators.  Additions in memory take what is subnormal for zero.  Sums of 2^-102 and
// more (and zeros) add up to nothing subnormal, as their last bits are 2^-125 and more; a smaller one becomes a NaN, and the
// result is computed again.
constexpr uint32_t LEAST = (uint32_t)(127 - 102) << 24;    // 2^-102, without its sign
__device__ __forceinline__ float range_sum(float v) {
  return (__float_as_uint(v) << 1) - 1u < LEAST - 1u ? __uint_as_float(0x7fffffffu) : v;
}
// 0xff000000 - LEAST and more: v is zero, smaller than 2^-102 or not finite.
__device__ __forceinline__ uint32_t unusual(float v) { return (__float_as_uint(v) << 1) - LEAST; }
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// The sum of a range of an item, columns c0 .. of one of its rows: behind the item's first range it joins what this thread
// has written of the ranges before.  `broken`: some sum was not finite.
template <int BT, int COLS>
__device__ __forceinline__ void put_range(const Cut& cut, int item, int end, int row, int c0, const float (&acc)[COLS],
                                          float* out, int M, int N, int64_t ldo, bool& broken) {
  int n0, m0, kb_begin, kb_end, range;
  place<BT>(cut, item, n0, m0, kb_begin, kb_end, range);
  const int n = n0 + row, m = m0 + c0, tokens = min(COLS, M - m);
  if (n >= N || tokens <= 0) return;
  float* const dst = out + (int64_t)m * ldo + n;
  const bool joins = end > cut.range_blocks;
  float v[COLS];
  uint32_t most = 0;
#pragma unroll
  for (int i = 0; i < COLS; ++i) {
    v[i] = acc[i] * DOWN;
    most = max(most, unusual(v[i]));
  }
  if (most >= 0xff000000u - LEAST) {                       // (the columns behind the last token are zero: rare but there)
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
      if (cut.ranges > 1) v[i] = range_sum(v[i]);
      broken = broken || !is_finite(v[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < COLS; ++i) {
    if (i < tokens) {
      if (joins) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(dst + i * ldo), "f"(v[i]) : "memory");   // (nothing to wait for)
      else dst[i * ldo] = v[i];
    }
  }
}

// Warps 0..15 cut the operands into parts (the weight's into tensor memory, the MMA's A operand; the tokens' into shared
// memory, its B operand) and keep the sums: warp w the tile's rows 32 (w % 4) .. and a quarter of its columns.  Warp 16
// requests the operands by TMA, warp 17 issues the products.  Weight parts in tensor memory: a product of 16 tokens
// then takes 16 cycles, with both operands in shared memory 40; of 96 tokens 49 cycles for 3 KB of shared memory instead of 7, and
// what is left of the 128 bytes a cycle is needed for the cutting.
template <int BT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_parts_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ out, int M, int N, int K,
                      int64_t ldx, int64_t ldw, int64_t ldo, Cut cut, int num_items, int* __restrict__ status) {
  using S = Shape<BT>;
  constexpr int COLS = BT / 4;      // columns of a worker
  extern __shared__ unsigned char smem_dyn[];
  __shared__ __align__(8) uint64_t raw_full[S::STAGES], raw_empty[S::STAGES], cut_full[S::CUT], cut_empty[S::CUT], main_full[2],
      main_empty[2], cross_empty[S::CROSS];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t raw_base = (smem_addr(smem_dyn) + 1023u) & ~1023u, parts_base = raw_base + S::STAGES * S::RAW;
  unsigned char* raw_ptr = smem_dyn + (raw_base - smem_addr(smem_dyn));
  unsigned char* parts_ptr = raw_ptr + S::STAGES * S::RAW;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) mbar_init(smem_addr(&raw_full[s]), 1), mbar_init(smem_addr(&raw_empty[s]), WORKERS / GROUPS);
    for (int s = 0; s < S::CUT; ++s) mbar_init(smem_addr(&cut_full[s]), WORKERS / GROUPS), mbar_init(smem_addr(&cut_empty[s]), 1);
    for (int b = 0; b < 2; ++b) mbar_init(smem_addr(&main_full[b]), 1), mbar_init(smem_addr(&main_empty[b]), WORKERS);
    for (int b = 0; b < S::CROSS; ++b) mbar_init(smem_addr(&cross_empty[b]), WORKERS);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WORKERS + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)),
                 "r"((uint32_t)S::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_main = tmem_base_slot, tmem_cross = tmem_main + 2 * BT, tmem_parts = tmem_cross + S::CROSS * BT;

  if (warp == WORKERS) {
    // ------------------------------------------------------------ operands by TMA
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      pdl_wait();                                          // (either operand may be what the kernel before writes)
      for (int w = blockIdx.x; w < num_items && ok; w += gridDim.x) {
        int n0, m0, kb_begin, kb_end, range;
        place<BT>(cut, w, n0, m0, kb_begin, kb_end, range);
        for (int kb = kb_begin; kb < kb_end; ++kb, ++it) {
          const uint32_t s = it % S::STAGES, round = it / S::STAGES, bar = smem_addr(&raw_full[s]);
          const uint32_t dst = raw_base + s * S::RAW;
          if (round > 0) {
            ok = mbar_wait(smem_addr(&raw_empty[s]), (round & 1u) ^ 1u, status, &abort_flag);
            if (!ok) break;
          }
          mbar_expect_tx(bar, (uint32_t)S::RAW);
          tma_load_2d(dst, &map_w, kb * KB, n0, bar);
          tma_load_2d(dst + ROWS * KB * 4, &map_x, kb * KB, m0, bar);
        }
      }
      if (abort_flag) {
        // let the copies already issued land before the CTA leaves (bounded)
        const uint32_t first = it > (uint32_t)S::STAGES ? it - S::STAGES : 0u;
        for (uint32_t i = first; i < it; ++i) {
          const unsigned long long t0 = global_timer();
          while (!mbar_try_wait(smem_addr(&raw_full[i % S::STAGES]), (i / S::STAGES) & 1u)) {
            if (global_timer() - t0 > UMMA_WAIT_LIMIT_NS) break;
          }
        }
      }
    }
    __syncwarp();
    if (cut.split) cluster_barrier(), cluster_barrier();
  } else if (warp == WORKERS + 1) {
    // ------------------------------------------------------------ products (the whole warp converged, one elected thread)
    const bool leader = elect_one();
    auto wait_u = [&](uint64_t* bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, mbar_wait(smem_addr(bar), parity, status, &abort_flag)) != 0;
    };
    constexpr uint32_t idesc = umma_idesc(ROWS, BT);
    uint32_t it = 0, chunks = 0, segments = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < num_items && ok; w += gridDim.x) {
      int n0, m0, kb_begin, kb_end, range;
      place<BT>(cut, w, n0, m0, kb_begin, kb_end, range);
      for (int r0 = kb_begin; r0 < kb_end && ok; r0 += cut.range_blocks, ++segments) {
        const int r1 = min(kb_end, r0 + cut.range_blocks);
        const uint32_t cb = segments % S::CROSS;
        ok = wait_u(&cross_empty[cb], ((segments / S::CROSS) & 1u) ^ 1u);
        if (!ok) break;
        const uint32_t d_cross = tmem_cross + cb * BT;
        for (int kb = r0, in_chunk = 0, len = cut.chunk + cut.extra; kb < r1; ++kb, ++it) {
          const bool chunk_first = in_chunk == 0, chunk_last = in_chunk + 1 == len || kb + 1 == r1;
          const uint32_t mb = chunks & 1u, d_main = tmem_main + mb * BT;
          if (chunk_first) {
            ok = wait_u(&main_empty[mb], ((chunks >> 1) & 1u) ^ 1u);
            if (!ok) break;
          }
          const uint32_t s = it % S::CUT;
          ok = wait_u(&cut_full[s], (it / S::CUT) & 1u);
          if (!ok) break;
          const uint32_t a0 = tmem_parts + s * A_COLS;
          const uint64_t b0 = desc64(parts_base + s * S::PARTS);
          constexpr uint64_t PART = (BT * KB * 2) >> 4;    // from one part of the tokens to the next
          if (leader) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int k = 0; k < KB / 16; ++k) {
              const uint32_t a = a0 + k * 8;
              const uint64_t b = b0 + (uint64_t)((k * 32) >> 4);
              umma_bf16_ts(d_main, a, b, idesc, (!chunk_first || k > 0) ? 1u : 0u);
              umma_bf16_ts(d_cross, a, b + PART, idesc, (kb > r0 || k > 0) ? 1u : 0u);
              umma_bf16_ts(d_cross, a + KB / 2, b, idesc, 1u);
              umma_bf16_ts(d_cross, a, b + 2 * PART, idesc, 1u);
              umma_bf16_ts(d_cross, a + KB / 2, b + PART, idesc, 1u);
              umma_bf16_ts(d_cross, a + KB, b, idesc, 1u);
            }
            umma_commit(smem_addr(&cut_empty[s]));
            if (chunk_last) umma_commit(smem_addr(&main_full[mb]));
          }
          __syncwarp();
          if (chunk_last) ++chunks, in_chunk = 0, len = cut.chunk;
          else ++in_chunk;
        }
      }
    }
    if (cut.split) cluster_barrier(), cluster_barrier();
  } else {
    // ------------------------------------------------------------ parts and sums
    pdl_wait();                                            // nothing is written before the previous kernel is done
    // the sums: this warp's rows 32 * quarter .., columns side * COLS ..
    const int quarter = warp & 3, side = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    // the parts: blocks are taken in turn by GROUPS groups of warps; of a block, a thread cuts A_K of its weight row's 32 k
    // and B_PIECES times eight k of a token's row
    constexpr int SIDES = WORKERS / GROUPS / 4, A_K = KB / SIDES;
    constexpr int GROUP_THREADS = WORKERS / GROUPS * 32;
    constexpr int B_PIECES = 4 * BT <= GROUP_THREADS ? 1 : 4 * BT <= 2 * GROUP_THREADS ? 2 : 4;
    const uint32_t group = (uint32_t)side / SIDES;
    const int a_side = side % SIDES;
    const int g_tid = (int)threadIdx.x - (int)group * GROUP_THREADS;
    const int b_row = g_tid / (4 / B_PIECES), b_piece = g_tid % (4 / B_PIECES) * B_PIECES;
    const bool has_b = b_row < BT;
    float acc[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
    uint32_t it = 0, chunks = 0, segments = 0;
    bool ok = true;
    auto wait_u = [&](uint64_t* bar, uint32_t parity) -> bool {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_addr(bar), parity, status, &abort_flag)) != 0;
      return ok;
    };
    // the chunk that waits to be added: of which item; where its range ends, if with it
    bool pending = false, broken = false;                  // (broken: some sum was not finite)
    int p_item = 0, p_end = 0;
    for (int item = blockIdx.x; ok; item += gridDim.x) {
      int n0, m0, kb_begin = 0, kb_end = 1, range;
      const bool more = item < num_items;                  // (behind the last item the pending chunk is left)
      if (more) place<BT>(cut, item, n0, m0, kb_begin, kb_end, range);
      for (int r0 = kb_begin; r0 < kb_end && ok; r0 += cut.range_blocks) {
        const int r1 = min(kb_end, r0 + cut.range_blocks);
        for (int c0 = r0, len = cut.chunk + cut.extra; c0 < r1 && ok; c0 += len, len = cut.chunk) {
          const int blocks = more ? min(len, r1 - c0) : 0;
          // this group's blocks of the chunk
          for (int j = (group - it) % GROUPS; ok; j += GROUPS) {
            if (j < blocks) {
              const uint32_t at = it + j, rs = at % S::STAGES, cs = at % S::CUT;
              if (!wait_u(&cut_empty[cs], ((at / S::CUT) & 1u) ^ 1u) || !wait_u(&raw_full[rs], (at / S::STAGES) & 1u)) break;
              const unsigned char* raw = raw_ptr + rs * S::RAW;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint32_t ta = tmem_parts + cs * A_COLS + lanes + a_side * (A_K / 2);
#pragma unroll
              for (int i = 0; i < A_K / 8; ++i) {
                const int e = a_side * (A_K / 4) + 2 * i;
                const float4 lo = *reinterpret_cast<const float4*>(raw + row * 128 + ((e ^ (row & 7)) << 4));
                const float4 hi = *reinterpret_cast<const float4*>(raw + row * 128 + (((e + 1) ^ (row & 7)) << 4));
                uint32_t parts[3][4];
                cut8(lo, hi, parts);
#pragma unroll
                for (int p = 0; p < 3; ++p) tmem_st4(ta + p * (KB / 2) + i * 4, parts[p]);
              }
              if (has_b) {
                const unsigned char* b_raw = raw + ROWS * 128 + b_row * 128;
                unsigned char* b_parts = parts_ptr + cs * S::PARTS + b_row * 64;
#pragma unroll
                for (int i = 0; i < B_PIECES; ++i) {
                  const int e = b_piece + i;
                  const float4 lo = *reinterpret_cast<const float4*>(b_raw + (((2 * e) ^ (b_row & 7)) << 4));
                  const float4 hi = *reinterpret_cast<const float4*>(b_raw + (((2 * e + 1) ^ (b_row & 7)) << 4));
                  uint32_t parts[3][4];
                  cut8(lo, hi, parts);
#pragma unroll
                  for (int p = 0; p < 3; ++p)
                    *reinterpret_cast<uint4*>(b_parts + p * (BT * KB * 2) + ((e ^ ((b_row >> 1) & 3)) << 4)) =
                        make_uint4(parts[p][0], parts[p][1], parts[p][2], parts[p][3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              }
              __syncwarp();
              tmem_wait_st();
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              __syncwarp();
              if (lane == 0) {
                mbar_arrive(smem_addr(&raw_empty[rs]));
                mbar_arrive(smem_addr(&cut_full[cs]));
              }
            }
            // The chunk before is added while the products of this block run: ahead of the next of the group's, as that stage
            // comes free only behind products that may wait for these sums to be taken.
            if (pending) {
              const uint32_t mb = chunks & 1u, cb = segments % S::CROSS;
              if (!wait_u(&main_full[mb], (chunks >> 1) & 1u)) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              add_columns<COLS>(tmem_main + mb * BT + lanes + side * COLS, acc);
              if (p_end) add_columns<COLS>(tmem_cross + cb * BT + lanes + side * COLS, acc);
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              __syncwarp();
              if (lane == 0) {
                mbar_arrive(smem_addr(&main_empty[mb]));
                if (p_end) mbar_arrive(smem_addr(&cross_empty[cb]));
              }
              ++chunks;
              pending = false;
              if (p_end) {
                ++segments;
                if (cut.split) break;                      // (the block's only item and range; `more` is false)
                put_range<BT, COLS>(cut, p_item, p_end, row, side * COLS, acc, out, M, N, ldo, broken);
#pragma unroll
                for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
              }
            }
            if (j + GROUPS >= blocks) break;
          }
          it += blocks;
          pending = true;
          p_item = item;
          p_end = c0 + len >= r1 ? r1 : 0;
        }
      }
      if (!more) break;
    }
    if (cut.split) {
      // Every block's sums to the blocks of the cluster, 1/ranges of the tile's rows to each, where they lie [range][column]
      // [row]: over the raw stages, which every block is done with behind the first barrier.
      const int each = (ROWS + cut.ranges - 1) / cut.ranges, owner = row / each;
      const uint32_t mine = (uint32_t)(blockIdx.x % (unsigned)cut.ranges);
      cluster_barrier();
      uint32_t dst;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                   : "=r"(dst)
                   : "r"(raw_base + ((mine * BT + side * COLS) * each + row - owner * each) * 4u), "r"(owner));
#pragma unroll
      for (int i = 0; i < COLS; ++i)
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)(i * each) * 4u), "f"(acc[i]) : "memory");
      cluster_barrier();
      int n0, m0, kb_begin, kb_end, range;
      place<BT>(cut, blockIdx.x, n0, m0, kb_begin, kb_end, range);
      const float* parts = reinterpret_cast<const float*>(raw_ptr);
      for (int i = threadIdx.x; i < BT * each; i += WORKERS * 32) {
        const int c = i / each, r = (int)mine * each + i - c * each, m = m0 + c, n = n0 + r;
        if (r >= ROWS || m >= M || n >= N) continue;
        float v = 0.f;
        for (int j = 0; j < cut.ranges; ++j) v += range_sum(parts[j * BT * each + i] * DOWN);
        broken = broken || !is_finite(v);
        out[(int64_t)m * ldo + n] = v;
      }
    }
    if (any_of_workers(broken))
      for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
        int n0, m0, kb_begin, kb_end, range;
        place<BT>(cut, item, n0, m0, kb_begin, kb_end, range);
        const int each = cut.split ? (ROWS + cut.ranges - 1) / cut.ranges : ROWS, first = cut.split ? range * each : 0;
        once_more<BT>(X, W, out, M, N, K, ldx, ldw, ldo, n0 + first, min(each, ROWS - first), m0);
      }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == WORKERS + 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_main), "r"((uint32_t)S::TMEM_COLS)
                 : "memory");
  }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A [rows, cols] fp32 matrix with `ld` elements between rows; boxes of KB columns x box_rows rows.
bool make_map(CUtensorMap* map, const float* base, int rows, int cols, int64_t ld, int box_rows) {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                       q == cudaDriverEntryPointSuccess;
    return found ? (EncodeTiledFn)p : nullptr;
  }();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {(cuuint32_t)KB, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How many clusters of `blocks` blocks this device runs at once, one block an SM (clusters do not reach across the SMs' groups).
int clusters_of(int blocks) {
  static const struct Table {
    int count[MOST_BLOCKS + 1] = {};
    Table() {
      if (cudaFuncSetAttribute(gemm_f32_parts_kernel<96>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<96>::SMEM) != cudaSuccess)
        return;
      for (int c = 2; c <= MOST_BLOCKS; ++c) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = Shape<96>::SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr, cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_parts_kernel<96>, &cfg) == cudaSuccess) count[c] = n;
      }
    }
  } table;
  return table.count[blocks];
}

// Ranges of K: a function of (N, K) alone, also on a device that holds fewer clusters or none (there the ranges of a tile follow
// one another; the order of the sums is the same).  As many blocks to a cluster as leave all tiles of one step of few tokens
// running at once on a B200, each range at least eight blocks of K long, and enough that none is longer than RANGE_BLOCKS.
constexpr int AT_ONCE[MOST_BLOCKS + 1] = {0, 0, 74, 45, 33, 26, 22, 15, 15};   // clusters_of() on 148 SMs
void ranges_of(int N, int K, int& ranges, int& range_blocks) {
  const int blocks = (K + KB - 1) / KB, tiles = (N + ROWS - 1) / ROWS;
  int want = 1;
  for (int c = 2; c <= MOST_BLOCKS; ++c)
    if (AT_ONCE[c] >= tiles) want = c;
  if (want > blocks / 8) want = blocks / 8;
  const int least = (blocks + RANGE_BLOCKS - 1) / RANGE_BLOCKS;
  if (want < least) want = least;
  if (want > MOST_RANGES) want = MOST_RANGES;
  if (want < 1) want = 1;
  range_blocks = (blocks + want - 1) / want;
  ranges = (blocks + range_blocks - 1) / range_blocks;     // (none is empty)
}

// Blocks between two visits to the leading accumulator.  Its truncations err to one side, so where all products have one sign a
// sum errs by half a chunk's additions whatever K is (1.7e-7 with 4 blocks, 2.1e-7 with 6, 2.8e-7 with 7, 3.8e-7 with 8), while
// the rounding of multiply-adds errs by the root of K (1.9e-7 at 640, 2.6e-7 at 1,280, 3.5e-7 at 2,048, 5.0e-7 at 4,096): no chunk
// is longer than leaves such a sum as close to 64 bits as multiply-adds leave it.
int chunk_of(int K) { return K < 1280 ? 4 : K < 2048 ? 6 : K < 4096 ? 7 : 8; }
// A range's blocks in as few chunks as that allows, of equal length (a range of 8 as 4 + 4: 2,048 x 2,048 x 1,536 131 us, 147 as 6 + 2).
// 8 + 7 + .. + 7 where that saves one: 3.0e-7 .. 3.3e-7, and 700 x 16,384 x 2,048 (64 blocks) 264 us for 271.
void chunks_of(Cut& cut, int K) {
  const int most = chunk_of(K);
  cut.extra = most == 7 && cut.range_blocks > 8 && cut.range_blocks % 7 == 1;
  const int visits = (cut.range_blocks + most - 1) / most;
  cut.chunk = cut.extra ? most : (cut.range_blocks + visits - 1) / visits;
}

// Tokens per tile and whether an item is one range: the layout whose fullest SM ends first.
struct Plan { int bt, split; };
Plan plan_of(int M, int N, int K) {
  int ranges, range_blocks;
  ranges_of(N, K, ranges, range_blocks);
  const int64_t blocks = (K + KB - 1) / KB, tiles_n = (N + ROWS - 1) / ROWS, sms = gllm_sm_count();
  // a block's time, in ns: up to 64 tokens the cutting of the weight's 128 rows, beyond the tokens' as well
  // and what a range's end costs where all are one item's (96 columns have one accumulator of the smaller products)
  static const int widths[] = {16, 32, 64, 80, 96};
  static const float block_ns[] = {445.f, 450.f, 455.f, 530.f, 565.f}, end_ns[] = {1000.f, 1000.f, 1000.f, 1000.f, 2500.f};
  Plan best{96, 0};
  float best_time = 0.f;
  for (int i = 0; i < 5; ++i) {
    const int64_t tiles = tiles_n * ((M + widths[i] - 1) / widths[i]);
    for (int split = 0; split < 2; ++split) {
      const int64_t at_once = !split ? sms : ranges > 1 && ranges <= MOST_BLOCKS ? clusters_of(ranges) : 0;
      if (at_once <= 0) continue;
      const int64_t waves = (tiles + at_once - 1) / at_once;
      // (a range's start and the sum through shared memory: measured 3 us)
      const float time = (float)waves * ((float)(split ? range_blocks : blocks) * block_ns[i] + (split ? 3000.f : end_ns[i] * (float)ranges));
      if (best_time == 0.f || time < best_time) best = Plan{widths[i], split}, best_time = time;
    }
  }
  return best;
}

template <int BT>
int launch(const float* X, const float* W, float* out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo, int split,
           int* status, cudaStream_t stream) {
  CUtensorMap map_w, map_x;
  if (!make_map(&map_w, W, N, K, ldw, ROWS) || !make_map(&map_x, X, M, K, ldx, BT)) return (int)cudaErrorInvalidValue;
  Cut cut;
  ranges_of(N, K, cut.ranges, cut.range_blocks);
  cut.blocks = (K + KB - 1) / KB;
  cut.tiles_n = (N + ROWS - 1) / ROWS, cut.tiles_m = (M + BT - 1) / BT;
  cut.split = split;
  chunks_of(cut, K);
  const int64_t items = (int64_t)cut.tiles_n * cut.tiles_m * (split ? cut.ranges : 1);
  if (items > 0x7fffffff - 4096) return (int)cudaErrorInvalidValue;
  auto kernel = gemm_f32_parts_kernel<BT>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<BT>::SMEM);
  if (e != cudaSuccess) return (int)e;
  if (split)
    return gllm_launch_cluster(kernel, dim3((unsigned)items), dim3(THREADS), (size_t)Shape<BT>::SMEM, stream,
                               (unsigned)cut.ranges, map_w, map_x, X, W, out, M, N, K, ldx, ldw, ldo, cut, (int)items, status);
  const int grid = items < gllm_sm_count() ? (int)items : gllm_sm_count();
  return gllm_launch(kernel, dim3(grid), dim3(THREADS), (size_t)Shape<BT>::SMEM, stream, map_w, map_x, X, W, out, M, N, K, ldx,
                     ldw, ldo, cut, (int)items, status);
}
}  // namespace parts3

bool on_vectors(const float* X, const float* W, int K, int64_t ldx, int64_t ldw) {
  return K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(W) & 15) == 0;
}
// Sums of up to 512 products stay with multiply-adds: by K alone, as a token's result may not depend on its batch.  The
// tensor-core kernel costs a start and an end of 4 us whatever K is (us, multiply-adds against parts: 8 x 1,024 x 256 3.9 against 6.3,
// 8 x 512 x 512 6.4 : 7.4, 8 x 1,024 x 1,024 11.7 : 7.4); with many tokens it is ahead from K = 256 on (2,048 x 512 x 512 33 : 16),
// which a decode step between two prompts does not get back.
constexpr int SHORT_SUM = 512;
}  // namespace

// Blocks of 32 k in a range of a sum of K products on the tensor cores.
GLLM_API int gllm_gemm_f32_range_blocks(int N, int K) {
  int ranges, range_blocks;
  parts3::ranges_of(N, K, ranges, range_blocks);
  return range_blocks;
}

GLLM_API int gllm_gemm_f32(const float* X, const float* W, float* C, int M, int N, int K, int64_t ldx, int64_t ldw,
                           int64_t ldc, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return (int)cudaErrorInvalidValue;
  const bool vectors = on_vectors(X, W, K, ldx, ldw);
  if (M > (vectors ? 128 : BM) * 65535) return (int)cudaErrorInvalidValue;
  if (vectors && K <= SHORT_SUM) {
    switch (pairs_tile_of(M, N)) {
      case 0: return gemm_f32_pairs<16, 16, 2, 2, 6, 8>(X, W, C, M, N, K, ldx, ldw, ldc, stream);
      case 1: return gemm_f32_pairs<32, 16, 4, 2, 6, 8>(X, W, C, M, N, K, ldx, ldw, ldc, stream);
      case 2: return gemm_f32_pairs<32, 32, 4, 4, 4, 8>(X, W, C, M, N, K, ldx, ldw, ldc, stream);
      case 3: return gemm_f32_pairs<64, 32, 8, 4, 4, 8>(X, W, C, M, N, K, ldx, ldw, ldc, stream);
      case 4: return gemm_f32_pairs<64, 64, 8, 4, 3, 8>(X, W, C, M, N, K, ldx, ldw, ldc, stream);
      default: return gemm_f32_pairs<64, 64, 8, 8, 3, 1>(X, W, C, M, N, K, ldx, ldw, ldc, stream);
    }
  }
  if (vectors) {
    const parts3::Plan plan = parts3::plan_of(M, N, K);
    switch (plan.bt) {
      case 16: return parts3::launch<16>(X, W, C, M, N, K, ldx, ldw, ldc, plan.split, status, stream);
      case 32: return parts3::launch<32>(X, W, C, M, N, K, ldx, ldw, ldc, plan.split, status, stream);
      case 64: return parts3::launch<64>(X, W, C, M, N, K, ldx, ldw, ldc, plan.split, status, stream);
      case 80: return parts3::launch<80>(X, W, C, M, N, K, ldx, ldw, ldc, plan.split, status, stream);
      default: return parts3::launch<96>(X, W, C, M, N, K, ldx, ldw, ldc, plan.split, status, stream);
    }
  }
  for (int m0 = 0; m0 < M; m0 += BM * 65535) {               // (tiles of rows lie along y, at most 65,535 a launch)
    const int rows = M - m0 < BM * 65535 ? M - m0 : BM * 65535;
    const int rc = gllm_launch(gemm_f32_kernel, dim3((N + BN - 1) / BN, (rows + BM - 1) / BM), dim3(256), 0, stream,
                               X + (int64_t)m0 * ldx, W, C + (int64_t)m0 * ldc, rows, N, K, ldx, ldw, ldc);
    if (rc != 0) return rc;
  }
  return 0;
}
