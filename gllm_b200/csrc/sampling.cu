// Sampling from fp32 logits: greedy, temperature, top-k, top-p, log-probabilities.
//
// The semantics are the reference sampler's (gllm/sample/sampler.py:67-107):
//   z = logits / temperature; keep the top_k highest z (0 = whole vocabulary);
//   over those, in descending order, keep the entries whose cumulative softmax
//   probability is <= top_p and always the first (the entry that crosses top_p
//   is dropped); draw from the softmax of what is left; log-probabilities are
//   log_softmax of the RAW logits at the highest candidates, at most
//   min(max_num_logprobs, number of candidates) of them, in descending order.
// Added here: temperature == 0 or top_k == 1 is an exact argmax (the reference
// divides by zero at temperature 0); the draw uses a counter-based generator
// keyed by (seed, counter) of the row, so a request's tokens do not depend on
// what else is in the batch; the sampled token's own log-probability is
// returned as well.
//
// No sort.  A cluster of blocks shares a row (sample_kernel below): every block copies its stretch of the row into
// shared memory once and all passes read that copy.  Requests with a moderate top_k finish on a short list of
// candidates in one block; the rest find the k-th largest value and the top-p cut by a search over the digits of
// order-preserving 32-bit keys.  Entries equal to the k-th largest value are all kept; entries equal to the value at
// which the cumulative probability crosses top_p are all dropped.
#include "common.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace {
constexpr int MAX_LOGPROBS = 32;

// Keys in the order of the numbers, NaN at the ends.  raw_key puts -0 right below +0; for to_key they are equal.
__device__ __forceinline__ uint32_t raw_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ uint32_t to_key(float v) {
  const uint32_t key = raw_key(v);
  return key == 0x7fffffffu ? 0x80000000u : key;
}

// Philox4x32-10, one block of four words for (seed, counter).
__device__ __forceinline__ float philox_uniform(uint64_t seed, uint32_t counter) {
  uint32_t c0 = counter, c1 = 0u, c2 = 0x5eedu, c3 = 0u;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  return (float)(c0 >> 8) * (1.0f / 16777216.0f);  // [0, 1)
}

// The largest value of a block and its lowest index; every thread gets both.  `sv` and `si` hold one entry per warp.
template <int N_WARPS>                           // (a power of two)
__device__ float block_max_arg(float v, int idx, int* out_idx, float* sv, int* si) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
  }
  __syncthreads();
  if (lane == 0) { sv[warp] = v; si[warp] = idx; }
  __syncthreads();
  float bv = sv[lane & (N_WARPS - 1)];
  int bi = si[lane & (N_WARPS - 1)];
#pragma unroll
  for (int o = N_WARPS / 2; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  *out_idx = bi;
  return bv;
}

// ---- sampling: a cluster of 2, 4 or 8 blocks per row (by the vocabulary alone: the order of every sum, and so a
// row's token, does not depend on what else is in the batch).
//
// What bounds it: the row's one trip from memory, then a chain of block-wide passes and cluster barriers.  The form
// before this one, a block per row with nine passes over the row through L2 and histograms of floats in shared memory
// (a compare-and-swap loop per element), took 270 us a call for 64 rows of 128,256 (top_k 40, top_p 0.9).  With 32 elements a
// thread, what every thread does once weighs as much as its elements: sums over a block's warps by shuffles, the bound
// by sixteen counting barriers over a maximum a thread and a look at the numbers ahead of their keys took it from 45.5 to 38.5 us.
//
// Threshold without a histogram: a block's stretch is cut into 64 groups (eight lanes of a warp each).  The K-th
// largest of all groups' maxima has at least K elements at or above it, so it (and its sixteen leading bits) bounds the
// K-th largest element from below, and only a few more than K elements lie above it when the row is in no particular
// order.  Those are handed, in index order, to block 0 of the cluster, which finds the exact K-th value, the top-p cut, the
// draw and the log-probabilities among them.  K is limited to half the groups (the bound gets loose beyond) and the list to
// LIST_CAP entries a block; rows that do not fit (and top_k 0) take the search over digits instead: eight rounds of
// sixteen bins, each bin's mass summed in a fixed order, one exchange between the blocks a round.
constexpr int SAMPLE_THREADS = 512;
constexpr int SAMPLE_WARPS = SAMPLE_THREADS / 32;
constexpr int GROUPS = SAMPLE_WARPS * 4;          // groups of eight lanes in a block
constexpr int MAX_RANKS = 8;
constexpr int BINS = 16;                          // values of a digit of the search
constexpr int LIST_CAP = 256;                     // candidates a block hands over
constexpr int SAMPLE_STAGE_BYTES = 160 * 1024;    // a stretch beyond this is read from global memory in every pass

struct SampleSmem {
  // written by every block of the cluster
  float group_max[MAX_RANKS][GROUPS];
  float max_v[MAX_RANKS];
  int max_i[MAX_RANKS];
  float sum_exp[MAX_RANKS];
  int list_n[MAX_RANKS];
  float bins[2][MAX_RANKS][BINS];
  union {
    struct {
      float list_v[MAX_RANKS * LIST_CAP];         // block r's at r * LIST_CAP (used in block 0)
      int list_i[MAX_RANKS * LIST_CAP];
      float packed_v[MAX_RANKS * LIST_CAP];       // the block's own from here on
      int packed_i[MAX_RANKS * LIST_CAP];
    };
    float lane_bins[SAMPLE_WARPS][BINS][32];      // during a search (no list is handed over or read meanwhile)
  };
  float kept_v[MAX_LOGPROBS];                     // the top elements in order, of a row whose token comes from a search
  int kept_i[MAX_LOGPROBS];
  float result[2];                                // key of the cut (as bits) and kept mass, for the distribution
  // the block's own
  float scratch[32];
  int scratch_i[32];
  float warp_bins[SAMPLE_WARPS][BINS];
  uint32_t word[2];
  float value[2];
  float packed_e[MAX_RANKS * LIST_CAP];
};

// What a block needs to walk its stretch: warp w owns the elements [w0, w1), in steps of 32.
struct Stretch {
  const float* x;      // the stretch (shared memory, or the row itself)
  int first;           // index of x[0] in the row
  int w0, w1;          // this warp's elements
  bool quads;          // x[w0] lies on a 16-byte boundary, and whole steps of 128 may be read four elements a lane

  // Calls f(j, value) for this warp's elements, a lane's in ascending order; every lane of the warp takes part.
  template <typename F> __device__ __forceinline__ void each(F f) const {
    const int lane = threadIdx.x & 31;
    int j0 = w0;
    if (quads) {
#pragma unroll 2
      for (; j0 + 128 <= w1; j0 += 128) {
        const int j = j0 + lane * 4;
        const float4 v = *reinterpret_cast<const float4*>(x + j);
        f(j, v.x), f(j + 1, v.y), f(j + 2, v.z), f(j + 3, v.w);
      }
    }
    for (int j = j0 + lane; j < w1; j += 32) f(j, x[j]);
  }
  // The same, four elements at once where that is possible: four(j, values) for j .. j + 3, one(j, value) for the others.
  template <typename Four, typename One> __device__ __forceinline__ void each_four(Four four, One one) const {
    const int lane = threadIdx.x & 31;
    int j0 = w0;
    if (quads) {
#pragma unroll 2
      for (; j0 + 128 <= w1; j0 += 128) four(j0 + lane * 4, *reinterpret_cast<const float4*>(x + j0 + lane * 4));
    }
    for (int j = j0 + lane; j < w1; j += 32) one(j, x[j]);
  }
};

// Mass of the sixteen values that digit `shift` of the key can take, over the elements whose key is at least `floor`
// and agrees with `prefix` under `mask`; an element weighs exp((v - xmax) * inv_t), or 1 with COUNT.  All blocks of
// the cluster get all sixteen sums (`total[BINS]` in the caller's registers, the same in every thread).  Every lane has its own
// sixteen sums in shared memory, one to a bank: an element costs a load, an addition and a store where sums in registers took
// sixteen comparisons and additions, and what is not in the prefix costs its key: 64 rows of 128,256 without top_k, top_p 0.9,
// 379 -> 213 us, one row 92 -> 70.  (The same sums in the same order.)
template <bool COUNT>
__device__ void digit_mass(const Stretch& s, cg::cluster_group& cluster, SampleSmem& sm, int parity, uint32_t floor,
                           uint32_t prefix, uint32_t mask, int shift, float xmax, float inv_t, float (&total)[BINS]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* mine = &sm.lane_bins[warp][0][lane];
#pragma unroll
  for (int b = 0; b < BINS; ++b) mine[b * 32] = 0.f;
  constexpr int AHEAD = 4;
  for (int j0 = s.w0 + lane; j0 < s.w1; j0 += 32 * AHEAD) {
    float v[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) v[u] = j0 + 32 * u < s.w1 ? s.x[j0 + 32 * u] : 0.f;
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const uint32_t key = to_key(v[u]);
      if (j0 + 32 * u < s.w1 && key >= floor && (key & mask) == prefix)
        mine[((key >> shift) & (BINS - 1)) * 32] += COUNT ? 1.f : expf((v[u] - xmax) * inv_t);
    }
  }
#pragma unroll
  for (int b = 0; b < BINS; ++b) {
    const float sum = warp_sum(mine[b * 32]);
    if (lane == 0) sm.warp_bins[warp][b] = sum;
  }
  __syncthreads();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  if (threadIdx.x < BINS * ranks) {
    const int b = threadIdx.x % BINS;
    float m = 0.f;
    for (int w = 0; w < SAMPLE_WARPS; ++w) m += sm.warp_bins[w][b];
    *cluster.map_shared_rank(&sm.bins[parity][rank][b], threadIdx.x / BINS) = m;
  }
  cluster.sync();
#pragma unroll
  for (int b = 0; b < BINS; ++b) {
    float m = 0.f;
    for (int r = 0; r < ranks; ++r) m += sm.bins[parity][r][b];
    total[b] = m;
  }
}

// The largest key T whose set {key >= floor, key >= T} has a mass above `limit` (with FRACTION: above `limit` times
// the mass of {key >= floor}).  False when not even the whole set has.
template <bool COUNT, bool FRACTION>
__device__ bool find_cut(const Stretch& s, cg::cluster_group& cluster, SampleSmem& sm, uint32_t floor, float limit,
                         float xmax, float inv_t, uint32_t* cut) {
  uint32_t prefix = 0, mask = 0;
  float above = 0.f;
  for (int round = 0; round < 8; ++round) {
    const int shift = 28 - 4 * round;
    float total[BINS];
    digit_mass<COUNT>(s, cluster, sm, round & 1, floor, prefix, mask, shift, xmax, inv_t, total);
    if (FRACTION && round == 0) {
      float all = 0.f;
#pragma unroll
      for (int b = BINS - 1; b >= 0; --b) all += total[b];
      limit *= all;
    }
    int pick = -1, last = -1;
    float run = above, run_pick = above, run_last = above;
#pragma unroll
    for (int b = BINS - 1; b >= 0; --b) {
      if (total[b] > 0.f) {
        if (pick < 0) { last = b; run_last = run; }
        if (pick < 0 && run + total[b] > limit) { pick = b; run_pick = run; }
      }
      run += total[b];
    }
    if (pick < 0) {
      if (round == 0) return false;
      // rounding: the digits sum to a hair less than their prefix did; the cut is then its smallest element
      pick = max(last, 0), run_pick = run_last;
    }
    above = run_pick;
    prefix |= (uint32_t)pick << shift;
    mask |= (uint32_t)(BINS - 1) << shift;
  }
  *cut = prefix;
  return true;
}

// This block's elements whose key is at least `floor`, above it or equal to it, in index order, to block 0's list.  Every
// block of the cluster learns how many each found; no more than LIST_CAP are handed over.
enum Wanted { FROM, ABOVE, EQUAL };
template <Wanted W> __device__ __forceinline__ bool wanted(float v, uint32_t floor) {
  return W == FROM ? raw_key(v) >= floor : (W == ABOVE ? to_key(v) > floor : to_key(v) == floor);
}
template <Wanted W>
__device__ void hand_over(const Stretch& s, cg::cluster_group& cluster, SampleSmem& sm, uint32_t floor) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = (int)cluster.block_rank();
  if (W == FROM && floor == 0x80000000u) floor = 0x7fffffffu;          // both zeros, as raw keys
  // Few elements are wanted: a look at the numbers themselves (NaN pass it) keeps the keys for those.
  const float least = W == EQUAL || floor < 0x00800000u ? -INFINITY : __uint_as_float((floor & 0x80000000u) ? floor ^ 0x80000000u : ~floor);
  auto maybe = [&](float v) { return !(v < least); };
  int mine = 0;
  s.each_four(
      [&](int, const float4& q) {
        if (maybe(q.x) || maybe(q.y) || maybe(q.z) || maybe(q.w))
          mine += wanted<W>(q.x, floor) + wanted<W>(q.y, floor) + wanted<W>(q.z, floor) + wanted<W>(q.w, floor);
      },
      [&](int, float v) { mine += wanted<W>(v, floor); });
  mine = __reduce_add_sync(0xffffffffu, mine);
  __syncthreads();
  if (lane == 0) sm.scratch_i[warp] = mine;
  __syncthreads();
  const int theirs = lane < SAMPLE_WARPS ? sm.scratch_i[lane] : 0;
  int at = __reduce_add_sync(0xffffffffu, lane < warp ? theirs : 0);
  const int all = __reduce_add_sync(0xffffffffu, theirs);
  if ((int)threadIdx.x < (int)cluster.num_blocks()) *cluster.map_shared_rank(&sm.list_n[rank], threadIdx.x) = all;
  if (mine > 0 && at < LIST_CAP) {
    float* list_v = cluster.map_shared_rank(sm.list_v, 0) + rank * LIST_CAP;
    int* list_i = cluster.map_shared_rank(sm.list_i, 0) + rank * LIST_CAP;
    int j0 = s.w0;
    if (s.quads) {
      for (; j0 + 128 <= s.w1; j0 += 128) {
        const int j = j0 + lane * 4;
        const float4 q = *reinterpret_cast<const float4*>(s.x + j);
        if (!__any_sync(0xffffffffu, maybe(q.x) || maybe(q.y) || maybe(q.z) || maybe(q.w))) continue;
        const float v[4] = {q.x, q.y, q.z, q.w};
        int found = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) found += wanted<W>(v[e], floor);
        if (!__any_sync(0xffffffffu, found)) continue;
        int upto = found;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += t;
        }
        int slot = at + upto - found;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (wanted<W>(v[e], floor)) {
            if (slot < LIST_CAP) { list_v[slot] = v[e]; list_i[slot] = s.first + j + e; }
            ++slot;
          }
        at += __shfl_sync(0xffffffffu, upto, 31);
      }
    }
    for (; j0 < s.w1; j0 += 32) {
      const int j = j0 + lane;
      const float v = j < s.w1 ? s.x[j] : 0.f;
      const bool in = j < s.w1 && wanted<W>(v, floor);
      const uint32_t votes = __ballot_sync(0xffffffffu, in);
      const int slot = at + __popc(votes & ((1u << lane) - 1));
      if (in && slot < LIST_CAP) { list_v[slot] = v; list_i[slot] = s.first + j; }
      at += __popc(votes);
    }
  }
  cluster.sync();
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int64_t row_stride, int V, int per, int staged, int vectors,
              const float* __restrict__ temperature, const int* __restrict__ top_k, const float* __restrict__ top_p,
              const int64_t* __restrict__ seed, const int* __restrict__ counter, const int* __restrict__ n_logprobs,
              int lp_stride, int* __restrict__ out_token, float* __restrict__ out_logprob, int* __restrict__ out_ncand,
              float* __restrict__ out_top_lp, int* __restrict__ out_top_id, float* __restrict__ probs_out) {
  extern __shared__ __align__(16) float stage[];
  __shared__ SampleSmem sm;
  pdl_trigger();
  cluster_arrive_started();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const int row = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = min(V, rank * per), n = min(V, first + per) - first;
  // (stretches of 2,048 elements and more are walked four elements a lane; shorter ones leave no warp without work)
  Stretch s;
  s.quads = staged && per >= SAMPLE_WARPS * 128;
  const int step = s.quads ? 128 : 32, seg = (n + SAMPLE_WARPS * step - 1) / (SAMPLE_WARPS * step) * step;
  s.first = first;
  s.w0 = min(n, warp * seg), s.w1 = min(n, s.w0 + seg);
  pdl_wait();
  const float* x = logits + (int64_t)row * row_stride;
  s.x = x + first;
  if (staged) {
    const float* src = x + first;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage);
    if (vectors) {
      for (int j = tid * 4; j + 3 < n; j += SAMPLE_THREADS * 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + j * 4), "l"(src + j) : "memory");
      for (int j = (n & ~3) + tid; j < n; j += SAMPLE_THREADS) stage[j] = src[j];
    } else {
      for (int j = tid; j < n; j += SAMPLE_THREADS)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + j * 4), "l"(src + j) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    s.x = stage;
  }
  const float temp = temperature ? temperature[row] : 0.f;
  const int k_in = top_k ? top_k[row] : 0;
  const float p_in = top_p ? top_p[row] : 1.f;
  const int n_lp_in = min(n_logprobs ? n_logprobs[row] : 0, min(MAX_LOGPROBS, lp_stride));
  const bool greedy = !(temp > 0.f) || k_in == 1;

  // maxima of the groups, of the block and (after the exchange) of the row; log-sum-exp of the raw logits
  float vmax = -INFINITY;
  int imax = 0x7fffffff;
  s.each_four(
      [&](int j, const float4& q) {
        const float v = fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w));
        if (v > vmax) { vmax = v; imax = j; }
      },
      [&](int j, float v) {
        if (v > vmax) { vmax = v; imax = j; }
      });
  if (imax < n) {                                  // (of four, the first that is the maximum)
    while (s.x[imax] != vmax) ++imax;
    imax += first;
  }
  float gmax = vmax;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
  int barg;
  const float bmax = block_max_arg<SAMPLE_WARPS>(vmax, imax, &barg, sm.scratch, sm.scratch_i);
  // (a stretch without a number above -inf adds nothing, unless it holds a NaN: then the sum is one, as in any other)
  float se = 0.f;
  const float base = bmax > -INFINITY ? bmax : 0.f;
  s.each([&](int, float v) { se += expf(v - base); });
  se = warp_sum(se);
  __syncthreads();
  if (lane == 0) sm.scratch[warp] = se;
  __syncthreads();
  se = warp_sum(lane < SAMPLE_WARPS ? sm.scratch[lane] : 0.f);
  cluster_wait_started();
  if ((lane & 7) == 0)
    for (int r = 0; r < ranks; ++r) *cluster.map_shared_rank(&sm.group_max[rank][warp * 4 + (lane >> 3)], r) = gmax;
  if (tid < ranks) {
    *cluster.map_shared_rank(&sm.max_v[rank], tid) = bmax;
    *cluster.map_shared_rank(&sm.max_i[rank], tid) = barg;
    *cluster.map_shared_rank(&sm.sum_exp[rank], tid) = se;
  }
  cluster.sync();
  float xmax = sm.max_v[0];
  int arg = sm.max_i[0];
  for (int r = 1; r < ranks; ++r)
    if (sm.max_v[r] > xmax) { xmax = sm.max_v[r]; arg = sm.max_i[r]; }
  if (arg >= V) arg = 0;                           // nothing above -inf in the row
  float z = 0.f;
  if (lane < ranks) z = sm.max_v[lane] > -INFINITY ? sm.sum_exp[lane] * expf(sm.max_v[lane] - xmax) : sm.sum_exp[lane];
#pragma unroll
  for (int o = MAX_RANKS / 2; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  z = __shfl_sync(0xffffffffu, z, 0);
  const float log_z = xmax + logf(z);
  const uint32_t key_max = to_key(xmax);

  const uint32_t k = (k_in <= 0 || k_in >= V) ? (uint32_t)V : (uint32_t)k_in;
  const int groups = ranks * GROUPS;
  bool listed = !greedy && k <= (uint32_t)groups / 2;             // the token comes from the list
  const int want = listed ? (int)k : (greedy ? 0 : n_lp_in);      // how many elements the list has to hold
  int n_list = 0;                                                 // entries of block 0's list, packed below
  // f(place, value, index) for the `most` highest of them
  auto rank_top = [&](int most, auto f) {
    for (int i = tid; i < n_list; i += SAMPLE_THREADS) {
      const float v = sm.packed_v[i];
      const int id = sm.packed_i[i];
      int place = 0;
      for (int o = 0; o < n_list && place < most; ++o) {
        const float ov = sm.packed_v[o];
        place += ov > v || (ov == v && sm.packed_i[o] < id);
      }
      if (place < most) f(place, v, id);
    }
  };
  if (want > 0) {
    // A lower bound of the want-th largest element: the largest key of sixteen leading bits at or above which lie `want`
    // of the groups' maxima, bit by bit, a maximum a thread.
    static_assert(MAX_RANKS * GROUPS <= SAMPLE_THREADS, "a maximum a thread");
    const uint32_t key = tid < groups ? to_key((&sm.group_max[0][0])[tid]) : 0u;
    uint32_t floor = 0;
#pragma unroll 1
    for (int bit = 31; bit >= 16; --bit) {
      const uint32_t trial = floor | 1u << bit;
      if (__syncthreads_count(key >= trial) >= want) floor = trial;
    }
    // block 0 packs what lies in its list, at most `most` entries of each block
    auto pack = [&](int most) {
      if (rank != 0) return;
      for (int r = 0; r < ranks; ++r) {
        const int c = min(sm.list_n[r], most);
        for (int i = tid; i < c; i += SAMPLE_THREADS) {
          sm.packed_v[n_list + i] = sm.list_v[r * LIST_CAP + i];
          sm.packed_i[n_list + i] = sm.list_i[r * LIST_CAP + i];
        }
        n_list += c;
      }
      __syncthreads();
    };
    hand_over<FROM>(s, cluster, sm, floor);
    bool fits = true;
    for (int r = 0; r < ranks; ++r) fits = fits && sm.list_n[r] <= LIST_CAP;
    if (fits) {
      pack(LIST_CAP);
    } else {
      listed = false;
      if (n_lp_in > 0) {
        // the elements above the n-th largest, fewer than MAX_LOGPROBS, then as many of those equal to it as can be reported
        floor = 0;
        find_cut<true, false>(s, cluster, sm, 0u, (float)n_lp_in - 0.5f, xmax, 1.f, &floor);
        hand_over<ABOVE>(s, cluster, sm, floor);
        pack(LIST_CAP);
        cluster.sync();                            // block 0 has taken them from its list
        hand_over<EQUAL>(s, cluster, sm, floor);
        pack(MAX_LOGPROBS);
      }
    }
    if (!listed && !greedy && rank == 0) {         // the searches for the token go over the lists' place
      rank_top(n_lp_in, [&](int place, float v, int id) { sm.kept_v[place] = v, sm.kept_i[place] = id; });
      __syncthreads();
    }
  }

  int ncand = 1;
  uint32_t key_cut = key_max;
  float inv_t = 1.f, z_kept = 1.f;
  if (greedy) {
    if (rank == 0 && tid == 0) {
      out_token[row] = arg;
      out_logprob[row] = x[arg] - log_z;
      out_ncand[row] = 1;
      if (n_lp_in > 0) {
        out_top_lp[(int64_t)row * lp_stride] = x[arg] - log_z;
        out_top_id[(int64_t)row * lp_stride] = arg;
      }
    }
  } else {
    inv_t = 1.0f / temp;
    const float u = philox_uniform((uint64_t)(seed ? seed[row] : 0), (uint32_t)(counter ? counter[row] : 0));
    if (listed) {
      if (rank == 0) {
        // the exact k-th largest value, then the top-p cut, among the list's entries
        if (tid == 0) sm.word[0] = 0xffffffffu, sm.word[1] = 0u;
        __syncthreads();
        for (int i = tid; i < n_list; i += SAMPLE_THREADS) {
          const float v = sm.packed_v[i];
          int larger = 0;
          for (int o = 0; o < n_list; ++o) larger += sm.packed_v[o] > v;
          if (larger < (int)k) atomicMin(&sm.word[0], to_key(v));
        }
        __syncthreads();
        const uint32_t key_k = sm.word[0];
        key_cut = key_k;
        float mass = 0.f;
        for (int i = tid; i < n_list; i += SAMPLE_THREADS) {
          const float v = sm.packed_v[i];
          const float e = to_key(v) >= key_k ? expf((v - xmax) * inv_t) : 0.f;
          sm.packed_e[i] = e;
          mass += e;
        }
        mass = block_sum(mass, sm.scratch);
        if (p_in < 1.f) {
          const float limit = p_in * mass;
          for (int i = tid; i < n_list; i += SAMPLE_THREADS) {
            const float v = sm.packed_v[i];
            float above = 0.f;                     // mass of everything at or above this value
            for (int o = 0; o < n_list; ++o) above += sm.packed_v[o] >= v ? sm.packed_e[o] : 0.f;
            if (to_key(v) >= key_k && above > limit) atomicMax(&sm.word[1], to_key(v));
          }
          __syncthreads();
          const uint32_t cross = sm.word[1];
          // everything above the crossing value is kept; the maximum always is
          if (cross) key_cut = cross >= key_max ? key_max : max(key_k, cross + 1u);
        }
        if (warp == 0) {
          // kept mass and count, then the draw by an index-ordered prefix of the kept masses
          float total = 0.f;
          int count = 0;
          for (int i0 = 0; i0 < n_list; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < n_list && to_key(sm.packed_v[i]) >= key_cut;
            total += warp_sum(in ? sm.packed_e[i] : 0.f);
            count += __popc(__ballot_sync(0xffffffffu, in));
          }
          const float target = u * total;
          float run = 0.f;
          int pick = -1;
          for (int i0 = 0; i0 < n_list && pick < 0; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < n_list && to_key(sm.packed_v[i]) >= key_cut;
            float inc = in ? sm.packed_e[i] : 0.f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const float t = __shfl_up_sync(0xffffffffu, inc, o);
              if (lane >= o) inc += t;
            }
            const uint32_t hit = __ballot_sync(0xffffffffu, in && target < run + inc);
            if (hit) pick = i0 + __ffs(hit) - 1;
            run += __shfl_sync(0xffffffffu, inc, 31);
          }
          if (lane == 0) {
            // rounding can leave the target past the end: take the maximum then
            out_token[row] = pick < 0 ? arg : sm.packed_i[pick];
            out_logprob[row] = (pick < 0 ? xmax : sm.packed_v[pick]) - log_z;
            out_ncand[row] = count;
            sm.scratch_i[0] = count;
            sm.value[0] = total;
          }
        }
        __syncthreads();
        ncand = sm.scratch_i[0];
        z_kept = sm.value[0];
        if (probs_out && tid < ranks) {
          float* result = cluster.map_shared_rank(sm.result, tid);
          result[0] = __uint_as_float(key_cut);
          result[1] = z_kept;
        }
      }
      if (probs_out) {
        cluster.sync();
        key_cut = __float_as_uint(sm.result[0]);
        z_kept = sm.result[1];
      }
    } else {
      uint32_t key_k = 0u;
      if (k < (uint32_t)V) find_cut<true, false>(s, cluster, sm, 0u, (float)k - 0.5f, xmax, 1.f, &key_k);
      key_cut = key_k;
      if (p_in < 1.f) {
        uint32_t cross = 0u;
        if (find_cut<false, true>(s, cluster, sm, key_k, p_in, xmax, inv_t, &cross))
          key_cut = cross >= key_max ? key_max : max(key_k, cross + 1u);
      }
      // kept mass and count of every warp's elements, of every block and of the row
      float mine = 0.f;
      int count = 0;
      for (int j = s.w0 + lane; j < s.w1; j += 32) {
        const float v = s.x[j];
        if (to_key(v) >= key_cut) { mine += expf((v - xmax) * inv_t); ++count; }
      }
      mine = warp_sum(mine);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
      __syncthreads();
      if (lane == 0) { sm.scratch[warp] = mine; sm.scratch_i[warp] = count; }
      __syncthreads();
      float block_mass = 0.f;
      int block_count = 0;
      for (int w = 0; w < SAMPLE_WARPS; ++w) block_mass += sm.scratch[w], block_count += sm.scratch_i[w];
      cluster.sync();                              // the last round's bins have been read everywhere
      if (tid < ranks) {
        float* dst = cluster.map_shared_rank(&sm.bins[0][rank][0], tid);
        dst[0] = block_mass;
        dst[1] = __int_as_float(block_count);
      }
      cluster.sync();
      float total = 0.f;
      ncand = 0;
      for (int r = 0; r < ranks; ++r) total += sm.bins[0][r][0], ncand += __float_as_int(sm.bins[0][r][1]);
      z_kept = total;
      const float target = u * total;
      float before = 0.f;
      int owner = -1;
      for (int r = 0; r < ranks && owner < 0; ++r) {
        if (target < before + sm.bins[0][r][0]) owner = r;
        else before += sm.bins[0][r][0];
      }
      if (owner < 0 && rank == 0 && tid == 0) {    // rounding can leave the target past the end: the maximum then
        out_token[row] = arg;
        out_logprob[row] = xmax - log_z;
      }
      if (owner == rank) {
        float run = before;
        int w_own = -1, w_last = 0;
        for (int w = 0; w < SAMPLE_WARPS && w_own < 0; ++w) {
          if (sm.scratch_i[w] > 0) w_last = w;
          if (target < run + sm.scratch[w]) w_own = w;
          else run += sm.scratch[w];
        }
        if (w_own < 0) w_own = w_last;
        if (warp == w_own) {
          int pick = -1, last = -1;
          for (int j0 = s.w0; j0 < s.w1 && pick < 0; j0 += 32) {
            const int j = j0 + lane;
            const float v = j < s.w1 ? s.x[j] : 0.f;
            const bool in = j < s.w1 && to_key(v) >= key_cut;
            const float e = in ? expf((v - xmax) * inv_t) : 0.f;
            float inc = e;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const float t = __shfl_up_sync(0xffffffffu, inc, o);
              if (lane >= o) inc += t;
            }
            const uint32_t kept = __ballot_sync(0xffffffffu, in);
            const uint32_t hit = __ballot_sync(0xffffffffu, in && target < run + inc);
            if (kept) last = j0 + 31 - __clz(kept);
            if (hit) pick = j0 + __ffs(hit) - 1;
            run += __shfl_sync(0xffffffffu, inc, 31);
          }
          if (pick < 0) pick = last;
          if (lane == 0) {
            out_token[row] = pick < 0 ? arg : first + pick;
            out_logprob[row] = (pick < 0 ? xmax : s.x[pick]) - log_z;
          }
        }
      }
      if (rank == 0 && tid == 0) out_ncand[row] = ncand;
    }
    // log-probabilities of the highest candidates
    const int n_lp = min(n_lp_in, ncand);
    if (rank == 0 && n_lp > 0) {
      auto put = [&](int place, float v, int id) {
        out_top_lp[(int64_t)row * lp_stride + place] = v - log_z;
        out_top_id[(int64_t)row * lp_stride + place] = id;
      };
      if (listed) rank_top(n_lp, put);
      else if (tid < min(n_lp, n_list)) put(tid, sm.kept_v[tid], sm.kept_i[tid]);
    }
  }
  if (probs_out) {
    float* po = probs_out + (int64_t)row * V + first;
    for (int j = s.w0 + lane; j < s.w1; j += 32) {
      const float v = s.x[j];
      float p = 0.f;
      if (greedy) p = first + j == arg ? 1.f : 0.f;
      else if (to_key(v) >= key_cut) p = expf((v - xmax) * inv_t) / z_kept;
      po[j] = p;
    }
  }
}

// A cluster of ARGMAX_CLUSTER blocks shares one row (a row of a large vocabulary read through one
// SM's port takes longer than the rest of a decode step's tail): each block takes a stretch of the
// row, pushes its (maximum, index) into every block's shared memory, and after one cluster barrier
// rank 0 picks the winner (the lowest index among equal maxima, as a single block would).
constexpr int THREADS = 1024;
constexpr int ARGMAX_CLUSTER = 8;
__global__ void __launch_bounds__(THREADS)
argmax_kernel(const float* __restrict__ logits, int64_t row_stride, int V, int* __restrict__ out_token,
              const int* __restrict__ out_index) {
  __shared__ float warp_v[THREADS / 32];
  __shared__ int warp_i[THREADS / 32];
  __shared__ float peer_v[ARGMAX_CLUSTER];
  __shared__ int peer_i[ARGMAX_CLUSTER];
  pdl_trigger();
  cluster_arrive_started();
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), n_ranks = (int)cluster.num_blocks();
  const int row = blockIdx.y;
  const int per = (V + n_ranks - 1) / n_ranks;
  const int j0 = rank * per, j1 = min(V, j0 + per);
  pdl_wait();
  const float* x = logits + (int64_t)row * row_stride;
  float vmax = -INFINITY;
  int imax = 0x7fffffff;
  for (int j = j0 + threadIdx.x; j < j1; j += THREADS) {
    const float v = x[j];
    if (v > vmax) { vmax = v; imax = j; }
  }
  int arg;
  const float best = block_max_arg<THREADS / 32>(vmax, imax, &arg, warp_v, warp_i);
  cluster_wait_started();
  if (threadIdx.x == 0) {
    *cluster.map_shared_rank(&peer_v[rank], 0) = best;
    *cluster.map_shared_rank(&peer_i[rank], 0) = arg;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    float bv = peer_v[0];
    int bi = peer_i[0];
    for (int r = 1; r < n_ranks; ++r)
      if (peer_v[r] > bv || (peer_v[r] == bv && peer_i[r] < bi)) { bv = peer_v[r]; bi = peer_i[r]; }
    out_token[out_index ? out_index[row] : row] = bi;
  }
}
}  // namespace

GLLM_API int gllm_sample(const float* logits, int64_t row_stride, int rows, int V, const float* temperature,
                         const int* top_k, const float* top_p, const int64_t* seed, const int* counter,
                         const int* n_logprobs, int lp_stride, int* out_token, float* out_logprob,
                         int* out_ncand, float* out_top_lp, int* out_top_id, float* probs_out,
                         cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0) return (int)cudaErrorInvalidValue;
  // 16,000 elements a block at 128,256: two blocks of 512 threads fit an SM.  Fewer blocks a row for small
  // vocabularies, whose passes are short beside the barriers between the blocks.
  const int ranks = V > 32768 ? 8 : (V > 8192 ? 4 : 2);
  const int per = (((V + ranks - 1) / ranks) + 3) & ~3;
  const int staged = (size_t)per * sizeof(float) <= (size_t)SAMPLE_STAGE_BYTES;
  const int vectors = row_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  const size_t smem = staged ? (size_t)per * sizeof(float) : 0;
  const cudaError_t e = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_STAGE_BYTES);
  if (e != cudaSuccess) return (int)e;
  // (rows lie along y, at most 65,535 a launch)
  for (int r0 = 0; r0 < rows; r0 += 65535) {
    const int nr = rows - r0 < 65535 ? rows - r0 : 65535;
    auto at = [r0](auto* p, int64_t step) { return p ? p + r0 * step : p; };
    const int rc = gllm_launch_cluster(
        sample_kernel, dim3(ranks, nr), dim3(SAMPLE_THREADS), smem, stream, (unsigned)ranks, at(logits, row_stride),
        row_stride, V, per, staged, vectors, at(temperature, 1), at(top_k, 1), at(top_p, 1), at(seed, 1),
        at(counter, 1), at(n_logprobs, 1), lp_stride, at(out_token, 1), at(out_logprob, 1), at(out_ncand, 1),
        at(out_top_lp, lp_stride), at(out_top_id, lp_stride), at(probs_out, V));
    if (rc != 0) return rc;
  }
  return 0;
}

// out_index (optional): row r's result goes to out_token[out_index[r]] instead of out_token[r].
GLLM_API int gllm_argmax(const float* logits, int64_t row_stride, int rows, int V, int* out_token,
                         const int* out_index, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0) return (int)cudaErrorInvalidValue;
  return gllm_launch_cluster(argmax_kernel, dim3(ARGMAX_CLUSTER, rows), dim3(THREADS), 0, stream,
                             (unsigned)ARGMAX_CLUSTER, logits, row_stride, V, out_token, out_index);
}
