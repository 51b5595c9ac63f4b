// Device-resident beam search: the generation loop of
// src/no_three_75/gpu_device_search.py:254-432 (gpu_device_beam_search) on the
// GPU.  Per generation, five launches on one stream and no host round trip:
//   mutate_kernel      children from the ranked elites (gpu_device_search.py:27-114),
//                      recording each child's parent and swaps
//   child_delta_kernel E and badness of every child from its parent's by the exact
//                      delta of each swap (the reference rescores every child)
//   select_kernel      stable score order prefix, the children within the energy
//                      window in index order, their random.Random shuffle, the
//                      pick of elite_size children (gpu_device_search.py:343-373)
//   gather_kernel      the picked children's rows, E and badness
//   rank_kernel        rank_elites order (gpu_device_search.py:185-197) and the
//                      best-so-far update by elite_key (:200-203, :388-396)
// The reference does the selection and ranking on the host with a copy of
// every child's score each generation.  Here the selection is one CTA: a
// one-pass histogram (or radix) select of the elite_size-th smallest score, a
// bitonic sort of the scores below it, ordered compactions by per-warp counts,
// the MT19937 state blocks twisted by the whole CTA, the shuffle's draws (exactly
// CPython's), and the first elite_size shuffled positions traced back through
// the draws.
#include <stdint.h>

#include <climits>

#include "dirs.cuh"
#include "pair_move.cuh"
#include "pyrandom.cuh"
#include "n3_common.cuh"

namespace n3 {
namespace beam {

// --------------------------------------------------------------------------
// xorshift64* (Vigna), the reference's per-child RNG (gpu_device_search.py:18-25).
// --------------------------------------------------------------------------
__device__ __forceinline__ uint64_t xs64(uint64_t& s) {
  uint64_t x = s;
  x ^= x >> 12;
  x ^= x << 25;
  x ^= x >> 27;
  s = x;
  return x * 2685821657736338717ULL;
}

struct MutArgs {
  const int32_t* pp;
  const int32_t* pq;
  const int32_t* pbad;
  int parent_count, quality_count, active_strength;  // used when status == nullptr
  const int64_t* status;                              // beam status: counts and strength derive from it
  int elite_size, n, population, max_strength, bad_bias, generation;
  uint64_t seed;
  int32_t* cp;
  int32_t* cq;
  int32_t* child_parent;  // optional: each child's parent and swaps (u | v << 8), for the delta scoring
  int32_t* child_moves;
  int32_t* child_nmoves;
  int moves_cap;
  int prefix_cap;  // parents whose badness prefix sums the CTA stages in shared memory
};

// One thread per child, the reference's draws in the reference's order.  The
// CTA's children live in shared memory (slot layout s = 2 * row + layer) from the
// parent copy to one coalesced write of their rows: in 16 bits (short2) in a beam,
// whose states lie on a grid, in 32 (int2) for n3_beam_mutate, which returns any
// columns as they came.  When the
// parents' badness prefix sums fit in shared memory (prefix_cap parents), the CTA
// builds them once, a warp per parent, and the roulette draw becomes a binary
// search: with no negative badness, the linear scan `t -= bad[u]` stops at the
// first u whose inclusive prefix exceeds t, which the search finds.  A negative
// badness anywhere, or one large enough for a sum to overflow (neither is a
// state's badness), sends the CTA back to the linear scan, so every draw and
// result stays the reference's for any input.  The parent's total badness is
// taken once per child instead of once per attempt (it does not change), and its
// draws' remainders by a reciprocal.
//
// A child is one thread's serial chain (about five draws a swap), so what counts
// besides is the staging, which every CTA repeats: with as many threads as spread
// the children over the SMs once (64 .. 256), 32,768 children of 64 parents at
// n = 75 take 31 us, 71 us in CTAs of 64.
constexpr int kMutThreads = 256;  // at most; half of it in 32 bits
constexpr size_t kMutPrefixMaxBytes = 96 * 1024;

constexpr size_t kMutSmemMax = sizeof(int16_t) * kMutThreads * kMaxM + kMutPrefixMaxBytes;
static_assert(kMutSmemMax <= 227 * 1024 - 2048, "mutate_kernel shared memory");

// x % d by a reciprocal: the quotient's estimate is at most two short.
struct Remainder {
  uint64_t d, inverse;
  __device__ explicit Remainder(uint64_t divisor) : d(divisor), inverse(~0ull / divisor) {}
  __device__ __forceinline__ uint64_t of(uint64_t x) const {
    uint64_t r = x - __umul64hi(x, inverse) * d;
    if (r >= d) r -= d;
    if (r >= d) r -= d;
    return r;
  }
};

template <class Row>
__global__ void __launch_bounds__(kMutThreads) mutate_kernel(const MutArgs A) {
  using Cell = decltype(Row::x);
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_parent[kMutThreads];
  int parent_count = A.parent_count, quality_count = A.quality_count, active = A.active_strength;
  if (A.status != nullptr) {
    if (A.status[1] == 0) return;  // uniform: the search has reached E = 0
    parent_count = (int)A.status[0];
    quality_count = max(1, min(parent_count, A.elite_size / 4));
    active = min(A.max_strength, 2 + (A.generation - (int)A.status[4]) / 10);
  }
  const int n = A.n, m = 2 * n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int threads = blockDim.x, warps = threads / 32;
  const int child0 = blockIdx.x * threads, child = child0 + tid;
  const int nc = min(threads, A.population - child0);
  int32_t* prefix = reinterpret_cast<int32_t*>(smem);                       // [prefix_cap][m] inclusive prefix sums
  Row* rows = reinterpret_cast<Row*>(prefix + (size_t)A.prefix_cap * m);  // [threads][n] both layers of a row
  uint64_t rng = A.seed ^ (0x9e3779b97f4a7c15ULL * (uint64_t)(child + 1)) ^
                 (0xbf58476d1ce4e5b9ULL * (uint64_t)(A.generation + 1));
  int parent = child;
  if (child < A.population && child >= parent_count) {
    const uint64_t pick = xs64(rng);
    const int pool = (pick & 255ULL) < 160ULL ? quality_count : parent_count;
    parent = (int)(xs64(rng) % (uint64_t)pool);
  }
  s_parent[tid] = parent;
  __syncthreads();
#pragma unroll 4
  for (int c = warp; c < nc; c += warps) {  // the parents' rows into the children's, a warp per child
    const int32_t* src_p = A.pp + (size_t)s_parent[c] * n;
    const int32_t* src_q = A.pq + (size_t)s_parent[c] * n;
#pragma unroll
    for (int k = 0; k < (kMaxN + 31) / 32; ++k) {
      const int r = lane + 32 * k;
      if (r < n) rows[c * n + r] = Row{(Cell)src_p[r], (Cell)src_q[r]};
    }
  }
  bool use_prefix = parent_count <= A.prefix_cap;  // uniform
  if (use_prefix) {
    bool negative = false;
#pragma unroll 4
    for (int p = warp; p < parent_count; p += warps) {
      int acc[kMaxM / 32 + 1];
#pragma unroll
      for (int k = 0; k < kMaxM / 32 + 1; ++k) {
        const int e = 32 * k + lane;
        acc[k] = e < m ? A.pbad[p * m + e] : 0;
        negative |= acc[k] < 0 || acc[k] > 0x7fffffff / kMaxM;  // keeps every prefix sum below 2^31
      }
      int before = 0;
#pragma unroll
      for (int k = 0; k < kMaxM / 32 + 1; ++k) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, acc[k], o);
          if (lane >= o) acc[k] = (int)((unsigned)acc[k] + (unsigned)y);
        }
        const int e = 32 * k + lane;
        if (e < m) prefix[p * m + e] = (int)((unsigned)acc[k] + (unsigned)before);
        before = (int)((unsigned)before + (unsigned)__shfl_sync(0xffffffffu, acc[k], 31));
      }
    }
    use_prefix = !__syncthreads_or(negative);
  } else {
    __syncthreads();
  }
  const bool record = A.child_moves != nullptr;
  if (child < A.population) {
    if (record) A.child_parent[child] = parent;
    if (child < parent_count) {
      if (record) A.child_nmoves[child] = 0;
    } else {
      Cell* cs = reinterpret_cast<Cell*>(rows + tid * n);
      const int32_t* bad = A.pbad + (size_t)parent * m;
      const int32_t* pre = prefix + parent * m;
      int total = 0;
      if (use_prefix) {
        total = pre[m - 1];
      } else {
        for (int e = 0; e < m; ++e) total += bad[e];
      }
      const Remainder by_total((uint64_t)(int64_t)(total ? total : 1)), by_slots((uint64_t)m);
      int strength, nmoves = 0;
      if ((xs64(rng) & 31ULL) == 0ULL)
        strength = 1 + (int)(xs64(rng) % (uint64_t)A.max_strength);
      else
        strength = 1 + (int)(xs64(rng) % (uint64_t)active);
      for (int step = 0; step < strength; ++step) {
        for (int attempt = 0; attempt < 32; ++attempt) {
          int u;
          if ((int)(xs64(rng) % 100ULL) < A.bad_bias) {
            if (total) {
              const int t = (int)by_total.of(xs64(rng));
              if (use_prefix) {  // first u with prefix[u] > t; prefix[m - 1] = total > t
                int lo = 0, hi = m - 1;
                while (lo < hi) {
                  const int mid = (lo + hi) >> 1;
                  if (pre[mid] > t) hi = mid;
                  else lo = mid + 1;
                }
                u = lo;
              } else {
                int r = t;
                for (u = 0; u < m - 1; ++u) {
                  r -= bad[u];
                  if (r < 0) break;
                }
              }
            } else {
              u = (int)by_slots.of(xs64(rng));
            }
          } else {
            u = (int)by_slots.of(xs64(rng));
          }
          const int v = (int)by_slots.of(xs64(rng));
          if ((u >> 1) == (v >> 1)) continue;
          const int cu = cs[u], cv = cs[v];
          if (cu == cv) continue;
          if (cv == cs[u ^ 1] || cu == cs[v ^ 1]) continue;  // the other point of each row
          cs[u] = (Cell)cv;
          cs[v] = (Cell)cu;
          if (record && nmoves < A.moves_cap) A.child_moves[(size_t)child * A.moves_cap + nmoves] = u | (v << 8);
          ++nmoves;
          break;
        }
      }
      if (record) A.child_nmoves[child] = nmoves;
    }
  }
  __syncthreads();
  for (int c = warp; c < nc; c += warps) {  // coalesced rows, a warp per child
    int32_t* dst_p = A.cp + (size_t)(child0 + c) * n;
    int32_t* dst_q = A.cq + (size_t)(child0 + c) * n;
    for (int r = lane; r < n; r += 32) {
      const Row both = rows[c * n + r];
      dst_p[r] = both.x;
      dst_q[r] = both.y;
    }
  }
}

// --------------------------------------------------------------------------
// Children's scores by exact deltas: warp per child, the parent's columns and
// badness in shared memory, then each recorded swap applied with its exact dE
// and the exact update of every badness (pair_move, accepting every move).  E
// and badness equal a full recount.
// --------------------------------------------------------------------------
constexpr int kDeltaWarps = 26;
constexpr size_t kDeltaWarpBytes = 2 * sizeof(uint32_t) * DenseNumbering::kWords + sizeof(int) * kMaxM + 152;
constexpr size_t kDeltaSmem = kCompactLutBytes + kDeltaWarps * kDeltaWarpBytes;
static_assert(kDeltaSmem <= 227 * 1024 && kDeltaWarpBytes % 8 == 0, "child_delta_kernel shared memory");

struct DeltaArgs {
  const int32_t* ep;
  const int32_t* eq;
  const int32_t* ebad;
  const int32_t* es;
  const int32_t* parent;
  const int32_t* moves;
  const int32_t* nmoves;
  int moves_cap, n, population;
  const int64_t* status;
  const uint16_t* lut4;
  int32_t* scores;
  int32_t* badness;
  uint32_t* error_word;
};

__global__ void __launch_bounds__(kDeltaWarps * 32, 1) child_delta_kernel(const DeltaArgs A) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem[];
  if (A.status[1] == 0) return;  // uniform: the search has reached E = 0
  uint16_t* lut4 = reinterpret_cast<uint16_t*>(smem);
  compact_lut_copy(lut4, A.lut4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* hist = reinterpret_cast<uint32_t*>(smem + kCompactLutBytes + (size_t)warp * kDeltaWarpBytes);
  for (int i = lane; i < 2 * DenseNumbering::kWords; i += 32) hist[i] = 0u;
  __syncthreads();
  const int n = A.n, m = 2 * n, nt = (m + 31) >> 5;
  WarpState W;
  W.m = m;
  W.lane = lane;
  W.bs = reinterpret_cast<int*>(hist + 2 * DenseNumbering::kWords);
  W.cs = reinterpret_cast<uint8_t*>(W.bs + kMaxM);
  uint32_t err = 0;
  for (int c = blockIdx.x * kDeltaWarps + warp; c < A.population; c += gridDim.x * kDeltaWarps) {
    const int par = A.parent[c];
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {
      const int s = W.slot(t);
      W.key2[t] = 0;
      if (s < m) {
        const int col = (s & 1) ? A.eq[(size_t)par * n + (s >> 1)] : A.ep[(size_t)par * n + (s >> 1)];
        W.cs[s] = (uint8_t)col;
        W.key2[t] = 2 * ((s >> 1) * kLutW + col);
        W.bs[s] = A.ebad[(size_t)par * m + s];
      }
    }
    __syncwarp();
    int E = A.es[par];
    const int k_end = min(A.nmoves[c], A.moves_cap);
    for (int k = 0; k < k_end; ++k) {
      const int mv = A.moves[(size_t)c * A.moves_cap + k];
      int dE;
      pair_move_any<DenseNumbering>(W, lut4, hist, nt, prepare_move(W, mv & 0xFF, (mv >> 8) & 0xFF),
                                    [](int) { return true; }, E, err, &dE);
    }
    if (lane == 0) A.scores[c] = E;
    for (int s = lane; s < m; s += 32) A.badness[(size_t)c * m + s] = W.bs[s];
    __syncwarp();
  }
  if (lane == 0 && err && A.error_word) atomicOr(A.error_word, err);
}


// One thread seeds (each word follows from the one before) in shared memory.
__global__ void __launch_bounds__(32) py_seed_kernel(uint32_t* state, uint64_t seed) {
  __shared__ uint32_t mt[kMT];
  if (threadIdx.x == 0) {
    const uint32_t key[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
    const int len = (seed >> 32) ? 2 : 1;
    uint32_t last = mt[0] = 19650218u;
    for (int i = 1; i < kMT; ++i) mt[i] = last = 1812433253u * (last ^ (last >> 30)) + (uint32_t)i;
    int i = 1, j = 0;
    last = mt[0];
    for (int k = kMT > len ? kMT : len; k; --k) {
      mt[i] = last = (mt[i] ^ ((last ^ (last >> 30)) * 1664525u)) + key[j] + (uint32_t)j;
      ++i;
      ++j;
      if (i >= kMT) {
        mt[0] = last;
        i = 1;
      }
      if (j >= len) j = 0;
    }
    for (int k = kMT - 1; k; --k) {
      mt[i] = last = (mt[i] ^ ((last ^ (last >> 30)) * 1566083941u)) - (uint32_t)i;
      ++i;
      if (i >= kMT) {
        mt[0] = last;
        i = 1;
      }
    }
    mt[0] = 0x80000000u;
  }
  __syncwarp();
  for (int i = threadIdx.x; i < kMT; i += 32) state[i] = mt[i];
  if (threadIdx.x == 0) state[kMT] = kMT;  // position: the first draw twists
}

__global__ void py_shuffle_kernel(uint32_t* state, int32_t* values, int count) {
  __shared__ uint32_t mt[kMT], out[kMT], seen[65536 / 32];
  for (int i = threadIdx.x; i < kMT; i += blockDim.x) mt[i] = state[i];
  for (int i = threadIdx.x; i < 65536 / 32; i += blockDim.x) seen[i] = 0u;
  __syncthreads();
  if (threadIdx.x < 32) {
    int idx = (int)state[kMT];
    py_shuffle_warp(mt, out, idx, values, count, seen, threadIdx.x);
    if (threadIdx.x == 0) state[kMT] = (uint32_t)idx;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kMT; i += blockDim.x) state[i] = mt[i];
}

// The state twist by part of a CTA, out of place: dst = twist(src).  Word k of the
// sequential in-place update reads the old words k, k + 1 and k + 397 (k < 227)
// or the new word k - 227 (k >= 227; for k = 623 also the new word 0), so three
// phases of at most 227 words each reproduce it.
__device__ __forceinline__ uint32_t mt_mix(uint32_t hi_word, uint32_t lo_word, uint32_t far) {
  const uint32_t y = (hi_word & 0x80000000u) | (lo_word & 0x7fffffffu);
  return far ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}

// Eight warps do it, with barriers of their own; the callers' __syncthreads follows.
constexpr int kTwistThreads = 256;
__device__ __forceinline__ void twist_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kTwistThreads) : "memory"); }
__device__ void mt_twist(const uint32_t* src, uint32_t* dst) {
  const int t = threadIdx.x;  // < kTwistThreads
  if (t < 227) dst[t] = mt_mix(src[t], src[t + 1], src[t + 397]);
  twist_barrier();
  if (t < 227) dst[227 + t] = mt_mix(src[227 + t], src[228 + t], dst[t]);
  twist_barrier();
  if (t < 170) {
    const int k = 454 + t;
    dst[k] = mt_mix(src[k], k == kMT - 1 ? dst[0] : src[k + 1], dst[k - 227]);
  }
  twist_barrier();
}

// Exclusive scan over the CTA (thread order) of a 32-bit value, with the total.
// wsum: 32 words of shared memory; consecutive calls must alternate between
// two such buffers (a call's buffer is rewritten only after every thread has
// passed the next call's barriers).  blockDim.x == 1024.
__device__ __forceinline__ uint32_t cta_exscan32(uint32_t v, uint32_t* wsum, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  total = wsum[31];
  return (warp ? wsum[warp - 1] : 0u) + x - v;
}

// The shuffle's draws for the steps i, i - 1, ..., 1 from the tempered outputs
// out[pos, avail) (consecutive blocks of the stream): step s takes words in order
// until one has r = word >> (32 - bit_length(s + 1)) <= s, and j = r goes to
// jstep[s].  No swap is made.  Word w (w = 0, 1, ... from pos) serves step
// i - A_w, A_w the number of accepted words before it, so the accepted words are
// the one fixed point of "accept w if it fits step i - A_w": word 0's answer is
// right in any iteration, word w's in the one after those before it.  Iterating
// over all words at once is much faster than that bound, as a wrong A_w misjudges
// only words whose r lies between the two steps.  It starts from the expected
// number of acceptances (below), and 5000 words take 2 to 8 iterations while
// steps are many and 10 to 20 at the end, all widths together.
//
// Warp v holds the words 160 v .. 160 v + 159, lane by lane; ballots give A_w
// inside the warp, one barrier per iteration the counts of the warps before.  A warp
// whose count before and whose answers did not change keeps them.  Every thread calls it with the same i >= 1 and
// pos < avail; i and pos advance.  tot: 64 words, cut: one, of shared memory.
// blockDim.x == 1024.
//
// A window of 10,000 steps: its draws with the twists take 26 us, 63 us by a call
// per draw width with scans of thread counts and the last 2048 steps by one warp.
constexpr int kDrawPer = 5;  // 5120 words per call: one batch of kSelBatch blocks
// Whether step >= 1 takes the word: word >> clz(step + 1) <= step, that is
// word < (step + 1) << clz(step + 1), which a float's mantissa holds (step < 2^23; a
// conversion of its own, as clz and int-to-float run at a quarter of the rate or less).
__device__ __forceinline__ bool draw_fits(uint32_t word, int step) {
  const float x = __uint_as_float(0x4B000000u | (uint32_t)(step + 1)) - 8388608.0f;
  return step >= 1 && word < (__float_as_uint(x) << 8 | 0x80000000u);
}
__device__ void shuffle_draws_cta(const uint32_t* out, int avail, int& pos, int& i, uint16_t* jstep, uint32_t* tot,
                                  int* cut) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int nw = min(min(avail - pos, (int)blockDim.x * kDrawPer), 2 * i + 64);
  const int w0 = warp * 32 * kDrawPer + lane;
  // Steps of bit length k (2^(k - 1) - 1 <= s) accept with probability (s + 1) / 2^k,
  // so s + 1 falls by 1 / 2^k of itself per word: from 2^k to 2^(k - 1) in
  // 2^k ln 2 words, and with l ln 2 words left at bit length k,
  // s + 1 = 2^(k - 2 + l / 2^k).
  const int bits = 32 - __clz((uint32_t)i + 1u);
  const float size = (float)(1u << bits);
  const float left = size * (2.0f + __log2f((float)(i + 1) / size));  // l at word 0
  uint32_t word[kDrawPer], accepted[kDrawPer];
  int each[kDrawPer], count = 0;
#pragma unroll
  for (int e = 0; e < kDrawPer; ++e) {
    const int w = w0 + 32 * e;
    const bool in = w < nw;
    word[e] = in ? out[pos + w] : ~0u;  // a word that never fits
    const float l = left - (float)w * 1.442695f;
    int step = 0;
    if (l >= 1.0f) {  // k from the exponent, l / 2^k from the mantissa
      const uint32_t l_bits = __float_as_uint(l);
      const float quarter = __uint_as_float((l_bits & 0x7F800000u) - (2u << 23));  // 2^(k - 2)
      const float ratio = __uint_as_float((l_bits & 0x007FFFFFu) | 0x3F800000u);
      step = min(i, (int)(quarter * exp2f(ratio)) - 1);
    }
    accepted[e] = __ballot_sync(0xffffffffu, draw_fits(word[e], step));
    count += each[e] = __popc(accepted[e]);
  }
  int before = -1, all, changed = 1;
  for (int it = 0;; it ^= 32) {
    if (lane == 0) tot[it + warp] = (uint32_t)count;
    const int any = __syncthreads_or(changed);
    const uint32_t c = tot[it + lane];
    if (!any) {
      all = (int)__reduce_add_sync(0xffffffffu, c);
      break;
    }
    const int now_before = (int)__reduce_add_sync(0xffffffffu, lane < warp ? c : 0u);
    const bool settled = !changed && now_before == before;  // uniform in the warp
    before = now_before;
    changed = 0;
    if (settled) continue;
    // the counts of the previous answers: no word waits for another
    int first = i - before;
    count = 0;
#pragma unroll
    for (int e = 0; e < kDrawPer; ++e) {
      const int step = first - __popc(accepted[e] & below);
      const unsigned now = __ballot_sync(0xffffffffu, draw_fits(word[e], step));
      first -= each[e];
      changed |= now != accepted[e];
      accepted[e] = now;
      count += each[e] = __popc(now);
    }
  }
  // the words up to the last step's, or all
#pragma unroll
  for (int e = 0; e < kDrawPer; ++e) {
    if ((accepted[e] >> lane) & 1u) {
      const int step = i - (before + __popc(accepted[e] & below));
      jstep[step] = (uint16_t)(word[e] >> __clz((uint32_t)step + 1u));
      if (step == 1) *cut = w0 + 32 * e + 1;
    }
    before += each[e];
  }
  __syncthreads();
  pos += all == i ? *cut : nw;
  i -= all;
}

// --------------------------------------------------------------------------
// Selection (one CTA of kSelThreads threads).
// --------------------------------------------------------------------------
constexpr int kSelThreads = 1024;
constexpr int kMaxPopulation = 65536;
constexpr int kMaxElite = 2048;
constexpr int kSelBatch = 8;  // MT state blocks generated per batch for the shuffle's draws
constexpr int kSelHistBins = 4096;  // one-pass selection when every score is below this
static_assert(kSelBatch * kMT <= kSelThreads * kDrawPer, "one resolver call covers a batch");
static_assert(kSelHistBins <= kSelBatch * kMT && kSelHistBins % 1024 == 0, "histogram in the MT words' space");

constexpr int kSelWarps = kSelThreads / 32;
static_assert(kSelWarps == 32, "a warp's lanes hold the counts of all warps");

struct SelArgs {
  const int32_t* scores;  // [population]
  int population, elite_size, energy_window;
  int64_t* status;
  uint32_t* rng;          // [625]
  int32_t* selected;      // [elite_size]
};

// The draws of random.shuffle over `count` items (steps s = count - 1 .. 1,
// j_s = _randbelow(s + 1)) into jstep[s], from the state in shared memory (mt,
// the current block; idx the position in it, 624 when it is used up), with
// no swap made.  The CTA twists and tempers the state blocks up to kSelBatch
// at a time (words: kSelBatch blocks; out: their outputs) and resolves the draws
// (shuffle_draws_cta).  On return mt and idx are the state CPython leaves: the
// block of the last draw and the position after it.  Every thread calls it; idx
// is uniform.
__device__ void shuffle_steps_cta(uint32_t* mt, int& idx, int count, uint16_t* jstep, uint32_t* words, uint32_t* out,
                                  uint32_t* tot, int* cut) {
  const int tid = threadIdx.x;
  int steps_left = count - 1;
  if (steps_left >= 1) {
    int pos = idx;
    if (pos < kMT) {
      for (int k = tid; k < kMT; k += blockDim.x) words[k] = mt[k];
      __syncthreads();
    } else {  // the current block is used up: the first draw twists
      if (tid < kTwistThreads) mt_twist(mt, words);
      pos = 0;
    }
    for (;;) {
      // a step takes 1.4 words on average
      const int blocks = min(kSelBatch, (pos + steps_left + steps_left / 2 + 64) / kMT + 1);
      if (tid < kTwistThreads)
        for (int g = 1; g < blocks; ++g) mt_twist(words + (g - 1) * kMT, words + g * kMT);
      __syncthreads();
      for (int k = tid; k < blocks * kMT; k += blockDim.x) out[k] = mt_temper(words[k]);
      __syncthreads();
      while (steps_left >= 1 && pos < blocks * kMT)
        shuffle_draws_cta(out, blocks * kMT, pos, steps_left, jstep, tot, cut);
      if (steps_left < 1) break;  // uniform
      // the next batch's first block, twisted out of place: a batch of one block
      // moves to the outputs, which are used up
      const uint32_t* from = words + (blocks - 1) * kMT;
      if (blocks == 1) {  // uniform
        for (int k = tid; k < kMT; k += blockDim.x) out[k] = words[k];
        __syncthreads();
        from = out;
      }
      if (tid < kTwistThreads) mt_twist(from, words);
      pos = 0;
    }
    const int last = pos - 1;  // >= 0: every round uses at least one word
    for (int k = tid; k < kMT; k += blockDim.x) mt[k] = words[(last / kMT) * kMT + k];
    idx = last % kMT + 1;
  }
  __syncthreads();
}

// The scores are read from memory once: they stay in shared memory in 16 bits (in
// jstep's space, free until the shuffle) if none is larger.  One CTA's latency
// bounds it.  32,768 children, 64 picks, a window of 10,000: 41 us, of which the
// draws take 26; 163 us with a score pass per step and the window traced by
// warps reading all steps.
struct SelSmem {
  uint64_t keys[kMaxElite];              // the keys below T; then picked, start_next
  uint32_t mt[kMT];
  int32_t order[kMaxElite];              // score-order prefix
  uint32_t mark[kMaxPopulation / 32];    // children picked
  uint32_t window[kMaxPopulation / 32];  // children within the energy window
  uint32_t offset[kMaxPopulation / 32];  // of these, those before the word's first
  // draws' outputs and state blocks; before, the histogram; after, with what the
  // window leaves of jstep, the table of step 5
  uint16_t jstep[kMaxPopulation];  // j of shuffle step s; before, the scores
  uint32_t words[2 * kSelBatch * kMT];
  uint32_t hist[256];
  uint32_t wsum[64];
  int misc[4];
};
static_assert(sizeof(SelSmem) <= 227 * 1024, "select_kernel shared memory");

__global__ void __launch_bounds__(kSelThreads, 1) select_kernel(const SelArgs A) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char smem[];
  SelSmem& S = *reinterpret_cast<SelSmem*>(smem);
  const int P = A.population, E = A.elite_size, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  if (A.status[1] == 0) return;  // uniform: the search has reached E = 0
  const int64_t limit = A.status[1] + (int64_t)A.energy_window;
  for (int i = tid; i < kMaxPopulation / 32; i += kSelThreads) S.mark[i] = 0u;
  for (int i = tid; i < kMT; i += kSelThreads) S.mt[i] = A.rng[i];

  // 1. T = the E-th smallest score.  One pass counts the scores below 4096, one
  //    bin per value (in the MT words' space), and finds the highest; if all are
  //    counted a scan over the bins tells T, otherwise a radix select over the
  //    32-bit scores, 8 bits a pass, from the highest byte that any score uses.
  uint32_t* const bins = S.words;
  uint16_t* const kept = S.jstep;
  for (int i = tid; i < kSelHistBins; i += kSelThreads) bins[i] = 0u;
  if (tid == 0) S.misc[2] = 0;
  __syncthreads();
  uint32_t top = 0u;
#pragma unroll 8
  for (int i = tid; i < P; i += kSelThreads) {
    const uint32_t x = (uint32_t)A.scores[i];
    top = max(top, x);
    kept[i] = (uint16_t)x;
    if (x < (uint32_t)kSelHistBins) atomicAdd(&bins[x], 1u);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) S.hist[warp] = top;
  __syncthreads();
  top = __reduce_max_sync(0xffffffffu, S.hist[lane]);
  __syncthreads();
  uint32_t T;
  int remaining;  // 1-based rank of the E-th element among the scores equal to T
  const bool in_16 = top <= 0xFFFFu;  // uniform
  if (top < (uint32_t)kSelHistBins) {
    constexpr int kPerT = kSelHistBins / kSelThreads;
    uint32_t c[kPerT], local = 0u;
#pragma unroll
    for (int k = 0; k < kPerT; ++k) {
      c[k] = bins[kPerT * tid + k];
      local += c[k];
    }
    uint32_t tot;
    int run = (int)cta_exscan32(local, S.wsum, tot);
    if (run < E && run + (int)local >= E) {  // this thread's bins hold the E-th smallest score
#pragma unroll
      for (int k = 0; k < kPerT; ++k) {
        if (run + (int)c[k] >= E) {
          S.misc[0] = kPerT * tid + k;
          S.misc[1] = E - run;
          break;
        }
        run += (int)c[k];
      }
    }
    __syncthreads();
    T = (uint32_t)S.misc[0];
    remaining = S.misc[1];
  } else {
    int shift = 24;
    while (shift > 0 && (top >> shift) == 0u) shift -= 8;  // the skipped high bytes are zero in every score
    uint32_t prefix = 0u, mask = 0u;
    remaining = E;
    for (; shift >= 0; shift -= 8) {
      for (int i = tid; i < 256; i += kSelThreads) S.hist[i] = 0u;
      __syncthreads();
#pragma unroll 4
      for (int b = 32 * warp; b < P; b += kSelThreads) {  // warp-uniform trip count; equal digits add once per warp
        const int i = b + lane;
        const uint32_t x = i < P ? (uint32_t)A.scores[i] : 0u;
        const bool valid = i < P && (x & mask) == prefix;
        const unsigned act = __ballot_sync(0xffffffffu, valid);
        if (valid) {
          const uint32_t digit = (x >> shift) & 255u;
          const unsigned peers = __match_any_sync(act, digit);
          if (lane == __ffs(peers) - 1) atomicAdd(&S.hist[digit], (uint32_t)__popc(peers));
        }
      }
      __syncthreads();
      if (tid == 0) {
        int before = 0, d = 0;
        for (; d < 255; ++d) {
          if (before + (int)S.hist[d] >= remaining) break;
          before += (int)S.hist[d];
        }
        S.misc[0] = d;
        S.misc[1] = remaining - before;
      }
      __syncthreads();
      prefix |= (uint32_t)S.misc[0] << shift;
      mask |= 255u << shift;
      remaining = S.misc[1];
      __syncthreads();
    }
    T = prefix;
  }
  const int n_less = E - remaining;  // scores below T; then `remaining` ties at T by index

  // 2. a thread per 32 children: the keys below T (at most E - 1) in any order,
  //    the first `remaining` ties at T in index order, and the children within
  //    the energy window
  int n_window = 0, n_tie = 0;
  for (int w0 = 0; w0 < (P + 31) / 32; w0 += kSelThreads) {
    const int w = w0 + tid, i0 = 32 * w;
    uint32_t lt = 0u, tie = 0u, within = 0u;
    if (i0 < P) {
      if (in_16) {
        const uint32_t* const two = reinterpret_cast<const uint32_t*>(kept) + 16 * w;
        const int turn = tid & 15;  // the lanes in different banks
        const int low = (int)min(limit, (int64_t)0xFFFF);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const uint32_t v = two[(k + turn) & 15];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int x = h ? (int)(v >> 16) : (int)(v & 0xFFFFu);
            if (x < (int)T) lt |= 1u << (2 * k + h);
            if (x == (int)T) tie |= 1u << (2 * k + h);
            if (x <= low) within |= 1u << (2 * k + h);
          }
        }
        lt = __funnelshift_l(lt, lt, 2 * turn);
        tie = __funnelshift_l(tie, tie, 2 * turn);
        within = __funnelshift_l(within, within, 2 * turn);
      } else {
        for (int k = 0; k < 32; ++k) {
          const int x = A.scores[min(i0 + k, P - 1)];
          if ((uint32_t)x < T) lt |= 1u << k;
          if ((uint32_t)x == T) tie |= 1u << k;
          if ((int64_t)x <= limit) within |= 1u << k;
        }
      }
      const uint32_t valid = P - i0 < 32 ? (1u << (P - i0)) - 1u : ~0u;
      lt &= valid;
      tie &= valid;
      within &= valid;
    }
    uint32_t tot;  // at most 32768 of each in a round
    const uint32_t before = cta_exscan32((uint32_t)__popc(tie) << 16 | (uint32_t)__popc(within),
                                         S.wsum + ((w0 / kSelThreads) & 1) * 32, tot);
    if (i0 < P) {
      S.window[w] = within;
      S.offset[w] = (uint32_t)n_window + (before & 0xFFFFu);
      int at = lt ? atomicAdd(&S.misc[2], __popc(lt)) : 0;
      for (; lt; lt &= lt - 1u) {
        const int i = i0 + __ffs(lt) - 1;
        S.keys[at++] = (uint64_t)(uint32_t)(in_16 ? (int)kept[i] : A.scores[i]) << 32 | (uint32_t)i;
      }
      for (int r = n_tie + (int)(before >> 16); tie && r < remaining; tie &= tie - 1u, ++r)
        S.order[n_less + r] = i0 + __ffs(tie) - 1;
    }
    n_window += (int)(tot & 0xFFFFu);
    n_tie += (int)(tot >> 16);
  }
  // 3. the keys below T sorted by (score, index): up to 512 by counting the lower
  //    ones, a warp per key (64 keys: 0.5 us, bitonic 2.9 us), more with a bitonic sort
  if (n_less <= 512) {
    __syncthreads();
    for (int k = warp; k < n_less; k += kSelWarps) {
      const uint64_t key = S.keys[k];
      int lower = 0;
      for (int j = lane; j < n_less; j += 32) lower += S.keys[j] < key;
      lower = __reduce_add_sync(0xffffffffu, lower);
      if (lane == 0) S.order[lower] = (int32_t)(uint32_t)key;
    }
  } else {
    int width = 1;
    while (width < n_less) width <<= 1;
    for (int i = n_less + tid; i < width; i += kSelThreads) S.keys[i] = ~0ull;
    __syncthreads();
    for (int size = 2; size <= width; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = tid; i < width; i += kSelThreads) {
          const int j = i ^ stride;
          if (j > i) {
            const bool up = (i & size) == 0;
            const uint64_t a = S.keys[i], b = S.keys[j];
            if ((a > b) == up) {
              S.keys[i] = b;
              S.keys[j] = a;
            }
          }
        }
        __syncthreads();
      }
    }
    for (int i = tid; i < n_less; i += kSelThreads) S.order[i] = (int32_t)(uint32_t)S.keys[i];
  }
  __syncthreads();  // the scores are no longer read, nor the keys

  // 4. the draws of the window list's shuffle (gpu_device_search.py:340-373):
  //    the j of every step s in jstep[s], no swap made (shuffle_steps_cta).
  {
    int idx = (int)A.rng[kMT];  // uniform
    shuffle_steps_cta(S.mt, idx, n_window, S.jstep, S.words, S.words + kSelBatch * kMT, S.wsum, &S.misc[0]);
    if (tid == 0) A.rng[kMT] = (uint32_t)idx;
  }

  // 5. the first K = min(E, window) shuffled positions.  Step s fixes position s
  //    for good, so position p holds what sat at j_p before step p; going back
  //    through the later steps p+1, p+2, ... (applied before it), the item moves
  //    only where a step's j equals its position, to that step.  From then on its
  //    position is the step it came from, so what it needs is next[x], the first
  //    step s > x with j_s = x; and for the start, the first step s > p with
  //    j_s = j_p: j_p <= p < K, so a search of the steps below K, then start_next,
  //    the first step from K on.  One pass over the steps fills both, the table
  //    of next for a part of the positions at a time if the window leaves no room
  //    for all (above 28,500).
  const int K = min(E, n_window);
  int32_t* const picked = reinterpret_cast<int32_t*>(S.keys);        // [K] positions, then children
  uint32_t* const start_next = reinterpret_cast<uint32_t*>(S.keys) + kMaxElite;  // [K]
  const int table_at = (n_window + 1) & ~1;
  uint32_t* const next = reinterpret_cast<uint32_t*>(S.jstep + table_at);
  const int room = (kMaxPopulation - table_at) / 2 + 2 * kSelBatch * kMT;
  for (int i = tid; i < K; i += kSelThreads) start_next[i] = UINT32_MAX;
  for (int lo = 0; lo < n_window; lo += room) {
    const int hi = min(n_window, lo + room);
    for (int i = tid; i < hi - lo; i += kSelThreads) next[i] = UINT32_MAX;
    __syncthreads();
    for (int s = 1 + tid; s < n_window; s += kSelThreads) {
      const int j = S.jstep[s];
      if (j < s && j >= lo && j < hi) atomicMin(&next[j - lo], (uint32_t)s);
      if (lo == 0 && s >= K && j < K) atomicMin(&start_next[j], (uint32_t)s);
    }
    __syncthreads();
    if (lo == 0) {  // the starts, a warp each
      for (int p = warp; p < K; p += kSelWarps) {
        const int j = p ? (int)S.jstep[p] : 0;
        uint32_t first = start_next[j];
        for (int s0 = p + 1; s0 < K; s0 += 32) {
          const unsigned m = __ballot_sync(0xffffffffu, s0 + lane < K && (int)S.jstep[s0 + lane] == j);
          if (m) {  // uniform
            first = (uint32_t)(s0 + __ffs(m) - 1);
            break;
          }
        }
        if (lane == 0) picked[p] = first == UINT32_MAX ? ~j : (int32_t)first;  // complemented: it stays there
      }
      __syncthreads();
    }
    for (int p = tid; p < K; p += kSelThreads) {
      if (picked[p] < 0) continue;
      uint32_t at = (uint32_t)picked[p];
      while (at < (uint32_t)hi) {
        const uint32_t to = next[at - (uint32_t)lo];
        if (to == UINT32_MAX) break;
        at = to;
      }
      picked[p] = at < (uint32_t)hi ? ~(int32_t)at : (int32_t)at;
    }
    __syncthreads();
  }
  // the window's position to its child
  for (int p = tid; p < K; p += kSelThreads) {
    const uint32_t pos = (uint32_t)~picked[p];
    int w = 0, w_end = (P + 31) / 32;  // the last word whose offset is not above pos
    while (w_end - w > 1) {
      const int mid = (w + w_end) >> 1;
      if (S.offset[mid] <= pos) w = mid;
      else w_end = mid;
    }
    uint32_t m = S.window[w];
    for (uint32_t r = pos - S.offset[w]; r > 0u; --r) m &= m - 1u;
    picked[p] = 32 * w + __ffs(m) - 1;
  }

  // 6. the pick (gpu_device_search.py:340-373): the best quarter, the shuffled
  //    window without them (its children are distinct), then the score order
  const int quality = max(1, E / 4);
  for (int r = tid; r < quality; r += kSelThreads) {
    const int c = S.order[r];
    atomicOr(&S.mark[c >> 5], 1u << (c & 31));
    A.selected[r] = c;
  }
  __syncthreads();
  int sel = quality;
  for (int part = 0; part < 2; ++part) {
    const int32_t* const list = part ? S.order : picked;
    const int end = part ? E : K;
    for (int r0 = 0; r0 < end && sel < E; r0 += kSelThreads) {  // uniform
      const int r = r0 + tid;
      const int c = r < end ? list[r] : 0;
      const bool open = r < end && !((S.mark[c >> 5] >> (c & 31)) & 1u);
      uint32_t tot;
      const int at = sel + (int)cta_exscan32(open, S.wsum + ((r0 / kSelThreads + part) & 1) * 32, tot);
      if (open && at < E) {
        A.selected[at] = c;
        if (part == 0) atomicOr(&S.mark[c >> 5], 1u << (c & 31));
      }
      sel += (int)tot;
      __syncthreads();
    }
  }
  for (int i = tid; i < kMT; i += kSelThreads) A.rng[i] = S.mt[i];
}

// The shuffle's draws alone (shuffle_steps_cta), for callers that apply the
// permutation themselves and for tests: j of step s in jout[s], jout[0] = 0.
constexpr size_t kStepsSmem = sizeof(uint32_t) * (kMT + 2 * kSelBatch * kMT) + sizeof(uint16_t) * kMaxPopulation;
__global__ void __launch_bounds__(kSelThreads, 1) py_steps_kernel(uint32_t* state, int count, int32_t* jout) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* mt = reinterpret_cast<uint32_t*>(smem);
  uint32_t* words = mt + kMT;
  uint32_t* out = words + kSelBatch * kMT;
  uint16_t* jstep = reinterpret_cast<uint16_t*>(out + kSelBatch * kMT);
  __shared__ uint32_t tot[64];
  __shared__ int cut;
  for (int i = threadIdx.x; i < kMT; i += blockDim.x) mt[i] = state[i];
  __syncthreads();
  int idx = (int)state[kMT];
  shuffle_steps_cta(mt, idx, count, jstep, words, out, tot, &cut);
  for (int s = threadIdx.x; s < count; s += blockDim.x) jout[s] = s == 0 ? 0 : (int32_t)jstep[s];
  for (int i = threadIdx.x; i < kMT; i += blockDim.x) state[i] = mt[i];
  if (threadIdx.x == 0) state[kMT] = (uint32_t)idx;
}

// pick rows r = child rows selected[r]
__global__ void gather_kernel(const int32_t* cp, const int32_t* cq, const int32_t* cs, const int32_t* cbad,
                              const int32_t* selected, int n, const int64_t* status, int32_t* __restrict__ pp,
                              int32_t* __restrict__ pq, int32_t* __restrict__ ps, int32_t* __restrict__ pbad) {
  chain_begin();
  if (status[1] == 0) return;
  const int r = blockIdx.x, c = selected[r];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    pp[(size_t)r * n + i] = cp[(size_t)c * n + i];
    pq[(size_t)r * n + i] = cq[(size_t)c * n + i];
  }
  for (int i = threadIdx.x; i < 2 * n; i += blockDim.x) pbad[(size_t)r * 2 * n + i] = cbad[(size_t)c * 2 * n + i];
  if (threadIdx.x == 0) ps[r] = cs[c];
}

// --------------------------------------------------------------------------
// Ranking (one CTA): rank_elites (gpu_device_search.py:185-197) is a stable
// sort by elite_key = (E, max badness, sum of squared badness); each element's
// rank is the number of keys before it.  Then the best-so-far update
// (gpu_device_search.py:388-396; set-up: :305-310).  A warp per state: 64 states
// at n = 75 take 11 us, 23 us by a thread each.
// --------------------------------------------------------------------------
constexpr int kRankThreads = 1024;

struct RankArgs {
  const int32_t* pp;
  const int32_t* pq;
  const int32_t* pbad;
  const int32_t* ps;
  int count;       // picks to rank (set-up: the base count; a generation: elite_size)
  int n, generation;
  int32_t* ep;
  int32_t* eq;
  int32_t* ebad;
  int32_t* es;
  int64_t* status;
  int32_t* best_p;
  int32_t* best_q;
  int32_t* history;
  int history_len;
};

__global__ void __launch_bounds__(kRankThreads, 1) rank_kernel(const RankArgs A) {
  chain_begin();
  __shared__ int32_t s_score[kMaxElite], s_max[kMaxElite], s_rank[kMaxElite];
  __shared__ int64_t s_ss[kMaxElite];
  __shared__ int s_first, s_improved;
  if (A.generation > 0 && A.status[1] == 0) return;  // uniform
  const int C = A.count, m = 2 * A.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = warp; i < C; i += kRankThreads / 32) {  // a warp per state
    int mx = INT32_MIN;
    int64_t ss = 0;
#pragma unroll
    for (int k = 0; k < kSlotsPerLane; ++k) {
      const int s = lane + 32 * k;
      const int b = s < m ? A.pbad[(size_t)i * m + s] : INT32_MIN;
      mx = max(mx, b);
      if (s < m) ss += (int64_t)b * b;
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) {
      s_score[i] = A.ps[i];
      s_max[i] = mx;
      s_ss[i] = ss;
    }
  }
  __syncthreads();
  for (int i = warp; i < C; i += kRankThreads / 32) {
    const int a0 = s_score[i], a1 = s_max[i];
    const int64_t a2 = s_ss[i];
    int r = 0;
    for (int j = lane; j < C; j += 32) {
      const int b0 = s_score[j], b1 = s_max[j];
      const int64_t b2 = s_ss[j];
      const bool less = b0 < a0 || (b0 == a0 && (b1 < a1 || (b1 == a1 && (b2 < a2 || (b2 == a2 && j < i)))));
      r += less;
    }
    r = __reduce_add_sync(0xffffffffu, r);
    if (lane == 0) {
      s_rank[i] = r;
      if (r == 0) s_first = i;
    }
  }
  __syncthreads();
  for (int i = warp; i < C; i += kRankThreads / 32) {  // a warp per state
    const size_t to = (size_t)s_rank[i], from = (size_t)i;
#pragma unroll
    for (int k = 0; k < kSlotsPerLane; ++k) {
      const int s = lane + 32 * k;
      if (s < m) A.ebad[to * m + s] = A.pbad[from * m + s];
      if (s < A.n) {
        A.ep[to * A.n + s] = A.pp[from * A.n + s];
        A.eq[to * A.n + s] = A.pq[from * A.n + s];
      }
    }
  }
  for (int i = tid; i < C; i += kRankThreads) A.es[s_rank[i]] = s_score[i];
  if (tid == 0) {
    const int f = s_first;
    const int64_t k0 = s_score[f], k1 = s_max[f], k2 = s_ss[f];
    int64_t* st = A.status;
    const bool improved = A.generation == 0 || k0 < st[1] || (k0 == st[1] && (k1 < st[2] || (k1 == st[2] && k2 < st[3])));
    if (improved) {
      st[1] = k0;
      st[2] = k1;
      st[3] = k2;
      if (A.generation > 0) st[4] = A.generation;
    }
    st[0] = C;
    if (A.generation == 0) st[4] = 0;
    st[5] = A.generation;
    st[6] = k0;
    st[7] = improved && A.generation > 0;
    if (A.history != nullptr && A.generation >= 1 && A.generation <= A.history_len) {
      A.history[2 * (A.generation - 1)] = (int32_t)k0;
      A.history[2 * (A.generation - 1) + 1] = (int32_t)st[1];
    }
    s_improved = improved;
  }
  __syncthreads();
  if (s_improved) {
    const int f = s_first;
    for (int k = tid; k < A.n; k += kRankThreads) {
      A.best_p[k] = A.pp[(size_t)f * A.n + k];
      A.best_q[k] = A.pq[(size_t)f * A.n + k];
    }
  }
}

}  // namespace beam
}  // namespace n3

namespace n3host {

// mutate_kernel over `population` children; the parents' prefix sums are staged
// when at most `parents_bound` parents fit in kMutPrefixMaxBytes.
template <class Row>
static int launch_mutate(n3::beam::MutArgs A, int parents_bound, cudaStream_t st) {
  using namespace n3::beam;
  constexpr int kMost = kMutThreads * (int)sizeof(short2) / (int)sizeof(Row);
  const int m = 2 * A.n;
  const int cap = (int)(kMutPrefixMaxBytes / (sizeof(int32_t) * (size_t)m));
  A.prefix_cap = parents_bound <= cap ? parents_bound : 0;
  int threads = 64;
  while (threads < kMost && (A.population + threads - 1) / threads > sm_count()) threads *= 2;
  const size_t bytes = (size_t)m * (sizeof(Row) / 2 * (size_t)threads + sizeof(int32_t) * (size_t)A.prefix_cap);
  N3_TRY(allow_smem(reinterpret_cast<const void*>(mutate_kernel<Row>), kMutSmemMax));
  return launch_chained("beam mutate_kernel", mutate_kernel<Row>, (A.population + threads - 1) / threads, threads, bytes,
                        st, A);
}

static int check_beam(const n3_beam* b) {
  if (b == nullptr) return set_error(N3_ERR_ARG, "null beam descriptor");
  if (b->n < 3 || b->n > N3_MAX_N) return set_error(N3_ERR_RANGE, "beam: n must lie in [3, %d]", N3_MAX_N);
  if (b->elite_size < 2 || b->elite_size > n3::beam::kMaxElite)
    return set_error(N3_ERR_RANGE, "beam: elite_size must lie in [2, %d]", n3::beam::kMaxElite);
  if (b->population < b->elite_size || b->population > n3::beam::kMaxPopulation)
    return set_error(N3_ERR_RANGE, "beam: population must lie in [elite_size, %d]", n3::beam::kMaxPopulation);
  if (b->max_strength < 1 || b->max_strength > 4096)
    return set_error(N3_ERR_RANGE, "beam: max_strength must lie in [1, 4096]");
  if (b->bad_bias < 0 || b->bad_bias > 100) return set_error(N3_ERR_RANGE, "beam: bad_bias must lie in [0, 100]");
  if (b->energy_window < 0) return set_error(N3_ERR_RANGE, "beam: energy_window must be non-negative");
  const void* ptrs[] = {b->elite_p, b->elite_q, b->elite_badness, b->elite_scores, b->child_p, b->child_q,
                        b->child_scores, b->pick_p, b->pick_q, b->pick_badness, b->pick_scores, b->selected,
                        b->rng, b->status, b->best_p, b->best_q, b->child_parent, b->child_moves,
                        b->child_nmoves, b->child_badness};
  for (const void* p : ptrs)
    if (p == nullptr) return set_error(N3_ERR_ARG, "beam: null buffer");
  return N3_OK;
}

static n3::beam::RankArgs rank_args(const n3_beam* b, int count, int generation) {
  n3::beam::RankArgs R;
  R.pp = b->pick_p;
  R.pq = b->pick_q;
  R.pbad = b->pick_badness;
  R.ps = b->pick_scores;
  R.count = count;
  R.n = b->n;
  R.generation = generation;
  R.ep = b->elite_p;
  R.eq = b->elite_q;
  R.ebad = b->elite_badness;
  R.es = b->elite_scores;
  R.status = b->status;
  R.best_p = b->best_p;
  R.best_q = b->best_q;
  R.history = b->history;
  R.history_len = b->history_len;
  return R;
}

}  // namespace n3host

extern "C" {

int n3_beam_mutate(const int32_t* parent_p, const int32_t* parent_q, const int32_t* parent_badness,
                   int parent_count, int quality_count, int n, int population, int active_strength,
                   int max_strength, int bad_bias, uint64_t seed, int generation, int32_t* child_p,
                   int32_t* child_q, void* stream) {
  if (!parent_p || !parent_q || !parent_badness || !child_p || !child_q)
    return n3host::set_error(N3_ERR_ARG, "beam mutate: null buffer");
  if (n < 2 || n > N3_MAX_N || parent_count < 1 || population < 0 || quality_count < 1 ||
      quality_count > parent_count || active_strength < 1 || max_strength < 1 || bad_bias < 0 || bad_bias > 100)
    return n3host::set_error(N3_ERR_RANGE, "beam mutate: argument out of range");
  if (population == 0) return N3_OK;
  n3::beam::MutArgs A;
  A.pp = parent_p;
  A.pq = parent_q;
  A.pbad = parent_badness;
  A.parent_count = parent_count;
  A.quality_count = quality_count;
  A.active_strength = active_strength;
  A.status = nullptr;
  A.elite_size = parent_count;
  A.n = n;
  A.population = population;
  A.max_strength = max_strength;
  A.bad_bias = bad_bias;
  A.generation = generation;
  A.seed = seed;
  A.cp = child_p;
  A.cq = child_q;
  A.child_parent = A.child_moves = A.child_nmoves = nullptr;
  A.moves_cap = 0;
  return n3host::launch_mutate<int2>(A, parent_count, (cudaStream_t)stream);
}

int n3_py_random_seed(uint32_t* state, uint64_t seed, void* stream) {
  if (!state) return n3host::set_error(N3_ERR_ARG, "null RNG state");
  n3::beam::py_seed_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(state, seed);
  return n3host::check_launch("py_seed_kernel");
}

int n3_py_random_shuffle(uint32_t* state, int32_t* values, int count, void* stream) {
  if (!state || (!values && count > 0)) return n3host::set_error(N3_ERR_ARG, "null shuffle buffer");
  if (count < 0 || count > n3::beam::kMaxPopulation) return n3host::set_error(N3_ERR_RANGE, "shuffle: bad count");
  n3::beam::py_shuffle_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(state, values, count);
  return n3host::check_launch("py_shuffle_kernel");
}

int n3_py_shuffle_steps(uint32_t* state, int count, int32_t* steps_j, void* stream) {
  if (!state || (!steps_j && count > 0)) return n3host::set_error(N3_ERR_ARG, "null shuffle-steps buffer");
  if (count < 0 || count > n3::beam::kMaxPopulation)
    return n3host::set_error(N3_ERR_RANGE, "shuffle steps: count %d outside [0, %d]", count, n3::beam::kMaxPopulation);
  N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(n3::beam::py_steps_kernel), n3::beam::kStepsSmem));
  n3::beam::py_steps_kernel<<<1, n3::beam::kSelThreads, n3::beam::kStepsSmem, (cudaStream_t)stream>>>(state, count,
                                                                                                      steps_j);
  return n3host::check_launch("py_steps_kernel");
}

int n3_beam_init(const n3_beam* b, int base_count, void* stream) {
  N3_TRY(n3host::check_beam(b));
  if (base_count < 1 || base_count > b->elite_size) return n3host::set_error(N3_ERR_RANGE, "beam: bad base count");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t rows = sizeof(int32_t) * (size_t)base_count * b->n;
  if (cudaMemcpyAsync(b->pick_p, b->elite_p, rows, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(b->pick_q, b->elite_q, rows, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return n3host::set_error(N3_ERR_CUDA, "beam init: copy failed");
  N3_TRY(n3_score_population(b->pick_p, b->pick_q, base_count, b->n, b->pick_scores, b->pick_badness, stream));
  n3::beam::rank_kernel<<<1, n3::beam::kRankThreads, 0, st>>>(n3host::rank_args(b, base_count, 0));
  N3_TRY(n3host::check_launch("beam rank_kernel"));
  return n3_py_random_seed(b->rng, b->seed, stream);
}

int n3_beam_generation(const n3_beam* b, int generation, void* stream) {
  N3_TRY(n3host::check_beam(b));
  if (generation < 1) return n3host::set_error(N3_ERR_RANGE, "beam: generations count from 1");
  cudaStream_t st = (cudaStream_t)stream;
  n3::beam::MutArgs M;
  M.pp = b->elite_p;
  M.pq = b->elite_q;
  M.pbad = b->elite_badness;
  M.parent_count = M.quality_count = M.active_strength = 0;
  M.status = b->status;
  M.elite_size = b->elite_size;
  M.n = b->n;
  M.population = b->population;
  M.max_strength = b->max_strength;
  M.bad_bias = b->bad_bias;
  M.generation = generation;
  M.seed = b->seed;
  M.cp = b->child_p;
  M.cq = b->child_q;
  M.child_parent = b->child_parent;
  M.child_moves = b->child_moves;
  M.child_nmoves = b->child_nmoves;
  M.moves_cap = b->max_strength;
  N3_TRY(n3host::launch_mutate<short2>(M, b->elite_size, st));
  N3_TRY(n3host::ensure_device_tables());
  N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(n3::beam::child_delta_kernel), n3::beam::kDeltaSmem));
  n3::beam::DeltaArgs D;
  D.ep = b->elite_p;
  D.eq = b->elite_q;
  D.ebad = b->elite_badness;
  D.es = b->elite_scores;
  D.parent = b->child_parent;
  D.moves = b->child_moves;
  D.nmoves = b->child_nmoves;
  D.moves_cap = b->max_strength;
  D.n = b->n;
  D.population = b->population;
  D.status = b->status;
  D.lut4 = n3host::dir4_lut_device_ptr();
  D.scores = b->child_scores;
  D.badness = b->child_badness;
  D.error_word = b->error_word;
  const int dgrid = (b->population + n3::beam::kDeltaWarps - 1) / n3::beam::kDeltaWarps;
  N3_TRY(n3host::launch_chained("beam child_delta_kernel", n3::beam::child_delta_kernel,
                                dgrid < n3host::sm_count() ? dgrid : n3host::sm_count(), n3::beam::kDeltaWarps * 32,
                                n3::beam::kDeltaSmem, st, D));
  N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(n3::beam::select_kernel), sizeof(n3::beam::SelSmem)));
  n3::beam::SelArgs S;
  S.scores = b->child_scores;
  S.population = b->population;
  S.elite_size = b->elite_size;
  S.energy_window = b->energy_window;
  S.status = b->status;
  S.rng = b->rng;
  S.selected = b->selected;
  N3_TRY(n3host::launch_chained("beam select_kernel", n3::beam::select_kernel, 1, n3::beam::kSelThreads,
                                sizeof(n3::beam::SelSmem), st, S));
  N3_TRY(n3host::launch_chained("beam gather_kernel", n3::beam::gather_kernel, b->elite_size, 128, 0, st, b->child_p,
                                b->child_q, b->child_scores, b->child_badness, b->selected, b->n, b->status, b->pick_p,
                                b->pick_q, b->pick_scores, b->pick_badness));
  return n3host::launch_chained("beam rank_kernel", n3::beam::rank_kernel, 1, n3::beam::kRankThreads, 0, st,
                                n3host::rank_args(b, b->elite_size, generation));
}

}  // extern "C"
