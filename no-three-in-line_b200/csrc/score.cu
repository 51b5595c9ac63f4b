// (a) Population scoring: exact collinear-triple counts of populations of states.
//
// Two independent kernels and a cross-checked pair of launches:
//
// * Determinant count (replaces src/no_three_75/gpu.py:13-42 and
//   src/no_three_75/gpu_device_search.py:118-161).  Every triple i<j<k is
//   tested once with an exact cross product, at its middle slot j.  The
//   two slots of j's row are pivots together; the triple's other two points
//   lie in rows above and below that row.  The larger side sits in lane
//   registers, the smaller side is broadcast from shared memory one row (two
//   slots) at a time, so one pair of products serves four tests.  Triples
//   holding j's row partner are skipped: two points of a row and a third point
//   in another row are never collinear.
//
// * Normalised-slope line count (the counting form of
//   src/no_three_75/verifier_b.py:8-33).  From every slot, the later slots are
//   told apart by gcd-reduced undirected direction; C(c,2) pairs of a
//   direction's c slots make collinear triples with it.  The gcd reduction is
//   tabulated once per device by build_dir_lut_kernel.
//
// The plain scores (n3_score_population, n3_score_columns) take the faster of
// the two for the grid size; n3_score_determinants is the first alone,
// n3_score_slope the second, n3_score_checked runs both and flags disagreement on
// the device.
//
// What bounds them, at 4096 n = 75 states:
//   det_kernel<.., 1, false>   278 us (304 us on 32-bit integers).  Four tests are
//       four packed multiply-add-pipe instructions, two compares and two adds
//       that read 22 registers; at two register reads a cycle and scheduler that
//       is 11 cycles (11.5 measured for the loop alone), the loop runs 4850 times
//       per state on 592 schedulers: 194 us.  The rest is the loop's overhead
//       over 19 rows on average and the pivots' set-up.
//   tag_kernel, E alone         74 us, with badness 88 us (86 and 122 us with
//       4-bit counters; the determinant count with badness took 464 us).  Shared
//       memory is busy 87 % of the cycles: a direction load (3.5 cycles for 32
//       random 2-byte words), a tag store and a tag load (2.9 each) per 32 slots.
#include <cstdio>
#include <type_traits>

#include "score_impl.cuh"

namespace n3 {

__device__ __align__(16) uint16_t g_dir_lut[kCompactLutBytes / 2];
__device__ __align__(16) uint16_t g_dir_lut_full[kFullLutBytes / 2];
__device__ __align__(16) uint16_t g_prim4_lut[kCompactLutBytes / 2];
__device__ __align__(16) uint16_t g_dir4_lut[kCompactLutBytes / 2];
__device__ int g_dir_count;

__device__ __forceinline__ int gcd_dev(int a, int b) {
  a = a < 0 ? -a : a;
  b = b < 0 ? -b : b;
  while (b) {
    const int t = a % b;
    a = b;
    b = t;
  }
  return a;
}

// Entry e = p * kLutW + (q + kMaxN - 1) names a primitive direction iff
// gcd(p, |q|) == 1 with p > 0, or (p, q) == (0, 1).
__device__ __forceinline__ bool is_primitive(int e) {
  const int p = e / kLutW, q = e % kLutW - (kMaxN - 1);
  return p == 0 ? q == 1 : gcd_dev(p, q) == 1;
}

// One block: numbers the primitive directions in (p, q) order, then maps every
// difference vector to the id of its gcd-reduced direction, to four times that
// (kDirCount for (0, 0)) and to four times the key p * kLutW + q of the direction.
__global__ void __launch_bounds__(1024) build_dir_lut_kernel() {
  __shared__ uint16_t prim[kLutSize];
  __shared__ int scan[1024];
  const int tid = threadIdx.x;
  constexpr int per = (kLutSize + 1023) / 1024;
  const int lo = tid * per, hi = min(lo + per, kLutSize);
  int c = 0;
  for (int e = lo; e < hi; ++e) c += is_primitive(e);
  scan[tid] = c;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {  // inclusive Hillis-Steele scan
    const int v = tid >= off ? scan[tid - off] : 0;
    __syncthreads();
    scan[tid] += v;
    __syncthreads();
  }
  int id = scan[tid] - c;
  for (int e = lo; e < hi; ++e) prim[e] = is_primitive(e) ? (uint16_t)id++ : (uint16_t)0xFFFFu;
  if (tid == 1023) g_dir_count = scan[1023];
  __syncthreads();
  for (int e = tid; e < kLutSize; e += 1024) {
    const int dx = e / kLutW, dy = e % kLutW - (kMaxN - 1);
    const int g = gcd_dev(dx, dy);
    uint16_t v = 0xFFFFu, step = 0;  // (0, 0) has no direction
    if (g) {
      const int p = dx / g;
      const int q = p == 0 ? 1 : dy / g;  // (0, -1) ~ (0, 1)
      v = prim[p * kLutW + q + (kMaxN - 1)];
      step = (uint16_t)(4 * (p * kLutW + q));
    }
    g_dir_lut[e] = v;
    g_prim4_lut[e] = step;
    g_dir4_lut[e] = (uint16_t)(4 * (g ? v : kDirCount));
  }
}

// The full signed table from the compact one (one entry per thread).
__global__ void build_full_lut_kernel() {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= kFullLutSize) return;
  const int dx = e / kLutW - (kMaxN - 1), dy = e % kLutW - (kMaxN - 1);
  g_dir_lut_full[e] = (dx == 0 && dy == 0) ? (uint16_t)0 : (uint16_t)dir_id(g_dir_lut, dx, dy);
}

struct PQSource {
  const int32_t* p;
  const int32_t* q;
  __device__ __forceinline__ int col(int b, int n, int s) const {
    const size_t base = (size_t)b * n + (s >> 1);
    return (s & 1) ? q[base] : p[base];
  }
};

struct ColSource {
  const int16_t* c;
  __device__ __forceinline__ int col(int b, int n, int s) const { return c[(size_t)b * 2 * n + s]; }
};

constexpr int kDetWarps = 4;  // small CTAs: 4096 states spread evenly over 148 SMs

// E by determinants: on packed floats when every column lies on the grid, else
// on 32-bit integers (det_state), as the count has always taken any columns.  On
// small grids, with a warp per state, integers are ahead whatever the columns (their
// set-up is shorter; 20,011 states, us, packed floats against integers: n = 10 20.8
// and 19.5, n = 14 32.4 and 31.5, n = 20 56.0 and 56.7; with badness n = 20 81.2 and
// 83.5, but 5000 of them 28.3 and 27.1).
// PARTS = 1: a warp per state, kDetWarps states per CTA.  PARTS > 1, for fewer
// states than warps that the GPU can hold: a CTA of PARTS warps per state,
// which share its pivot rows.
template <class Src, int PARTS, bool BAD>
__global__ void __launch_bounds__((PARTS > 1 ? PARTS : kDetWarps) * 32)
    det_kernel(Src src, int B, int n, int32_t* __restrict__ scores, int32_t* __restrict__ badness) {
  __shared__ float4 rows_all[PARTS > 1 ? 1 : kDetWarps][kMaxN];
  __shared__ int bad_all[PARTS > 1 || !BAD ? 1 : kDetWarps][BAD ? kMaxM : 1];
  __shared__ int total;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = PARTS > 1 ? blockIdx.x : blockIdx.x * kDetWarps + warp;
  if (b >= B) return;
  constexpr int kIntegersMaxN = PARTS > 1 ? 0 : BAD ? 20 : 16;
  float4* rows4 = rows_all[PARTS > 1 ? 0 : warp];
  int* bad = BAD ? bad_all[PARTS > 1 ? 0 : warp] : nullptr;
  const int first = PARTS > 1 ? threadIdx.x : lane, stride = PARTS > 1 ? PARTS * 32 : 32;
  bool on_grid = n > kIntegersMaxN;
  if (BAD)
    for (int s = first; s < 2 * n; s += stride) bad[s] = 0;
  for (int r = first; on_grid && r < n; r += stride) {
    const int c0 = src.col(b, n, 2 * r), c1 = src.col(b, n, 2 * r + 1);
    on_grid = on_grid && (unsigned)c0 < (unsigned)kMaxN && (unsigned)c1 < (unsigned)kMaxN;
    rows4[r] = make_float4((float)c0, (float)c0, (float)c1, (float)c1);
  }
  if (PARTS > 1) {
    if (threadIdx.x == 0) total = 0;
    on_grid = __syncthreads_and(on_grid);
  } else {
    on_grid = __all_sync(0xffffffffu, on_grid);
    __syncwarp();
  }
  int cnt = 0;
  if (on_grid) {  // uniform
    cnt = det_state_f<BAD>(rows4, n, lane, PARTS > 1 ? warp : 0, PARTS, bad);
  } else if (PARTS == 1 || warp == 0) {
    int* cs = reinterpret_cast<int*>(rows4);
    for (int s = lane; s < 2 * n; s += 32) cs[s] = src.col(b, n, s);
    __syncwarp();
    cnt = det_state<BAD>(cs, n, lane, bad);
  }
  cnt = warp_sum(cnt);
  if (PARTS > 1) {
    if (lane == 0 && cnt) atomicAdd(&total, cnt);
    __syncthreads();
    cnt = total;
  } else {
    __syncwarp();
  }
  if (first == 0) scores[b] = cnt;
  if (BAD)
    for (int s = first; s < 2 * n; s += stride) badness[(size_t)b * 2 * n + s] = bad[s];
}

// The slope count (tag_state): the warps of a CTA share one compact direction table
// and take consecutive states, a warp each; where fewer states than warps are left,
// `parts` warps (a power of two) share a state's centres, so that few states fill
// the SMs too (64 n = 75 states with badness: 8.9 us; 51 us with a warp each) and a
// batch just above a round of all warps does not cost two (4300 n = 75 states with
// badness: 96 us, 167 with the last 156 states on six CTAs, a warp each).
//   kCount   E and, if wanted, badness of any states: one with a column off the
//            grid or two equal points in a row, which has no line count, is
//            counted by determinants (det_state), so the results are the
//            determinant count's for every input.
//   kSlope   the same, but such a state gets -1 (and the error bits, if wanted).
//   kChecked E and the badness's sum compared with the determinant counts already
//            in `scores` (written by det_kernel on the same stream).
// NT, the slots a lane holds, bounds the unrolled work per centre and, with the ids of
// the directions that a grid of 16 NT rows has, a warp's shared memory: 32 warps fit
// up to n = 48 (4096 n = 14 states with badness: 8.6 us, 16.4 with NT = 5 and 28
// warps).
enum TagMode { kCount, kSlope, kChecked };
// What a CTA does with its states: whole rounds of a warp each, a state shared by several
// warps, or rounds and then the last states shared.  (A kernel that can do both takes 2
// to 10 % longer where it needs only one.)
enum TagPlan { kRounds, kShared, kRoundsThenShared };
constexpr int kTagMaxParts = 16;     // warps that share a state
constexpr int kTagMinThreads = 256;  // threads that copy the table when few states are scored
// Compact ids of the directions with dx < 16 NT (any dy), rounded up to 8: ids go by (dx, dy).
__host__ __device__ constexpr int tag_ids(int nt) {
  return nt == 1 ? 1400 : nt == 2 ? 2896 : nt == 3 ? 4352 : kDirCount;
}
__host__ __device__ constexpr int tag_warps(int nt) { return nt <= 3 ? 32 : 28; }  // 28 x 148 = 4144 states at once
__host__ __device__ constexpr size_t tag_warp_bytes(int nt) { return tag_ids(nt) + sizeof(uint32_t) * 32 * nt; }
__host__ __device__ constexpr size_t tag_smem(int nt, int warps) {
  return kCompactLutBytes + (size_t)warps * tag_warp_bytes(nt);
}
static_assert(tag_smem(3, tag_warps(3)) <= 227 * 1024 && tag_smem(5, tag_warps(5)) <= 227 * 1024,
              "tag_kernel shared memory");
static_assert(tag_ids(1) >= (int)sizeof(int) * 32 && tag_ids(2) >= (int)sizeof(int) * 64, "columns fit in a warp's tags");
static_assert(tag_ids(1) % 8 == 0 && tag_ids(2) % 8 == 0 && tag_ids(3) % 8 == 0 && tag_ids(5) % 8 == 0, "alignment");

// State b's table keys for tag_state, its word[] cleared; returns the error bits of
// columns outside [0, limit) and equal points in a row (the same in every lane), which
// are told after such columns have been moved to the edge, as they always were.
template <class Src, int NT>
__device__ __forceinline__ uint32_t tag_load(const Src& src, int b, int n, int limit, int lane, int (&key)[NT],
                                             uint32_t* __restrict__ word) {
  uint32_t err = 0;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int s = lane + 32 * t;
    const bool in = s < 2 * n;
    const int c = in ? src.col(b, n, s) : 0;
    const int inside = min(max(c, 0), limit - 1);
    // the two points of a row are neighbouring lanes
    const int other = __shfl_xor_sync(0xffffffffu, inside, 1);
    if (in && inside != c) err |= kErrColumnRange;
    if (in && inside == other) err |= kErrDuplicate;
    key[t] = in ? (s >> 1) * kLutW + c : -1;
    if (in) word[s] = 0u;
  }
  return __reduce_or_sync(0xffffffffu, err);
}

// The states without a line count among first, first + step, ... below end, and
// `extra` if it is not negative, by determinants.  Called once at a warp's end, so that
// the code of these rare states takes no registers from tag_kernel's loops (inlined
// there it cost 20,011 n = 17 states 47 us against 36).
template <class Src, bool BAD>
static __device__ __noinline__ void count_rare(Src src, int n, int lane, int first, int end, int step, int extra,
                                               int* __restrict__ cs, int* __restrict__ bad,
                                               int32_t* __restrict__ scores, int32_t* __restrict__ badness) {
  for (int i = first;; i += step) {
    const int b = i < end ? i : extra;
    bool rare = false;
    for (int r = lane; b >= 0 && r < n; r += 32) {
      const int c0 = src.col(b, n, 2 * r), c1 = src.col(b, n, 2 * r + 1);
      rare = rare || (unsigned)c0 >= (unsigned)kMaxN || (unsigned)c1 >= (unsigned)kMaxN || c0 == c1;
    }
    if (__any_sync(0xffffffffu, rare)) {
      for (int s = lane; s < 2 * n; s += 32) {
        cs[s] = src.col(b, n, s);
        if (BAD) bad[s] = 0;
      }
      __syncwarp();
      const int e = warp_sum(det_state<BAD>(cs, n, lane, bad));
      if (lane == 0) scores[b] = e;
      __syncwarp();
      if (BAD)
        for (int s = lane; s < 2 * n; s += 32) badness[(size_t)b * 2 * n + s] = bad[s];
      __syncwarp();
    }
    if (i >= end) return;
  }
}

template <class Src, int MODE, bool BAD, int NT, int PLAN>
__global__ void __launch_bounds__(tag_warps(NT) * 32, 1) tag_kernel(Src src, int B, int n, int W,
                                                                     const uint16_t* __restrict__ g_lut,
                                                                     int32_t* __restrict__ scores,
                                                                     int32_t* __restrict__ badness,
                                                                     int32_t* __restrict__ mismatch,
                                                                     uint32_t* __restrict__ error_word) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int total_all[tag_warps(NT)];
  __shared__ volatile uint8_t rare[tag_warps(NT)];  // kCount: the warp met a state without a line count
  uint16_t* lut = reinterpret_cast<uint16_t*>(smem);
  compact_lut_copy(lut, g_lut);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp >= W) return;  // it only helped to copy the table
  const int m = 2 * n;
  uint8_t* tag = smem + kCompactLutBytes + (size_t)warp * tag_warp_bytes(NT);
  uint32_t* word = reinterpret_cast<uint32_t*>(tag + tag_ids(NT));
  if (MODE == kCount && lane == 0) rare[warp] = 0;

  // State b by `parts` warps, this one `part` of them; the group's badness and count live with its first
  // warp.  sync: the group's barrier.
  const auto score = [&](auto split, int b, int group, int part, int parts, const auto& sync) {
    constexpr bool SPLIT = decltype(split)::value;
    uint32_t* bad = word - (size_t)part * (tag_warp_bytes(NT) / sizeof(uint32_t));
    int* total = total_all + group;
    int key[NT];
    const uint32_t err = tag_load<Src, NT>(src, b, n, MODE == kCount ? kMaxN : n, lane, key, word);
    if (SPLIT && part == 0 && lane == 0) *total = 0;
    sync();
    if (err) {  // no line count exists
      if (part == 0) {
        if (MODE == kCount) {
          if (lane == 0) rare[warp] = 1;
        } else {
          if (lane == 0) {
            scores[b] = -1;
            if (error_word) atomicOr(error_word, err);
            if (MODE == kChecked) atomicAdd(mismatch, 1);
          }
          if (BAD)
            for (int s = lane; s < m; s += 32) badness[(size_t)b * m + s] = -1;
        }
      }
      sync();
      return;
    }
    int e = tag_state<BAD, SPLIT, NT>(key, m, lut, tag, lane, word, bad, part, parts);
    if (SPLIT) {
      if (lane == 0) atomicAdd(total, e);
      sync();
      e = *total;
    } else {
      __syncwarp();
    }
    if (part == 0) {
      int bad_sum = 0;
      if (BAD)
        for (int s = lane; s < m; s += 32) {
          const int v = (int)bad[s];
          badness[(size_t)b * m + s] = v;
          bad_sum += v;
        }
      if (MODE == kChecked) {  // scores[b] holds the determinant count of this state
        if (BAD) bad_sum = warp_sum(bad_sum);
        const uint32_t differ = checked_error(scores[b], e, BAD, bad_sum);
        if (lane == 0 && differ) {
          atomicAdd(mismatch, 1);
          if (error_word) atomicOr(error_word, differ);
        }
      } else if (lane == 0) {
        scores[b] = e;
      }
    }
    sync();
  };

  const int b_begin = (int)((int64_t)B * blockIdx.x / gridDim.x);
  const int b_end = (int)((int64_t)B * (blockIdx.x + 1) / gridDim.x);
  int b = b_begin;
  if (PLAN != kShared)
    for (; PLAN == kRounds ? b + warp < b_end : 2 * (b_end - b) > W; b += W)
      if (PLAN == kRounds || b + warp < b_end) score(std::false_type{}, b + warp, 0, 0, 1, [] { __syncwarp(); });
  int shared = -1;  // the state that this warp led a group at
  if (const int left = b_end - b; PLAN != kRounds && left > 0) {
    int parts = 2;
    while (parts < kTagMaxParts && 2 * parts * left <= W) parts *= 2;
    const int group = warp / parts, part = warp % parts;
    if (group < left) {
      if (part == 0) shared = b + group;
      // at most 16 groups: barrier ids 0 .. 15, the block's own is done with
      score(std::true_type{}, b + group, group, part, parts,
            [&] { asm volatile("barrier.sync %0, %1;" ::"r"(group), "r"(32 * parts) : "memory"); });
    }
  }
  __syncwarp();
  if (MODE == kCount && rare[warp])
    count_rare<Src, BAD>(src, n, lane, b_begin + warp, PLAN == kRounds ? b_end : b, W, shared, reinterpret_cast<int*>(tag),
                         reinterpret_cast<int*>(word), scores, badness);
}

// Both counts of the checked score side by side: the determinants wait for the
// multiply-add pipe (71 % of issue slots used), the tags for shared memory (70 %), so
// `tag_warps` of a CTA's 32 warps take the tags and the rest the determinants, a
// quarter of a state's pivot rows at a time.  A CTA owns `per` consecutive states
// and compares the counts (checked_error) kCheckedStates states at a time.
constexpr int kCheckedStates = 56;
struct CheckedShared {
  int det[kCheckedStates], slope[kCheckedStates], bad_sum[kCheckedStates];
  uint32_t err[kCheckedStates], off_grid[kCheckedStates];
  int next_det, next_tag;
};
__host__ __device__ constexpr size_t checked_smem(int tag_warps, int n) {
  return kCompactLutBytes + (size_t)tag_warps * kTagWarpBytes + (size_t)kCheckedStates * n * sizeof(float4) +
         sizeof(CheckedShared);
}

constexpr size_t kCheckedMaxSmem = checked_smem(14, kMaxN);
static_assert(kCheckedMaxSmem <= 227 * 1024, "checked_kernel shared memory");

template <bool BAD>
__global__ void __launch_bounds__(1024, 1) checked_kernel(ColSource src, int B, int n, int per, int tag_warps,
                                                          const uint16_t* __restrict__ g_lut,
                                                          int32_t* __restrict__ scores,
                                                          int32_t* __restrict__ badness,
                                                          int32_t* __restrict__ mismatch,
                                                          uint32_t* __restrict__ error_word) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* lut = reinterpret_cast<uint16_t*>(smem);
  float4* rows = reinterpret_cast<float4*>(smem + kCompactLutBytes);  // [kCheckedStates][n]
  unsigned char* tags = smem + kCompactLutBytes + (size_t)kCheckedStates * n * sizeof(float4);
  CheckedShared& S = *reinterpret_cast<CheckedShared*>(tags + (size_t)tag_warps * kTagWarpBytes);
  compact_lut_copy(lut, g_lut);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, det_warps = 32 - tag_warps, m = 2 * n;
  const int b_end = min(B, (int)(blockIdx.x + 1) * per);
  for (int b0 = blockIdx.x * per; b0 < b_end; b0 += kCheckedStates) {
    const int count = min(kCheckedStates, b_end - b0);
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      S.det[i] = 0;
      S.off_grid[i] = 0u;
    }
    if (threadIdx.x == 0) S.next_det = S.next_tag = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < count * n; i += blockDim.x) {
      const int k = i / n, r = i - k * n;
      const int c0 = src.col(b0 + k, n, 2 * r), c1 = src.col(b0 + k, n, 2 * r + 1);
      if ((unsigned)c0 >= (unsigned)kMaxN || (unsigned)c1 >= (unsigned)kMaxN) S.off_grid[k] = 1u;
      rows[i] = make_float4((float)c0, (float)c0, (float)c1, (float)c1);
    }
    __syncthreads();
    if (warp < det_warps) {
      for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(&S.next_det, 1);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= 4 * count) break;
        const int k = task >> 2, part = task & 3;
        float4* rows4 = rows + k * n;
        int cnt = 0;
        if (!S.off_grid[k]) {  // uniform
          cnt = det_state_f<false>(rows4, n, lane, part, 4, nullptr);
        } else if (part == 0) {
          int* cs = reinterpret_cast<int*>(rows4);
          for (int s = lane; s < m; s += 32) cs[s] = src.col(b0 + k, n, s);
          __syncwarp();
          cnt = det_state<false>(cs, n, lane, nullptr);
        }
        cnt = warp_sum(cnt);
        if (lane == 0 && cnt) atomicAdd(&S.det[k], cnt);
      }
    } else {
      uint8_t* tag = tags + (size_t)(warp - det_warps) * kTagWarpBytes;
      uint32_t* word = reinterpret_cast<uint32_t*>(tag + kDirCount);
      for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(&S.next_tag, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= count) break;
        int key[kSlotsPerLane], e = -1;
        const uint32_t err = tag_load(src, b0 + k, n, n, lane, key, word);
        __syncwarp();
        if (!err) e = tag_state<BAD>(key, m, lut, tag, lane, word, word);
        __syncwarp();
        int bad_sum = 0;
        if (BAD) {
          for (int s = lane; s < m; s += 32) {
            const int v = err ? -1 : (int)word[s];
            badness[(size_t)(b0 + k) * m + s] = v;
            bad_sum += v;
          }
          bad_sum = warp_sum(bad_sum);
        }
        if (lane == 0) {
          S.slope[k] = e;
          S.bad_sum[k] = bad_sum;
          S.err[k] = err;
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < count; k += blockDim.x) {
      uint32_t err = S.err[k];
      scores[b0 + k] = err ? -1 : S.det[k];
      if (!err) err = checked_error(S.det[k], S.slope[k], BAD, S.bad_sum[k]);
      if (err) {
        atomicAdd(mismatch, 1);
        if (error_word) atomicOr(error_word, err);
      }
    }
    __syncthreads();
  }
}

}  // namespace n3

namespace n3host {

int build_dir_lut(cudaStream_t st) {
  n3::build_dir_lut_kernel<<<1, 1024, 0, st>>>();
  N3_TRY(check_launch("build_dir_lut_kernel"));
  n3::build_full_lut_kernel<<<(n3::kFullLutSize + 255) / 256, 256, 0, st>>>();
  N3_TRY(check_launch("build_full_lut_kernel"));
  int count = 0;
  if (cudaMemcpyFromSymbolAsync(&count, n3::g_dir_count, sizeof(int), 0, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return check_launch("direction table read-back");
  if (count != n3::kDirCount)
    return set_error(N3_ERR_CUDA, "direction table has %d ids, expected %d", count, n3::kDirCount);
  return N3_OK;
}

const uint16_t* dir_lut_device_ptr() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, n3::g_dir_lut) != cudaSuccess) return nullptr;
  return static_cast<const uint16_t*>(p);
}

const uint16_t* prim4_lut_device_ptr() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, n3::g_prim4_lut) != cudaSuccess) return nullptr;
  return static_cast<const uint16_t*>(p);
}

const uint16_t* dir4_lut_device_ptr() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, n3::g_dir4_lut) != cudaSuccess) return nullptr;
  return static_cast<const uint16_t*>(p);
}

const uint16_t* dir_lut_full_device_ptr() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, n3::g_dir_lut_full) != cudaSuccess) return nullptr;
  return static_cast<const uint16_t*>(p);
}

static int check_common(int B, int n, const void* a, const void* out) {
  if (n < 2 || n > N3_MAX_N) return set_error(N3_ERR_RANGE, "n=%d outside [2, %d]", n, N3_MAX_N);
  if (B < 0) return set_error(N3_ERR_ARG, "negative batch size %d", B);
  if (B > 0 && (a == nullptr || out == nullptr)) return set_error(N3_ERR_ARG, "null device pointer");
  return N3_OK;
}

template <class Src, int MODE, bool BAD, int NT, int PLAN>
static int launch_tag_plan(Src src, int sms, int B, int n, int W, int32_t* scores, int32_t* badness, int32_t* mismatch,
                           uint32_t* error_word, cudaStream_t st) {
  using namespace n3;
  const auto kernel = tag_kernel<Src, MODE, BAD, NT, PLAN>;
  N3_TRY(allow_smem(reinterpret_cast<const void*>(kernel), tag_smem(NT, tag_warps(NT))));
  const int threads = W * 32 > kTagMinThreads ? W * 32 : kTagMinThreads;
  kernel<<<B < sms ? B : sms, threads, tag_smem(NT, W), st>>>(src, B, n, W, dir_lut_device_ptr(), scores, badness,
                                                              mismatch, error_word);
  return check_launch("tag_kernel");
}

template <class Src, int MODE, bool BAD, int NT>
static int launch_tag_nt(Src src, int sms, int B, int n, int32_t* scores, int32_t* badness, int32_t* mismatch,
                         uint32_t* error_word, cudaStream_t st) {
  using namespace n3;
  N3_TRY(ensure_device_tables());
  const int most = tag_warps(NT);
  const int per = (B + sms - 1) / sms;  // states per SM
  if (2 * per <= most) {
    int parts = 2;
    while (parts < kTagMaxParts && 2 * parts * per <= most) parts *= 2;
    return launch_tag_plan<Src, MODE, BAD, NT, kShared>(src, sms, B, n, per * parts, scores, badness, mismatch,
                                                        error_word, st);
  }
  const int last = per % most;
  if (per > most && last > 0 && 2 * last <= most)
    return launch_tag_plan<Src, MODE, BAD, NT, kRoundsThenShared>(src, sms, B, n, most, scores, badness, mismatch,
                                                                  error_word, st);
  return launch_tag_plan<Src, MODE, BAD, NT, kRounds>(src, sms, B, n, per < most ? per : most, scores, badness, mismatch,
                                                      error_word, st);
}

template <class Src, int MODE, bool BAD>
static int launch_tag(Src src, int sms, int B, int n, int32_t* scores, int32_t* badness, int32_t* mismatch,
                      uint32_t* error_word, cudaStream_t st) {
  switch ((2 * n + 31) / 32) {
    case 1: return launch_tag_nt<Src, MODE, BAD, 1>(src, sms, B, n, scores, badness, mismatch, error_word, st);
    case 2: return launch_tag_nt<Src, MODE, BAD, 2>(src, sms, B, n, scores, badness, mismatch, error_word, st);
    case 3: return launch_tag_nt<Src, MODE, BAD, 3>(src, sms, B, n, scores, badness, mismatch, error_word, st);
    default: return launch_tag_nt<Src, MODE, BAD, 5>(src, sms, B, n, scores, badness, mismatch, error_word, st);
  }
}

template <int MODE>
static int launch_slope(const int16_t* cols, int B, int n, int32_t* scores, int32_t* badness, int32_t* mismatch,
                        uint32_t* error_word, cudaStream_t st) {
  if (B == 0) return N3_OK;
  const n3::ColSource src{cols};
  const int sms = sm_count();
  return badness ? launch_tag<n3::ColSource, MODE, true>(src, sms, B, n, scores, badness, mismatch, error_word, st)
                 : launch_tag<n3::ColSource, MODE, false>(src, sms, B, n, scores, nullptr, mismatch, error_word, st);
}

template <class Src, bool BAD>
static int launch_det(Src src, int sms, int B, int n, int32_t* scores, int32_t* badness, cudaStream_t st) {
  using namespace n3;
  // warps per state: 16 while two such CTAs fit every SM, 4 while eight do (64
  // n = 75 states: 14 us against 79 us with one warp a state; 1024: 76 and 105), seven
  // on the smallest grids (1184 n = 10 states: 4.5 us, 4.2 with one)
  if (B <= 2 * sms)
    det_kernel<Src, 16, BAD><<<B, 16 * 32, 0, st>>>(src, B, n, scores, badness);
  else if (B <= (n <= 12 ? 7 : 8) * sms)
    det_kernel<Src, 4, BAD><<<B, 4 * 32, 0, st>>>(src, B, n, scores, badness);
  else
    det_kernel<Src, 1, BAD><<<(B + kDetWarps - 1) / kDetWarps, kDetWarps * 32, 0, st>>>(src, B, n, scores, badness);
  return check_launch("det_kernel");
}

// Whether the determinants are the faster count: they grow with n^3, the tags with
// n^2, but every centre costs the tags two round trips to shared memory, and every CTA
// the copy of a table.  So on the smallest grids, for up to two states an SM (16 warps
// share each) on those up to n = 28, and in between for little work, where they may take
// a microsecond more: the tags' tables cost the host 0.6, and it is the slower of the
// two for such calls (413 n = 22 states with badness 16.5 us a call, 17.1).  us, determinants
// against tags, E alone: 20,011 states n = 5 9.4 / 10.0, n = 10 20.8 / 16.2, n = 24 83 / 49;
// n = 8, 5000 6.2 / 6.9 and 8300 8.0 / 8.0; n = 10, 4096 6.1 / 6.0; n = 12, 2100 5.3 / 5.6;
// n = 20, 600 4.7 / 5.1 and 1184 7.7 / 6.0; n = 28, 296 4.3 / 4.7 and 297 5.8 / 4.7.  With
// badness: 20,011 states n = 10 28 / 21, n = 20 81 / 53; n = 8, 4096 5.9 / 6.1; n = 10, 3000
// 6.8 / 7.0; n = 12, 1036 4.5 / 4.9 and 1184 6.5 / 5.1; n = 20, 1036 7.4 / 6.8; n = 22, 600
// 6.9 / 6.5 and 1036 8.6 / 7.2; n = 26, 296 5.1 / 5.1.
static bool determinants_faster(int sms, int B, int n, bool badness) {
  if (n <= 5) return true;
  if (B <= 2 * sms) return n <= (badness ? 26 : 28);
  const int64_t work = (int64_t)B * n * n;
  if (B <= 7 * sms) return n <= (badness ? 22 : 24) && work <= (badness ? 400000 : 500000);
  return n <= (badness ? 10 : 12) && work <= (badness ? 300000 : 400000);
}

template <class Src>
static int launch_count(Src src, int B, int n, int32_t* scores, int32_t* badness, cudaStream_t st) {
  if (B == 0) return N3_OK;
  const int sms = sm_count();
  const bool det = determinants_faster(sms, B, n, badness != nullptr);
  if (badness)
    return det ? launch_det<Src, true>(src, sms, B, n, scores, badness, st)
               : launch_tag<Src, n3::kCount, true>(src, sms, B, n, scores, badness, nullptr, nullptr, st);
  return det ? launch_det<Src, false>(src, sms, B, n, scores, nullptr, st)
             : launch_tag<Src, n3::kCount, false>(src, sms, B, n, scores, nullptr, nullptr, nullptr, st);
}

template <class Src, int MODE, int NT, int PLAN>
static int prepare_tag_plan() {
  using namespace n3;
  const size_t smem = tag_smem(NT, tag_warps(NT));
  N3_TRY((allow_smem(reinterpret_cast<const void*>(tag_kernel<Src, MODE, true, NT, PLAN>), smem)));
  return allow_smem(reinterpret_cast<const void*>(tag_kernel<Src, MODE, false, NT, PLAN>), smem);
}

template <class Src, int MODE, int NT>
static int prepare_tag_nt() {
  N3_TRY((prepare_tag_plan<Src, MODE, NT, n3::kRounds>()));
  N3_TRY((prepare_tag_plan<Src, MODE, NT, n3::kShared>()));
  return prepare_tag_plan<Src, MODE, NT, n3::kRoundsThenShared>();
}

template <class Src, int MODE>
static int prepare_tag() {
  N3_TRY((prepare_tag_nt<Src, MODE, 1>()));
  N3_TRY((prepare_tag_nt<Src, MODE, 2>()));
  N3_TRY((prepare_tag_nt<Src, MODE, 3>()));
  return prepare_tag_nt<Src, MODE, 5>();
}

// The two counts of the checked score in one kernel (checked_kernel) for many
// states of larger grids.  us with badness, two kernels against one: 4096 states
// n = 75 364 / 346, 60 224 / 212, 49 148 / 140; 20,011 states 1668 / 1630, 1020 / 988,
// 663 / 655; 4300 states, which leave the determinants a last wave of few blocks,
// 414 / 365, 258 / 226, 173 / 165; 1300 states, which four warps each no longer take,
// 171 / 119, 109 / 77, 73 / 58; n = 75, 900 states 109 / 118 (fewer states get more warps
// each in the two kernels).  Up to n = 48 the tags alone have 32 warps of less work:
// one kernel only where the determinants have many states for four warps and few for
// one (n = 48: 1184 states 43 / 54, 1300 65 / 56, 2000 79 / 71, 4096 130 / 133, 4300
// 144 / 160, 20,011 582 / 625; n = 44: 37 / 49, 56 / 51, 68 / 61, 110 / 115, 122 / 144, 495 / 544).
// Warps for the tags: 12 from n = 56 on, 14 below (n = 50: 14 take 150 us for 4096
// states, 12 take 173; n = 75: 352 both).
static bool checked_in_one(int B, int n) {
  if (n < 44) return false;
  const int sms = sm_count();
  return n > 48 ? B >= 8 * sms : B > 8 * sms && B <= 20 * sms;
}
constexpr int kCheckedTagWarps = 12, kCheckedTagWarpsSmall = 14, kCheckedSmallN = 56;

static int launch_checked(const int16_t* cols, int B, int n, int32_t* scores, int32_t* badness, int32_t* mismatch,
                          uint32_t* error_word, cudaStream_t st) {
  using namespace n3;
  N3_TRY(ensure_device_tables());
  const int sms = sm_count(), per = (B + sms - 1) / sms;
  const int tag_warps = n < kCheckedSmallN ? kCheckedTagWarpsSmall : kCheckedTagWarps;
  const auto kernel = badness ? checked_kernel<true> : checked_kernel<false>;
  N3_TRY(allow_smem(reinterpret_cast<const void*>(kernel), kCheckedMaxSmem));
  kernel<<<(B + per - 1) / per, 1024, checked_smem(tag_warps, n), st>>>(
      ColSource{cols}, B, n, per, tag_warps, dir_lut_device_ptr(), scores, badness, mismatch, error_word);
  return check_launch("checked_kernel");
}

int prepare_score() {
  using namespace n3;
  N3_TRY(allow_smem(reinterpret_cast<const void*>(checked_kernel<true>), kCheckedMaxSmem));
  N3_TRY(allow_smem(reinterpret_cast<const void*>(checked_kernel<false>), kCheckedMaxSmem));
  N3_TRY((prepare_tag<n3::PQSource, n3::kCount>()));
  N3_TRY((prepare_tag<n3::ColSource, n3::kCount>()));
  N3_TRY((prepare_tag<n3::ColSource, n3::kSlope>()));
  return prepare_tag<n3::ColSource, n3::kChecked>();
}

}  // namespace n3host

extern "C" {

int n3_score_population(const int32_t* p, const int32_t* q, int B, int n, int32_t* scores, int32_t* badness,
                        void* stream) {
  N3_TRY(n3host::check_common(B, n, p, scores));
  if (B > 0 && q == nullptr) return n3host::set_error(N3_ERR_ARG, "null Q pointer");
  return n3host::launch_count(n3::PQSource{p, q}, B, n, scores, badness, (cudaStream_t)stream);
}

int n3_score_columns(const int16_t* cols, int B, int n, int32_t* scores, int32_t* badness, void* stream) {
  N3_TRY(n3host::check_common(B, n, cols, scores));
  return n3host::launch_count(n3::ColSource{cols}, B, n, scores, badness, (cudaStream_t)stream);
}

int n3_score_determinants(const int16_t* cols, int B, int n, int32_t* scores, int32_t* badness, void* stream) {
  N3_TRY(n3host::check_common(B, n, cols, scores));
  if (B == 0) return N3_OK;
  const n3::ColSource src{cols};
  const int sms = n3host::sm_count();
  return badness ? n3host::launch_det<n3::ColSource, true>(src, sms, B, n, scores, badness, (cudaStream_t)stream)
                 : n3host::launch_det<n3::ColSource, false>(src, sms, B, n, scores, nullptr, (cudaStream_t)stream);
}

int n3_score_slope(const int16_t* cols, int B, int n, int32_t* scores, int32_t* badness, void* stream) {
  N3_TRY(n3host::check_common(B, n, cols, scores));
  return n3host::launch_slope<n3::kSlope>(cols, B, n, scores, badness, nullptr, nullptr, (cudaStream_t)stream);
}

int n3_checked_error(int determinant_e, int slope_e, int has_badness, int badness_sum) {
  return (int)n3::checked_error(determinant_e, slope_e, has_badness != 0, badness_sum);
}

int n3_score_checked(const int16_t* cols, int B, int n, int32_t* scores, int32_t* badness, int32_t* mismatch,
                     uint32_t* error_word, void* stream) {
  N3_TRY(n3host::check_common(B, n, cols, scores));
  if (B > 0 && mismatch == nullptr) return n3host::set_error(N3_ERR_ARG, "null mismatch counter");
  if (B == 0) return N3_OK;
  if (n3host::checked_in_one(B, n))
    return n3host::launch_checked(cols, B, n, scores, badness, mismatch, error_word, (cudaStream_t)stream);
  // Two launches on one stream: the determinant count at full occupancy, then
  // the independent slope count, which validates each state, compares, and
  // gives the badness if it is wanted.
  N3_TRY((n3host::launch_det<n3::ColSource, false>(n3::ColSource{cols}, n3host::sm_count(), B, n, scores, nullptr,
                                                   (cudaStream_t)stream)));
  return n3host::launch_slope<n3::kChecked>(cols, B, n, scores, badness, mismatch, error_word, (cudaStream_t)stream);
}

}  // extern "C"
