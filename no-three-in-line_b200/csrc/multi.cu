// Multi-point moves: the three-cycle scores of src/no_three_75/accelerated.py:196-276
// (evaluate_three_cycles) and the four-cycle / double-switch neighbourhood scans
// of src/no_three_75/gpu_neighborhood.py:70-211 (best_four_cycle,
// best_double_switch).
//
// A move that relocates the points of a slot set M (k points in k distinct
// rows; columns permuted among them) changes E by
//   dE = side(new positions) - side(old positions),
//   side(X) = sum_i t_A(x_i) + sum_{i<j} j_A(x_i, x_j) + #collinear triples within X,
// where A = S \ M, t_A(x) = pairs of A collinear with x (a direction histogram
// around x over A) and j_A(x, y) = points of A on the line x-y (the count of
// that direction in x's histogram).  Both sides count exactly the collinear
// triples that contain a point of M, before and after.  The reference scores a
// three-cycle by its O(n^2) pair loops and a four-point move by materialising
// the whole candidate state and rescoring it (O(n^3)); here each is O(n) per
// position, and the scan shares positions: for a slot set (anchor + 3 slots)
// every four-cycle and double switch puts each target at one of 12 possible
// positions, and for a state with two points in every column three of the slots
// already fix 6 of these (scan_kernel).
#include <stdint.h>

#include "cover.cuh"
#include "dirs.cuh"
#include "n3_common.cuh"

namespace n3 {
namespace multi {

constexpr int kT = kSlotsPerLane;  // 5 slots per lane

// This lane's slots' direction-table keys row * kLutW + column (the state is
// fixed for the whole kernel, so the keys stay in registers).
__device__ __forceinline__ void lane_keys(const int* __restrict__ cs, int m, int lane, int (&key)[kT]) {
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const int k = lane + 32 * t;
    key[t] = k < m ? (k >> 1) * kLutW + cs[k] : 0;
  }
}

// Direction histogram of centre (rx, cx) over A, on the full signed table:
// slots whose bit t is set in `skip` (this lane's slot lane + 32 t is a moved
// one) are left out, and so are the points in row rx.  key: lane_keys of the
// state.
__device__ __forceinline__ int hist_build_excl(const int (&key)[kT], int m, int rx, int cx, uint32_t skip,
                                               const uint16_t* __restrict__ lutf, uint32_t* __restrict__ hist,
                                               int lane, int (&ids)[kT]) {
  const uint16_t* base = lutf + kFullLutCentre - (rx * kLutW + cx);
  int pairs = 0;
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const int k = lane + 32 * t;
    ids[t] = -1;
    if (k < m && !((skip >> t) & 1u) && (k >> 1) != rx) {
      const int id = base[key[t]];
      ids[t] = id;
      pairs += hist_add(hist, id);
    }
  }
  return pairs;
}

__device__ __forceinline__ uint32_t skip_mask(int lane, const int* moved, int count) {
  uint32_t s = 0;
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const int k = lane + 32 * t;
    for (int i = 0; i < count; ++i) s |= (uint32_t)(k == moved[i]) << t;
  }
  return s;
}

__device__ __forceinline__ int collinear(int r0, int c0, int r1, int c1, int r2, int c2) {
  return (r1 - r0) * (c2 - c0) == (c1 - c0) * (r2 - r0);
}

// side() of `count` positions (distinct rows) over A; all lanes return the sum.
__device__ __forceinline__ int side_sum(const int (&key)[kT], int m, const int* rows, const int* cols, int count, uint32_t skip,
                        const uint16_t* __restrict__ lutf, uint32_t* __restrict__ hist, int lane) {
  int total = 0;
  for (int i = 0; i < count; ++i) {
    int ids[kT];
    const int part = hist_build_excl(key, m, rows[i], cols[i], skip, lutf, hist, lane, ids);
    __syncwarp();
    int pair_lines = 0;
    if (lane == 0)
      for (int j = i + 1; j < count; ++j)
        pair_lines += hist_get(hist, dir_id_full(lutf, rows[j] - rows[i], cols[j] - cols[i]));
    __syncwarp();
    hist_release(hist, ids);
    __syncwarp();
    total += warp_sum(part) + __shfl_sync(0xffffffffu, pair_lines, 0);
  }
  for (int i = 0; i < count; ++i)
    for (int j = i + 1; j < count; ++j)
      for (int k = j + 1; k < count; ++k) total += collinear(rows[i], cols[i], rows[j], cols[j], rows[k], cols[k]);
  return total;
}

// --------------------------------------------------------------------------
// Three-cycles: warp per candidate (u, v, w, orientation).
// --------------------------------------------------------------------------
constexpr int kWarps = 8;
constexpr size_t kSmem = kFullLutBytes + kWarps * sizeof(uint32_t) * kDirWords + sizeof(int) * kMaxM;

__global__ void __launch_bounds__(kWarps * 32) three_cycle_kernel(const int32_t* __restrict__ p,
                                                                  const int32_t* __restrict__ q, int n,
                                                                  const int32_t* __restrict__ cand, int count,
                                                                  int64_t current, const uint16_t* __restrict__ g_lut,
                                                                  int64_t* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* lutf = reinterpret_cast<uint16_t*>(smem);
  uint32_t* hist_all = reinterpret_cast<uint32_t*>(smem + kFullLutBytes);
  int* cs = reinterpret_cast<int*>(hist_all + kWarps * kDirWords);
  full_lut_copy(lutf, g_lut);
  for (int i = threadIdx.x; i < kWarps * kDirWords; i += blockDim.x) hist_all[i] = 0u;
  const int m = 2 * n;
  for (int s = threadIdx.x; s < m; s += blockDim.x) cs[s] = (s & 1) ? q[s >> 1] : p[s >> 1];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* hist = hist_all + warp * kDirWords;
  int key[kT];
  lane_keys(cs, m, lane, key);
  for (int c = blockIdx.x * kWarps + warp; c < count; c += gridDim.x * kWarps) {
    const int u = cand[4 * c], v = cand[4 * c + 1], w = cand[4 * c + 2], o = cand[4 * c + 3];
    // the moves search.py:38-65 generates: three slots in three rows, three
    // distinct columns, no row left with a repeated column
    bool ok = u >= 0 && v >= 0 && w >= 0 && u < m && v < m && w < m && (o == 0 || o == 1);
    int nu = 0, nv = 0, nw = 0;
    if (ok) {
      const int ru = u >> 1, rv = v >> 1, rw = w >> 1;
      ok = ru != rv && ru != rw && rv != rw && cs[u] != cs[v] && cs[u] != cs[w] && cs[v] != cs[w];
      nu = o == 0 ? cs[v] : cs[w];
      nv = o == 0 ? cs[w] : cs[u];
      nw = o == 0 ? cs[u] : cs[v];
      ok = ok && nu != cs[u ^ 1] && nv != cs[v ^ 1] && nw != cs[w ^ 1];
    }
    if (!ok) {
      if (lane == 0) out[c] = (int64_t)1 << 60;
      continue;
    }
    const int moved[3] = {u, v, w};
    const uint32_t skip = skip_mask(lane, moved, 3);
    const int rows[3] = {u >> 1, v >> 1, w >> 1};
    const int old_cols[3] = {cs[u], cs[v], cs[w]};
    const int new_cols[3] = {nu, nv, nw};
    const int before = side_sum(key, m, rows, old_cols, 3, skip, lutf, hist, lane);
    const int after = side_sum(key, m, rows, new_cols, 3, skip, lutf, hist, lane);
    if (lane == 0) out[c] = current - before + after;
  }
}

// --------------------------------------------------------------------------
// Neighbourhood scan around an anchor slot.
// Enumeration order and tie rule of gpu_neighborhood.py:108-116 / :181-190: row
// triples in itertools.combinations order, layers in itertools.product order,
// then orderings (itertools.permutations) or the three pairings; the result is
// the first candidate (in that order) with the lowest score, kept only if it
// improves on the base.
//
// Two kernels, of which the state's columns choose one (both are launched, the
// other returns at once): scan_kernel for states with two points in every
// column, in cells of their own; scan_any_kernel for all others, and for small
// grids (kScanSmallN).
// --------------------------------------------------------------------------
struct ScanArgs {
  const int32_t* p;
  const int32_t* q;
  int n, anchor;
  int64_t base;          // E of the state
  int combos;            // C(n - 1, 3)
  const uint16_t* lut;    // scan_any_kernel's table
  const uint16_t* prim4;  // scan_kernel's
  const uint16_t* dir4;
  unsigned long long* best;   // [2]: (score << 32 | index) for four-cycles, double switches
  unsigned long long* legal;  // [2]
};

// j-th (0-based, lexicographic) 3-subset {a < b < c} of {0 .. N-1}
__device__ __forceinline__ void unrank3(int x, int N, int& a, int& b, int& c) {
  a = 0;
  for (;; ++a) {
    const int k = N - 1 - a, cnt = k * (k - 1) / 2;
    if (x < cnt) break;
    x -= cnt;
  }
  b = a + 1;
  for (;; ++b) {
    const int cnt = N - 1 - b;
    if (x < cnt) break;
    x -= cnt;
  }
  c = b + 1 + x;
}

// Whether every column of the state holds two points and no row the same cell
// twice, columns on the grid; all threads of the block call it (at least m).
__device__ __forceinline__ bool regular_state(const ScanArgs& A, int* __restrict__ columns) {
  const int n = A.n, r = threadIdx.x;
  for (int i = r; i < kMaxN; i += blockDim.x) columns[i] = 0;
  __syncthreads();
  bool regular = true;
  if (r < n) {
    const int p = A.p[r], q = A.q[r];
    regular = p >= 0 && p < n && q >= 0 && q < n && p != q;
    if (regular) {
      atomicAdd(&columns[p], 1);
      atomicAdd(&columns[q], 1);
    }
  }
  __syncthreads();
  if (r < n) regular = regular && columns[r] == 2;
  return __syncthreads_and(regular);
}

// The nine candidates of slot set gw by a warp, from 4 + 12 histograms.
__device__ __forceinline__ void scan_slot_set(const ScanArgs& A, const int* __restrict__ cs, int gw, int lane,
                                              const uint16_t* __restrict__ lutf, uint32_t* __restrict__ hist,
                                              int (*jt)[12], int* tn) {
  const int n = A.n, m = 2 * n;
  const int combo = gw >> 3, layers = gw & 7;
  const int arow = A.anchor >> 1;
  int r[3];
  unrank3(combo, n - 1, r[0], r[1], r[2]);
  int T[4];
  T[0] = A.anchor;
  for (int i = 0; i < 3; ++i) {
    const int row = r[i] < arow ? r[i] : r[i] + 1;  // i-th row other than the anchor's
    T[i + 1] = 2 * row + ((layers >> (2 - i)) & 1);
  }
  int rowT[4], colT[4], partner[4];
  for (int i = 0; i < 4; ++i) {
    rowT[i] = T[i] >> 1;
    colT[i] = cs[T[i]];
    partner[i] = cs[T[i] ^ 1];
  }
  const uint32_t skip = skip_mask(lane, T, 4);
  int key[kT];
  lane_keys(cs, m, lane, key);
  const int before = side_sum(key, m, rowT, colT, 4, skip, lutf, hist, lane);
  // the 12 candidate positions: target i with the column of source j != i (index 3 i + (j > i ? j - 1 : j))
  for (int a = 0; a < 12; ++a) {
    const int i = a / 3, jj = a % 3, j = jj >= i ? jj + 1 : jj;
    const int rx = rowT[i], cx = colT[j];
    int ids[kT];
    const int part = hist_build_excl(key, m, rx, cx, skip, lutf, hist, lane, ids);
    __syncwarp();
    if (lane < 12) {
      const int b = lane, ib = b / 3, jb = b % 3 >= ib ? b % 3 + 1 : b % 3;
      jt[a][b] = ib != i ? hist_get(hist, dir_id_full(lutf, rowT[ib] - rx, colT[jb] - cx)) : 0;
    }
    __syncwarp();
    hist_release(hist, ids);
    const int t = warp_sum(part);
    if (lane == 0) tn[a] = t;
    __syncwarp();
  }
  // the moves: sigma[i] = source of target i
  if (lane < 9) {
    int sigma[4];
    unsigned int idx;
    if (lane < 6) {  // four-cycle with ordering number `lane` of (T1, T2, T3)
      const int perm[6][3] = {{1, 2, 3}, {1, 3, 2}, {2, 1, 3}, {2, 3, 1}, {3, 1, 2}, {3, 2, 1}};
      const int o0 = perm[lane][0], o1 = perm[lane][1], o2 = perm[lane][2];
      sigma[0] = o0;
      sigma[o0] = o1;
      sigma[o1] = o2;
      sigma[o2] = 0;
      idx = (unsigned)((combo * 8 + layers) * 6 + lane);
    } else {  // double switch pairing lane - 6: (a, anchor, c, b), (b, c, anchor, a), (c, b, a, anchor)
      const int pairs[3][4] = {{1, 0, 3, 2}, {2, 3, 0, 1}, {3, 2, 1, 0}};
      for (int i = 0; i < 4; ++i) sigma[i] = pairs[lane - 6][i];
      idx = (unsigned)((combo * 8 + layers) * 3 + (lane - 6));
    }
    bool legal = true;
    int after = 0, pos[4], nr[4], nc[4];
    for (int i = 0; i < 4; ++i) {
      const int j = sigma[i];
      legal = legal && colT[j] != partner[i];
      pos[i] = 3 * i + (j > i ? j - 1 : j);
      nr[i] = rowT[i];
      nc[i] = colT[j];
      after += tn[pos[i]];
    }
    for (int i = 0; i < 4; ++i)
      for (int k = i + 1; k < 4; ++k) after += jt[pos[i]][pos[k]];
    for (int i = 0; i < 4; ++i)
      for (int j = i + 1; j < 4; ++j)
        for (int k = j + 1; k < 4; ++k) after += collinear(nr[i], nc[i], nr[j], nc[j], nr[k], nc[k]);
    if (legal) {
      const int64_t score = A.base + after - before;
      const unsigned long long key = ((unsigned long long)score << 32) | idx;
      const int which = lane < 6 ? 0 : 1;
      atomicMin(A.best + which, key);
      atomicAdd(A.legal + which, 1ull);
    }
  }
}

// SMALL: every state, a warp per slot set (n = 5: 14.4 us, 17.1 with the loop and the test of
// the state); else irregular ones only, in loops.
template <bool SMALL>
__global__ void __launch_bounds__(kWarps * 32) scan_any_kernel(const ScanArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* lutf = reinterpret_cast<uint16_t*>(smem);
  uint32_t* hist_all = reinterpret_cast<uint32_t*>(smem + kFullLutBytes);
  int* cs = reinterpret_cast<int*>(hist_all + kWarps * kDirWords);
  __shared__ int jt_all[kWarps][12][12];  // points of A on the line between two candidate positions
  __shared__ int tn_all[kWarps][12];      // t_A of each candidate position
  __shared__ int columns[kMaxN];
  const int n = A.n, m = 2 * n;
  if (!SMALL && regular_state(A, columns)) return;
  full_lut_copy(lutf, A.lut);
  for (int i = threadIdx.x; i < kWarps * kDirWords; i += blockDim.x) hist_all[i] = 0u;
  for (int s = threadIdx.x; s < m; s += blockDim.x) cs[s] = (s & 1) ? A.q[s >> 1] : A.p[s >> 1];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* hist = hist_all + warp * kDirWords;
  const int first = blockIdx.x * kWarps + warp;
  if (SMALL) {
    if (first < A.combos * 8) scan_slot_set(A, cs, first, lane, lutf, hist, jt_all[warp], tn_all[warp]);
  } else {
    for (int gw = first; gw < A.combos * 8; gw += gridDim.x * kWarps) {
      scan_slot_set(A, cs, gw, lane, lutf, hist, jt_all[warp], tn_all[warp]);
      __syncwarp();
    }
  }
}

// --------------------------------------------------------------------------
// The scan of a state with two points in every column.  A warp takes three slots
// T0 (the anchor), T1, T2 and its lanes 32 slots T3 of later rows: 9 candidates
// each.  Write o_k for the point of T_k, x_ab = (row of a, column of b) for a, b
// in {0, 1, 2}, y_a = (row of a, column of T3), z_b = (row of T3, column of b).  A
// candidate is named by the a that takes T3's column and the b whose column T3
// takes: y_a and z_b, and with c the third of {0, 1, 2} x_bc and x_ca (a != b), or
// the two x of the others (a = b: a double switch).
//
// Points are taken out and put in one after the other, so that every count is one
// counter of a histogram and nothing is subtracted twice:
//   out  o_0, o_1, o_2, o_3: t(o_k) over what is left = T[o_k] less the earlier
//        o_j's counts (the cover table T counts pairs of the whole state);
//   t_A of y_a and z_b likewise: T[cell] less the count in o_k's histogram, k = 0 .. 2
//        (o_3 shares its column with y and its row with z);
//   t_A of x_ab: the pair sum of its histogram over B = S \ {o_0, o_1, o_2} less
//        the count of o_3;
//   j_A of x_ab with any other new point: a counter of that histogram, and
//        triples of new points: equal directions from x_ab;
//   j_A of y_a with z_b: a walk along their line over B's occupancy bits, if without
//        it the candidate is no worse than the block's best so far.
// So 3 + 6 histograms per warp, 45 counters and 36 comparisons per lane serve 9
// candidates, where a warp took 4 + 12 histograms.  Points in a
// histogram's own row and column are not counted (no row or column ever holds a
// third point), so a counter of a vertical line is 0.  Where T3's column is
// a's (q[a]), z_a is o_3's own cell and y_a is o_a's: their own points are taken
// off the counts that hold them.
//
// Both issue and latency bound it (66 % of issue slots, 5 warps a scheduler), a
// fifth of it the cover table, which every block builds.  n = 20: 26 us, 83 us by
// scan_any_kernel; 40: 42 and 588; 75: 133 and 4100 (238 with every line walked).
// --------------------------------------------------------------------------
constexpr int kScanWarps = 20;
constexpr int kScanSmallN = 12;  // below, scan_any_kernel alone (n = 8: 16 us, 22 with both; 12: 24 and 24)
constexpr int kScanRegion = ((kMaxN * kMaxN + 1) / 2 + 3) / 4 * 4;  // words of the cover table

struct ScanSmem {
  uint16_t prim4[kCompactLutBytes / 2];
  uint16_t dir4[kCompactLutBytes / 2];
  uint32_t recip[kMaxN + 1];
  uint32_t T[kScanRegion];
  uint32_t occ[kOccWords + 3];
  uint32_t occ_b[kScanWarps][kOccWords + 3];  // without the warp's three points
  uint32_t hist[kScanWarps][kDirWords];
  uint2 scratch[kScanWarps][32];
  int columns[kMaxN];
  int first[kMaxN + 1];  // tasks before those of row r2 (numbered without the anchor's)
  int next;
  int bound[2];  // lowest dE of the block's four-cycles, double switches
  uint8_t cs[152];
};
static_assert(sizeof(ScanSmem) <= 227 * 1024, "scan_kernel shared memory");

// A histogram of centre (rx, cx) over the lane's slots that `in` has set, without
// the centre's row and column: the lane's share of the pair sum.
__device__ __forceinline__ int scan_centre(const int (&key)[kT], int lane, uint32_t in, int rx, int cx,
                                           const uint16_t* __restrict__ dir4_, uint32_t* __restrict__ hist,
                                           int (&ids)[kT]) {
  const int centre = rx * kLutW + cx;
  int pairs = 0;
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const int row = (lane + 32 * t) >> 1;
    const bool counted = ((in >> t) & 1u) && row != rx && key[t] - row * kLutW != cx;
    ids[t] = counted ? (int)(dir4(dir4_, key[t], centre) >> 2) : -1;
    if (counted) pairs += hist_add(hist, ids[t]);
  }
  return pairs;
}

// points_on_line, not inlined: nine places call it.
static __device__ __noinline__ int line_points(const uint32_t* __restrict__ occ, int n,
                                               const uint16_t* __restrict__ prim4, int r0, int c0, int r1, int c1) {
  return points_on_line(occ, n, prim4, r0, c0, r1, c1);
}

__device__ __forceinline__ int choose2(int k) { return k * (k - 1) / 2; }

__global__ void __launch_bounds__(kScanWarps * 32, 1) scan_kernel(const ScanArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  ScanSmem& S = *reinterpret_cast<ScanSmem*>(smem);
  const int n = A.n, m = 2 * n, N = n - 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (!regular_state(A, S.columns)) return;
  compact_lut_copy(S.prim4, A.prim4);
  compact_lut_copy(S.dir4, A.dir4);
  for (int a = tid; a <= kMaxN; a += blockDim.x) S.recip[a] = a ? (65536u + (uint32_t)a - 1u) / (uint32_t)a : 0u;
  for (int i = tid; i < kScanRegion; i += blockDim.x) S.T[i] = 0u;
  for (int i = tid; i < kOccWords; i += blockDim.x) S.occ[i] = 0u;
  uint32_t* hist = S.hist[warp];
  for (int i = lane; i < kDirWords; i += 32) hist[i] = 0u;
  if (tid == 0) {
    // 4 r2 pairs (row and layer of T1, layer of T2), their later slots 32 at a time
    int tasks = 0;
    for (int r2 = 0; r2 <= N; ++r2) {
      S.first[r2] = tasks;
      if (r2 < N) tasks += 4 * r2 * ((2 * (N - 1 - r2) + 31) / 32);
    }
    S.next = 0;
    S.bound[0] = S.bound[1] = INT32_MAX;
  }
  __syncthreads();
  for (int s = tid; s < m; s += blockDim.x) {
    const int c = (s & 1) ? A.q[s >> 1] : A.p[s >> 1];
    S.cs[s] = (uint8_t)c;
    atomicOr(&S.occ[3 * (s >> 1) + (c >> 5)], 1u << (c & 31));
  }
  __syncthreads();
  cover_build(S.cs, S.T, n, S.prim4, S.recip, S.scratch[warp], lane, warp, kScanWarps);
  int key[kT];
  uint32_t present = 0u;
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const int k = lane + 32 * t;
    key[t] = k < m ? (k >> 1) * kLutW + S.cs[k] : 0;
    present |= (uint32_t)(k < m) << t;
  }
  __syncthreads();
  const int arow = A.anchor >> 1;
  const int tasks = S.first[N];
  uint32_t* occ_b = S.occ_b[warp];
  unsigned long long best4 = ~0ull, best2 = ~0ull;
  uint32_t legal4 = 0u, legal2 = 0u;
  for (;;) {
    int task = 0;
    if (lane == 0) task = atomicAdd(&S.next, 1);
    task = __shfl_sync(0xffffffffu, task, 0) * (int)gridDim.x + (int)blockIdx.x;
    if (task >= tasks) break;
    int r2 = -1;  // the last row whose tasks do not begin after this one
    for (int r0 = 0; r0 < N; r0 += 32) r2 += __popc(__ballot_sync(0xffffffffu, r0 + lane < N && S.first[r0 + lane] <= task));
    const int in_row = task - S.first[r2], pair = in_row % (4 * r2), chunk = in_row / (4 * r2);
    const int r1 = pair >> 2, l1 = (pair >> 1) & 1, l2 = pair & 1;
    const int i3 = 2 * (r2 + 1) + 32 * chunk + lane;  // T3 among the slots without the anchor's row
    const bool active = i3 < 2 * N;
    const int r3 = min(i3 >> 1, N - 1), l3 = i3 & 1;
    int row[3], col[3], other[3];  // T0 .. T2 and their row partners' columns
    {
      const int slot[3] = {A.anchor, 2 * (r1 + (r1 >= arow)) + l1, 2 * (r2 + (r2 >= arow)) + l2};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        row[k] = slot[k] >> 1;
        col[k] = S.cs[slot[k]];
        other[k] = S.cs[slot[k] ^ 1];
      }
    }
    const int row3 = r3 + (r3 >= arow), slot3 = 2 * row3 + l3, col3 = S.cs[slot3], other3 = S.cs[slot3 ^ 1];
    const int key3 = row3 * kLutW + col3;
    int q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = col[k] == col3;

    // B's occupancy
    for (int i = lane; i < 3 * n; i += 32) {
      uint32_t w = S.occ[i];
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (i == 3 * row[k] + (col[k] >> 5)) w &= ~(1u << (col[k] & 31));
      occ_b[i] = w;
    }

    // out: o_0 .. o_3, and t_A of the y and z
    int ty[3], tz[3], before = cover_get(S.T, row3 * n + col3);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ty[a] = cover_get(S.T, row[a] * n + col3);
      tz[a] = cover_get(S.T, row3 * n + col[a]);
      before += cover_get(S.T, row[a] * n + col[a]);
    }
    uint32_t in = present;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      int ids[kT];
#pragma unroll
      for (int t = 0; t < kT; ++t)
        if (key[t] == row[k] * kLutW + col[k]) in &= ~(1u << t);  // o_k is not counted from here on
      scan_centre(key, lane, in, row[k], col[k], S.dir4, hist, ids);
      __syncwarp();
      const int centre = row[k] * kLutW + col[k];
      const auto count = [&](int at) { return hist_get(hist, (int)(dir4(S.dir4, at, centre) >> 2)); };
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (a > k) before -= max(count(row[a] * kLutW + col[a]) - 1, 0);
        if (a != k) {
          ty[a] -= count(row[a] * kLutW + col3) - (a > k ? q[a] : 0);
          tz[a] -= count(row3 * kLutW + col[a]) - q[a];
        }
      }
      before -= max(count(key3) - 1, 0);
      __syncwarp();
      hist_release(hist, ids);
      __syncwarp();
    }

    // in: the x, each with its partners
    int acc[3][3];  // [a][b]
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) acc[a][b] = ty[a] + tz[b];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (a == b) continue;
        const int c = 3 - a - b;
        int ids[kT];
        const int part = scan_centre(key, lane, in, row[a], col[b], S.dir4, hist, ids);
        const int t_b = __reduce_add_sync(0xffffffffu, part);
        __syncwarp();
        const int centre = row[a] * kLutW + col[b];
        const auto direction = [&](int r, int cc) { return (int)(dir4(S.dir4, r * kLutW + cc, centre) >> 2); };
        const int d3 = direction(row3, col3);
        const int yb = direction(row[b], col3), yc = direction(row[c], col3);
        const int za = direction(row3, col[a]), zc = direction(row3, col[c]);
        const int t_x = t_b - max(hist_get(hist, d3) - 1, 0);
        const int jyb = hist_get(hist, yb), jyc = hist_get(hist, yc);
        const int jza = hist_get(hist, za) - q[a], jzc = hist_get(hist, zc) - q[c];
        acc[c][c] += t_x + jyc + jzc + (yc == zc);
        acc[c][a] += t_x + jyc + jza + (yc == za);
        acc[b][c] += t_x + jyb + jzc + (yb == zc);
        {  // with x_bc, both in the candidate (c, a)
          const int d = direction(row[b], col[c]);
          acc[c][a] += hist_get(hist, d) - (d == d3) + (d == yc) + (d == za);
        }
        if (a < b) {  // with x_ba, both in (c, c)
          const int d = direction(row[b], col[a]);
          acc[c][c] += hist_get(hist, d) - (d == d3) + (d == yc) + (d == zc);
        }
        __syncwarp();
        hist_release(hist, ids);
        __syncwarp();
      }
    }

    // y with z, legality, the index of each candidate
    const int rank = choose2(N) * (N - 2) / 3 - choose2(N - r1) * (N - r1 - 2) / 3 + choose2(N - 1 - r1) -
                     choose2(N - r2) + (r3 - r2 - 1);
    const unsigned set = (unsigned)(rank * 8 + l1 * 4 + l2 * 2 + l3);
    int bound[2] = {*(volatile int*)&S.bound[0], *(volatile int*)&S.bound[1]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        bool legal = active && col3 != other[a] && col[b] != other3;
        const int c = 3 - a - b, which = a == b;
        if (a != b) {
          legal = legal && col[c] != other[b] && col[a] != other[c];
        } else {
          const int u = (a + 1) % 3, v = (a + 2) % 3;
          legal = legal && col[v] != other[u] && col[u] != other[v];
        }
        (which ? legal2 : legal4) += legal;
        int dE = acc[a][b] - before;
        const bool open = legal && dE <= bound[which];
        if (!__any_sync(0xffffffffu, open)) continue;
        // orderings (T1, T2, T3), (1, 3, 2), (2, 1, 3), (2, 3, 1), (3, 1, 2), (3, 2, 1) of the cycle
        // through the anchor: T3's source b and taker a tell which; pairings 0 .. 2: T3 with c, b, anchor
        constexpr unsigned kOrder[3][3] = {{2, 4, 5}, {2, 1, 1}, {0, 3, 0}};
        if (open) {
          dE += line_points(occ_b, n, S.prim4, row[a], col3, row3, col[b]);
          const unsigned long long found =
              (unsigned long long)(A.base + dE) << 32 | (set * (which ? 3u : 6u) + kOrder[a][b]);
          if (which) best2 = min(best2, found); else best4 = min(best4, found);
        }
        const int low = __reduce_min_sync(0xffffffffu, open ? dE : INT32_MAX);
        if (low < bound[which]) {
          bound[which] = low;
          if (lane == 0) atomicMin(&S.bound[which], low);
        }
      }
    }
    __syncwarp();
  }
  legal4 = __reduce_add_sync(0xffffffffu, legal4);
  legal2 = __reduce_add_sync(0xffffffffu, legal2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    best4 = min(best4, __shfl_xor_sync(0xffffffffu, best4, o));
    best2 = min(best2, __shfl_xor_sync(0xffffffffu, best2, o));
  }
  if (lane == 0) {
    if (legal4) {
      atomicMin(A.best, best4);
      atomicAdd(A.legal, (unsigned long long)legal4);
    }
    if (legal2) {
      atomicMin(A.best + 1, best2);
      atomicAdd(A.legal + 1, (unsigned long long)legal2);
    }
  }
}

}  // namespace multi
}  // namespace n3

extern "C" {

int n3_three_cycle_scores(const int32_t* p, const int32_t* q, int n, const int32_t* candidates, int count,
                          int64_t current, int64_t* scores, void* stream) {
  if (n < 3 || n > N3_MAX_N) return n3host::set_error(N3_ERR_RANGE, "three cycles: n=%d outside [3, %d]", n, N3_MAX_N);
  if (count < 0) return n3host::set_error(N3_ERR_ARG, "three cycles: negative count");
  if (count == 0) return N3_OK;
  if (!p || !q || !candidates || !scores) return n3host::set_error(N3_ERR_ARG, "three cycles: null buffer");
  N3_TRY(n3host::ensure_device_tables());
  N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(n3::multi::three_cycle_kernel), n3::multi::kSmem));
  const int want = (count + n3::multi::kWarps - 1) / n3::multi::kWarps;
  const int grid = want < 2 * n3host::sm_count() ? want : 2 * n3host::sm_count();
  n3::multi::three_cycle_kernel<<<grid, n3::multi::kWarps * 32, n3::multi::kSmem, (cudaStream_t)stream>>>(
      p, q, n, candidates, count, current, n3host::dir_lut_full_device_ptr(), scores);
  return n3host::check_launch("three_cycle_kernel");
}

int n3_neighborhood_scan(const int32_t* p, const int32_t* q, int n, int anchor, int64_t current,
                         unsigned long long* best, unsigned long long* legal, void* stream) {
  if (n < 5 || n > N3_MAX_N) return n3host::set_error(N3_ERR_RANGE, "neighbourhood scan: n=%d outside [5, %d]", n,
                                                      N3_MAX_N);
  if (anchor < 0 || anchor >= 2 * n) return n3host::set_error(N3_ERR_RANGE, "anchor index outside point slots");
  if (!p || !q || !best || !legal) return n3host::set_error(N3_ERR_ARG, "neighbourhood scan: null buffer");
  N3_TRY(n3host::ensure_device_tables());
  const bool small = n < n3::multi::kScanSmallN;
  const auto scan_any = small ? n3::multi::scan_any_kernel<true> : n3::multi::scan_any_kernel<false>;
  N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(scan_any), n3::multi::kSmem));
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(best, 0xFF, 2 * sizeof(unsigned long long), st) != cudaSuccess ||
      cudaMemsetAsync(legal, 0, 2 * sizeof(unsigned long long), st) != cudaSuccess)
    return n3host::set_error(N3_ERR_CUDA, "neighbourhood scan: memset failed");
  n3::multi::ScanArgs A;
  A.p = p;
  A.q = q;
  A.n = n;
  A.anchor = anchor;
  A.base = current;
  A.combos = (n - 1) * (n - 2) * (n - 3) / 6;
  A.lut = n3host::dir_lut_full_device_ptr();
  A.best = best;
  A.legal = legal;
  int grid = (A.combos * 8 + n3::multi::kWarps - 1) / n3::multi::kWarps;
  if (!small) {
    A.prim4 = n3host::prim4_lut_device_ptr();
    A.dir4 = n3host::dir4_lut_device_ptr();
    N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(n3::multi::scan_kernel), sizeof(n3::multi::ScanSmem)));
    const int sms = n3host::sm_count(), pairs = 2 * (n - 2) * (n - 3);  // (T1, T2) with a later row
    n3::multi::scan_kernel<<<pairs < sms ? pairs : sms, n3::multi::kScanWarps * 32, sizeof(n3::multi::ScanSmem), st>>>(
        A);
    N3_TRY(n3host::check_launch("scan_kernel"));
    if (grid > 2 * sms) grid = 2 * sms;
  }
  scan_any<<<grid, n3::multi::kWarps * 32, n3::multi::kSmem, st>>>(A);
  return n3host::check_launch("scan_any_kernel");
}

}  // extern "C"
