// (b) Exact incremental deltas of row-pair column swaps.
//
// A move exchanges the columns of slots u and v (different rows): u' takes
// (r_u, c_v), v' takes (r_v, c_u).  It is legal iff the columns differ and
// neither new point duplicates the other point of its row
// (src/no_three_75/tempering.py:58, accelerated.py:145-151).  With
// A = S \ {u, v} and, for a centre X, t(X) = number of pairs of A collinear
// with X and j(X, Y) = number of points of A collinear with X and Y:
//
//   dE = t(u') + t(v') + j(u', v') - t(u) - t(v) - j(u, v)
//
// which is the reference's "triples through a moved point" accounting
// (tempering.py:68-89: pairs through one moved point plus triples through
// both).  Only pairs through the moved points are touched, and they are counted
// by direction class: t(X) = sum over directions from X of C(count, 2), one
// direction-histogram insertion per point of A (dirs.cuh).  The same
// histograms give every other point's badness change:
//
//   dbad[k] = sum over new centres (count - 1) - sum over old centres (count - 1)
//             + [k on line(u', v')] - [k on line(u, v)]
//
// and dbad[u] = t(u') + j(u',v') - t(u) - j(u,v) (likewise v).
//
// A second, independent kernel evaluates the reference formulation literally
// (every pair (i<j) outside {u,v} tested against u, u', v, v' with int32 cross
// products, plus every k against (u,v) and (u',v')); tests compare the two.
#include <type_traits>

#include "cover.cuh"
#include "dirs.cuh"
#include "n3_common.cuh"

namespace n3 {

// One legal move by 8-bit histograms over A, one centre at a time, for what
// swap_delta_pair leaves: its dE and badness changes (BAD; change[t] for slot lane +
// 32 t).  hist: kDirWords words, zero, left zero.
template <bool BAD>
__device__ __noinline__ int swap_delta_slow(const int (&key2)[kSlotsPerLane], int m, int lane, int u, int v, int cu,
                                            int cv, const uint16_t* __restrict__ lut4, uint32_t* __restrict__ hist,
                                            int (&change)[kSlotsPerLane]) {
  const int ru = u >> 1, rv = v >> 1;
  int t_sum[4], line_count[2] = {0, 0};
  for (int t = 0; t < kSlotsPerLane; ++t) change[t] = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {  // u, v, u', v'
    const int rx = (c & 1) ? rv : ru, centre = rx * kLutW + (c == 0 || c == 3 ? cu : cv);
    int ids[kSlotsPerLane], part = 0;
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {
      const int k = lane + 32 * t;
      ids[t] = -1;
      if (k < m && k != u && k != v && (k >> 1) != rx) {
        ids[t] = (int)(dir4(lut4, key2[t] >> 1, centre) >> 2);
        part += hist_add(hist, ids[t]);
      }
    }
    __syncwarp();
    t_sum[c] = warp_sum(part);
    int line = -1;  // direction of the other moved point, for u and u'
    if (!(c & 1)) {
      line = (int)(dir4(lut4, rv * kLutW + (c ? cu : cv), centre) >> 2);
      line_count[c >> 1] = hist_get(hist, line);
    }
    if (BAD) {
#pragma unroll
      for (int t = 0; t < kSlotsPerLane; ++t)
        if (ids[t] >= 0) change[t] += (c < 2 ? -1 : 1) * (hist_get(hist, ids[t]) - 1 + (ids[t] == line));
    }
    __syncwarp();
    hist_release(hist, ids);
    __syncwarp();
  }
  const int before_u = t_sum[0] + line_count[0], before_v = t_sum[1] + line_count[0];
  const int after_u = t_sum[2] + line_count[1], after_v = t_sum[3] + line_count[1];
  if (BAD) {
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {
      if (lane + 32 * t == u) change[t] = after_u - before_u;
      if (lane + 32 * t == v) change[t] = after_v - before_v;
    }
  }
  return after_u + after_v - line_count[1] - (before_u + before_v - line_count[0]);
}

// The same with 4-bit counters, u' and v' side by side and then u and v
// (pair_move.cuh).  False, with nothing to use, if a counter may have wrapped.
template <bool BAD, int NT>
__device__ __forceinline__ bool swap_delta_pair(const WarpState& W, int u, int v, int cu, int cv,
                                                const uint16_t* __restrict__ lut4, uint32_t* __restrict__ hist,
                                                int& dE, int (&change)[kSlotsPerLane]) {
  using Num = DenseNumbering;
  uint32_t* const h1 = hist + Num::kWords;
  const int ru = u >> 1, rv = v >> 1;
  Directions a, b;
  uint32_t line_new;
  const PairCount p = count_pair<Num, NT, false>(W, lut4, hist, ru, rv, cu, cv, a, b, line_new);
  if (BAD) {  // as pair_move takes them
#pragma unroll
    for (int t = 0; t < NT; ++t)
      change[t] = centre_get(a, t) + centre_get(b, t) - (a.e[t] == Num::kRow || a.e[t] == Num::kCol) -
                  (b.e[t] == Num::kRow || b.e[t] == Num::kCol) + (a.e[t] == line_new);
  }
  __syncwarp();
  clear_centre<NT>(a);
  clear_centre<NT>(b);
  const int kU = 2 * (ru * kLutW + cu), kV = 2 * (rv * kLutW + cv);
  const uint32_t line_old = dir4_2(lut4, kV, kU);
  find_centre<Num, NT>(W, lut4, hist, kU, a);
  find_centre<Num, NT>(W, lut4, h1, kV, b);
  __syncwarp();
  const uint32_t part = count_centres<NT>(W, a, b);
  __syncwarp();
  const int joint = (int)counter_of(hist, line_old) - 1;
  if (BAD) {
#pragma unroll
    for (int t = 0; t < NT; ++t) change[t] -= centre_get(a, t) + centre_get(b, t) - (b.e[t] == line_old);
  }
  const uint32_t sums = __reduce_add_sync(0xffffffffu, part);
  const int bad_u = (int)(sums & 0xFFFu), bad_v = (int)(sums >> 12);
  __syncwarp();
  clear_centre<NT>(a);
  clear_centre<NT>(b);
  __syncwarp();
  dE = p.ta + p.tb + p.j_new - (bad_u + bad_v - joint);
  if (BAD) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      if (W.slot(t) == u) change[t] = p.ta + p.j_new - bad_u;
      if (W.slot(t) == v) change[t] = p.tb + p.j_new - bad_v;
    }
  }
  return !p.wide && bad_u < kMoveSum && bad_v < kMoveSum;
}

// The reference formulation (tempering.py:68-89), pair by pair.  Returns this
// lane's share of dE; badness changes are added to the warp's smem array `db`.
__device__ __forceinline__ int aligned(int a, int ca, int b, int cb, int c, int cc) {
  return (b - a) * (cc - ca) == (cb - ca) * (c - a);
}

__device__ int swap_delta_pairs(const int* __restrict__ cs, int m, int u, int v, int lane, int* db) {
  const int ru = u >> 1, rv = v >> 1, cu = cs[u], cv = cs[v];
  int delta = 0;
  for (int i = 0; i < m - 1; ++i) {
    if (i == u || i == v) continue;
    const int ri = i >> 1, ci = cs[i];
    for (int j = i + 1 + lane; j < m; j += 32) {
      if (j == u || j == v) continue;
      const int rj = j >> 1, cj = cs[j];
      int d = aligned(ru, cv, ri, ci, rj, cj) - aligned(ru, cu, ri, ci, rj, cj);
      if (d) {
        delta += d;
        if (db) {
          atomicAdd(db + u, d);
          atomicAdd(db + i, d);
          atomicAdd(db + j, d);
        }
      }
      d = aligned(rv, cu, ri, ci, rj, cj) - aligned(rv, cv, ri, ci, rj, cj);
      if (d) {
        delta += d;
        if (db) {
          atomicAdd(db + v, d);
          atomicAdd(db + i, d);
          atomicAdd(db + j, d);
        }
      }
    }
  }
  for (int k = lane; k < m; k += 32) {
    if (k == u || k == v) continue;
    const int d = aligned(ru, cv, rv, cu, k >> 1, cs[k]) - aligned(ru, cu, rv, cv, k >> 1, cs[k]);
    if (d) {
      delta += d;
      if (db) {
        atomicAdd(db + u, d);
        atomicAdd(db + v, d);
        atomicAdd(db + k, d);
      }
    }
  }
  return delta;
}

// Batched swap deltas: moves[mv] = (state, u, v), a warp each.  dE = N3_SENTINEL
// for illegal moves or bad indices (then the badness changes are 0).
struct MoveArgs {
  const int16_t* cols;
  const int32_t* moves;
  int B, n, M;
  const uint16_t* lut4;
  int32_t* dE;
  int32_t* dbad;  // [M][2n] or nullptr
};

// The reference formulation.
constexpr int kPairsWarps = 8;
__global__ void __launch_bounds__(kPairsWarps * 32) swap_delta_pairs_kernel(const MoveArgs A) {
  __shared__ int cs_all[kPairsWarps][kMaxM], db_all[kPairsWarps][kMaxM];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = 2 * A.n;
  int *cs = cs_all[warp], *db = db_all[warp];
  for (int mv = blockIdx.x * kPairsWarps + warp; mv < A.M; mv += gridDim.x * kPairsWarps) {
    const int b = A.moves[3 * mv], u = A.moves[3 * mv + 1], v = A.moves[3 * mv + 2];
    const bool in_range = b >= 0 && b < A.B && u >= 0 && u < m && v >= 0 && v < m;
    if (in_range)
      for (int s = lane; s < m; s += 32) cs[s] = A.cols[(size_t)b * m + s];
    for (int s = lane; s < m; s += 32) db[s] = 0;
    __syncwarp();
    int d = N3_SENTINEL;
    if (in_range && legal_swap(cs, u, v)) d = warp_sum(swap_delta_pairs(cs, m, u, v, lane, A.dbad ? db : nullptr));
    __syncwarp();
    if (A.dbad)
      for (int s = lane; s < m; s += 32) A.dbad[(size_t)mv * m + s] = db[s];
    if (lane == 0) A.dE[mv] = d;
    __syncwarp();
  }
}

// By direction histograms.  Shared-memory operations bound it: 20 table loads, 20
// counts and 20 clears per move, 3 to 3.5 cycles each for 32 lanes at random (95 %
// of the cycles).  65,536 moves of 4096 n = 75 states: 63 us, 77 us with four 8-bit
// histograms one after the other; with badness changes 89 and 103 us.
constexpr int kDeltaWarps = 30;
constexpr size_t kDeltaSmem = kCompactLutBytes + sizeof(uint32_t) * 2 * DenseNumbering::kWords * kDeltaWarps;
static_assert(kDeltaSmem <= 227 * 1024, "swap_delta_kernel shared memory");
static_assert(2 * DenseNumbering::kWords >= kDirWords, "swap_delta_slow's counters");

template <bool BAD, int NT>
__global__ void __launch_bounds__(kDeltaWarps * 32, 1) swap_delta_kernel(const MoveArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* lut4 = reinterpret_cast<uint16_t*>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, m = 2 * A.n;
  uint32_t* hist = reinterpret_cast<uint32_t*>(smem + kCompactLutBytes) + warp * 2 * DenseNumbering::kWords;
  compact_lut_copy(lut4, A.lut4);
  for (int i = lane; i < 2 * DenseNumbering::kWords; i += 32) hist[i] = 0u;
  __syncthreads();
  WarpState W;
  W.m = m;
  W.lane = lane;
  W.cs = nullptr;
  W.bs = nullptr;
  for (int mv = blockIdx.x * warps + warp; mv < A.M; mv += gridDim.x * warps) {
    const int b = A.moves[3 * mv], u = A.moves[3 * mv + 1], v = A.moves[3 * mv + 2];
    int d = N3_SENTINEL, change[kSlotsPerLane];
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) change[t] = 0;
    if (b >= 0 && b < A.B && u >= 0 && u < m && v >= 0 && v < m) {  // uniform in the warp
      const int16_t* cols = A.cols + (size_t)b * m;
#pragma unroll
      for (int t = 0; t < kSlotsPerLane; ++t) {
        const int k = W.slot(t);
        W.key2[t] = t < NT && k < m ? 2 * ((k >> 1) * kLutW + cols[k]) : 0;
      }
      const int cu = cols[u], cv = cols[v], pu = cols[u ^ 1], pv = cols[v ^ 1];
      if ((u >> 1) != (v >> 1) && cu != cv && pu != cv && pv != cu) {  // uniform
        // a cell held twice has no direction to itself
        const bool twin = pu == cu || pv == cv;
        if (twin || !swap_delta_pair<BAD, NT>(W, u, v, cu, cv, lut4, hist, d, change))
          d = swap_delta_slow<BAD>(W.key2, m, lane, u, v, cu, cv, lut4, hist, change);
      }
    }
    if (BAD) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int k = W.slot(t);
        if (k < m) A.dbad[(size_t)mv * m + k] = change[t];
      }
    }
    if (lane == 0) A.dE[mv] = d;
  }
}

// Scores of every partner of anchor slots (the reference plugin
// two_switch_scores, src/no_three_75/gpu_delta.py:19-75, and
// evaluate_two_switches / evaluate_transpositions, accelerated.py:40-195):
//   out = current - (bad[u] + bad[v] - joint(u, v)) + t(u') + t(v') + j(u', v')
// SAME_LAYER restricts partners to slots of u's layer and indexes the output by
// partner row.  The partner rule is the reference's (accelerated.py:146-151,
// gpu_delta.py:175-180): another row, and neither new point duplicates its row
// partner; equal columns are allowed (the move is then the identity).
//
// For a state with two points in every column, t(u') over A = S \ {u, v} depends
// on the cell u' = (r_u, c_v) alone: no pair with u or v lines up with it off its
// row and column, so it is the cell's cover entry (cover.cuh).  One CTA takes a
// run of consecutive anchors of one state:
//   kRunCover or more   the CTA builds the cover table of the state once; then a
//       warp per anchor takes joint(u, v) of all partners from one histogram
//       around u, t(u') and t(v') from the table, and j(u', v') by the cells of
//       32 partners' lines numbered through (4.6 on average, but 40 in the longest,
//       so a walk per lane took 8 us more); the last anchors of a run share
//       their partners among the warps left (4 us)
//   fewer               a warp per partner, both new centres' histograms side by
//       side (pair_move.cuh), whatever the columns hold; each warp holds the state
//       itself, so that short runs follow each other without a barrier, and the next
//       run's first partners go to the warps that the last one left idle (512 n = 20
//       states with a slot each: 14.0 us, 17.7 with the state shared by the CTA, 14.8 with
//       a CTA of eight warps per anchor)
// 64 n = 75 states, every slot: 70 us, 834 us with two histograms per partner one
// after the other; 1024 states with a slot each, partners of its layer: 48 and 60 us.
constexpr int kPartnerWarps = 24;
// Anchors of one state from which its cover table is built (512 states, us: n = 75, 5 anchors each by
// pairs 177, 7 by pairs 245, 8 by the table 142; n = 40 74, 100, 57; n = 20 38, 50, 30; n = 10 18, 23, 19;
// n = 4 13, 15, 17: from five on the table would do as well on larger grids).
constexpr int kRunCover = 8;
constexpr int kPartnerRegion = ((kMaxN * kMaxN + 1) / 2 + 3) / 4 * 4;  // words of the cover table

struct PartnerSmem {
  uint16_t prim4[kCompactLutBytes / 2];
  uint16_t dir4[kCompactLutBytes / 2];
  uint32_t recip[kMaxN + 1];
  uint32_t T[kPartnerRegion];
  uint32_t bits[(kMaxN * kMaxN + 31) / 32];  // the state's cells
  uint32_t hist[kPartnerWarps][2 * DenseNumbering::kWords];
  uint2 scratch[kPartnerWarps][32];
  uint32_t count[kPartnerWarps][32];
  int columns[kMaxN];
  uint8_t cs[152];
};
static_assert(sizeof(PartnerSmem) <= 227 * 1024, "partner_scores_kernel shared memory");

// One partner's score by 8-bit histograms over A, one centre at a time: for equal
// columns and where a 4-bit counter may have wrapped.
__device__ __noinline__ int partner_by_histograms(const uint16_t* __restrict__ lut4, const uint8_t* __restrict__ cs,
                                                  uint32_t* __restrict__ hist, int m, int u, int v, int cur,
                                                  int bad_uv, int lane) {
  const int ru = u >> 1, rv = v >> 1, cu = cs[u], cv = cs[v];
  int part = 0, j_new = 0;
  for (int c = 0; c < 2; ++c) {
    const int rx = c ? rv : ru, centre = c ? rv * kLutW + cu : ru * kLutW + cv;
    int ids[kSlotsPerLane];
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {
      const int k = lane + 32 * t;
      ids[t] = -1;
      if (k < m && k != u && k != v && (k >> 1) != rx) {
        const int ck = cs[k];
        ids[t] = (int)(dir4(lut4, (k >> 1) * kLutW + ck, centre) >> 2);
        part += hist_add(hist, ids[t]);
        if (c == 0) part += ((rv - ru) * (ck - cu) == (cv - cu) * ((k >> 1) - ru)) << 16;  // joint
      } else if (c == 0 && k < m && k != u && k != v) {  // u's row partner
        part += ((rv - ru) * (cs[k] - cu) == (cv - cu) * ((k >> 1) - ru)) << 16;
      }
    }
    __syncwarp();
    if (c == 0) j_new = hist_get(hist, (int)(dir4(lut4, rv * kLutW + cu, centre) >> 2));
    __syncwarp();
    hist_release(hist, ids);
    __syncwarp();
  }
  const int sum = warp_sum(part);
  return cur - (bad_uv - (sum >> 16)) + (sum & 0xFFFF) + j_new;
}

// A state's column as the partner scores hold it: the histograms take columns beyond n as well.
__device__ __forceinline__ uint8_t partner_column(int c) { return (uint8_t)min(max(c, 0), kMaxN - 1); }

// The partners of the anchors [a0, a1) of one state (`cols`, m columns) by a warp each.  cs: the
// warp's 152 bytes; turn: the warp that the next partner is for; await: the block's barrier comes
// first (the same in every warp), for the tables to be in place and the space of cs to be free.
template <bool SAME_LAYER, int NT>
__device__ __forceinline__ void partners_by_pairs(const uint16_t* __restrict__ lut4, uint8_t* __restrict__ cs,
                                                  uint32_t* __restrict__ hist, int n,
                                                  const int16_t* __restrict__ cols,
                                                  const int32_t* __restrict__ anchors, int a0, int a1,
                                                  const int32_t* __restrict__ bad, int cur, int warp, int lane,
                                                  int& turn, bool& await, int32_t* __restrict__ out) {
  const int m = 2 * n, width = SAME_LAYER ? n : m;
  WarpState W;
  W.m = m;
  W.lane = lane;
  W.cs = nullptr;
  W.bs = nullptr;
#pragma unroll
  for (int t = 0; t < kSlotsPerLane; ++t) {
    const int s = W.slot(t);
    W.key2[t] = 0;
    if (t < NT && s < m) W.key2[t] = 2 * ((s >> 1) * kLutW + partner_column(cols[s]));
  }
  if (await)
    __syncthreads();
  else
    __syncwarp();  // done with the state before
  await = false;
#pragma unroll
  for (int t = 0; t < NT; ++t)
    if (W.slot(t) < m) cs[W.slot(t)] = (uint8_t)(W.key2[t] / 2 - (W.slot(t) >> 1) * kLutW);
  __syncwarp();
  for (int a = a0; a < a1; ++a) {
    const int u = anchors[2 * a + 1];
    const bool in_range = u >= 0 && u < m;
    int w = warp - turn;
    if (w < 0) w += kPartnerWarps;
    for (; w < width; w += kPartnerWarps) {
      int score = N3_SENTINEL;
      if (in_range) {  // uniform
        const int v = SAME_LAYER ? 2 * w + (u & 1) : w;
        const int ru = u >> 1, rv = v >> 1, cu = cs[u], cv = cs[v];
        if (rv != ru && cv != cs[u ^ 1] && cu != cs[v ^ 1]) {  // uniform in the warp
          const int bad_uv = bad[u] + bad[v];
          bool redo = cu == cv;
          if (!redo) {
            Directions x, y;
            uint32_t line_new;
            const PairCount p = count_pair<DenseNumbering, NT>(W, lut4, hist, ru, rv, cu, cv, x, y, line_new);
            __syncwarp();
            clear_centre<NT>(x);
            clear_centre<NT>(y);
            __syncwarp();
            score = cur - (bad_uv - p.joint) + p.ta + p.tb + p.j_new;
            redo = p.wide;
          }
          if (redo) score = partner_by_histograms(lut4, cs, hist, m, u, v, cur, bad_uv, lane);
        }
      }
      if (lane == 0) out[(size_t)a * width + w] = score;
    }
    turn = (turn + width) % kPartnerWarps;
  }
}

template <bool SAME_LAYER>
__global__ void __launch_bounds__(kPartnerWarps * 32, 1) partner_scores_kernel(
    const int16_t* __restrict__ cols, const int32_t* __restrict__ badness, const int32_t* __restrict__ current,
    int B, int n, const int32_t* __restrict__ anchors, int A, int per_cta, const uint16_t* __restrict__ g_prim4,
    const uint16_t* __restrict__ g_dir4, int32_t* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  PartnerSmem& S = *reinterpret_cast<PartnerSmem*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m = 2 * n, width = SAME_LAYER ? n : m;
  compact_lut_copy(S.prim4, g_prim4);
  compact_lut_copy(S.dir4, g_dir4);
  for (int a = tid; a <= kMaxN; a += blockDim.x) S.recip[a] = a ? (65536u + (uint32_t)a - 1u) / (uint32_t)a : 0u;
  uint32_t* hist = S.hist[warp];
  for (int i = lane; i < 2 * DenseNumbering::kWords; i += 32) hist[i] = 0u;
  // the warp's own state, in the cover table's space
  uint8_t* const mine = reinterpret_cast<uint8_t*>(S.T) + 152 * warp;
  static_assert(152 * kPartnerWarps <= sizeof(S.T), "the warps' states");
  int turn = 0;
  bool await = true;
  const int a_end = min(A, (int)(blockIdx.x + 1) * per_cta);
  for (int a0 = blockIdx.x * per_cta; a0 < a_end;) {
    // the run of anchors of one state (the same in every warp)
    const int b = anchors[2 * a0];
    int a1 = a0 + 1;
    for (;;) {
      const int a = a1 + lane;
      const unsigned same = __ballot_sync(0xffffffffu, a < a_end && anchors[2 * a] == b);
      const int more = __ffs(~same) - 1;  // -1 if all 32
      a1 += more < 0 ? 32 : more;
      if (more >= 0) break;
    }
    if (b < 0 || b >= B) {  // uniform
      for (int i = tid; i < (a1 - a0) * width; i += blockDim.x) out[(size_t)a0 * width + i] = N3_SENTINEL;
      a0 = a1;
      continue;
    }
    const int cur = current[b];
    const int32_t* bad = badness + (size_t)b * m;
    const int16_t* state = cols + (size_t)b * m;
    bool cover = a1 - a0 >= kRunCover;
    if (cover) {
      __syncthreads();  // the warps are done with the table, or with their own states
      for (int i = tid; i < kMaxN; i += blockDim.x) S.columns[i] = 0;
      for (int i = tid; i < (kMaxN * kMaxN + 31) / 32; i += blockDim.x) S.bits[i] = 0u;
      for (int i = tid; i < kPartnerRegion; i += blockDim.x) S.T[i] = 0u;
      __syncthreads();
      bool regular = true;  // two points in every column, in cells of their own
      for (int s = tid; s < m; s += blockDim.x) {
        const int c = state[s];
        const bool on_grid = c >= 0 && c < n;
        regular = regular && on_grid;
        S.cs[s] = partner_column(c);
        if (on_grid) {
          atomicAdd(&S.columns[c], 1);
          const int cell = (s >> 1) * n + c;
          const uint32_t bit = 1u << (cell & 31);
          if (atomicOr(&S.bits[cell >> 5], bit) & bit) regular = false;
        }
      }
      __syncthreads();
      for (int c = tid; c < n; c += blockDim.x) regular = regular && S.columns[c] == 2;
      cover = __syncthreads_and(regular);
    }
    if (cover) {
      cover_build(S.cs, S.T, n, S.prim4, S.recip, S.scratch[warp], lane, warp, kPartnerWarps);
      __syncthreads();
      for (int first = a0; first < a1; first += kPartnerWarps) {
        // a warp per anchor; the last ones share their partners among several warps
        const int left = a1 - first, parts = left < kPartnerWarps ? kPartnerWarps / left : 1;
        const int a = first + warp / parts, w_first = 32 * (warp % parts), w_step = 32 * parts;
        if (a >= a1) break;  // uniform in the warp
        const int u = anchors[2 * a + 1];
        if (u < 0 || u >= m) {  // uniform in the warp
          for (int w0 = w_first; w0 < width; w0 += w_step)
            if (w0 + lane < width) out[(size_t)a * width + w0 + lane] = N3_SENTINEL;
          continue;
        }
        const int ru = u >> 1, cu = S.cs[u], centre = ru * kLutW + cu, bad_u = bad[u];
        int ids[kSlotsPerLane];  // 8-bit counters of the directions from u
#pragma unroll
        for (int t = 0; t < kSlotsPerLane; ++t) {
          const int k = lane + 32 * t;
          ids[t] = k < m && k != u ? (int)(dir4(S.dir4, (k >> 1) * kLutW + S.cs[k], centre) >> 2) : -1;
          if (ids[t] >= 0) hist_add(hist, ids[t]);
        }
        __syncwarp();
        for (int w0 = w_first; w0 < width; w0 += w_step) {
          const int w = w0 + lane, v = min(SAME_LAYER ? 2 * w + (u & 1) : w, m - 1);
          const int rv = v >> 1, cv = S.cs[v];
          const bool legal = w < width && rv != ru && cv != S.cs[u ^ 1] && cu != S.cs[v ^ 1];
          const int line = count_lines(S.bits, n, ru, cv, rv, cu, legal, S.prim4, S.recip, S.scratch[warp],
                                       S.count[warp], lane);
          if (w >= width) continue;
          int score = N3_SENTINEL;
          if (legal) {
            // the others on the line (u, v) (a column holds no third point)
            const int joint = hist_get(hist, (int)(dir4(S.dir4, rv * kLutW + cv, centre) >> 2)) - 1;
            score = cur - (bad_u + bad[v] - joint) + cover_get(S.T, ru * n + cv) + cover_get(S.T, rv * n + cu) + line;
          }
          out[(size_t)a * width + w] = score;
        }
        __syncwarp();
        hist_release(hist, ids);
        __syncwarp();
      }
      await = true;
    } else {
      const auto pairs = [&](auto nt) {
        partners_by_pairs<SAME_LAYER, decltype(nt)::value>(S.dir4, mine, hist, n, state, anchors, a0, a1, bad, cur, warp,
                                                           lane, turn, await, out);
      };
      switch ((m + 31) >> 5) {
        case 5: pairs(std::integral_constant<int, 5>{}); break;
        case 4: pairs(std::integral_constant<int, 4>{}); break;
        case 3: pairs(std::integral_constant<int, 3>{}); break;
        case 2: pairs(std::integral_constant<int, 2>{}); break;
        default: pairs(std::integral_constant<int, 1>{}); break;
      }
    }
    a0 = a1;
  }
}

}  // namespace n3

namespace n3host {

template <class K>
static int prepare(K kernel, size_t bytes) {
  return allow_smem(reinterpret_cast<const void*>(kernel), bytes);
}

// swap_delta_kernel for 2n slots, NT = ceil(2n / 32) a lane.
static void (*delta_kernel(bool bad, int n))(const n3::MoveArgs) {
  using namespace n3;
  switch ((2 * n + 31) / 32) {
    case 5: return bad ? swap_delta_kernel<true, 5> : swap_delta_kernel<false, 5>;
    case 4: return bad ? swap_delta_kernel<true, 4> : swap_delta_kernel<false, 4>;
    case 3: return bad ? swap_delta_kernel<true, 3> : swap_delta_kernel<false, 3>;
    case 2: return bad ? swap_delta_kernel<true, 2> : swap_delta_kernel<false, 2>;
    default: return bad ? swap_delta_kernel<true, 1> : swap_delta_kernel<false, 1>;
  }
}

int prepare_delta() {
  for (int n = 16; n <= 80; n += 16) {
    N3_TRY(prepare(delta_kernel(true, n), n3::kDeltaSmem));
    N3_TRY(prepare(delta_kernel(false, n), n3::kDeltaSmem));
  }
  N3_TRY(prepare(n3::partner_scores_kernel<true>, sizeof(n3::PartnerSmem)));
  return prepare(n3::partner_scores_kernel<false>, sizeof(n3::PartnerSmem));
}

static int check_state_args(int B, int n, const void* cols) {
  if (n < 2 || n > N3_MAX_N) return set_error(N3_ERR_RANGE, "n=%d outside [2, %d]", n, N3_MAX_N);
  if (B < 0) return set_error(N3_ERR_ARG, "negative batch size %d", B);
  if (B > 0 && cols == nullptr) return set_error(N3_ERR_ARG, "null state pointer");
  return N3_OK;
}

static int launch_swap(bool pairs, const int16_t* cols, int B, int n, const int32_t* moves, int M, int32_t* dE,
                       int32_t* dbad, cudaStream_t st) {
  N3_TRY(check_state_args(B, n, cols));
  if (M < 0) return set_error(N3_ERR_ARG, "negative move count");
  if (M == 0) return N3_OK;
  if (moves == nullptr || dE == nullptr) return set_error(N3_ERR_ARG, "null move or output pointer");
  N3_TRY(ensure_device_tables());
  const n3::MoveArgs A = {cols, moves, B, n, M, dir4_lut_device_ptr(), dE, dbad};
  const int sms = sm_count();
  if (pairs) {
    const int want = (M + n3::kPairsWarps - 1) / n3::kPairsWarps;
    n3::swap_delta_pairs_kernel<<<want < 8 * sms ? want : 8 * sms, n3::kPairsWarps * 32, 0, st>>>(A);
    return check_launch("swap_delta_pairs_kernel");
  }
  // One CTA per SM, with as many warps as share its moves evenly, but enough to copy
  // the table.  (With 30 warps for any number of moves above 4440, the last round was
  // almost empty: 4500 n = 75 moves 11.0 us, now 7.4; 9000 14.7, now 11.4.)
  const int per_sm = (M + sms - 1) / sms, rounds = (per_sm + n3::kDeltaWarps - 1) / n3::kDeltaWarps;
  int warps = (per_sm + rounds - 1) / rounds;
  if (warps < 8) warps = 8;
  const int want = (M + warps - 1) / warps;
  const auto kernel = delta_kernel(dbad != nullptr, n);
  N3_TRY(prepare(kernel, n3::kDeltaSmem));
  kernel<<<want < sms ? want : sms, warps * 32, n3::kDeltaSmem, st>>>(A);
  return check_launch("swap_delta_kernel");
}

static int launch_partners(bool same_layer, const int16_t* cols, const int32_t* badness, const int32_t* current, int B,
                           int n, const int32_t* anchors, int A, int32_t* out, cudaStream_t st) {
  N3_TRY(check_state_args(B, n, cols));
  if (A < 0) return set_error(N3_ERR_ARG, "negative anchor count");
  if (A == 0) return N3_OK;
  if (!badness || !current || !anchors || !out) return set_error(N3_ERR_ARG, "null pointer");
  N3_TRY(ensure_device_tables());
  const int sms = sm_count();
  // Consecutive anchors to a CTA, one CTA per SM.  Callers list a state's anchors
  // together; with enough of them each CTA gets whole states or a share of one, as
  // it would if all states had the same number, so that few build two cover tables
  // (64 states of 150 anchors, with a walk per lane: 128 CTAs of 75 took 85 us, 148 of
  // 65 took 111 us).
  int per_cta = (A + sms - 1) / sms;
  const int each = B > 0 ? A / B : 0;
  if (each >= 2 * n3::kRunCover && each * (int64_t)B == A) {
    const int parts = B < sms ? sms / B : 1;
    const int share = (each + parts - 1) / parts;
    if (share > per_cta) per_cta = share;
  }
  const int grid = (A + per_cta - 1) / per_cta;
  const auto kernel = same_layer ? n3::partner_scores_kernel<true> : n3::partner_scores_kernel<false>;
  N3_TRY(prepare(kernel, sizeof(n3::PartnerSmem)));
  kernel<<<grid, n3::kPartnerWarps * 32, sizeof(n3::PartnerSmem), st>>>(
      cols, badness, current, B, n, anchors, A, per_cta, prim4_lut_device_ptr(), dir4_lut_device_ptr(), out);
  return check_launch("partner_scores_kernel");
}

}  // namespace n3host

extern "C" {

int n3_swap_delta(const int16_t* cols, int B, int n, const int32_t* moves, int M, int32_t* dE, int32_t* dbad,
                  void* stream) {
  return n3host::launch_swap(false, cols, B, n, moves, M, dE, dbad, (cudaStream_t)stream);
}

int n3_swap_delta_pairs(const int16_t* cols, int B, int n, const int32_t* moves, int M, int32_t* dE, int32_t* dbad,
                        void* stream) {
  return n3host::launch_swap(true, cols, B, n, moves, M, dE, dbad, (cudaStream_t)stream);
}

int n3_two_switch_scores(const int16_t* cols, const int32_t* badness, const int32_t* current, int B, int n,
                         const int32_t* anchors, int A, int32_t* out, void* stream) {
  return n3host::launch_partners(false, cols, badness, current, B, n, anchors, A, out, (cudaStream_t)stream);
}

int n3_transposition_scores(const int16_t* cols, const int32_t* badness, const int32_t* current, int B, int n,
                            const int32_t* anchors, int A, int32_t* out, void* stream) {
  return n3host::launch_partners(true, cols, badness, current, B, n, anchors, A, out, (cudaStream_t)stream);
}

}  // extern "C"
