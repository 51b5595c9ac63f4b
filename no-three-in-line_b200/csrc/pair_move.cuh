// Exact dE of a swap by one warp from direction histograms with 4-bit counters,
// two centres at a time.
//
// A histogram tells the points of the state S apart by their direction from a
// centre; its pair sum is the number of pairs collinear with the centre.  The new
// centres u' and v' are counted side by side (for an accepted move then u and v),
// each in counters of its own: a lane owns slots lane, lane + 32, ..., and its ten
// table loads and then its ten atomics are in flight together.  A chain's moves
// follow each other, so what counts is one move's latency, at about four cycles
// per instruction; no slot is tested or left out, which saves a third of them:
//  - u and v are counted with the rest.  As u' shares a row with u and a column
//    with v, they add only to those two classes: the row's one pair, and for a
//    column of x points x - 1 pairs, so t(u') over A = S \ {u, v} is the sum less
//    the column's counter x (likewise v').  The sum around u itself is its badness.
//  - a lane's missing slots add 0 to a word that stays 0.
// The counters have 4 bits, so that two histograms of each of 16 chains fit an
// SM.  A counter that reaches 16 has by then added 0 + 1 + ... + 15 = 120 pairs to
// its centre's sum, so a move with a sum of 120 or more is evaluated again by
// slow_move with 8-bit counters.
//
// The direction table maps |key(k) - key(centre)| (key = row * kLutW + column;
// the sign of the difference only turns the direction round) to four times the
// direction's number: the low five bits are the counter's shift in its word,
// the rest is the word.  Two numberings, with their tables:
//   StepNumbering   the direction (p, q) is p * kLutW + q (n3host::prim4_lut_device_ptr);
//                   the table gives the steps of a walk as well
//   DenseNumbering  the compact ids 0 .. kDirCount - 1 (n3host::dir4_lut_device_ptr)
// In both the difference 0 has a counter of its own, and a histogram's last word
// belongs to no direction.
#pragma once

#include "dirs.cuh"
#include "n3_common.cuh"

namespace n3 {

struct StepNumbering {
  static constexpr uint32_t kRow = 4u * 1u, kCol = 4u * kLutW;  // the directions (0, 1) and (1, 0)
  static constexpr int kWords = 1408;                           // up to 74 * kLutW + 74, and one
};
struct DenseNumbering {
  static constexpr uint32_t kRow = 0u, kCol = 4u * kMaxN;  // ids in (p, q) order: (0, 1), then (1, -74) ..
  static constexpr int kWords = kDirCount / 8 + 2;         // the centre's word, and one
};
static_assert(StepNumbering::kWords * 8 > (kMaxN - 1) * (kLutW + 1) + 8, "a 4-bit counter per step, and a word");

constexpr int kMoveSum = 120;  // pair sums from which a 4-bit counter may have wrapped

__device__ __forceinline__ uint32_t dir4(const uint16_t* __restrict__ lut4, int key, int centre) {
  return lut4[abs(key - centre) + kMaxN - 1];
}
// The same for doubled keys, which are byte offsets into the table.
__device__ __forceinline__ uint32_t dir4_2(const uint16_t* __restrict__ lut4, int key2, int centre2) {
  return *reinterpret_cast<const uint16_t*>(reinterpret_cast<const char*>(lut4 + kMaxN - 1) + abs(key2 - centre2));
}

// One chain's state as its warp holds it: twice the table key of each of the
// lane's slots in registers, every slot's column and badness in shared memory.
struct WarpState {
  int key2[kSlotsPerLane];  // 0 for a slot beyond m
  int m;         // slots
  int lane;
  uint8_t* cs;   // [m] columns
  int* bs;       // [m] badness
  __device__ __forceinline__ int slot(int t) const { return lane + 32 * t; }
  __device__ __forceinline__ void swap_keys(int u, int v, int dc) {
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) key2[t] += slot(t) == u ? 2 * dc : (slot(t) == v ? -2 * dc : 0);
  }
  // The lane's points among slots lane, ..., lane + 32 (NT - 1) on the line through
  // (ru, cu) with direction (dr, dc); with ck = key - rk * kLutW,
  //   dr (ck - cu) - dc (rk - ru) = dr key - rk (kLutW dr + dc) - (dr cu - dc ru).
  template <int NT>
  __device__ __forceinline__ int on_line(int ru, int cu, int dr, int dc) const {
    const int q = kLutW * dr + dc, w = 2 * (dr * cu - dc * ru) + (lane & ~1) * q;
    int c = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t) c += dr * key2[t] == w + t * 32 * q && (t < NT - 1 || slot(t) < m);
    return c;
  }
};

// A proposed move as its lane prepares it: the slots, their columns and the sum of
// their badness, in two words that a shuffle hands to the warp.
struct PreparedMove {
  uint32_t slots;  // u | v << 8 | cu << 16 | cv << 24
  int bad;         // badness of u plus badness of v
};

// The histogram of one centre: the directions of the lane's slots and their words.
struct Directions {
  uint32_t e[kSlotsPerLane];
  uint32_t* word[kSlotsPerLane];
};

// NT: the slots a lane may hold, ceil(m / 32); only the last can be missing.
template <class Num, int NT>
__device__ __forceinline__ void find_centre(const WarpState& W, const uint16_t* __restrict__ lut4, uint32_t* hist,
                                            int centre2, Directions& d) {
#pragma unroll
  for (int t = 0; t < NT; ++t) d.e[t] = dir4_2(lut4, W.key2[t], centre2);
  if (W.slot(NT - 1) >= W.m) d.e[NT - 1] = 32u * (Num::kWords - 1);
#pragma unroll
  for (int t = 0; t < NT; ++t) d.word[t] = hist + (d.e[t] >> 5);
}

// Counts the slots of two centres; returns this lane's share of the pair sums, the
// second's from bit 12 on (at most 150 counters of 15 each).
template <int NT>
__device__ __forceinline__ uint32_t count_centres(const WarpState& W, const Directions& a, const Directions& b) {
  uint32_t olda[NT], oldb[NT], sum = 0u;
  const uint32_t last = W.slot(NT - 1) < W.m ? 1u : 0u;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const uint32_t one = t < NT - 1 ? 1u : last;  // the funnel shifts take e modulo 32
    olda[t] = atomicAdd(a.word[t], __funnelshift_l(0u, one, a.e[t]));
    oldb[t] = atomicAdd(b.word[t], __funnelshift_l(0u, one, b.e[t]));
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
    sum += (__funnelshift_r(olda[t], 0u, a.e[t]) & 15u) + ((__funnelshift_r(oldb[t], 0u, b.e[t]) & 15u) << 12);
  return sum;
}

__device__ __forceinline__ uint32_t counter_of(const uint32_t* hist, uint32_t e) {
  return __funnelshift_r(hist[e >> 5], 0u, e) & 15u;
}
__device__ __forceinline__ int centre_get(const Directions& d, int t) {
  return (int)(__funnelshift_r(*d.word[t], 0u, d.e[t]) & 15u);
}
template <int NT>
__device__ __forceinline__ void clear_centre(const Directions& d) {
#pragma unroll
  for (int t = 0; t < NT; ++t) *d.word[t] = 0u;
}

// The same move with 8-bit counters, a centre at a time, in `hist` (kWords words,
// zero, left zero).  accept(dE) decides (the same in every lane); an accepted
// move is made, but for the keys.  (Not inlined: rare.)
template <int kWords, class Accept>
static __device__ __noinline__ bool slow_move(int m, int lane, uint8_t* __restrict__ cs, int* __restrict__ bs,
                                              const uint16_t* __restrict__ lut4, uint32_t* __restrict__ hist, int u,
                                              int v, Accept accept, uint32_t* err, int* dE_out) {
  constexpr int kT = kSlotsPerLane;
  static_assert(kWords * 4 >= kDirCount, "a byte per direction");
  const int ru = u >> 1, rv = v >> 1, cu = cs[u], cv = cs[v];
  const int centre[4] = {ru * kLutW + cv, rv * kLutW + cu, ru * kLutW + cu, rv * kLutW + cv};  // u', v', u, v
  int t_sum[4], change[kT], line_count[4] = {0, 0, 0, 0};
  int joint = 0;
  for (int t = 0; t < kT; ++t) {
    change[t] = 0;
    const int k = lane + 32 * t;
    if (k < m && k != u && k != v) joint += (rv - ru) * (cs[k] - cu) == (cv - cu) * ((k >> 1) - ru);
  }
  joint = warp_sum(joint);
  for (int c = 0; c < 4; ++c) {
    // the direction of the other moved point, for u' and u
    const int line = (c & 1) ? -1 : (int)(dir4(lut4, centre[c + 1], centre[c]) >> 2);
    int part = 0;
    for (int pass = 0; pass < 3; ++pass) {  // add, read, clear
      for (int t = 0; t < kT; ++t) {
        const int k = lane + 32 * t;
        if (k >= m || k == u || k == v) continue;
        const int id = (int)(dir4(lut4, (k >> 1) * kLutW + cs[k], centre[c]) >> 2);
        if (pass == 0) part += hist_add(hist, id);
        if (pass == 1) change[t] += (c < 2 ? 1 : -1) * (hist_get(hist, id) - 1 + (id == line));
        if (pass == 2) hist_clear(hist, id);
      }
      __syncwarp();
      if (pass == 0) {
        t_sum[c] = warp_sum(part);
        if (line >= 0) line_count[c] = hist_get(hist, line);
      }
      if (pass == 1) __syncwarp();
    }
  }
  const int dE = (t_sum[0] + t_sum[1] + line_count[0]) - (bs[u] + bs[v] - joint);
  *dE_out = dE;
  if (!accept(dE)) return false;
  if (bs[u] != t_sum[2] + line_count[2] || bs[v] != t_sum[3] + line_count[2] || line_count[2] != joint)
    *err |= kErrAudit;
  __syncwarp();
  for (int t = 0; t < kT; ++t) {
    const int k = lane + 32 * t;
    if (k < m && k != u && k != v) bs[k] += change[t];
  }
  if (lane == 0) {
    bs[u] = t_sum[0] + line_count[0];
    bs[v] = t_sum[1] + line_count[0];
    cs[u] = (uint8_t)cv;
    cs[v] = (uint8_t)cu;
  }
  __syncwarp();
  return true;
}

template <int kWords, class Accept>
__device__ __forceinline__ bool call_slow_move(WarpState& W, const uint16_t* __restrict__ lut4,
                                               uint32_t* __restrict__ hist, int u, int v, Accept accept, int& E,
                                               uint32_t& err, int* dE_out) {
  const int dc = (int)W.cs[v] - (int)W.cs[u];
  uint32_t e = 0u;  // copies, so that only they live in memory
  int dE = 0;
  const bool accepted = slow_move<kWords>(W.m, W.lane, W.cs, W.bs, lut4, hist, u, v, accept, &e, &dE);
  err |= e;
  *dE_out = dE;
  if (!accepted) return false;
  W.swap_keys(u, v, dc);
  E += dE;
  return true;
}

// What the histograms around the new centres u' = (r_u, c_v) and v' = (r_v, c_u)
// tell about the swap of slots u and v in different rows and columns.
struct PairCount {
  int ta, tb;    // t(u'), t(v') over A
  int j_new;     // points of A on the line (u', v')
  int joint;     // points of A on the line (u, v) (JOINT)
  bool wide;     // a counter may have wrapped: the rest is not to be used
};

// Counts them into hist (two zero histograms of Num::kWords words each) and leaves
// the centres' directions in a and b: the caller clears those words.
template <class Num, int NT, bool JOINT = true>
__device__ __forceinline__ PairCount count_pair(const WarpState& W, const uint16_t* __restrict__ lut4,
                                                uint32_t* __restrict__ hist, int ru, int rv, int cu, int cv,
                                                Directions& a, Directions& b, uint32_t& line_new) {
  uint32_t* const h0 = hist;
  uint32_t* const h1 = hist + Num::kWords;
  const int kA = 2 * (ru * kLutW + cv), kB = 2 * (rv * kLutW + cu);  // u', v'
  line_new = dir4_2(lut4, kB, kA);
  find_centre<Num, NT>(W, lut4, h0, kA, a);
  find_centre<Num, NT>(W, lut4, h1, kB, b);
  // pair sums in 12 bits each, the points on the line (u, v), both included, in the top byte
  uint32_t part = count_centres<NT>(W, a, b);
  if (JOINT) part += (uint32_t)W.on_line<NT>(ru, cu, rv - ru, cv - cu) << 24;
  __syncwarp();
  PairCount p;
  p.j_new = (int)counter_of(h0, line_new);
  const int xa = (int)counter_of(h0, Num::kCol), xb = (int)counter_of(h1, Num::kCol);
  const uint32_t sums = __reduce_add_sync(0xffffffffu, part);
  const int sa = (int)(sums & 0xFFFu), sb = (int)((sums >> 12) & 0xFFFu);
  p.ta = sa - xa;
  p.tb = sb - xb;
  p.joint = (int)(sums >> 24) - 2;
  p.wide = sa >= kMoveSum || sb >= kMoveSum;
  return p;
}

// One legal move, prepared as `mv` on the current state.  lut4: Num's table; hist:
// two histograms of Num::kWords words each, zero, left zero.  NT = ceil(m / 32).
// accept(dE) as in slow_move.
template <class Num, int NT, class Accept>
__device__ __forceinline__ bool pair_move(WarpState& W, const uint16_t* __restrict__ lut4,
                                          uint32_t* __restrict__ hist, PreparedMove mv, Accept accept, int& E,
                                          uint32_t& err, int* dE_out) {
  constexpr uint32_t e_row = Num::kRow, e_col = Num::kCol;
  uint32_t* const h0 = hist;
  uint32_t* const h1 = hist + Num::kWords;
  const int u = (int)(mv.slots & 0xFFu), v = (int)((mv.slots >> 8) & 0xFFu);
  const int cu = (int)((mv.slots >> 16) & 0xFFu), cv = (int)(mv.slots >> 24);
  const int ru = u >> 1, rv = v >> 1, dc = cv - cu;
  Directions a, b;
  uint32_t line_new;
  const PairCount p = count_pair<Num, NT>(W, lut4, hist, ru, rv, cu, cv, a, b, line_new);
  const int dE = p.ta + p.tb + p.j_new + p.joint - mv.bad;
  *dE_out = dE;
  if (p.wide || !accept(dE)) {  // uniform
    __syncwarp();
    clear_centre<NT>(a);
    clear_centre<NT>(b);
    __syncwarp();
    return p.wide ? call_slow_move<2 * Num::kWords>(W, lut4, hist, u, v, accept, E, err, dE_out) : false;
  }
  // every other point's badness change: the points it shares a line through u' and v' with, less
  // those through u and v.  At the new centres u or v is counted too for a point of their row or
  // column; the other moved point counts for one of two centres only.
  int change[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t)
    change[t] = centre_get(a, t) + centre_get(b, t) - (a.e[t] == e_row || a.e[t] == e_col) -
                (b.e[t] == e_row || b.e[t] == e_col) + (a.e[t] == line_new);
  __syncwarp();
  clear_centre<NT>(a);
  clear_centre<NT>(b);
  const int kU = 2 * (ru * kLutW + cu), kV = 2 * (rv * kLutW + cv);
  const uint32_t line_old = dir4_2(lut4, kV, kU);
  find_centre<Num, NT>(W, lut4, h0, kU, a);
  find_centre<Num, NT>(W, lut4, h1, kV, b);
  __syncwarp();
  const uint32_t old_part = count_centres<NT>(W, a, b);
  __syncwarp();
  const int jo = (int)counter_of(h0, line_old) - 1;
#pragma unroll
  for (int t = 0; t < NT; ++t) change[t] -= centre_get(a, t) + centre_get(b, t) - (b.e[t] == line_old);
  const uint32_t old_sums = __reduce_add_sync(0xffffffffu, old_part);
  const int tc = (int)(old_sums & 0xFFFu), td = (int)(old_sums >> 12);
  __syncwarp();
  clear_centre<NT>(a);
  clear_centre<NT>(b);
  if (tc >= kMoveSum || td >= kMoveSum) {  // uniform
    __syncwarp();
    return call_slow_move<2 * Num::kWords>(W, lut4, hist, u, v, accept, E, err, dE_out);
  }
  if (mv.bad != tc + td || jo != p.joint) err |= kErrAudit;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int k = W.slot(t);
    if (t < NT - 1 || k < W.m) W.bs[k] += change[t];
  }
  W.swap_keys(u, v, dc);
  __syncwarp();
  if (W.lane == 0) {
    W.bs[u] = p.ta + p.j_new;
    W.bs[v] = p.tb + p.j_new;
    W.cs[u] = (uint8_t)cv;
    W.cs[v] = (uint8_t)cu;
  }
  __syncwarp();
  E += dE;
  return true;
}

// pair_move for any m: nt = ceil(m / 32).
template <class Num, class Accept>
__device__ __forceinline__ bool pair_move_any(WarpState& W, const uint16_t* __restrict__ lut4,
                                              uint32_t* __restrict__ hist, int nt, PreparedMove mv, Accept accept,
                                              int& E, uint32_t& err, int* dE_out) {
  switch (nt) {
    case 5: return pair_move<Num, 5>(W, lut4, hist, mv, accept, E, err, dE_out);
    case 4: return pair_move<Num, 4>(W, lut4, hist, mv, accept, E, err, dE_out);
    case 3: return pair_move<Num, 3>(W, lut4, hist, mv, accept, E, err, dE_out);
    case 2: return pair_move<Num, 2>(W, lut4, hist, mv, accept, E, err, dE_out);
    default: return pair_move<Num, 1>(W, lut4, hist, mv, accept, E, err, dE_out);
  }
}

// A move prepared by the whole warp, and the legality rule (tempering.py:58).
__device__ __forceinline__ PreparedMove prepare_move(const WarpState& W, int u, int v) {
  return PreparedMove{(uint32_t)u | ((uint32_t)v << 8) | ((uint32_t)W.cs[u] << 16) | ((uint32_t)W.cs[v] << 24),
                      W.bs[u] + W.bs[v]};
}
__device__ __forceinline__ bool legal_swap(const uint8_t* cs, int u, int v) {
  const int cu = cs[u], cv = cs[v];
  return (u >> 1) != (v >> 1) && cu != cv && cs[u ^ 1] != cv && cs[v ^ 1] != cu;
}

}  // namespace n3
