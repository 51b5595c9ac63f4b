// Cover table of a state: T[cell] = pairs of points of S \ {cell} whose line
// runs through the cell, rows and columns of the grid left out, for every cell
// of the n x n grid.
//
// It makes the dE of a swap of a row/column 2-factor a matter of four loads.
// u' = (r_u, c_v) shares its row with u and its column with v, so no pair that
// holds u or v and no row or column counts at u': t(u') over A = S \ {u, v} is
// T[u'], and likewise t(v') = T[v'].  The badness of u is T[u].  With j, j' the
// points of A on the lines (u, v) and (u', v'):
//   dE = T[u'] + T[v'] - T[u] - T[v] + j + j'
// and as j, j' >= 0 the four loads alone reject most moves of a cold chain
// exactly (column multiplicities other than 2 would cancel in dE too, but not
// in the badness).  An accepted move changes T by the lines from u and v (minus
// one per cell) and from u' and v' (plus one) to every other point: 4 x 148
// lines of 4.6 cells on average, half of them of one.
#pragma once

#include "dirs.cuh"
#include "n3_common.cuh"
#include "pair_move.cuh"

namespace n3 {

// Adds `delta` to every cell of the line through (rx, cx) and (rk, ck) except
// those two, for each lane with `valid` set (nothing for points of one row or
// one column).  rx, cx, delta uniform; all lanes call it.  T: two 16-bit entries a
// word (no entry exceeds C(149, 2)).  prim4: four times the primitive step's key
// a * kLutW + b.  recip[a] = ceil(65536 / a), so x * recip[a] >> 16 is x / a for
// x < kMaxN.  scratch: the warp's 32 uint2 of shared memory.
//
// The lines of 32 points have 4.6 cells each on average but 40 in the longest,
// so a lane per line would leave most lanes waiting.  Instead the cells of all
// lines are numbered through and taken 32 at a time: each line's start sets a bit
// of the chunk's word, so the bits up to a lane's number tell its line.
static __device__ __noinline__ void cover_line(uint32_t* __restrict__ T, int n, int rx, int cx, int rk, int ck,
                                               int delta, bool valid, const uint16_t* __restrict__ prim4,
                                               const uint32_t* __restrict__ recip, uint2* __restrict__ scratch,
                                               int lane) {
  const int key = (int)(dir4(prim4, rk * kLutW + ck, rx * kLutW + cx) >> 2);
  int a = (key + kMaxN - 1) / kLutW, b = key - a * kLutW;
  valid = valid && a != 0 && b != 0;
  if (!valid) a = b = 1;
  const uint32_t ia = recip[a], ib = recip[abs(b)];
  const int right = n - 1 - cx, down = n - 1 - rx;
  // steps of (a, b) that stay on the grid from (rx, cx), forward and back, and those to (rk, ck)
  const int fwd = min((int)((uint32_t)down * ia >> 16), (int)((uint32_t)(b > 0 ? right : cx) * ib >> 16));
  const int back = min((int)((uint32_t)rx * ia >> 16), (int)((uint32_t)(b > 0 ? cx : right) * ib >> 16));
  const int apart = (int)((uint32_t)abs(rk - rx) * ia >> 16);
  const int step = a * n + b, first = rx * n + cx - back * step;
  const int at_x = back, at_k = rk > rx ? back + apart : back - apart;  // positions of the two points on the line
  const int cells = valid ? fwd + back - 1 : 0;                         // without the two
  // number the cells: offset of this line's first, and the line's place among those that have any
  int offset = cells;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, offset, o);
    if (lane >= o) offset += y;
  }
  const int total = __shfl_sync(0xffffffffu, offset, 31);
  offset -= cells;
  const unsigned some = __ballot_sync(0xffffffffu, cells > 0);
  __syncwarp();
  if (cells > 0)
    scratch[__popc(some & ((1u << lane) - 1u))] =
        make_uint2((uint32_t)first | ((uint32_t)min(at_x, at_k) << 16) | ((uint32_t)max(at_x, at_k) << 23),
                   (uint32_t)step | ((uint32_t)offset << 16));
  __syncwarp();
  int line = -1;  // lines begun before the chunk, less one
#pragma unroll 2
  for (int base = 0; base < total; base += 32) {
    const unsigned in_chunk = (unsigned)(offset - base);
    const unsigned starts = __reduce_or_sync(0xffffffffu, cells > 0 && in_chunk < 32u ? 1u << in_chunk : 0u);
    const int i = base + lane;
    if (i < total) {
      const uint2 d = scratch[line + __popc(starts & (0xffffffffu >> (31 - lane)))];
      int s = i - (int)(d.y >> 16);
      s += s >= (int)((d.x >> 16) & 127u);
      s += s >= (int)(d.x >> 23);
      const int cell = (int)(d.x & 0xFFFFu) + s * (int)(d.y & 0xFFFFu);
      atomicAdd(T + (cell >> 1), (uint32_t)delta << ((cell & 1) * 16));
    }
    line += __popc(starts);
  }
}

__device__ __forceinline__ int cover_get(const uint32_t* __restrict__ T, int cell) {
  return reinterpret_cast<const uint16_t*>(T)[cell];
}

// The pairs of slots part, part + parts, ... with the later ones, into T of the
// state in cs (`parts` warps build zeroed T together).
static __device__ __noinline__ void cover_build(const uint8_t* __restrict__ cs, uint32_t* __restrict__ T, int n,
                                                const uint16_t* __restrict__ prim4,
                                                const uint32_t* __restrict__ recip, uint2* __restrict__ scratch,
                                                int lane, int part = 0, int parts = 1) {
  const int m = 2 * n;
  for (int i = part; i + 1 < m; i += parts) {
    const int ri = i >> 1, ci = cs[i];
    for (int k0 = (i | 1) + 1; k0 < m; k0 += 32) {  // the slots after i's row
      const int k = k0 + lane;
      const bool in = k < m;
      cover_line(T, n, ri, ci, in ? k >> 1 : ri, in ? (int)cs[k] : ci, 1, in, prim4, recip, scratch, lane);
    }
  }
}

// The changes of T for the swap of slots u and v (the columns are the caller's to change).
static __device__ __noinline__ void cover_swap(const uint8_t* __restrict__ cs, uint32_t* __restrict__ T, int n, int u, int v,
                                               const uint16_t* __restrict__ prim4,
                                               const uint32_t* __restrict__ recip, uint2* __restrict__ scratch,
                                               int lane) {
  const int m = 2 * n, ru = u >> 1, rv = v >> 1, cu = cs[u], cv = cs[v];
  for (int c = 0; c < 4; ++c) {  // from u, v (removed), u', v' (added)
    const int rx = (c & 1) ? rv : ru, cx = c == 0 || c == 3 ? cu : cv;
    const int other = (c & 1) ? -1 : (c == 0 ? cv : cu);  // v's column as seen from u, v' from u'
    for (int k0 = 0; k0 < m; k0 += 32) {
      const int k = k0 + lane;
      bool in = k < m && k != u;
      int ck = in ? (int)cs[k] : 0;
      if (k == v) {
        in = other >= 0;
        ck = max(other, 0);
      }
      cover_line(T, n, rx, cx, in ? k >> 1 : rx, in ? ck : cx, c < 2 ? -1 : 1, in, prim4, recip, scratch, lane);
    }
  }
}

// Points of the state on each lane's line through (r0, c0) and (r1, c1), those two
// cells left out; 0 for lanes without `valid` and for cells of one row or column.  bits:
// a bit per cell, number row * n + column.  The cells are numbered through as in
// cover_line; a cell in 40 holds a point, which adds to its line's counter.  scratch:
// the warp's 32 uint2; count: its 32 words.  All lanes call it.
static __device__ __noinline__ int count_lines(const uint32_t* __restrict__ bits, int n, int r0, int c0, int r1, int c1,
                                               bool valid, const uint16_t* __restrict__ prim4,
                                               const uint32_t* __restrict__ recip, uint2* __restrict__ scratch,
                                               uint32_t* __restrict__ count, int lane) {
  const int key = (int)(dir4(prim4, r1 * kLutW + c1, r0 * kLutW + c0) >> 2);
  int a = (key + kMaxN - 1) / kLutW, b = key - a * kLutW;
  valid = valid && a != 0 && b != 0;
  if (!valid) a = b = 1;
  const uint32_t ia = recip[a], ib = recip[abs(b)];
  const int right = n - 1 - c0, down = n - 1 - r0;
  const int fwd = min((int)((uint32_t)down * ia >> 16), (int)((uint32_t)(b > 0 ? right : c0) * ib >> 16));
  const int back = min((int)((uint32_t)r0 * ia >> 16), (int)((uint32_t)(b > 0 ? c0 : right) * ib >> 16));
  const int apart = (int)((uint32_t)abs(r1 - r0) * ia >> 16);
  const int step = a * n + b, first = r0 * n + c0 - back * step;
  const int at_0 = back, at_1 = r1 > r0 ? back + apart : back - apart;
  const int cells = valid ? fwd + back - 1 : 0;
  int offset = cells;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, offset, o);
    if (lane >= o) offset += y;
  }
  const int total = __shfl_sync(0xffffffffu, offset, 31);
  offset -= cells;
  const unsigned some = __ballot_sync(0xffffffffu, cells > 0);
  const int mine = __popc(some & ((1u << lane) - 1u));
  __syncwarp();
  count[lane] = 0u;
  if (cells > 0)
    scratch[mine] = make_uint2((uint32_t)first | ((uint32_t)min(at_0, at_1) << 16) | ((uint32_t)max(at_0, at_1) << 23),
                               (uint32_t)step | ((uint32_t)offset << 16));
  __syncwarp();
  int line = -1;  // lines begun before the chunk, less one
#pragma unroll 2
  for (int base = 0; base < total; base += 32) {
    const unsigned in_chunk = (unsigned)(offset - base);
    const unsigned starts = __reduce_or_sync(0xffffffffu, cells > 0 && in_chunk < 32u ? 1u << in_chunk : 0u);
    const int i = base + lane;
    if (i < total) {
      const int at = line + __popc(starts & (0xffffffffu >> (31 - lane)));
      const uint2 d = scratch[at];
      int s = i - (int)(d.y >> 16);
      s += s >= (int)((d.x >> 16) & 127u);
      s += s >= (int)(d.x >> 23);
      const int cell = (int)(d.x & 0xFFFFu) + s * (int)(d.y & 0xFFFFu);
      if ((bits[cell >> 5] >> (cell & 31)) & 1u) atomicAdd(count + at, 1u);
    }
    line += __popc(starts);
  }
  __syncwarp();
  return cells > 0 ? (int)count[mine] : 0;
}

// Occupancy of the grid: three words a row, bit c & 31 of word c >> 5 for column c.
constexpr int kOccWords = 3 * kMaxN;

// Points of the state on the line through (r0, c0) and (r1, c1), the cell
// (r0, c0) left out; 0 if the two share a row or a column.
__device__ __forceinline__ int points_on_line(const uint32_t* __restrict__ occ, int n,
                                              const uint16_t* __restrict__ prim4, int r0, int c0, int r1, int c1) {
  if (r0 == r1 || c0 == c1) return 0;
  const int key = (int)(dir4(prim4, r1 * kLutW + c1, r0 * kLutW + c0) >> 2);
  const int a = (key + kMaxN - 1) / kLutW, b = key - a * kLutW;
  int count = 0;
  for (int r = r0 + a, c = c0 + b; r < n && (unsigned)c < (unsigned)n; r += a, c += b)
    count += (occ[3 * r + (c >> 5)] >> (c & 31)) & 1u;
  for (int r = r0 - a, c = c0 - b; r >= 0 && (unsigned)c < (unsigned)n; r -= a, c -= b)
    count += (occ[3 * r + (c >> 5)] >> (c & 31)) & 1u;
  return count;
}

}  // namespace n3
