// Device bodies of the two population scorers, shared by score.cu (the
// scoring entry points) and tempering.cu (the on-device energy audit).
// See score.cu for the method.
#pragma once

#include "dirs.cuh"
#include "n3_common.cuh"

namespace n3 {

// Tests of the two pivots of row `rho` against all pairs (x, y) with x on the
// larger side (R register slots per lane) and y on the smaller side.
// X=(r_x,c_x), J=(rho,c_j), Y=(r_y,c_y) are collinear iff
//   (r_x-rho)(c_y-c_j) == (c_x-c_j)(r_y-rho)
//   <=>  a_x*c_y == a_y*b_x + a_x*c_j,   a = r - rho, b_x = c_x - c_j.
template <int R, bool BAD>
__device__ __forceinline__ int det_pivot_row(const int* __restrict__ cs, int n, int rho, int lane, int* bad) {
  const int cj0 = cs[2 * rho], cj1 = cs[2 * rho + 1];
  const int above = rho, below = n - 1 - rho;
  const bool lanes_above = above >= below;
  const int L = 2 * (lanes_above ? above : below);
  const int lbase = lanes_above ? 0 : 2 * rho + 2;
  const int rb0 = lanes_above ? rho + 1 : 0;
  const int rb1 = lanes_above ? n : rho;
  int ax[R], bx0[R], bx1[R], k0[R], k1[R], sx[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int x = lane + 32 * r;
    if (x < L) {
      const int s = lbase + x;
      const int a = (s >> 1) - rho, c = cs[s];
      ax[r] = a;
      bx0[r] = c - cj0;
      bx1[r] = c - cj1;
      k0[r] = a * cj0;
      k1[r] = a * cj1;
      sx[r] = s;
    } else {  // idle slot: products are 0, targets -1, never a hit
      ax[r] = 0;
      bx0[r] = 0;
      bx1[r] = 0;
      k0[r] = -1;
      k1[r] = -1;
      sx[r] = 0;
    }
  }
  int cnt = 0;
  const int2* rows2 = reinterpret_cast<const int2*>(cs);
  // Each target T (one per pivot) matches at most one of the row's two
  // products: P0 == P1 needs a_x == 0 (a lane slot always has a_x != 0; an
  // idle slot has target -1).  So every target contributes one OR of two
  // compares, and the count needs no per-test conversion.  Two hits of one
  // register slot in one row do occur (two lines through x, one per pivot).
#pragma unroll 2
  for (int row = rb0; row < rb1; ++row) {
    const int2 cy = rows2[row];
    const int ay = row - rho;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int P0 = ax[r] * cy.x, P1 = ax[r] * cy.y;
      const int T0 = ay * bx0[r] + k0[r], T1 = ay * bx1[r] + k1[r];
      const bool g0 = (P0 == T0) | (P1 == T0), g1 = (P0 == T1) | (P1 == T1);
      cnt += (int)g0 + (int)g1;
      if (BAD && (g0 | g1)) {
        if (g0) {  // x, pivot 2 rho, and slot 2 row or 2 row + 1
          atomicAdd(bad + sx[r], 1);
          atomicAdd(bad + 2 * rho, 1);
          atomicAdd(bad + 2 * row + (P0 == T0 ? 0 : 1), 1);
        }
        if (g1) {
          atomicAdd(bad + sx[r], 1);
          atomicAdd(bad + 2 * rho + 1, 1);
          atomicAdd(bad + 2 * row + (P0 == T1 ? 0 : 1), 1);
        }
      }
    }
  }
  return cnt;
}

// The same tests on packed float pairs, for columns in [0, kMaxN) (every value
// below stays under 2^14 in magnitude, so float arithmetic is exact; a product
// of two non-zero differences is at least 1, so it is zero iff one of them is).
// Per register slot and row y: the targets of the two pivots advance by one
// packed add, two packed multiply-adds give the four differences
// a_x c_y - T (pivot 0 in the low half, pivot 1 in the high half), and one
// packed multiply joins the row's two points, which hit at most one of them
// (see above), so two compares and two adds count four tests: eight
// instructions, four on the multiply-add pipe (two results each) and four on
// the ALU pipe, against 12 with 32-bit integer multiplies and compares
// (integer multiply-adds run at half the float rate).
// rows4[row] = (c, c, c', c') of the row's two points.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// One compare and one predicated add (from the plain expression the compiler
// makes a select as well).
__device__ __forceinline__ void count_zero(int& cnt, float x) {
  asm("{\n\t.reg .pred p;\n\tsetp.eq.f32 p, %1, 0f00000000;\n\t@p add.s32 %0, %0, 1;\n\t}" : "+r"(cnt) : "f"(x));
}

template <int R, bool BAD>
__device__ __forceinline__ int det_pivot_row_f(const float4* __restrict__ rows4, int n, int rho, int lane,
                                               int* __restrict__ bad) {
  const float cj0 = rows4[rho].x, cj1 = rows4[rho].z;
  const int above = rho, below = n - 1 - rho;
  const bool lanes_above = above >= below;
  const int L = 2 * (lanes_above ? above : below);
  const int lbase = lanes_above ? 0 : 2 * rho + 2;
  const int rb0 = lanes_above ? rho + 1 : 0;
  const int rb1 = lanes_above ? n : rho;
  uint64_t ax[R], nb[R], nt[R];  // (a, a), (-b0, -b1), (-T0, -T1) of the current row
  const float ay0 = (float)(rb0 - rho);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int x = lane + 32 * r;
    if (x < L) {
      const int s = lbase + x;
      const float4 v = rows4[s >> 1];
      const float c = (s & 1) ? v.z : v.x, a = (float)((s >> 1) - rho);
      const float b0 = c - cj0, b1 = c - cj1;
      ax[r] = pack2(a, a);
      nb[r] = pack2(-b0, -b1);
      nt[r] = pack2(-(ay0 * b0 + a * cj0), -(ay0 * b1 + a * cj1));
    } else {  // idle slot: every difference is 1, never a hit
      ax[r] = 0ull;
      nb[r] = 0ull;
      nt[r] = pack2(1.f, 1.f);
    }
  }
  int cnt = 0, cnt1 = 0;
  const ulonglong2* rows2 = reinterpret_cast<const ulonglong2*>(rows4);
#pragma unroll 4
  for (int row = rb0; row < rb1; ++row) {
    const ulonglong2 cy = rows2[row];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint64_t d0 = fma2(ax[r], cy.x, nt[r]), p = mul2(d0, fma2(ax[r], cy.y, nt[r]));
      float p0, p1;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(p));
      if (BAD && (p0 == 0.f || p1 == 0.f)) {  // x, the pivot, and slot 2 row or 2 row + 1
        float e0, e1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(e0), "=f"(e1) : "l"(d0));
        if (p0 == 0.f) {
          atomicAdd(bad + lbase + lane + 32 * r, 1);
          atomicAdd(bad + 2 * rho, 1);
          atomicAdd(bad + 2 * row + (e0 == 0.f ? 0 : 1), 1);
        }
        if (p1 == 0.f) {
          atomicAdd(bad + lbase + lane + 32 * r, 1);
          atomicAdd(bad + 2 * rho + 1, 1);
          atomicAdd(bad + 2 * row + (e1 == 0.f ? 0 : 1), 1);
        }
      }
      count_zero(cnt, p0);
      count_zero(cnt1, p1);
      nt[r] = add2(nt[r], nb[r]);
    }
  }
  return cnt + cnt1;
}

// E's share of this lane from the pivot rows 1 + part, 1 + part + parts, ...;
// rows4 in shared memory, columns in [0, kMaxN).  BAD: bad[s] (shared memory,
// zeroed) receives the number of triples holding slot s.
template <bool BAD>
__device__ __forceinline__ int det_state_f(const float4* __restrict__ rows4, int n, int lane, int part, int parts,
                                           int* __restrict__ bad) {
  int cnt = 0;
  for (int rho = 1 + part; rho < n - 1; rho += parts) {
    const int L = 2 * max(rho, n - 1 - rho);
    switch ((L + 31) >> 5) {
      case 1: cnt += det_pivot_row_f<1, BAD>(rows4, n, rho, lane, bad); break;
      case 2: cnt += det_pivot_row_f<2, BAD>(rows4, n, rho, lane, bad); break;
      case 3: cnt += det_pivot_row_f<3, BAD>(rows4, n, rho, lane, bad); break;
      case 4: cnt += det_pivot_row_f<4, BAD>(rows4, n, rho, lane, bad); break;
      default: cnt += det_pivot_row_f<5, BAD>(rows4, n, rho, lane, bad); break;
    }
  }
  return cnt;
}

template <bool BAD>
__device__ __forceinline__ int det_state(const int* __restrict__ cs, int n, int lane, int* bad) {
  int cnt = 0;
  for (int rho = 1; rho < n - 1; ++rho) {
    const int L = 2 * max(rho, n - 1 - rho);
    switch ((L + 31) >> 5) {
      case 1: cnt += det_pivot_row<1, BAD>(cs, n, rho, lane, bad); break;
      case 2: cnt += det_pivot_row<2, BAD>(cs, n, rho, lane, bad); break;
      case 3: cnt += det_pivot_row<3, BAD>(cs, n, rho, lane, bad); break;
      case 4: cnt += det_pivot_row<4, BAD>(cs, n, rho, lane, bad); break;
      default: cnt += det_pivot_row<5, BAD>(cs, n, rho, lane, bad); break;
    }
  }
  return cnt;
}

// Error bits of a state whose counts are to agree: the determinants' E, the slope
// side's E and, if the slope side gave badness, its sum, which holds every triple
// three times (the badness is added up beside E, so E alone would not show a slip in it).
__host__ __device__ inline uint32_t checked_error(int det, int slope, bool has_badness, int badness_sum) {
  return det == slope && (!has_badness || badness_sum == 3 * det) ? 0u : kErrMismatch;
}

// Normalised-slope line count of one state by tags: E for the whole warp.
//
// From each centre a, in slot order, the later slots k of other rows are told
// apart by the gcd-reduced direction of k - a, so every collinear triple is
// found once, from its first slot.  Each k writes its slot number into the tag
// byte of its direction and reads it back: the last writer of a direction (the
// winner) reads itself, every other slot of the direction (a loser) reads the
// winner.  A few of the 148 slots lose, so most centres cost a load of the
// direction, a store and a load per slot; nothing is counted or cleared for a
// slot alone in its direction, and a slot only reads bytes that its own
// direction wrote at this centre.  The losers then count themselves in the top
// byte of their winner's word: a direction of c slots has c - 1 losers, which
// find 0, 1, ... there and add 1 + 2 + ... = C(c, 2) triples.
//
// NT: the slots a lane may hold, at least ceil(m / 32).
// key: this lane's slots' table keys row * kLutW + column, negative beyond m.
// lut: the compact direction table in shared memory, whose entry of the
// difference d = key(k) - key(a) > 0 is lut[d + kMaxN - 1].  tag: this warp's
// kDirCount bytes, any contents.  word[s] (shared memory, zeroed): with BAD, the
// number of triples holding slot s on return (at most C(149, 2), below 2^24).
constexpr size_t kTagWarpBytes = kDirCount + sizeof(uint32_t) * kMaxM;  // the tags, then word[]

// SPLIT: only the centres part, part + parts, ... are counted (parts a power of
// two up to 32), so that `parts` warps can share a state.  Each then counts its
// losers in words of its own, and the badness of all goes to `bad`, the first
// warp's (only that warp touches a top byte there).
template <bool BAD, bool SPLIT = false, int NT = kSlotsPerLane>
__device__ __forceinline__ int tag_state(const int (&key)[NT], int m, const uint16_t* __restrict__ lut,
                                         uint8_t* __restrict__ tag, int lane, uint32_t* word, uint32_t* bad,
                                         int part = 0, int parts = 1) {
  constexpr int kT = NT;
  constexpr uint32_t kOne = 1u << 24;
  volatile uint8_t* vtag = tag;
  int total = 0;  // this lane's triples
#pragma unroll
  for (int ta = 0; ta < kT; ++ta) {
    const int la_end = min(32, m - 32 * ta);  // centres 32 ta + la
    for (int la = SPLIT ? part : 0; la < la_end; la += SPLIT ? parts : 1) {
      const int ka = __shfl_sync(0xffffffffu, key[ta], la);
      const uint16_t* base = lut + (kMaxN - 1) - ka;
      int id[kT];
      unsigned lose = 0u;
#pragma unroll
      for (int t = ta; t < kT; ++t) {
        const bool in = key[t] >= 0 && (t > ta || lane > (la | 1));
        id[t] = in ? (int)base[key[t]] : -1;
        if (in) vtag[id[t]] = (uint8_t)(lane + 32 * t);
      }
      __syncwarp();
      int win[kT];
#pragma unroll
      for (int t = ta; t < kT; ++t) {
        win[t] = lane + 32 * t;
        if (id[t] >= 0) win[t] = vtag[id[t]];
        lose |= (unsigned)(win[t] != lane + 32 * t) << t;
      }
      __syncwarp();  // the next centre's tags come after every lane has read this one's
      if (__any_sync(0xffffffffu, lose != 0u)) {
        uint32_t before[kT];
#pragma unroll
        for (int t = ta; t < kT; ++t)
          if ((lose >> t) & 1u) {
            before[t] = atomicAdd(word + win[t], kOne) >> 24;
            total += (int)before[t] + 1;
          }
        __syncwarp();
        if (BAD) {
          uint32_t others[kT];  // the other slots of the direction
#pragma unroll
          for (int t = ta; t < kT; ++t)
            if ((lose >> t) & 1u) others[t] = *(volatile uint32_t*)(word + win[t]) >> 24;
          __syncwarp();
#pragma unroll
          for (int t = ta; t < kT; ++t)
            if ((lose >> t) & 1u) {
              if (before[t] == 0u) {  // the first loser speaks for the winner
                if (SPLIT && word != bad) {  // uniform
                  word[win[t]] = 0u;
                  atomicAdd(bad + win[t], others[t]);
                } else {
                  atomicAdd(word + win[t], others[t] - others[t] * kOne);
                }
              }
              atomicAdd(bad + lane + 32 * t, others[t]);
              atomicAdd(bad + 32 * ta + la, before[t] + 1u);
            }
        } else {
#pragma unroll
          for (int t = ta; t < kT; ++t)
            if ((lose >> t) & 1u) word[win[t]] = 0u;
        }
      }
    }
  }
  return warp_sum(total);
}

}  // namespace n3
