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
#include "cover.cuh"
#include "dirs.cuh"
#include "n3_common.cuh"

namespace n3 {

// Exact dE (and, if dbad != nullptr, this lane's badness changes for slots
// lane + 32 t, plus the moved slots' changes in *dbad_u, *dbad_v) of a legal
// move.  Uses the 4 centres u, v, u', v'; hist must be zeroed, is left zeroed.
// lutf: the full signed direction table; key: this lane's slots' table keys
// row * kLutW + column.
template <bool BAD>
__device__ __forceinline__ int swap_delta_hist(const int* __restrict__ cs, const int (&key)[kSlotsPerLane], int m,
                                               int u, int v, const uint16_t* __restrict__ lutf,
                                               uint32_t* __restrict__ hist, int lane, int (&dbad)[kSlotsPerLane],
                                               int* dbad_u, int* dbad_v) {
  const int ru = u >> 1, rv = v >> 1, cu = cs[u], cv = cs[v];
  // centre order: u, v, u', v'
  const int crow[4] = {ru, rv, ru, rv};
  const int ccol[4] = {cu, cv, cv, cu};
  int tX[4];
  int j_old = 0, j_new = 0;
  if (BAD) {
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) dbad[t] = 0;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    int ids[kSlotsPerLane];
    int part = 0;
    {
      const int rx = crow[c];
      const uint16_t* base = lutf + kFullLutCentre - (rx * kLutW + ccol[c]);
#pragma unroll
      for (int t = 0; t < kSlotsPerLane; ++t) {
        const int k = lane + 32 * t;
        ids[t] = -1;
        if (k < m && k != u && k != v && (k >> 1) != rx) {
          const int id = base[key[t]];
          ids[t] = id;
          part += hist_add(hist, id);
        }
      }
    }
    __syncwarp();
    tX[c] = warp_sum(part);
    const int sign = c < 2 ? -1 : 1;
    int line_id = -1;  // direction of the other moved point, for centres u and u'
    if (c == 0) {
      line_id = dir_id_full(lutf, rv - ru, cv - cu);
      j_old = hist_get(hist, line_id);
    } else if (c == 2) {
      line_id = dir_id_full(lutf, rv - ru, cu - cv);
      j_new = hist_get(hist, line_id);
    }
    if (BAD) {
#pragma unroll
      for (int t = 0; t < kSlotsPerLane; ++t) {
        if (ids[t] >= 0) dbad[t] += sign * (hist_get(hist, ids[t]) - 1 + (ids[t] == line_id));
      }
    }
    __syncwarp();
    hist_release(hist, ids);
    __syncwarp();
  }
  if (BAD) {
    *dbad_u = (tX[2] + j_new) - (tX[0] + j_old);
    *dbad_v = (tX[3] + j_new) - (tX[1] + j_old);
  }
  return (tX[2] + tX[3] + j_new) - (tX[0] + tX[1] + j_old);
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

constexpr int kDeltaWarps = 8;

struct DeltaSmem {
  static constexpr size_t lut_bytes = kFullLutBytes;  // the full signed direction table
  static constexpr size_t bytes =
      lut_bytes + sizeof(uint32_t) * kDirWords * kDeltaWarps + sizeof(int) * kMaxM * kDeltaWarps * 2;
};

__device__ __forceinline__ void load_lut_and_clear(unsigned char* smem, const uint16_t* __restrict__ g_lut,
                                                   uint16_t*& lut, uint32_t*& hist_all, int*& cs_all, int*& aux_all) {
  lut = reinterpret_cast<uint16_t*>(smem);
  hist_all = reinterpret_cast<uint32_t*>(smem + DeltaSmem::lut_bytes);
  cs_all = reinterpret_cast<int*>(hist_all + kDirWords * kDeltaWarps);
  aux_all = cs_all + kMaxM * kDeltaWarps;
  full_lut_copy(lut, g_lut);
  for (int i = threadIdx.x; i < kDirWords * kDeltaWarps; i += blockDim.x) hist_all[i] = 0u;
  __syncthreads();
}

// Batched swap deltas: moves[mv] = (state, u, v).  PAIRS selects the literal
// reference formulation.  dE = N3_SENTINEL for illegal moves or bad indices.
template <bool PAIRS>
__global__ void __launch_bounds__(kDeltaWarps * 32) swap_delta_kernel(const int16_t* __restrict__ cols, int B, int n,
                                                                        const int32_t* __restrict__ moves, int M,
                                                                        const uint16_t* __restrict__ g_lut,
                                                                        int32_t* __restrict__ dE,
                                                                        int32_t* __restrict__ dbad) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* lut;
  uint32_t* hist_all;
  int *cs_all, *aux_all;
  load_lut_and_clear(smem, g_lut, lut, hist_all, cs_all, aux_all);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = 2 * n;
  int* cs = cs_all + warp * kMaxM;
  int* db = aux_all + warp * kMaxM;
  uint32_t* hist = hist_all + warp * kDirWords;
  for (int mv = blockIdx.x * kDeltaWarps + warp; mv < M; mv += gridDim.x * kDeltaWarps) {
    const int b = moves[3 * mv], u = moves[3 * mv + 1], v = moves[3 * mv + 2];
    const bool in_range = b >= 0 && b < B && u >= 0 && u < m && v >= 0 && v < m;
    int key[kSlotsPerLane];
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {  // this lane's slots and their table keys
      const int k = lane + 32 * t;
      const int c = in_range && k < m ? (int)cols[(size_t)b * m + k] : 0;
      if (in_range && k < m) cs[k] = c;
      key[t] = (k >> 1) * kLutW + c;
    }
    __syncwarp();
    if (!in_range || !legal_swap(cs, u, v)) {
      if (lane == 0) dE[mv] = N3_SENTINEL;
      if (dbad)
        for (int s = lane; s < m; s += 32) dbad[(size_t)mv * m + s] = 0;
      __syncwarp();
      continue;
    }
    int d;
    if (PAIRS) {
      if (dbad)
        for (int s = lane; s < m; s += 32) db[s] = 0;
      __syncwarp();
      d = warp_sum(swap_delta_pairs(cs, m, u, v, lane, dbad ? db : nullptr));
      __syncwarp();
      if (dbad)
        for (int s = lane; s < m; s += 32) dbad[(size_t)mv * m + s] = db[s];
    } else {
      int local[kSlotsPerLane];
      int du = 0, dv = 0;
      if (dbad) {
        d = swap_delta_hist<true>(cs, key, m, u, v, lut, hist, lane, local, &du, &dv);
#pragma unroll
        for (int t = 0; t < kSlotsPerLane; ++t) {
          const int k = lane + 32 * t;
          if (k < m) dbad[(size_t)mv * m + k] = k == u ? du : (k == v ? dv : local[t]);
        }
      } else {
        d = swap_delta_hist<false>(cs, key, m, u, v, lut, hist, lane, local, &du, &dv);
      }
    }
    if (lane == 0) dE[mv] = d;
    __syncwarp();
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
//       around u, t(u') and t(v') from the table, and j(u', v') by walking the
//       line over the occupancy bits (4.6 cells on average), a lane per partner
//   fewer               a warp per partner, both new centres' histograms side by
//       side (pair_move.cuh), whatever the columns hold
// 64 n = 75 states, every slot: 85 us, 835 us with two histograms per partner one
// after the other; 1024 states with a slot each, partners of its layer: 48 and 60 us.
constexpr int kPartnerWarps = 24;
constexpr int kRunCover = 8;
constexpr int kPartnerRegion = ((kMaxN * kMaxN + 1) / 2 + 3) / 4 * 4;  // words of the cover table

struct PartnerSmem {
  uint16_t prim4[kCompactLutBytes / 2];
  uint16_t dir4[kCompactLutBytes / 2];
  uint32_t recip[kMaxN + 1];
  uint32_t T[kPartnerRegion];
  uint32_t occ[kOccWords + 3];
  uint32_t hist[kPartnerWarps][2 * DenseNumbering::kWords];
  uint2 scratch[kPartnerWarps][32];
  int columns[kMaxN];
  uint8_t cs[152];
};
static_assert(sizeof(PartnerSmem) <= 227 * 1024, "partner_scores_kernel shared memory");

// One partner's score by 8-bit histograms over A, one centre at a time: for equal
// columns and where a 4-bit counter may have wrapped.
__device__ __noinline__ int partner_by_histograms(const PartnerSmem& S, uint32_t* __restrict__ hist, int m, int u,
                                                  int v, int cur, int bad_uv, int lane) {
  const int ru = u >> 1, rv = v >> 1, cu = S.cs[u], cv = S.cs[v];
  int part = 0, j_new = 0;
  for (int c = 0; c < 2; ++c) {
    const int rx = c ? rv : ru, centre = c ? rv * kLutW + cu : ru * kLutW + cv;
    int ids[kSlotsPerLane];
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {
      const int k = lane + 32 * t;
      ids[t] = -1;
      if (k < m && k != u && k != v && (k >> 1) != rx) {
        const int ck = S.cs[k];
        ids[t] = (int)(dir4(S.dir4, (k >> 1) * kLutW + ck, centre) >> 2);
        part += hist_add(hist, ids[t]);
        if (c == 0) part += ((rv - ru) * (ck - cu) == (cv - cu) * ((k >> 1) - ru)) << 16;  // joint
      } else if (c == 0 && k < m && k != u && k != v) {  // u's row partner
        part += ((rv - ru) * (S.cs[k] - cu) == (cv - cu) * ((k >> 1) - ru)) << 16;
      }
    }
    __syncwarp();
    if (c == 0) j_new = hist_get(hist, (int)(dir4(S.dir4, rv * kLutW + cu, centre) >> 2));
    __syncwarp();
    hist_release(hist, ids);
    __syncwarp();
  }
  const int sum = warp_sum(part);
  return cur - (bad_uv - (sum >> 16)) + (sum & 0xFFFF) + j_new;
}

// A run's partners by a warp each.
template <bool SAME_LAYER, int NT>
__device__ __forceinline__ void partners_by_pairs(const PartnerSmem& S, uint32_t* __restrict__ hist, int n,
                                                  const int32_t* __restrict__ anchors, int a0, int a1,
                                                  const int32_t* __restrict__ bad, int cur, int warp, int lane,
                                                  int32_t* __restrict__ out) {
  const int m = 2 * n, width = SAME_LAYER ? n : m;
  WarpState W;
  W.m = m;
  W.lane = lane;
  W.cs = nullptr;
  W.bs = nullptr;
#pragma unroll
  for (int t = 0; t < kSlotsPerLane; ++t)
    W.key2[t] = W.slot(t) < m ? 2 * ((W.slot(t) >> 1) * kLutW + S.cs[W.slot(t)]) : 0;
  for (int a = a0; a < a1; ++a) {
    const int u = anchors[2 * a + 1];
    const bool in_range = u >= 0 && u < m;
    for (int w = warp; w < width; w += kPartnerWarps) {
      int score = N3_SENTINEL;
      if (in_range) {  // uniform
        const int v = SAME_LAYER ? 2 * w + (u & 1) : w;
        const int ru = u >> 1, rv = v >> 1, cu = S.cs[u], cv = S.cs[v];
        if (rv != ru && cv != S.cs[u ^ 1] && cu != S.cs[v ^ 1]) {  // uniform in the warp
          const int bad_uv = bad[u] + bad[v];
          bool redo = cu == cv;
          if (!redo) {
            Directions x, y;
            uint32_t line_new;
            const PairCount p = count_pair<DenseNumbering, NT>(W, S.dir4, hist, ru, rv, cu, cv, x, y, line_new);
            __syncwarp();
            clear_centre<NT>(x);
            clear_centre<NT>(y);
            __syncwarp();
            score = cur - (bad_uv - p.joint) + p.ta + p.tb + p.j_new;
            redo = p.wide;
          }
          if (redo) score = partner_by_histograms(S, hist, m, u, v, cur, bad_uv, lane);
        }
      }
      if (lane == 0) out[(size_t)a * width + w] = score;
    }
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
    __syncthreads();  // the previous run is done with the state
    if (b < 0 || b >= B) {  // uniform
      for (int i = tid; i < (a1 - a0) * width; i += blockDim.x) out[(size_t)a0 * width + i] = N3_SENTINEL;
      a0 = a1;
      continue;
    }
    const int cur = current[b];
    const int32_t* bad = badness + (size_t)b * m;
    bool cover = a1 - a0 >= kRunCover;
    if (cover) {
      for (int i = tid; i < kMaxN; i += blockDim.x) S.columns[i] = 0;
      for (int i = tid; i < kOccWords; i += blockDim.x) S.occ[i] = 0u;
      for (int i = tid; i < kPartnerRegion; i += blockDim.x) S.T[i] = 0u;
      __syncthreads();
    }
    bool regular = true;  // two points in every column, in cells of their own
    for (int s = tid; s < m; s += blockDim.x) {
      const int c = cols[(size_t)b * m + s];
      const bool on_grid = c >= 0 && c < n;
      regular = regular && on_grid;
      S.cs[s] = (uint8_t)min(max(c, 0), n - 1);
      if (cover && on_grid) {
        atomicAdd(&S.columns[c], 1);
        const uint32_t bit = 1u << (c & 31);
        if (atomicOr(&S.occ[3 * (s >> 1) + (c >> 5)], bit) & bit) regular = false;
      }
    }
    __syncthreads();
    if (cover) {
      for (int c = tid; c < n; c += blockDim.x) regular = regular && S.columns[c] == 2;
      cover = __syncthreads_and(regular);
    }
    if (cover) {
      cover_build(S.cs, S.T, n, S.prim4, S.recip, S.scratch[warp], lane, warp, kPartnerWarps);
      __syncthreads();
      for (int a = a0 + warp; a < a1; a += kPartnerWarps) {
        const int u = anchors[2 * a + 1];
        if (u < 0 || u >= m) {  // uniform in the warp
          for (int w = lane; w < width; w += 32) out[(size_t)a * width + w] = N3_SENTINEL;
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
        for (int w = lane; w < width; w += 32) {
          const int v = SAME_LAYER ? 2 * w + (u & 1) : w;
          const int rv = v >> 1, cv = S.cs[v];
          int score = N3_SENTINEL;
          if (rv != ru && cv != S.cs[u ^ 1] && cu != S.cs[v ^ 1]) {
            // the others on the line (u, v) (a column holds no third point)
            const int joint = hist_get(hist, (int)(dir4(S.dir4, rv * kLutW + cv, centre) >> 2)) - 1;
            score = cur - (bad_u + bad[v] - joint) + cover_get(S.T, ru * n + cv) + cover_get(S.T, rv * n + cu) +
                    points_on_line(S.occ, n, S.prim4, ru, cv, rv, cu);
          }
          out[(size_t)a * width + w] = score;
        }
        __syncwarp();
        hist_release(hist, ids);
        __syncwarp();
      }
    } else {
      switch ((m + 31) >> 5) {
        case 5: partners_by_pairs<SAME_LAYER, 5>(S, hist, n, anchors, a0, a1, bad, cur, warp, lane, out); break;
        case 4: partners_by_pairs<SAME_LAYER, 4>(S, hist, n, anchors, a0, a1, bad, cur, warp, lane, out); break;
        case 3: partners_by_pairs<SAME_LAYER, 3>(S, hist, n, anchors, a0, a1, bad, cur, warp, lane, out); break;
        case 2: partners_by_pairs<SAME_LAYER, 2>(S, hist, n, anchors, a0, a1, bad, cur, warp, lane, out); break;
        default: partners_by_pairs<SAME_LAYER, 1>(S, hist, n, anchors, a0, a1, bad, cur, warp, lane, out); break;
      }
    }
    a0 = a1;
  }
}

}  // namespace n3

namespace n3host {

template <class K>
static int prepare(K kernel, size_t bytes = n3::DeltaSmem::bytes) {
  return allow_smem(reinterpret_cast<const void*>(kernel), bytes);
}

int prepare_delta() {
  N3_TRY(prepare(n3::swap_delta_kernel<true>));
  N3_TRY(prepare(n3::swap_delta_kernel<false>));
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
  const uint16_t* lut = dir_lut_full_device_ptr();
  const int want = (M + n3::kDeltaWarps - 1) / n3::kDeltaWarps;
  const int grid = want < sm_count() * 2 ? want : sm_count() * 2;
  if (pairs) {
    N3_TRY(prepare(n3::swap_delta_kernel<true>));
    n3::swap_delta_kernel<true><<<grid, n3::kDeltaWarps * 32, n3::DeltaSmem::bytes, st>>>(cols, B, n, moves, M, lut,
                                                                                          dE, dbad);
  } else {
    N3_TRY(prepare(n3::swap_delta_kernel<false>));
    n3::swap_delta_kernel<false><<<grid, n3::kDeltaWarps * 32, n3::DeltaSmem::bytes, st>>>(cols, B, n, moves, M, lut,
                                                                                           dE, dbad);
  }
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
  // (64 states of 150 anchors: 128 CTAs of 75 take 85 us, 148 of 65 take 111 us).
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
