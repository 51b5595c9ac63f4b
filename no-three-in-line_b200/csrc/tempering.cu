// (c) Replica-exchange tempering: one persistent kernel over thousands of
// chains, ladders of neighbouring temperatures exchanged on the device.
//
// Reference: the per-replica walk kernel and host-side exchange of
// src/no_three_75/tempering.py:29-191.  Layout and scheduling here:
//
// * One warp per chain, `cpb` <= 16 chains per CTA.  A ladder of L temperatures
//   lives either inside one CTA (cpb a multiple of L) or across a thread-block
//   cluster of L / cpb CTAs; its exchange step uses the CTA barrier or the
//   cluster barrier and distributed shared memory, never a global spin-wait.
// * Every chain keeps its columns and badness in shared memory and proposes
//   row-pair column swaps (slots u, v from Philox4x32-10 with counter
//   (proposal index, chain), key = seed; u badness-weighted for bad_bias
//   percent of proposals, tempering.py:50-55).  An optional umbrella restraint
//   on the distance to a reference state enters the acceptance energy in
//   2^-24 fixed point (tempering.py:59-63, 93-94).  The lanes prepare 32 proposals
//   at a time on the current state; the legal ones are decided in order, and
//   after an accepted move the later ones are prepared again.
// * Acceptance falls from half the proposals at the hot end of a ladder to one in
//   thousands at the cold end (about exp(-3.2 / T)), and the two ends are decided
//   differently.  Hot chains take a move's exact dE from the maintained badness
//   (the reference identity bad[u]+bad[v]-joint, accelerated.py:78) and direction
//   histograms of the new positions, and an accepted move's badness changes from
//   histograms of the old ones too (pair_move.cuh).  Cold chains keep a cover
//   table instead (cover.cuh): four table entries bound each of 32 proposals at
//   once and reject most of them exactly; an accepted move costs about 20 times
//   a rejected one's histograms.
// * Metropolis acceptance compares a 32-bit uniform with a per-temperature
//   integer threshold table floor(2^32 exp(-dE/T)) built on the host, so the
//   CPU oracle replays every chain bit for bit.  Exchanges swap temperature
//   labels (not states) between neighbours with the reference's rule
//   (tempering.py:178-184, even/odd alternation), thresholds likewise tabled.
// * Results depend only on the seed, the chain index and the round structure,
//   not on cpb or on how rounds are split over launches.
#include <cooperative_groups.h>

#include "dirs.cuh"
#include "n3_common.cuh"
#include "philox.cuh"
#include "cover.cuh"
#include "pair_move.cuh"
#include "score_impl.cuh"

namespace cg = cooperative_groups;

namespace n3 {

struct TemperArgs {
  n3_chains ch;
  n3_temper_config cfg;
  const uint16_t* lut;  // table of primitive steps (device)
  int cluster;          // CTAs per ladder (1: whole ladders per CTA)
};

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Shared memory of the tempering kernel (dynamic): the table of primitive steps,
// the reciprocals, per chain a region that holds either the cover table or two
// histograms, the running badness sums (badness-weighted draws), badness,
// columns and cover_line's scratch; then the leader arrays.
constexpr int kRegionWords = ((kMaxN * kMaxN + 1) / 2 + 3) / 4 * 4;  // 2816: the cover table of 75 x 75 cells
static_assert(kRegionWords >= 2 * StepNumbering::kWords, "two histograms");
struct TemperSmem {
  static constexpr size_t tables = kCompactLutBytes + sizeof(uint32_t) * (kMaxN + 1);
  static __host__ __device__ constexpr size_t chain(bool bias) {
    return sizeof(uint32_t) * kRegionWords + sizeof(int) * kMaxM * (bias ? 2 : 1) + 152 + 32 * sizeof(uint2);
  }
  static __host__ __device__ constexpr size_t bytes(int cpb, bool bias) {
    return tables + (size_t)cpb * chain(bias) + 3 * sizeof(int) * 64 + 16;
  }
};
static_assert(TemperSmem::tables % 16 == 0 && TemperSmem::chain(true) % 8 == 0 && TemperSmem::chain(false) % 8 == 0 &&
                  sizeof(int) * kMaxM % 8 == 0, "alignment");
static_assert(TemperSmem::bytes(16, true) <= 227 * 1024, "16 chains of an SM");

// Metropolis test of an acceptance energy e = dE + umb_q / 2^24 (umb_q: an
// umbrella restraint term in units of 2^-24): accept iff e <= 0 or z is below
// thr[a] x f1[b >> 16] x f2[(b >> 8) & 255] x f3[b & 255] (32-bit fixed-point
// products), where e = a + b / 2^24.  thr[a] = floor(2^32 exp(-a/T)); frac
// holds f1, f2, f3 (256 each): floor(2^32 exp(-k/(2^8 T))), exp(-k/(2^16 T)),
// exp(-k/(2^24 T)).  A factor whose index is 0 is skipped, so umb_q = 0 is the
// plain test.
__device__ __forceinline__ bool umbrella_accept(int dE, int64_t umb_q, uint32_t z, const uint32_t* __restrict__ thr,
                                                int W, const uint32_t* __restrict__ frac) {
  const int64_t e = ((int64_t)dE << 24) + umb_q;
  if (e <= 0) return true;
  const int64_t a = e >> 24;
  if (a >= W) return false;
  uint32_t t = thr[a];
  const int b = (int)(e & 0xFFFFFF);
  if (b >> 16) t = (uint32_t)(((uint64_t)t * frac[b >> 16]) >> 32);
  if ((b >> 8) & 255) t = (uint32_t)(((uint64_t)t * frac[256 + ((b >> 8) & 255)]) >> 32);
  if (b & 255) t = (uint32_t)(((uint64_t)t * frac[512 + (b & 255)]) >> 32);
  return z < t;
}

// Change of the umbrella distance `removed` (reference points missing from the
// state) when slot u takes column c_v and slot v takes c_u: the reference's
// distance_delta (tempering.py:59-63) over the reference state's rows.
__device__ __forceinline__ int umbrella_distance_delta(const int16_t* __restrict__ ref, int u, int v, int cu, int cv) {
  const int ur = u & ~1, vr = v & ~1;
  const int a0 = ref[ur], a1 = ref[ur + 1], b0 = ref[vr], b1 = ref[vr + 1];
  return (int)(cu == a0 || cu == a1) + (int)(cv == b0 || cv == b1) - (int)(cv == a0 || cv == a1) -
         (int)(cu == b0 || cu == b1);
}

// Exchange step of one ladder (run by its leader thread).  tmp_chain[t] is the
// ladder-local chain at temperature t, tmp_temp[i] the temperature of chain i,
// e[i] the energy of chain i.
__device__ void exchange_ladder(int* tmp_chain, int* tmp_temp, const int* e, int L, int ladder, uint32_t round,
                                const uint32_t* __restrict__ xthr, int XW, uint32_t k0, uint32_t k1,
                                uint32_t& accepted) {
  for (int t = (int)(round & 1u); t < L - 1; t += 2) {
    const int a = tmp_chain[t], b = tmp_chain[t + 1];
    const int D = e[a] - e[b];  // chain a holds the lower temperature
    bool swap = D >= 0;
    if (!swap) {
      const U4 r = philox4x32_10(U4{round, (uint32_t)t, (uint32_t)ladder, kTagExchange}, k0, k1);
      const int d = -D;
      swap = d < XW && r.x < xthr[(size_t)t * XW + d];
    }
    if (swap) {
      tmp_chain[t] = b;
      tmp_chain[t + 1] = a;
      tmp_temp[a] = t + 1;
      tmp_temp[b] = t;
      ++accepted;
    }
  }
}

// Chains at temperatures whose acceptance of dE = 3 lies below kCoverAccept (in
// 2^-32) work from a cover table, the others from histograms.  Per chain alone on
// an SM, n = 75: a histogram move costs 940 cycles rejected and 2200 accepted, the
// cover table 15 per proposal, 36,000 per accepted move and 300,000 to build.  100
// sweeps of 2048 chains, ladders of 64 from 0.05 to 5.0: 16.8 ms with the line at
// 0.008, 16.5 ms at 0.039, 24.8 ms at 0.078 (38.3 ms with one 8-bit histogram at a
// time, a team barrier after each, and no cover table).  40 sweeps on other grids, ms with
// no table, the line at 0.02, 0.039 and 0.078, and one 8-bit histogram at a time:
//   2048 chains 0.05 .. 5.0   n = 8  0.49 0.52 0.57 0.70 0.94   n = 20 1.75 1.49 1.58 2.18 2.93
//                             n = 40 3.68 3.10 3.06 4.58 6.72   n = 75 8.6  6.4  6.4  11.1 15.3
//   512 chains 0.3 .. 1.2     n = 8  0.39 0.48 0.60 0.68 0.68   n = 20 1.31 1.17 1.52 1.88 2.07
//                             n = 40 2.67 2.24 2.85 4.13 4.47   n = 75 6.3  4.6  5.1  9.4  9.9
// So the line suits wide ladders from n = 16 on; for small grids, and for ladders that
// sit in the middle of it, 0.02 would do better.
constexpr uint32_t kCoverAccept = 0x0A000000u;  // 0.039
constexpr int kCoverMinProposals = 512;         // proposals left in the launch that pay for building the table

// What a chain's proposals need beyond its state; uniform across the warp.
struct Walk {
  const uint32_t* thr;  // threshold row of the chain's temperature
  int width;
  uint32_t k0, k1;
  int chain;
  int bad_bias;          // BIAS
  const int16_t* ref;    // umbrella (UMB): reference columns, fraction factors, coefficients
  const uint32_t* frac;
  int64_t s_q, c2s_q;
};

// A lane's proposal: proposal index p + lane of the chain.
struct Proposal {
  int u, v;
  uint32_t z;       // Metropolis uniform
  uint32_t bias_x;  // BIAS: the badness draw's uniform
  bool weighted;    // BIAS: u is drawn by badness
};

template <bool BIAS>
__device__ __forceinline__ Proposal draw_proposal(const Walk& w, uint64_t ctr, int m) {
  const U4 r = philox4x32_10(U4{(uint32_t)ctr, (uint32_t)(ctr >> 32), (uint32_t)w.chain, kTagPropose}, w.k0, w.k1);
  Proposal p;
  p.u = (int)__umulhi(r.x, (unsigned)m);
  p.v = (int)__umulhi(r.y, (unsigned)m);
  p.z = r.z;
  p.weighted = BIAS && __umulhi(r.w, 100u) < (unsigned)w.bad_bias;
  p.bias_x = 0u;
  if (BIAS)
    p.bias_x = philox4x32_10(U4{(uint32_t)ctr, (uint32_t)(ctr >> 32), (uint32_t)w.chain, kTagBias}, w.k0, w.k1).x;
  return p;
}

// Slot of a badness-weighted draw (tempering.py:52-54): the first slot whose
// running badness sum exceeds target, and at most m - 1.
__device__ __forceinline__ int weighted_slot(const int* __restrict__ prefix, int m, int target) {
  int lo = 0, hi = m - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] > target)
      hi = mid;
    else
      lo = mid + 1;
  }
  return lo;
}

// prefix[s] = badness of slots 0 .. s; bad(s) gives one slot's.  Lane l sums slots 5 l .. 5 l + 4.
template <class Bad>
__device__ __forceinline__ void running_sums(int* __restrict__ prefix, int m, int lane, const Bad& bad) {
  const int s0 = lane * kSlotsPerLane;
  int val[kSlotsPerLane], local = 0;
#pragma unroll
  for (int t = 0; t < kSlotsPerLane; ++t) {
    val[t] = s0 + t < m ? bad(s0 + t) : 0;
    local += val[t];
  }
  int run = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += y;
  }
  run -= local;
  __syncwarp();  // every lane is done with the sums before
#pragma unroll
  for (int t = 0; t < kSlotsPerLane; ++t) {
    run += val[t];
    if (s0 + t < m) prefix[s0 + t] = run;
  }
  __syncwarp();
}

__device__ __forceinline__ bool metropolis(const Walk& w, int dE, uint32_t z) {
  return dE <= 0 || (dE < w.width && z < w.thr[dE]);
}

// A legal move from the cover table: mv.bad is minus the bound on dE that the four
// entries give, and the points on the lines (u, v) and (u', v') complete it.
template <class Accept>
__device__ __forceinline__ bool cover_move(WarpState& W, uint32_t* __restrict__ T, int n,
                                           const uint16_t* __restrict__ prim4, const uint32_t* __restrict__ recip,
                                           uint2* __restrict__ scratch, PreparedMove mv, Accept accept, int& E) {
  const int u = (int)(mv.slots & 0xFFu), v = (int)((mv.slots >> 8) & 0xFFu);
  const int cu = (int)((mv.slots >> 16) & 0xFFu), cv = (int)(mv.slots >> 24);
  const int ru = u >> 1, dr = (v >> 1) - ru, dc = cv - cu;
  // u and v lie on the first line themselves
  const int hits = W.on_line<kSlotsPerLane>(ru, cu, dr, dc) + W.on_line<kSlotsPerLane>(ru, cv, dr, -dc);
  const int dE = warp_sum(hits) - 2 - mv.bad;
  if (!accept(dE)) return false;
  cover_swap(W.cs, T, n, u, v, prim4, recip, scratch, W.lane);
  W.swap_keys(u, v, dc);
  __syncwarp();
  if (W.lane == 0) {
    W.cs[u] = (uint8_t)cv;
    W.cs[v] = (uint8_t)cu;
  }
  __syncwarp();
  E += dE;
  return true;
}

// A legal move from histograms; nt = ceil(m / 32).
template <bool UMB>
__device__ __forceinline__ bool hist_move(WarpState& W, const uint16_t* __restrict__ prim4,
                                          uint32_t* __restrict__ hist, int nt, PreparedMove mv, const Walk& w,
                                          uint32_t z, int& removed, int& E, uint32_t& err) {
  int dE, dd = 0;
  int64_t umb = 0;
  if (UMB) {
    dd = umbrella_distance_delta(w.ref, (int)(mv.slots & 0xFFu), (int)((mv.slots >> 8) & 0xFFu),
                                 (int)((mv.slots >> 16) & 0xFFu), (int)(mv.slots >> 24));
    umb = w.s_q * (int64_t)(2 * removed * dd + dd * dd) - w.c2s_q * (int64_t)dd;
  }
  const auto accept = [=](int d) {
    return UMB ? umbrella_accept(d, umb, z, w.thr, w.width, w.frac) : metropolis(w, d, z);
  };
  const bool acc = pair_move_any<StepNumbering>(W, prim4, hist, nt, mv, accept, E, err, &dE);
  if (UMB && acc) removed += dd;
  return acc;
}

template <bool BIAS, bool UMB>
__global__ void __launch_bounds__(512, 1) temper_kernel(const TemperArgs A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const n3_chains& ch = A.ch;
  const n3_temper_config& cfg = A.cfg;
  const int cpb = cfg.chains_per_block, L = ch.ladder_size, CS = A.cluster;
  uint16_t* prim4 = reinterpret_cast<uint16_t*>(smem);
  uint32_t* recip = reinterpret_cast<uint32_t*>(smem + kCompactLutBytes);
  unsigned char* chains_base = smem + TemperSmem::tables;
  int* ld_e = reinterpret_cast<int*>(chains_base + (size_t)cpb * TemperSmem::chain(BIAS));  // leader arrays (64 each)
  int* ld_temp = ld_e + 64;
  int* ld_chain = ld_temp + 64;
  int* ld_stop = ld_chain + 64;

  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CS > 1 ? (int)cluster.block_rank() : 0;
  auto barrier = [&]() {
    if (CS > 1)
      cluster.sync();
    else
      __syncthreads();
  };
  // leader arrays: CTA rank 0 of the cluster (CS > 1) or this CTA (CS == 1)
  int* L_e = CS > 1 ? cluster.map_shared_rank(ld_e, 0) : ld_e;
  int* L_temp = CS > 1 ? cluster.map_shared_rank(ld_temp, 0) : ld_temp;
  int* L_stop = CS > 1 ? cluster.map_shared_rank(ld_stop, 0) : ld_stop;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A ladder's chains are dealt out to its cluster's CTAs one by one: a chain's
  // temperature drifts slowly from its own index, and hot chains take far
  // longer than cold ones, so every CTA gets its share of them.
  const int li = CS > 1 ? warp * CS + rank : warp % L;
  const int lad = CS > 1 ? blockIdx.x / CS : (blockIdx.x * cpb + warp) / L;
  const int c = lad * L + li;
  const int lidx = CS > 1 ? li : warp;              // index into the leader arrays
  const int lbase = CS > 1 ? 0 : (warp / L) * L;    // this ladder's block in them
  const int n = ch.ladder_n[lad], m = 2 * n, nt = (m + 31) >> 5;
  unsigned char* mine = chains_base + (size_t)warp * TemperSmem::chain(BIAS);
  uint32_t* region = reinterpret_cast<uint32_t*>(mine);
  int* bs = reinterpret_cast<int*>(region + kRegionWords);
  int* prefix = bs + kMaxM;  // BIAS
  uint8_t* cs = reinterpret_cast<uint8_t*>(bs + kMaxM * (BIAS ? 2 : 1));
  uint2* scratch = reinterpret_cast<uint2*>(cs + 152);

  compact_lut_copy(prim4, A.lut);
  for (int a = threadIdx.x; a <= kMaxN; a += blockDim.x) recip[a] = a ? (65536u + (uint32_t)a - 1u) / (uint32_t)a : 0u;
  WarpState W;
  W.m = m;
  W.lane = lane;
  W.cs = cs;
  W.bs = bs;
  for (int i = lane; i < kRegionWords; i += 32) region[i] = 0u;
  // The state; a column off the largest grid stops the chain (error bit 1), and one
  // off the state's own, columns that do not hold two points each, or a cell that
  // holds two, keep it from the cover table.
  bool on_grid = true, factor = true;
#pragma unroll
  for (int t = 0; t < kSlotsPerLane; ++t) {
    const int s = W.slot(t);
    W.key2[t] = 0;
    if (s < m) {
      const int col = ch.cols[(size_t)c * kMaxM + s];
      on_grid = on_grid && col >= 0 && col < kMaxN;
      factor = factor && col < n;
      W.key2[t] = 2 * ((s >> 1) * kLutW + col);
      cs[s] = (uint8_t)col;
      bs[s] = ch.badness[(size_t)c * kMaxM + s];
    }
    const int row_other = __shfl_xor_sync(0xffffffffu, W.key2[t], 1);
    factor = factor && (row_other != W.key2[t] || s >= m);
  }
  on_grid = __all_sync(0xffffffffu, on_grid);
  if (on_grid) {  // points per column
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t)
      if (W.slot(t) < m) atomicAdd(region + (W.key2[t] / 2 - (W.slot(t) >> 1) * kLutW), 1u);
    __syncwarp();
    for (int col = lane; col < n; col += 32) {
      factor = factor && region[col] == 2u;
      region[col] = 0u;
    }
    factor = __all_sync(0xffffffffu, factor);
    __syncwarp();
  }
  int E = ch.energy[c], bestE = ch.best_energy[c];
  int removed = UMB ? ch.removed[c] : 0;
  const uint64_t counter0 = ch.counter[c];
  uint64_t counter = counter0;
  uint32_t accepted = ch.accepted[c];
  uint32_t err = on_grid ? 0u : kErrColumnRange;
  bool hit_done = false;

  // The leader CTA loads the ladder bookkeeping of its ladder(s).
  const bool leader_cta = rank == 0;
  const int lad_first = (blockIdx.x * cpb) / L;          // first ladder of this CTA
  const int n_lad_here = CS > 1 ? 1 : cpb / L;
  if (leader_cta) {
    for (int i = threadIdx.x; i < n_lad_here * L; i += blockDim.x) {
      const int gl = lad_first + i / L;
      ld_chain[i] = ch.chain_at[(size_t)gl * L + i % L];
      ld_temp[i] = ch.temp_of[(size_t)gl * L + i % L];
    }
    if (threadIdx.x == 0) *ld_stop = 0;
  }
  uint32_t lround = 0, lexch = 0;  // leader-thread copies (one leader per ladder)
  const bool ladder_leader = leader_cta && lane == 0 && (CS > 1 ? warp == 0 : (warp % L) == 0);
  if (ladder_leader) {
    lround = ch.ladder_round[lad];
    lexch = ch.ladder_exchanges[lad];
  }
  barrier();

  const int rounds = cfg.ladder_rounds ? cfg.ladder_rounds[lad] : cfg.rounds;
  const int per_round = cfg.round_proposals > 0 ? cfg.round_proposals : cfg.round_sweeps * m;
  const uint32_t k0 = (uint32_t)cfg.seed, k1 = (uint32_t)(cfg.seed >> 32);
  Walk w;
  w.width = ch.acc_width;
  w.k0 = k0;
  w.k1 = k1;
  w.chain = c;
  w.bad_bias = cfg.bad_bias;
  w.ref = ch.reference;
  w.frac = nullptr;
  w.s_q = 0;
  w.c2s_q = 0;

  // bookkeeping of an accepted move, proposal p of the round
  auto moved = [&](int p) {
    ++accepted;
    if (E < bestE) {
      bestE = E;
      for (int s = lane; s < m; s += 32) ch.best_cols[(size_t)c * kMaxM + s] = (int16_t)cs[s];
    }
    if (cfg.target_energy >= 0 && E <= cfg.target_energy && !hit_done) {
      hit_done = true;
      if (lane == 0 && ch.hit != nullptr && atomicCAS(ch.hit, -1, c) == -1) {
        const uint64_t now = global_ns();
        ch.hit[1] = (int32_t)(uint32_t)(counter + (uint64_t)p + 1u);
        ch.hit[2] = (int32_t)(uint32_t)now;
        ch.hit[3] = (int32_t)(uint32_t)(now >> 32);
        if (ch.stop) atomicExch(ch.stop, 1);
      }
    }
  };

  bool covered = false;  // the region holds the cover table (else zeros), and bs is stale
  auto uncover = [&]() {
    __syncwarp();
    for (int s = lane; s < m; s += 32) bs[s] = cover_get(region, (s >> 1) * n + cs[s]);
    __syncwarp();
    for (int i = lane; i < kRegionWords; i += 32) region[i] = 0u;
    __syncwarp();
    covered = false;
  };
  for (int r = 0; r < rounds; ++r) {
    const int temp = L_temp[lidx];
    w.thr = ch.acc_thresh + (size_t)temp * w.width;
    if (UMB) {
      const size_t pos = (size_t)lad * L + temp;  // the replica position (temperature slot) of this chain
      w.frac = ch.acc_frac + (size_t)temp * 768;
      w.s_q = ch.umbrella[2 * pos];
      w.c2s_q = ch.umbrella[2 * pos + 1];
    }
    if (!UMB && on_grid && factor) {
      const bool cold = w.width <= 3 || w.thr[3] < kCoverAccept;
      if (covered && !cold) uncover();
      if (!covered && cold && (int64_t)(rounds - r) * per_round >= kCoverMinProposals) {
        cover_build(cs, region, n, prim4, recip, scratch, lane);
        __syncwarp();
        covered = true;
        for (int s = lane; s < m; s += 32)
          if (bs[s] != cover_get(region, (s >> 1) * n + cs[s])) err |= kErrAudit;
      }
    }
    for (int p = 0; on_grid && E > 0 && p < per_round; p += 32) {
      const int cnt = min(32, per_round - p);
      Proposal pr = draw_proposal<BIAS>(w, counter + (uint64_t)(p + lane), m);
      int from = 0;  // proposals before it are decided
      do {
        if (BIAS) {
          if (covered)
            running_sums(prefix, m, lane, [&](int s) { return cover_get(region, (s >> 1) * n + cs[s]); });
          else
            running_sums(prefix, m, lane, [&](int s) { return bs[s]; });
          if (pr.weighted) pr.u = weighted_slot(prefix, m, (int)__umulhi(pr.bias_x, 3u * (unsigned)E));
        }
        // every lane prepares its own proposal on the current state
        const int u = pr.u, v = pr.v, cu = cs[u], cv = cs[v];
        bool live = lane >= from && lane < cnt && legal_swap(cs, u, v);
        PreparedMove mine_mv;
        mine_mv.slots = (uint32_t)(u | (v << 8) | (cu << 16) | (cv << 24));
        if (!UMB && covered) {  // bad: less the new positions' entries, so that -bad is the bound on dE
          const int row_u = (u >> 1) * n, row_v = (v >> 1) * n;
          mine_mv.bad = cover_get(region, row_u + cu) + cover_get(region, row_v + cv) -
                        cover_get(region, row_u + cv) - cover_get(region, row_v + cu);
          live = live && metropolis(w, -mine_mv.bad, pr.z);
        } else {
          mine_mv.bad = bs[u] + bs[v];
        }
        unsigned open = __ballot_sync(0xffffffffu, live);
        from = 32;
        while (open) {
          const int j = __ffs(open) - 1;
          open &= open - 1u;
          PreparedMove mv;
          mv.slots = __shfl_sync(0xffffffffu, mine_mv.slots, j);
          mv.bad = __shfl_sync(0xffffffffu, mine_mv.bad, j);
          const uint32_t z = __shfl_sync(0xffffffffu, pr.z, j);
          bool acc;
          if (!UMB && covered)
            acc = cover_move(W, region, n, prim4, recip, scratch, mv, [=](int d) { return metropolis(w, d, z); }, E);
          else if (UMB)
            acc = hist_move<true>(W, prim4, region, nt, mv, w, z, removed, E, err);
          else
            acc = hist_move<false>(W, prim4, region, nt, mv, w, z, removed, E, err);
          if (acc) {
            moved(p + j);
            from = j + 1;
            break;
          }
        }
      } while (from < cnt && E > 0);
    }
    counter += (uint64_t)per_round;
    if (!cfg.exchange) continue;
    if (lane == 0) L_e[lidx] = E;
    barrier();
    if (ladder_leader) {
      exchange_ladder(ld_chain + lbase, ld_temp + lbase, ld_e + lbase, L, lad, lround, ch.exch_thresh,
                      ch.exch_width, k0, k1, lexch);
      ++lround;
      if (ch.stop != nullptr && warp == 0) *ld_stop = *((volatile int*)ch.stop);
    }
    barrier();
    if (*((volatile int*)L_stop)) break;
  }
  if (covered) uncover();

  // write back
  if (on_grid)
    for (int s = lane; s < m; s += 32) {
      ch.cols[(size_t)c * kMaxM + s] = (int16_t)cs[s];
      ch.badness[(size_t)c * kMaxM + s] = bs[s];
    }
  if (err && ch.error_word) atomicOr(ch.error_word, err);
  if (lane == 0) {
    ch.energy[c] = E;
    ch.best_energy[c] = bestE;
    ch.counter[c] = counter;
    ch.accepted[c] = accepted;
    if (UMB) ch.removed[c] = removed;
    if (ch.global_best) atomicMin(ch.global_best, bestE);
  }
  if (ladder_leader) {
    ch.ladder_round[lad] = lround;
    ch.ladder_exchanges[lad] = lexch;
  }
  barrier();  // the leader threads have finished their exchanges
  if (leader_cta) {
    for (int i = threadIdx.x; i < n_lad_here * L; i += blockDim.x) {
      const int gl = lad_first + i / L;
      ch.chain_at[(size_t)gl * L + i % L] = ld_chain[i];
      ch.temp_of[(size_t)gl * L + i % L] = ld_temp[i];
    }
  }
  barrier();  // keep the leader's shared memory alive until every CTA is done with it
}

// Full recompute of every chain's energy (determinant count) and badness
// (slope count) compared with the maintained values.  One warp per chain.
constexpr int kAuditWarps = 4;
constexpr size_t kAuditSmem = kCompactLutBytes + kAuditWarps * (kTagWarpBytes + sizeof(int) * kMaxM);

__global__ void __launch_bounds__(kAuditWarps * 32) audit_kernel(const n3_chains ch, const uint16_t* __restrict__ g_lut,
                                                                   int32_t* mismatch) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* lut = reinterpret_cast<uint16_t*>(smem);
  compact_lut_copy(lut, g_lut);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* tag = smem + kCompactLutBytes + warp * (kTagWarpBytes + sizeof(int) * kMaxM);
  uint32_t* bs = reinterpret_cast<uint32_t*>(tag + kDirCount);
  int* cs = reinterpret_cast<int*>(bs + kMaxM);
  for (int c = blockIdx.x * kAuditWarps + warp; c < ch.n_chains; c += gridDim.x * kAuditWarps) {
    const int n = ch.ladder_n[c / ch.ladder_size], m = 2 * n;
    int key[kSlotsPerLane];
    int ok = 1;
#pragma unroll
    for (int t = 0; t < kSlotsPerLane; ++t) {
      const int s = lane + 32 * t;
      const int col = s < m ? (int)ch.cols[(size_t)c * kMaxM + s] : 0;
      if (s < m) {
        ok &= col >= 0 && col < kMaxN;
        cs[s] = col;
        bs[s] = 0u;
      }
      key[t] = s < m ? (s >> 1) * kLutW + col : -1;
    }
    ok = __all_sync(0xffffffffu, ok);
    __syncwarp();
    if (ok) {  // uniform: every column is on the grid
      const int e = warp_sum(det_state<false>(cs, n, lane, nullptr));
      tag_state<true>(key, m, lut, tag, lane, bs, bs);
      __syncwarp();
      for (int s = lane; s < m; s += 32) ok &= (int)bs[s] == ch.badness[(size_t)c * kMaxM + s];
      ok = __all_sync(0xffffffffu, ok) && e == ch.energy[c];
    }
    if (lane == 0 && !ok) {
      atomicAdd(mismatch, 1);
      if (ch.error_word) atomicOr(ch.error_word, kErrAudit);
    }
    __syncwarp();
  }
}

}  // namespace n3

namespace n3host {

static int check_chains(const n3_chains* ch) {
  if (ch == nullptr) return set_error(N3_ERR_ARG, "null chains descriptor");
  const int L = ch->ladder_size;
  if (L < 2 || L > 64) return set_error(N3_ERR_ARG, "ladder_size %d outside [2, 64]", L);
  if (ch->n_chains <= 0 || ch->n_chains % L)
    return set_error(N3_ERR_ARG, "n_chains %d is not a positive multiple of ladder_size %d", ch->n_chains, L);
  if (!ch->cols || !ch->badness || !ch->energy || !ch->best_energy || !ch->best_cols || !ch->temp_of ||
      !ch->chain_at || !ch->counter || !ch->accepted || !ch->ladder_n || !ch->ladder_round ||
      !ch->ladder_exchanges || !ch->acc_thresh || !ch->exch_thresh)
    return set_error(N3_ERR_ARG, "null device pointer in chains descriptor");
  if (ch->acc_width < 2 || ch->exch_width < 2) return set_error(N3_ERR_ARG, "threshold tables too narrow");
  return N3_OK;
}

using TemperKernel = void (*)(const n3::TemperArgs);

static TemperKernel temper_instance(bool bias, bool umb) {
  return umb ? (bias ? n3::temper_kernel<true, true> : n3::temper_kernel<false, true>)
             : (bias ? n3::temper_kernel<true, false> : n3::temper_kernel<false, false>);
}

int temper_launch(const n3_chains* ch, const n3_temper_config* cfg, cudaStream_t st) {
  N3_TRY(check_chains(ch));
  if (cfg == nullptr) return set_error(N3_ERR_ARG, "null config");
  const int L = ch->ladder_size, cpb = cfg->chains_per_block;
  const int tpc = cfg->threads_per_chain == 0 ? 32 : cfg->threads_per_chain;
  if (tpc != 32 && tpc != 64 && tpc != 128 && tpc != 256)
    return set_error(N3_ERR_ARG, "threads_per_chain %d is not 32, 64, 128 or 256", cfg->threads_per_chain);
  const int wpc = tpc / 32;
  if (cpb < 1 || cpb * wpc > 16)
    return set_error(N3_ERR_ARG, "chains_per_block %d x %d warps per chain outside [1, 16] warps", cpb, wpc);
  int cluster = 1;
  if (cpb < L) {
    if (L % cpb) return set_error(N3_ERR_ARG, "chains_per_block %d does not divide ladder_size %d", cpb, L);
    cluster = L / cpb;
    if (cluster > 8) return set_error(N3_ERR_ARG, "a ladder would span %d CTAs (max 8)", cluster);
  } else if (cpb % L) {
    return set_error(N3_ERR_ARG, "chains_per_block %d is not a multiple of ladder_size %d", cpb, L);
  }
  if (ch->n_chains % cpb) return set_error(N3_ERR_ARG, "n_chains not a multiple of chains_per_block");
  if (cfg->rounds < 0 || cfg->round_proposals < 0 || cfg->round_sweeps < 0)
    return set_error(N3_ERR_ARG, "negative round count or length");
  if (!cfg->exchange && cfg->round_proposals == 0 && cfg->round_sweeps == 0)
    return set_error(N3_ERR_ARG, "a round without exchange needs proposals");
  if (cfg->bad_bias < 0 || cfg->bad_bias > 100) return set_error(N3_ERR_ARG, "bad_bias %d outside [0, 100]", cfg->bad_bias);
  const bool umb = ch->umbrella != nullptr;
  if (umb) {
    if (!ch->reference || !ch->removed || !ch->acc_frac)
      return set_error(N3_ERR_ARG, "umbrella needs reference, removed and acc_frac");
    if (cfg->exchange)
      return set_error(N3_ERR_ARG, "temperature-only exchange is disabled with umbrella potentials");
  }
  N3_TRY(ensure_device_tables());
  n3::TemperArgs args;
  args.ch = *ch;
  args.lut = prim4_lut_device_ptr();
  args.cfg = *cfg;
  args.cluster = cluster;
  const bool bias = cfg->bad_bias > 0;
  const size_t smem = n3::TemperSmem::bytes(cpb, bias);
  void (*kern)(const n3::TemperArgs) = temper_instance(bias, umb);
  N3_TRY(allow_smem(reinterpret_cast<const void*>(kern), n3::TemperSmem::bytes(16, bias)));
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ch->n_chains / cpb);
  lc.blockDim = dim3(cpb * 32);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&lc, kern, args);
  if (e != cudaSuccess) return set_error(N3_ERR_CUDA, "temper_kernel launch: %s", cudaGetErrorString(e));
  return check_launch("temper_kernel");
}

}  // namespace n3host

namespace n3host {
int prepare_tempering() {
  for (int b = 0; b < 2; ++b)
    for (int u = 0; u < 2; ++u)
      N3_TRY(allow_smem(reinterpret_cast<const void*>(temper_instance(b, u)), n3::TemperSmem::bytes(16, b)));
  return allow_smem(reinterpret_cast<const void*>(n3::audit_kernel), n3::kAuditSmem);
}
}  // namespace n3host

extern "C" {

int n3_temper_run(const n3_chains* chains, const n3_temper_config* config, void* stream) {
  return n3host::temper_launch(chains, config, (cudaStream_t)stream);
}

int n3_temper_audit(const n3_chains* chains, int32_t* mismatch, void* stream) {
  N3_TRY(n3host::check_chains(chains));
  if (mismatch == nullptr) return n3host::set_error(N3_ERR_ARG, "null mismatch counter");
  N3_TRY(n3host::ensure_device_tables());
  const n3_chains ch = *chains;
  const size_t smem = n3::kAuditSmem;
  N3_TRY(n3host::allow_smem(reinterpret_cast<const void*>(n3::audit_kernel), smem));
  const int want = (ch.n_chains + n3::kAuditWarps - 1) / n3::kAuditWarps;
  const int grid = want < n3host::sm_count() * 4 ? want : n3host::sm_count() * 4;
  n3::audit_kernel<<<grid, n3::kAuditWarps * 32, smem, (cudaStream_t)stream>>>(ch, n3host::dir_lut_device_ptr(),
                                                                                 mismatch);
  return n3host::check_launch("audit_kernel");
}

}  // extern "C"

namespace n3 {
__global__ void clock_kernel(int64_t* out) { out[0] = (int64_t)global_ns(); }
}  // namespace n3

extern "C" int n3_device_clock_ns(int64_t* out, void* stream) {
  if (out == nullptr) return n3host::set_error(N3_ERR_ARG, "null output");
  n3::clock_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(out);
  return n3host::check_launch("clock_kernel");
}
