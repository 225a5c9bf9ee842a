// The whole 2D substep of a small world as one cooperative launch.
//
// A world of a few thousand particles spends its substep between kernels: 51
// dependent launches of 1-3 us of work each took 167 us at 4,096 particles.
// Here one CTA per SM runs every phase of sim2d.cuh, the phases separated by
// grid barriers, and what a phase hands to itself in the next one stays on the
// SM:
//
//   * each CTA owns an equal share of every colour class (its particles are
//     contiguous in sorted space, colour by colour), and keeps their neighbour
//     lists, records and wall bounds in shared memory through all iterations,
//     with the kernel tables: what is left on a phase's critical path is one
//     load of the neighbours' records;
//   * the grid is a counting sort over the cells: the cell counts fit every
//     CTA, so each scans them by itself (no phase of its own, and the cell
//     ranges the list build needs are in shared memory). Arrival order inside
//     a cell is whatever the count's atomics gave; each particle then ranks
//     itself among its cell's slots, which puts the cell into ascending slot
//     order, the canonical order the radix sort of the large path gives (cells
//     of hundreds are put in order by a whole CTA, see rank_pile);
//   * the last CTA to finish folds the chain.
//
// The sums are those of the per-phase kernels (the same device functions), so
// the results are equal word by word. Every wait is bounded (grid_wait).
//
// Measured (us a substep, the per-phase graph it replaced -> this): 1.5 k particles
// 149 -> 82, 4.1 k 167 -> 84, 13 k 167 -> 92, 42 k 219 -> 129, 61 k 256 -> 145, 93 k
// 312 -> 208. A barrier costs 1.05-1.3 us and a colour pass about 2 us on its
// slowest CTA (two dependent L2 round trips); the limit is what fits an SM
// (fused_fits).
#pragma once
#include "gridsync.cuh"
#include "rigid.cuh"

namespace sn {
namespace d2 {

constexpr uint32_t FU_ROW = 52;  // words per list row: 8 lanes of 4 rows, or 4 of 8, fall on different banks
constexpr uint32_t FU_OWN_BYTES = 16 + 8 + 4 + 4 + 4 * FU_ROW;
constexpr uint32_t FU_TAIL_WORDS = 2 + FU_ROW;  // of these, what nothing uses before the owned share is known

struct FusedPar {
  uint32_t iters, friction, bonds, seal, chain;
  uint32_t slots;    // slots that can be active: [0, slots)
  uint32_t xWords;   // shared words for the cell ranges, then the CA table
  uint32_t ownCap;   // particles a CTA can own
  uint32_t bodies;   // rigid bodies, one CTA each in turn
  uint32_t* count;   // [K] cell counts, zero between launches
  uint32_t* tmp;     // slots by cell in arrival order
  GridBar bar;       // count[0] barrier arrivals, count[1] finished CTAs, zero between launches
};

// Neighbour access of an owned particle: its list row and the kernel tables in
// shared memory, records in the current buffer (or, in a colour pass, split as
// NbrSplit does).
struct NbrOwned {
  const int4* g;
  const uint32_t* rows;
  const int2* swg;
  const int2* sca;
  uint32_t cut, off;
  __device__ __forceinline__ uint32_t entry(uint32_t row, uint32_t k) const { return rows[row * FU_ROW + k]; }
  __device__ __forceinline__ int4 rec(uint32_t e) const {
    return g[(int32_t)(e < cut ? e + off : e)];
  }
  __device__ __forceinline__ int2 pred(uint32_t e) const { return ld_pred(g, e); }
  __device__ __forceinline__ int2 wg(const Bufs&, int id) const { return swg[id]; }
  __device__ __forceinline__ int2 ca(const Bufs&, int id) const { return sca[id]; }
};

// The sums of solveA and solveB with FU_B neighbours' records in flight at a
// time: the list entries are at hand, so a batch costs one L2 round trip (one
// ahead of the pair in hand, as the per-phase kernels have it, is one for every
// neighbour but the first when a CTA has a few warps). When they came in, with 16
// lanes to a colour's particle, a substep of 4.7 k particles went from 94 to 86 us, of
// 40 k from 145 to 128.
constexpr int FU_B = 3;
constexpr uint32_t FU_CHUNK = 16;  // particles of a colour dealt to a CTA at a time, in worlds with bodies
template <int L>
__device__ __forceinline__ void solveA_owned(const Bufs& b, const NbrOwned& nb, uint32_t row, uint32_t cnt,
                                             uint32_t sub, int2 pi, const Flags<false>& f, int32_t& rho, int32_t& S,
                                             int32_t& sgx, int32_t& sgy) {
  for (uint32_t k = sub; k < cnt; k += L * FU_B) {
    int2 pj[FU_B];
#pragma unroll
    for (int j = 0; j < FU_B; ++j) pj[j] = nb.pred(k + j * L < cnt ? nb.entry(row, k + j * L) : 0u);
#pragma unroll
    for (int j = 0; j < FU_B; ++j)
      if (k + j * L < cnt) solveA_pair<false>(b, nb, pi, pj[j], f, rho, S, sgx, sgy);
  }
  rho = gsum<L>(rho);
  S = gsum<L>(S);
  sgx = gsum<L>(sgx);
  sgy = gsum<L>(sgy);
}
// RIG: infoI is a rigid member's info, whose correction skips its own body, or 0.
template <int L, bool RIG>
__device__ __forceinline__ int2 solveB_owned(const Bufs& b, const NbrOwned& nb, uint32_t row, uint32_t cnt,
                                             uint32_t sub, int2 pi, int32_t li, uint32_t infoI,
                                             const Flags<false>& f) {
  int32_t dpx = 0, dpy = 0;
  for (uint32_t k = sub; k < cnt; k += L * FU_B) {
    int4 o[FU_B];
#pragma unroll
    for (int j = 0; j < FU_B; ++j) o[j] = nb.rec(k + j * L < cnt ? nb.entry(row, k + j * L) : 0u);
#pragma unroll
    for (int j = 0; j < FU_B; ++j)
      if (k + j * L < cnt && !(RIG && !is_wall(o[j].w) && same_body(infoI, (uint32_t)o[j].w)))
        solveB_pair<false>(b, nb, pi, li, o[j], f, dpx, dpy);
  }
  return make_int2(gsum<L>(dpx), gsum<L>(dpy));
}

// The pred box of cell k, [lo, hi) in sorted space, by the whole CTA.
__device__ __forceinline__ void pile_box(const Bufs& b, uint32_t k, uint32_t lo, uint32_t hi, uint32_t* ws) {
  int32_t* m = reinterpret_cast<int32_t*>(ws);
  if (threadIdx.x < 4u) m[threadIdx.x] = threadIdx.x < 2u ? INT32_MAX : INT32_MIN;
  __syncthreads();
  int4 box = make_int4(INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN);
  for (uint32_t q = lo + threadIdx.x; q < hi; q += FU_T) {
    const int2 pq = ld_pred(b.PL, q);
    box = make_int4(min(box.x, pq.x), min(box.y, pq.y), max(box.z, pq.x), max(box.w, pq.y));
  }
  box.x = __reduce_min_sync(0xffffffffu, box.x);
  box.y = __reduce_min_sync(0xffffffffu, box.y);
  box.z = __reduce_max_sync(0xffffffffu, box.z);
  box.w = __reduce_max_sync(0xffffffffu, box.w);
  if ((threadIdx.x & 31u) == 0u) {
    atomicMin(m, box.x);
    atomicMin(m + 1, box.y);
    atomicMax(m + 2, box.z);
    atomicMax(m + 3, box.w);
  }
  __syncthreads();
  if (threadIdx.x == 0u) b.CB[k] = make_int4(m[0], m[1], m[2], m[3]);
  __syncthreads();
}

// L lanes share a particle's list in the sweeps over every owned particle, LC
// in the colour passes (a quarter of the particles each). RIG: the world has
// rigid bodies. A body's passes run on one CTA (the bodies dealt round), between
// barriers of their own: rigidStep before the keys, rigidSolve beside the
// friction correction, which touches other particles, rigidMember after the
// owners, who have the lists, have marked the members that leave. Twins of this
// kernel without RIG keep the bodies out of worlds that have none.
template <int L, int LC, bool RIG>
__global__ void __launch_bounds__(FU_T, 1) k_substep_fused(Bufs b, FusedPar P) {
  extern __shared__ int4 dyn[];
  int4* rec = dyn;                                              // [ownCap] records
  int2* wall = reinterpret_cast<int2*>(rec + P.ownCap);         // [ownCap] domain - WALL
  int2* swg = wall + P.ownCap;                                  // [TN]
  uint32_t* X = reinterpret_cast<uint32_t*>(swg + TN);          // [xWords]
  uint32_t* pOf = X + P.xWords;                                 // [ownCap] sorted index
  uint32_t* word = pOf + P.ownCap;                              // [ownCap] NBRN words
  uint32_t* rows = word + P.ownCap;                             // [ownCap][FU_ROW]
  __shared__ uint32_t ws[64], mask[FU_T / 32];
  __shared__ int4 smat1[MAT_MAX], smat2[MAT_MAX];
  __shared__ int2 scol[MAT_MAX];  // {eps, dpMax}
  __shared__ bool sfric[MAT_MAX];  // the row rubs or bonds
  __shared__ uint32_t dsacc[8], dsscene, lastCta;
  __shared__ int32_t rsum[RIG ? FU_T / 32 : 1][RG_SUMS];
  const Flags<false> f{b.dbg};
  const uint32_t tid = threadIdx.x, lane = tid & 31u, G = gridDim.x, cta = blockIdx.x;
  const uint32_t K = b.world->K;
  uint32_t target = 0;
  // an earlier launch gave up: its counts are not zero, and the results are void
  if (*(volatile uint32_t*)b.err & ERR_BARRIER) return;

  // ---- predict and cell counts: one slot per thread, warps dealt round the CTAs
  if (cta == 0 && tid < 8 && tid != 4) b.work[tid] = 0u;
  const uint32_t slot = ((tid >> 5) * G + cta) * 32u + lane;
  bool on = false;
  uint32_t sc = 0, key = 0, arrival = 0, info = 0;
  int2 pos = make_int2(0, 0), pred = pos;
  int32_t temp = 0;
  if (slot < P.slots) {
    sc = b.sceneOf[slot];
    const ScenePar& S = b.scenes[sc];
    const uint32_t i = slot - S.slotBase;
    on = S.active && i < S.n;
    if (on) {
      if (i == 0) b.scenes[sc].formNow = form_now(S);
      const int4* w4 = reinterpret_cast<const int4*>(b.state + (size_t)slot * 8);
      const int4 a = w4[0], c = w4[1];
      pos = make_int2(a.x, a.y);
      temp = c.z;
      info = info_of((uint32_t)c.x, (uint32_t)c.y, i >= S.nFluid);
      pred = predict_pos(b, S, slot, i, a, c, f);
    }
  }
  if constexpr (RIG) {
    const bool member = on && (info & INFO_RIGID);
    if (member) b.predSlot[slot] = pred;
    if (!grid_wait(P.bar, target)) return;
    for (uint32_t k = cta; k < P.bodies; k += G) rigid_step_body<false, FU_T, false>(b, k, rsum, f);
    if (!grid_wait(P.bar, target)) return;
    if (member) pred = b.predSlot[slot];
  }
  if (on) {
    const ScenePar& S = b.scenes[sc];
    const int2 cc = cell_coord(S, pred);
    key = key_of(S, cc.x, cc.y);
    arrival = atomicAdd(P.count + key, 1u);
  }
  for (uint32_t k = tid; k < (uint32_t)TN; k += FU_T) swg[k] = __ldg(b.WG + k);
  post1_mats(b, smat1);
  post2_mats(b, smat2);
  if (tid < (uint32_t)MAT_MAX) {
    scol[tid] = make_int2(matw(b, tid, M_eps), matw(b, tid, M_dpMax));
    if (RIG) sfric[tid] = friction_row(b, tid);
  }
  if (!grid_wait(P.bar, target)) return;

  // ---- cell ranges (every CTA its own copy), slots to their cells
  for (uint32_t k = tid; k < K; k += FU_T) X[k] = __ldcg(P.count + k);
  __syncthreads();
  const uint32_t most = cta_scan(X, K, ws);
  const bool crowded = most > CELL_BIG, piled = most > CELL_PILE;
  // this thread's cell of those the CTA looks after (one at most: the cells' words
  // fit shared memory, so no CTA of 50 or more has over FU_T) is a pile
  const auto pileHere = [&]() {
    const uint32_t k = tid * G + cta;
    return k < K && X[k + 1] - X[k] > CELL_PILE;
  };
  for (uint32_t k = cta * FU_T + tid; k <= K; k += G * FU_T) b.cellStart[k] = X[k];
  if (on) P.tmp[X[key] + arrival] = slot;
  if (!grid_wait(P.bar, target)) return;

  // ---- canonical order inside the cell, working set into sorted space
  for (uint32_t k = cta * FU_T + tid; k < K; k += G * FU_T) P.count[k] = 0u;
  if (piled) {
    each_pile(pileHere(), mask, [&](uint32_t t) {
      const uint32_t k = t * G + cta;
      rank_pile(P.tmp, X[k], X[k + 1], (P.slots + 31u) / 32u, pOf, P.ownCap * FU_TAIL_WORDS, ws);
    });
    if (!grid_wait(P.bar, target)) return;
  }
  if (on) {
    const uint32_t lo = X[key], hi = X[key + 1];
    uint32_t p = lo;
    if (hi - lo > CELL_PILE) p = P.tmp[lo + arrival] & ~RANKED;
    else
      for (uint32_t q = lo; q < hi; ++q) p += P.tmp[q] < slot ? 1u : 0u;
    const int4 r = make_int4(pred.x, pred.y, 0, (int32_t)info);
    b.PL[p] = r;
    if (info & INFO_BOUNDARY) b.PL2[p] = r;
    b.QC[p] = (info & INFO_DEAD) ? CAND_DEAD : cand_code(b.scenes[sc], pred);
    b.RX[p] = make_int4(0, 0, temp, 0);
    b.POS[p] = pos;
    b.SCN[p] = sc;
    b.inv[slot] = p;
    b.sslot[p] = slot;
    gather_flags(b, b.scenes[sc], info);
    // containStress has work: a held fluid particle
    raise_work(b, 6, !(info & INFO_BOUNDARY) && (info & INFO_PINNED));
  }
  if (!grid_wait(P.bar, target)) return;

  // ---- the owned share of each colour class
  // One contiguous share, which has the best of L1, but in worlds with bodies
  // whole rounds of a chunk to each CTA first: their members, who rub and are
  // marked, lie together, on 8 of 152 CTAs. us a substep, contiguous / chunks of
  // 32, 16, 8: the site 304 / 286, 277, 279; worlds without bodies lose (40 k
  // 139 / 141, 142, 146, 16 twins 145 / 153, 162, 178).
  uint32_t own[5], first[4], lo4[4], dealt[4];
  own[0] = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    lo4[c] = X[b.world->colourBase[c]];
    const uint32_t n = X[b.world->colourBase[c + 1]] - lo4[c];
    dealt[c] = RIG ? n / (FU_CHUNK * G) * FU_CHUNK : 0u;
    const uint32_t rest = n - dealt[c] * G, per = (rest + G - 1) / G;
    const uint32_t s0 = min(cta * per, rest), e0 = min(s0 + per, rest);
    first[c] = lo4[c] + dealt[c] * G + s0;
    own[c + 1] = own[c] + dealt[c] + (e0 - s0);
  }
  for (uint32_t i = tid; i < own[4]; i += FU_T) {
    const int c = i < own[1] ? 0 : i < own[2] ? 1 : i < own[3] ? 2 : 3;
    const uint32_t k = i - (c == 0 ? 0u : c == 1 ? own[1] : c == 2 ? own[2] : own[3]);
    const uint32_t lo = c == 0 ? lo4[0] : c == 1 ? lo4[1] : c == 2 ? lo4[2] : lo4[3];
    const uint32_t d = c == 0 ? dealt[0] : c == 1 ? dealt[1] : c == 2 ? dealt[2] : dealt[3];
    const uint32_t f0 = c == 0 ? first[0] : c == 1 ? first[1] : c == 2 ? first[2] : first[3];
    const uint32_t p = RIG && k < d ? lo + (k / FU_CHUNK * G + cta) * FU_CHUNK + k % FU_CHUNK : f0 + (k - d);
    pOf[i] = p;
    rec[i] = b.PL[p];
    const ScenePar& S = b.scenes[b.SCN[p]];
    wall[i] = make_int2(S.domW - WALL, S.domH - WALL);
  }
  // pred boxes of crowded cells (k_cellbox), one warp per cell
  if (crowded) {
    for (uint32_t k = (tid >> 5) * G + cta; k < K; k += G * (FU_T / 32)) {
      const uint32_t lo = X[k], hi = X[k + 1];
      if (hi - lo <= CELL_BIG || hi - lo > CELL_PILE) continue;
      int4 box = make_int4(INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN);
      for (uint32_t q = lo + lane; q < hi; q += 32) {
        const int2 pq = ld_pred(b.PL, q);
        box = make_int4(min(box.x, pq.x), min(box.y, pq.y), max(box.z, pq.x), max(box.w, pq.y));
      }
      box.x = __reduce_min_sync(0xffffffffu, box.x);
      box.y = __reduce_min_sync(0xffffffffu, box.y);
      box.z = __reduce_max_sync(0xffffffffu, box.z);
      box.w = __reduce_max_sync(0xffffffffu, box.w);
      if (lane == 0) b.CB[k] = box;
    }
    if (piled)
      each_pile(pileHere(), mask, [&](uint32_t t) {
        const uint32_t k = t * G + cta;
        pile_box(b, k, X[k], X[k + 1], ws);
      });
    if (!grid_wait(P.bar, target)) return;
  }
  __syncthreads();

  // ---- neighbour lists
  const uint32_t sub = tid & (L - 1);
  const bool cutLists = *(volatile uint32_t*)(b.work + 1) == 0u;
  const auto lists = [&](auto cut) {  // the stopping scan without the other's flags
    for (uint32_t i = tid / L;; i += FU_T / L) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;  // warp-uniform exit
      const bool valid = i < own[4];
      const uint32_t r = valid ? i : 0u, p = pOf[r];
      const uint32_t w = nbr_lanes<false, L, false>(
          b, X, decltype(cut)::value, valid, p, rec[r],
          [&](uint32_t at, uint32_t q, uint32_t, uint32_t) { rows[r * FU_ROW + at] = q; }, f);
      if (valid && sub == 0) {
        word[r] = w;
        b.NBRN[p] = w;
      }
    }
  };
  if (cutLists) lists(std::true_type{});
  else lists(std::false_type{});
  __syncthreads();
  int2* sca = reinterpret_cast<int2*>(X);  // the cell ranges are not read again
  for (uint32_t k = tid; k < (uint32_t)TN; k += FU_T) sca[k] = __ldg(b.CA + k);

  // ---- solver iterations
  const int32_t W0 = swg[0].x;  // the tables' first entry: luts[0]
  const bool fric = P.friction && *(volatile uint32_t*)b.work != 0u;
  for (uint32_t it = 0; it < P.iters; ++it) {
    const bool last = it + 1 == P.iters;
    NbrOwned nb{b.PL, rows, swg, sca, 0u, (uint32_t)(b.PL2 - b.PL)};
    for (uint32_t i = tid / L;; i += FU_T / L) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
      const bool valid = i < own[4];
      const uint32_t r = valid ? i : 0u;
      const int4 me = rec[r];
      const bool act = valid && !((uint32_t)me.w & INFO_BOUNDARY);
      const uint32_t cnt = act ? (word[r] & NBRN_COUNT) : 0u;
      int32_t rho = 0, S = 0, sgx = 0, sgy = 0;
      solveA_owned<L>(b, nb, r, cnt, sub, xy(me), f, rho, S, sgx, sgy);
      if (!act || sub != 0) continue;
      int32_t rinv;
      const int32_t lam =
          solveA_lambda(b, scol[(uint32_t)me.w & INFO_MAT].x, W0, rho, S, sgx, sgy, last, rinv, f);
      const uint32_t p = pOf[r];
      rec[r].z = lam;
      b.PL[p].z = lam;
      b.RX[p].x = rho;
      if (last) b.RX[p].y = rinv;
    }
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      if (!grid_wait(P.bar, target)) return;
      nb.cut = c == 0 ? lo4[0] : c == 1 ? lo4[1] : c == 2 ? lo4[2] : lo4[3];
      const uint32_t i0 = c == 0 ? own[0] : c == 1 ? own[1] : c == 2 ? own[2] : own[3];
      const uint32_t i1 = c == 0 ? own[1] : c == 1 ? own[2] : c == 2 ? own[3] : own[4];
      const uint32_t subC = tid & (LC - 1);
      for (uint32_t i = i0 + tid / LC;; i += FU_T / LC) {
        if (__shfl_sync(0xffffffffu, i, 0) >= i1) break;
        const bool valid = i < i1;
        const uint32_t r = valid ? i : i0;
        int4 me = rec[r];
        const uint32_t inf = (uint32_t)me.w;
        const bool act = valid && !(inf & INFO_BOUNDARY);
        const uint32_t cnt = act ? (word[r] & NBRN_COUNT) : 0u;
        const int2 dp =
            solveB_owned<LC, RIG>(b, nb, r, cnt, subC, xy(me), me.z, (inf & INFO_RIGID) ? inf : 0u, f);
        if (!act || subC != 0) continue;
        if (RIG && (inf & INFO_RIGID)) b.DP[pOf[r]] = dp;
        if (!(inf & INFO_PINNED)) {
          const int2 pr = apply_dp_in(scol[inf & INFO_MAT].y, wall[r], xy(me), dp, f);
          me.x = pr.x;
          me.y = pr.y;
          rec[r] = me;
        }
        b.PL2[pOf[r]] = me;
      }
    }
    swap_records(b);
    if (!grid_wait(P.bar, target)) return;
    if (fric) {
      const NbrOwned nf{b.PL, rows, swg, sca, 0u, 0u};
      // beside bodies few rows rub: their lists over as many lanes as a colour pass
      // takes, warps without one go on
      constexpr int LF = RIG ? LC : L;
      for (uint32_t i = tid / LF;; i += FU_T / LF) {
        if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
        const uint32_t r = i < own[4] ? i : 0u;
        const bool valid = i < own[4] && !(RIG && (is_wall(rec[r].w) || !sfric[(uint32_t)rec[r].w & INFO_MAT]));
        if (!RIG || __any_sync(0xffffffffu, valid))
          friction_particle<false, LF>(b, nf, valid, pOf[r], r, tid & (LF - 1), f);
      }
      if (!grid_wait(P.bar, target)) return;
      for (uint32_t i = tid; i < own[4]; i += FU_T) {
        int4 me = rec[i];
        const uint32_t inf = (uint32_t)me.w, m = inf & INFO_MAT;
        if ((inf & (INFO_BOUNDARY | INFO_PINNED)) || !friction_row(b, m)) continue;
        const uint32_t p = pOf[i];
        const int2 pr = apply_dp_in(scol[m].y, wall[i], xy(me), b.DP[p], f);
        me.x = pr.x;
        me.y = pr.y;
        rec[i] = me;
        b.PL[p] = me;
      }
    }
    if constexpr (RIG)
      for (uint32_t k = cta; k < P.bodies; k += G) rigid_solve_body<false, FU_T>(b, k, P.seal != 0u, rsum, f);
    if (RIG || fric) {
      if (!grid_wait(P.bar, target)) return;
    }
    if constexpr (RIG) {
      for (uint32_t i = tid; i < own[4]; i += FU_T) {
        if (!((uint32_t)rec[i].w & INFO_RIGID)) continue;
        const int2 pr = ld_pred(b.PL, pOf[i]);
        rec[i].x = pr.x;
        rec[i].y = pr.y;
      }
      __syncthreads();
    }
  }

  // ---- containment, then the post sweeps
  const NbrOwned nb{b.PL, rows, swg, sca, 0u, 0u};
  if (P.seal && !cutLists) {
    for (uint32_t i = tid; i < own[4]; i += FU_T) contain_particle(b, nb, pOf[i], i, f);
    if (!grid_wait(P.bar, target)) return;
  }
  for (uint32_t i = tid / L;; i += FU_T / L) {
    if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
    const bool valid = i < own[4];
    const uint32_t r = valid ? i : 0u;
    post1_particle<false, L>(b, nb, smat1, valid, pOf[r], r, sub, f);
  }
  if (!grid_wait(P.bar, target)) return;
  for (uint32_t i = tid / L;; i += FU_T / L) {
    if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
    const bool valid = i < own[4];
    const uint32_t r = valid ? i : 0u, p = pOf[r];
    bool act;
    const int2 a2 = post2_sums<false, L>(b, nb, smat2, valid, p, r, sub, act, f);
    if (act && sub == 0) {
      const uint32_t sl = b.sslot[p];
      const ScenePar& S = b.scenes[b.SCN[p]];
      post2_finish(b, S, p, sl, sl - S.slotBase, a2, !P.bonds, b.state + (size_t)sl * 8, f);
    }
  }
  const bool stress = P.seal && *(volatile uint32_t*)(b.work + 6) != 0u;
  const bool forming = P.bonds && *(volatile uint32_t*)(b.work + 5) != 0u;
  if (RIG || stress) {
    if (!grid_wait(P.bar, target)) return;
  }
  if (stress) {
    const uint32_t subC = tid & (LC - 1);
    for (uint32_t i = tid / LC;; i += FU_T / LC) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
      const uint32_t r = i < own[4] ? i : 0u;
      const bool held = i < own[4] && !is_wall(rec[r].w) && ((uint32_t)rec[r].w & INFO_PINNED);
      if (__any_sync(0xffffffffu, held)) contain_stress_slot<false, LC>(b, nb, held, b.sslot[pOf[r]], r, subC, f);
    }
    // a burst takes a member out of its body: the marks below see it
    if (RIG && !grid_wait(P.bar, target)) return;
  }
  if constexpr (RIG) {
    const uint32_t subC = tid & (LC - 1);
    for (uint32_t i = tid / LC;; i += FU_T / LC) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
      const uint32_t r = i < own[4] ? i : 0u;
      const bool member = i < own[4] && !is_wall(rec[r].w) && ((uint32_t)rec[r].w & INFO_RIGID);
      if (!__any_sync(0xffffffffu, member)) continue;
      const uint32_t p = pOf[r], sl = b.sslot[p];
      const int32_t tag = (int32_t)((uint32_t)b.state[(size_t)sl * 8 + 5] & WELD_TAG_MASK);
      const bool leaves = rigid_leaves<false, LC>(b, nb, member, sl, p, r, subC, tag, f);
      if (member && subC == 0) b.rmark[sl] = leaves ? 1u : 0u;
    }
    if (!grid_wait(P.bar, target)) return;
    for (uint32_t k = cta; k < P.bodies; k += G) rigid_member_body<false, FU_T, true>(b, k, rsum, f);
    if (!forming && !grid_wait(P.bar, target)) return;
  }
  if (forming) {
    if (!grid_wait(P.bar, target)) return;
    for (uint32_t i = tid / L;; i += FU_T / L) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
      const bool valid = i < own[4];
      const uint32_t r = valid ? i : 0u;
      form1_particle<false, L>(b, nb, valid, pOf[r], r, sub, f);
    }
    if (!grid_wait(P.bar, target)) return;
    const bool live = *(volatile uint32_t*)(b.work + 4) != 0u;
    for (uint32_t i = tid / L;; i += FU_T / L) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own[4]) break;
      const bool valid = i < own[4];
      const uint32_t r = valid ? i : 0u, p = pOf[r], sl = b.sslot[p];
      const ScenePar& S = b.scenes[b.SCN[p]];
      form2_slot<L>(b, S, valid && !is_wall(rec[r].w) && S.formNow, sl, sl - S.slotBase, sub, live);
    }
  }

  // ---- digest and chain
  __syncthreads();
  if (P.chain) {
    digest_block_begin(dsacc, &dsscene);
    const bool live = P.bonds && *(volatile uint32_t*)(b.work + 4) != 0u;
    for (uint32_t i0 = 0; i0 < own[4]; i0 += FU_T) {
      const bool valid = i0 + tid < own[4];
      uint32_t s = 0, h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (valid) {
        const uint32_t p = pOf[i0 + tid], sl = b.sslot[p];
        s = b.SCN[p];
        const uint32_t idx = sl - b.scenes[s].slotBase;
        const bool fluid = !((uint32_t)rec[i0 + tid].w & INFO_BOUNDARY);
        particle_digest(b.state + (size_t)sl * 8, idx, live && fluid ? b.bond + (size_t)sl * BOND_CAP : nullptr, h);
      }
      digest_add_block(b.acc, dsacc, &dsscene, valid, s, h);
    }
    digest_block_end(b.acc, dsacc, &dsscene);
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    lastCta = atomicAdd(P.bar.count + 1, 1u) == G - 1 ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  if (!lastCta) return;
  for (uint32_t s = tid; s < b.world->numScenes; s += FU_T) fold_scene(b, s, P.chain != 0u);
  if (tid < 2) P.bar.count[tid] = 0u;
}

}  // namespace d2
}  // namespace sn
