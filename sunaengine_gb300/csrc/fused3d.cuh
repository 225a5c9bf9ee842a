// The whole 3D substep of a small world as one cooperative launch: the phases of
// sim3d.cuh with grid barriers between them, as fused2d.cuh does it in 2D. One CTA
// per SM owns an equal contiguous share of sorted space and keeps its particles'
// neighbour lists, positions and tags in shared memory with the kernel tables.
//
// The grid is a counting sort. A 3D box has more cells than a CTA can scan by
// itself (23,520 in the page's, 140,608 in the largest), so each CTA scans its
// slice of the cells and publishes the slice's total; every CTA then has the 152
// totals and with them every slice's base. Arrival order inside a cell is what the
// count's atomics gave; each particle ranks itself among its cell's slots, which
// puts the cell into the canonical ascending order.
//
// The sums are the per-phase kernels' own device functions: results are equal
// word by word. Every wait is bounded (grid_wait).
//
// Measured at 4 iterations (us a substep, the per-phase graph it replaced -> this):
// 4 k particles 88 -> 39, 16 k 100 -> 50, 60 k 146 -> 82, 91 k 236 -> 144, 125 k 277 ->
// 168; the limit is what fits an SM (fused_fits).
#pragma once
#include "gridsync.cuh"
#include "sim3d.cuh"

namespace sn {
namespace d3 {

constexpr uint32_t F3_ROW = 52;  // words per list row (see FU_ROW)
constexpr uint32_t F3_OWN_BYTES = 16 + 4 + 4 + 4 * F3_ROW;
constexpr uint32_t F3_TAIL_WORDS = 2 + F3_ROW;  // of these, what nothing uses before the owned share is known
constexpr uint32_t F3_MAX_GRID = 256;  // CTAs whose totals a CTA keeps
constexpr int F3_B = 3;                // neighbours' records in flight

struct Fused3Par {
  uint32_t iters, chain;
  uint32_t slots;     // slots that can be active: [0, slots)
  uint32_t slice;     // cells a CTA scans, at most FU_T
  uint32_t ownCap;    // particles a CTA can own
  uint32_t* count;    // [K] cell counts, zero between launches
  uint32_t* local;    // [K] cell starts inside their slice
  uint32_t* totals;   // [grid] particles of each slice
  uint32_t* tmp;      // slots by cell in arrival order
  GridBar bar;        // count[0] barrier arrivals, count[1] finished CTAs, zero between launches
};

// Particle s's list by L lanes (a warp calls it together; `valid` false for a lane
// group with none), the hits to out(position, sorted index); returns the count.
// The nine rows of the stencil are dealt to the lanes in order, and a prefix over
// the lanes places each row's hits.
template <int L, class OUT>
__device__ __forceinline__ uint32_t nbr_rows(const Bufs3& b, bool valid, uint32_t s, int4 me, OUT out) {
  const uint32_t sub = threadIdx.x & (L - 1);
  const Scene3& S = b.scenes[valid ? scene_of_tag((uint32_t)me.w) : 0u];
  const int32_t cx = me.x >> HSHIFT, cy = me.y >> HSHIFT, cz = me.z >> HSHIFT;
  const int32_t x0 = max(cx - 1, 0), x1 = min(cx + 1, (int32_t)S.gx - 1);
  uint32_t n = 0;
  for (uint32_t r0 = 0; r0 < 9u; r0 += L) {
    const int32_t r = (int32_t)(r0 + sub), z = cz + r / 3 - 1, y = cy + r % 3 - 1;
    uint32_t lo = 0, hi = 0;
    if (valid && r < 9 && z >= 0 && z < (int32_t)S.gz && y >= 0 && y < (int32_t)S.gy) {
      const uint32_t row = S.keyOff + ((uint32_t)z * S.gy + (uint32_t)y) * S.gx;
      lo = b.cellStart[row + x0];
      hi = b.cellStart[row + x1 + 1];
    }
    // the first two filter words are kept, a longer row's others found again
    const uint32_t base = lo & ~3u;
    uint32_t m[2] = {0u, 0u}, mine = 0;
    if (lo < hi) {
      m[0] = cand_row<4>(b.QC, b.PW, base, lo, hi, s, me);
      if (base + 32u < hi) m[1] = cand_row<4>(b.QC, b.PW, base + 32u, lo, hi, s, me);
      mine = (uint32_t)(__popc(m[0]) + __popc(m[1]));
      // (past MAXNBR the count no longer matters)
      for (uint32_t c = base + 64u; c < hi && mine < MAXNBR; c += 32u)
        mine += (uint32_t)__popc(cand_row<4>(b.QC, b.PW, c, lo, hi, s, me));
    }
    uint32_t inc = mine;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o, L);
      if (sub >= (uint32_t)o) inc += v;
    }
    uint32_t at = n + inc - mine;
    n += __shfl_sync(0xffffffffu, inc, L - 1, L);
    if (lo < hi)
      for (uint32_t c = base; c < hi && at < MAXNBR; c += 32u) {
        uint32_t w = c == base ? m[0] : c == base + 32u ? m[1] : cand_row<4>(b.QC, b.PW, c, lo, hi, s, me);
        for (; w && at < MAXNBR; ++at) {
          const uint32_t j = (uint32_t)__clz((int)w);
          w ^= 0x80000000u >> j;
          out(at, c + j);
        }
      }
    if (!__any_sync(0xffffffffu, valid && n < MAXNBR)) break;
  }
  return valid ? min(n, MAXNBR) : 0u;
}

template <int L>
__global__ void __launch_bounds__(FU_T, 1) k3_substep_fused(Bufs3 b, Fused3Par P) {
  extern __shared__ int4 dyn[];
  int4* rec = dyn;                                             // [ownCap] {position, tag}
  int2* swg = reinterpret_cast<int2*>(rec + P.ownCap);         // [LUT_N]
  int2* spg = swg + LUT_N;                                     // [PLANE_N]
  int32_t* lamS = reinterpret_cast<int32_t*>(spg + PLANE_N);   // [ownCap]
  uint32_t* cntS = reinterpret_cast<uint32_t*>(lamS + P.ownCap);  // [ownCap]
  uint32_t* rows = cntS + P.ownCap;                            // [ownCap][F3_ROW]
  __shared__ uint32_t ws[64], mask[FU_T / 32], X[FU_T + 1], bases[F3_MAX_GRID + 1];
  __shared__ uint32_t dsacc[8], dsscene, lastCta;
  const Flags<false> f{b.dbg};
  const uint32_t tid = threadIdx.x, lane = tid & 31u, G = gridDim.x, cta = blockIdx.x;
  const uint32_t K = b.world->K;
  uint32_t target = 0;
  // an earlier launch gave up: its counts are not zero, and the results are void
  if (*(volatile uint32_t*)P.bar.err & ERR_BARRIER) return;

  // ---- predict and cell counts: one slot per thread, warps dealt round the CTAs
  const uint32_t slot = ((tid >> 5) * G + cta) * 32u + lane;
  bool on = false;
  uint32_t key = 0, arrival = 0;
  int4 pr = make_int4(0, 0, 0, 0);
  if (slot < P.slots) {
    const uint32_t sc = b.sceneOf[slot];
    on = sc != NO_SCENE && slot - b.scenes[sc].slotBase < b.scenes[sc].n;
    if (on) {
      pr = predict_record(b, b.scenes[sc], sc, slot, f);
      key = key_of(b.scenes[sc], pr);
      arrival = atomicAdd(P.count + key, 1u);
    }
  }
  for (uint32_t k = tid; k < (uint32_t)LUT_N; k += FU_T) swg[k] = __ldg(b.WG + k);
  if (tid < (uint32_t)PLANE_N) spg[tid] = __ldg(b.PG + tid);
  if (!grid_wait(P.bar, target)) return;

  // ---- cell starts inside this CTA's slice of the cells
  const uint32_t c0 = min(cta * P.slice, K), cn = min(P.slice, K - c0);
  if (tid < cn) X[tid] = __ldcg(P.count + c0 + tid);
  __syncthreads();
  const uint32_t most = cta_scan(X, cn, ws);
  if (tid < cn) P.local[c0 + tid] = X[tid];
  if (tid == 0) P.totals[cta] = X[cn] | (most > CELL_PILE ? RANKED : 0u);
  if (!grid_wait(P.bar, target)) return;

  // ---- every slice's base; slots to their cells
  const uint32_t total = tid < G ? __ldcg(P.totals + tid) : 0u;
  if (tid < G) bases[tid] = total & ~RANKED;
  const bool piled = __syncthreads_or((int)(total & RANKED)) != 0;  // some slice has a pile
  cta_scan(bases, G, ws);
  if (tid < cn) {
    b.cellStart[c0 + tid] = bases[cta] + X[tid];
    P.count[c0 + tid] = 0u;
  }
  if (cta == 0 && tid == 0) b.cellStart[K] = bases[G];
  const uint32_t place = on ? bases[key / P.slice] + __ldcg(P.local + key) + arrival : 0u;
  if (on) P.tmp[place] = slot;
  if (!grid_wait(P.bar, target)) return;

  // ---- canonical order inside the cell, working set into sorted space
  if (piled) {
    each_pile(tid < cn && X[tid + 1] - X[tid] > CELL_PILE, mask, [&](uint32_t t) {
      rank_pile(P.tmp, bases[cta] + X[t], bases[cta] + X[t + 1], (P.slots + 31u) / 32u,
                reinterpret_cast<uint32_t*>(lamS), P.ownCap * F3_TAIL_WORDS, ws);
    });
    if (!grid_wait(P.bar, target)) return;
  }
  if (on) {
    const uint32_t lo = b.cellStart[key], hi = b.cellStart[key + 1];
    uint32_t p = lo;
    if (hi - lo > CELL_PILE) p = P.tmp[place] & ~RANKED;
    else
      for (uint32_t q = lo; q < hi; ++q) p += P.tmp[q] < slot ? 1u : 0u;
    b.PW[p] = pr;
    b.QC[p] = cand_code(pr);
    b.inv[slot] = p;
    b.sslot[p] = slot;
  }
  if (!grid_wait(P.bar, target)) return;

  // ---- the owned share; neighbour lists
  const uint32_t nAct = bases[G], per = (nAct + G - 1) / G;
  const uint32_t p0 = min(cta * per, nAct), own = min(per, nAct - p0);
  const uint32_t sub = tid & (L - 1);
  for (uint32_t i = tid / L;; i += FU_T / L) {
    if (__shfl_sync(0xffffffffu, i, 0) >= own) break;  // warp-uniform exit
    const bool valid = i < own;
    const uint32_t r = valid ? i : 0u;
    const int4 me = b.PW[p0 + r];
    const uint32_t n =
        nbr_rows<L>(b, valid, p0 + r, me, [&](uint32_t at, uint32_t q) { rows[r * F3_ROW + at] = q; });
    if (valid && sub == 0) {
      rec[r] = me;
      cntS[r] = n;
      b.NBRN[p0 + r] = n;
    }
  }
  __syncthreads();

  // ---- solver iterations
  const int32_t W0 = swg[0].x;
  int4 *cur = b.PW, *nxt = b.PW2;
  for (uint32_t it = 0; it < P.iters; ++it) {
    for (uint32_t i = tid / L;; i += FU_T / L) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own) break;
      const bool valid = i < own;
      const uint32_t r = valid ? i : 0u, cnt = valid ? cntS[r] : 0u;
      const int4 me = rec[r];
      int32_t rho = 0, St = 0, sgx = 0, sgy = 0, sgz = 0;
      for (uint32_t k = sub; k < cnt; k += L * F3_B) {
        int4 o[F3_B];
#pragma unroll
        for (int j = 0; j < F3_B; ++j) o[j] = cur[k + j * L < cnt ? rows[r * F3_ROW + k + j * L] : 0u];
#pragma unroll
        for (int j = 0; j < F3_B; ++j)
          if (k + j * L < cnt) density_pair(swg, me, o[j], rho, St, sgx, sgy, sgz, f);
      }
      rho = gsum3<L>(rho);
      St = gsum3<L>(St);
      sgx = gsum3<L>(sgx);
      sgy = gsum3<L>(sgy);
      sgz = gsum3<L>(sgz);
      if (!valid || sub != 0) continue;
      const int32_t lam = density_lambda(b, spg, W0, me, rho, St, sgx, sgy, sgz, f);
      lamS[r] = lam;
      b.PL[p0 + r] = make_int4(me.x, me.y, me.z, lam);
    }
    if (!grid_wait(P.bar, target)) return;
    const bool last = it + 1 == P.iters;
    for (uint32_t i = tid / L;; i += FU_T / L) {
      if (__shfl_sync(0xffffffffu, i, 0) >= own) break;
      const bool valid = i < own;
      const uint32_t r = valid ? i : 0u, cnt = valid ? cntS[r] : 0u;
      int4 me = rec[r];
      const int32_t tag = me.w;
      me.w = lamS[r];
      int32_t ax = 0, ay = 0, az = 0;
      for (uint32_t k = sub; k < cnt; k += L * F3_B) {
        int4 o[F3_B];
#pragma unroll
        for (int j = 0; j < F3_B; ++j) o[j] = b.PL[k + j * L < cnt ? rows[r * F3_ROW + k + j * L] : 0u];
#pragma unroll
        for (int j = 0; j < F3_B; ++j) {
          int32_t tx, ty, tz;
          if (k + j * L < cnt && dp_term(swg, me, o[j], tx, ty, tz, f)) {
            ax = wadd(ax, tx);
            ay = wadd(ay, ty);
            az = wadd(az, tz);
          }
        }
      }
      ax = gsum3<L>(ax);
      ay = gsum3<L>(ay);
      az = gsum3<L>(az);
      if (!valid || sub != 0) continue;
      const int3 np = solve_place(b, spg, me, tag, p0 + r, ax, ay, az, f);
      rec[r] = make_int4(np.x, np.y, np.z, tag);
      if (!last) nxt[p0 + r] = rec[r];
    }
    int4* t = cur;
    cur = nxt;
    nxt = t;
    if (!last && !grid_wait(P.bar, target)) return;
  }

  // ---- integrate (3d/sim3d.wgsl:542-552), digest and chain
  __syncthreads();
  if (P.chain) d2::digest_block_begin(dsacc, &dsscene);
  for (uint32_t i0 = 0; i0 < own; i0 += FU_T) {
    const bool valid = i0 + tid < own;
    uint32_t sc = 0, h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (valid) {
      const int4 q = rec[i0 + tid];
      const uint32_t sl = b.sslot[p0 + i0 + tid];
      sc = scene_of_tag((uint32_t)q.w);
      int4* w4 = reinterpret_cast<int4*>(b.state + (size_t)sl * 8);
      const int4 p = w4[0];
      const int4 np = make_int4(q.x, q.y, q.z, p.w);
      const int4 v = make_int4(sub_sat(q.x, p.x, f), sub_sat(q.y, p.y, f), sub_sat(q.z, p.z, f), 0);
      w4[0] = np;
      w4[1] = v;
      const int32_t w8[8] = {np.x, np.y, np.z, np.w, v.x, v.y, v.z, 0};
      if (P.chain) d2::particle_digest(w8, sl - b.scenes[sc].slotBase, nullptr, h);
    }
    if (P.chain) d2::digest_add_block(b.acc, dsacc, &dsscene, valid, sc, h);
  }
  if (P.chain) d2::digest_block_end(b.acc, dsacc, &dsscene);
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    lastCta = atomicAdd(P.bar.count + 1, 1u) == G - 1 ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  if (!lastCta) return;
  for (uint32_t s = tid; s < b.world->numScenes; s += FU_T) fold_scene3(b, s, P.chain != 0u);
  if (tid < 2) P.bar.count[tid] = 0u;
}

}  // namespace d3
}  // namespace sn
