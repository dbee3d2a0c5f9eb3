// imc_batch.cu — batched independent 1-D gray slab problems (imc_batch_* of
// include/imcb200.h): source fill, the persistent tracking kernel with one work queue over
// every instance's histories, the comb, and the C entry points.
//
// Layout.  Instance k owns cells [cell_off[k], cell_off[k+1]) of every per-cell array and
// bank slots [slot_off[k], slot_off[k+1]) of both banks.  Its live entries this step are
// its census followed by its new particles (left face | right face | emission), so the
// flattened index space "entry q of the batch" is instance-major: entry q belongs to the
// last k with live_pref[k] <= q.  Kernels that run over entries find k by a binary search
// of the (K+1)-entry prefix held in shared memory.
//
// Equivalence with the single-problem path.  Every per-particle computation (source
// sampling, event geometry, implicit capture, tallies, weight floor, comb copies) is the
// single-problem slab code with the instance's own Philox key and the entry's index inside
// its instance as the counter, so instance k reproduces an imc_step_transport / imc_comb
// run with seed[k] (IMC/IMC1D.py:75-200 events, 319-329 boundary, 203-291 emission,
// 770-828 comb).
#include <algorithm>
#include <cmath>
#include <cstring>
#include "imc_batch.h"
#include "imc_event.cuh"
#include "imc_internal.h"
#include "imc_sample.cuh"

using namespace imcdev;
using namespace imcsample;

namespace {

enum : int { B_FLOOR = 0, B_REFLECT, B_CAP, B_ESCAPE, B_N };

// last k with pref[k] <= q; for q < pref[K] this is the instance that owns entry q
// (instances without entries share their prefix value with the next one)
__device__ __forceinline__ int find_inst(const long long* pref, int K, long long q) {
  int lo = 0, hi = K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pref[mid] <= q) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void load_pref(long long* sh, const long long* pref, int K) {
  for (int q = threadIdx.x; q <= K; q += blockDim.x) sh[q] = pref[q];
  __syncthreads();
}

// ---------------------------------------------------------------- sources
// ic = 1: the initial census (tag IC, step 0, uniform in the cell, birth time 0).
__global__ void k_bfill(BatchArgs a, int ic) {
  extern __shared__ long long pref[];
  load_pref(pref, a.new_pref, a.K);
  const long long total = pref[a.K];
  const BatchBank B = a.bank[*a.sel];
  const uint32_t step = ic ? 0u : *a.step;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += stride) {
    const int k = find_inst(pref, a.K, q);
    const long long local = q - pref[k];
    const int cb = a.cell_off[k], nc = a.cell_off[k + 1] - cb;
    const double* e1 = a.edges + cb + k;
    const uint64_t seed = a.seed[k];
    const long long b = a.slot_off[k] + a.n_census[k] + local;
    const long long n0 = a.n_side[2 * k], n1 = a.n_side[2 * k + 1];
    if (local < n0 + n1) {
      // boundary particle (IMC/IMC1D.py:319-329): at the face, mu = +-sqrt(u), t ~ U(0, dt)
      const int side = local < n0 ? 0 : 1;
      const uint32_t kk = (uint32_t)(side == 0 ? local : local - n0);
      const U4 ra = draw(seed, kk, 0, step, TAG_BOUNDARY | (uint32_t)side);
      const U4 rb = draw(seed, kk, 1, step, TAG_BOUNDARY | (uint32_t)side);
      const double mu_n = sqrt(u01d(ra.z));
      const double t = u01d(rb.x) * a.dt;
      B.p1[b] = (float)(side == 0 ? e1[0] : e1[nc]);
      B.d1[b] = (float)(side == 0 ? mu_n : -mu_n);
      B.w[b] = a.w_side[2 * k + side];
      B.t[b] = (float)t;
      B.cell[b] = side == 0 ? 0 : nc - 1;
    } else {
      // emission / initial-census particle: cell from the instance's count prefix
      const long long m = local - (n0 + n1);
      const long long* off = a.emit_off + cb + k;
      int lo = 0, hi = nc;
      while (lo < hi) { const int mid = (lo + hi) >> 1; if (off[mid + 1] <= m) lo = mid + 1; else hi = mid; }
      const int c = lo;
      const uint32_t tag = ic ? TAG_IC : TAG_EMISSION;
      const U4 r = draw(seed, (uint32_t)m, 0, step, tag);
      const U4 s = draw(seed, (uint32_t)m, 1, step, tag);
      const double u0 = u01d(r.x), u2 = u01d(r.z), u3 = u01d(r.w);
      const double s0 = u01d(s.x);
      const double ea = e1[c], eb = e1[c + 1];
      double p1 = ea + (ic ? u0 * (eb - ea) : slab_linear(eb - ea, a.tilt[cb + c], a.T[cb + c], u0));
      p1 = fmin(fmax(p1, ea), eb);
      double d1, d2;
      iso_dir(G_SLAB, u2, u3, d1, d2);
      B.p1[b] = (float)p1;
      B.d1[b] = (float)d1;
      B.w[b] = a.emit_w[cb + c];
      B.t[b] = (float)(s0 * (ic ? 0.0 : a.dt));
      B.cell[b] = c;
    }
  }
}

// per-instance sum of the tracked entries' weights (the weight floor is 1e-10 * sum / n)
// wsum[k] = sum of instance k's live weights.  Block b sums the contiguous entries
// [b*per, (b+1)*per) (coalesced, block-strided by blockDim); each thread finds its entry's
// instance once and advances it as its index passes instance boundaries (the entry space is
// instance-major), adding its partial sum to wsum when it leaves an instance and, at the end,
// through one warp-aggregated add per instance.
__global__ void __launch_bounds__(256) k_bwsum(BatchArgs a) {
  extern __shared__ long long pref[];
  __shared__ WarpStage stages[8];
  load_pref(pref, a.live_pref, a.K);
  WarpStage* st = stages + (threadIdx.x >> 5);
  const BatchBank B = a.bank[*a.sel];
  const long long total = pref[a.K];
  const long long per = (total + gridDim.x - 1) / gridDim.x;
  const long long lo = min(total, per * (long long)blockIdx.x), hi = min(total, lo + per);
  int k = lo + threadIdx.x < hi ? find_inst(pref, a.K, lo + threadIdx.x) : 0;
  long long slot0 = a.slot_off[k] - pref[k];  // bank slot of entry q is slot0 + q within instance k
  double s = 0.0;
  for (long long q = lo + threadIdx.x; q < hi; q += blockDim.x) {
    if (q >= pref[k + 1]) {  // left instance k (k < K - 1 here: q < total = pref[K])
      if (s != 0.0) atomicAdd(a.wsum + k, s);
      s = 0.0;
      do { ++k; } while (q >= pref[k + 1]);
      slot0 = a.slot_off[k] - pref[k];
    }
    const float wf = B.w[slot0 + q];
    if (wf > 0.f) s += (double)wf;
  }
  warp_tally1(s != 0.0, k, s, a.wsum, st);
}

// ---------------------------------------------------------------- tracking
// The single-problem slab kernel's histories (k_track<G_SLAB>) over every instance: the same
// flights, Philox draws and end rules, in two forms of the work distribution.
struct BHist {
  uint32_t pid, ev;              // bank slot, events so far
  float x, u, w, dcen, w_in;     // w_in: the weight the current cell visit began with
  float2 tab;                    // cell table entry
  int ci;                        // cell inside the instance
  DrawKey key;
};
struct BOut {
  bool flush, finished;  // the cell visit / the history ended
  double lost;           // the visit's deposition (flush)
  float wd;              // w*s of a flight in a cell without absorption, else 0
  float kill;            // weight of a history killed after a crossing, to the cell it entered
  int escaped;           // face an escaping history left through (its weight in esc_w), else -1
  float esc_w;
};

// One event; e: the cell's edges.  After a crossing the caller loads the new cell's table entry.
__device__ __forceinline__ void batch_event(BHist& h, BOut& o, float2 e, const U4& r, int nc, int rmask, float wfloor,
                                            unsigned* blk_cnt, int* flags, unsigned& s_cen, unsigned& s_sc) {
  o = BOut{false, false, 0.0, 0.f, 0.f, -1, 0.f};
  if (h.ev >= (1u << 30)) {
    atomicAdd(&blk_cnt[B_CAP], 1u);
    atomicOr(flags, (int)IMC_FLAG_EVENT_CAP);
    o.finished = true;
  } else {
    ++h.ev;
    const Flight f = next_flight<G_SLAB, true>(e, e, h.tab.y, h.x, 0.f, h.u, 0.f, h.dcen, r);
    const float wn = h.w * __expf(-h.tab.x * f.d);
    if (!(h.tab.x > 0.f)) o.wd = h.w * f.d;
    h.dcen -= f.d;
    s_sc += f.evt == EV_SCATTER ? 1u : 0u;
    s_cen += f.evt == EV_CENSUS ? 1u : 0u;
    h.w = wn; h.x = f.x; h.u = f.u;
    if (f.di != 0) {
      o.flush = true; o.lost = (double)h.w_in - (double)h.w;
      h.w_in = h.w;
      const int ni = h.ci + f.di;
      if ((unsigned)ni >= (unsigned)nc) {
        const int side = ni < 0 ? 0 : 1;
        if ((rmask >> side) & 1) {  // stays in its cell
          h.u = -h.u;
          atomicAdd(&blk_cnt[B_REFLECT], 1u);
        } else {
          o.escaped = side; o.esc_w = h.w;
          atomicAdd(&blk_cnt[B_ESCAPE], 1u);
          h.w = 0.f;
          o.finished = true;
        }
      } else {
        h.ci = ni;
      }
    }
    if (!o.finished && h.w < wfloor) {
      // IMC/IMC1D.py:188-195: kill and deposit the remainder in the current cell.  Without a
      // crossing in this event the visit's flush at the history end (w_in - 0) carries it; after
      // one it goes to the new cell (its intensity follows from the deposition)
      atomicAdd(&blk_cnt[B_FLOOR], 1u);
      if (o.flush) o.kill = h.w;
      h.w = 0.f;
      o.finished = true;
    }
    if (!(h.dcen > 0.f)) o.finished = true;
  }
  if (o.finished && !o.flush) { o.flush = true; o.lost = (double)h.w_in - (double)h.w; }
}

// Stores an ended history.
__device__ __forceinline__ void batch_retire(const BatchBank& B, const BHist& h) {
  B.w[h.pid] = h.w;
  if (h.w > 0.f) { B.p1[h.pid] = h.x; B.d1[h.pid] = h.u; B.cell[h.pid] = h.ci; }
}

// the block's event counts to the global ones (every thread calls it)
__device__ __forceinline__ void batch_event_counts(const BatchArgs& a, const unsigned* blk_cnt,
                                                   unsigned long long events, unsigned s_cen, unsigned s_sc) {
  __shared__ unsigned long long tot[3];
  if (threadIdx.x < 3) tot[threadIdx.x] = 0ull;
  __syncthreads();
  if (events) atomicAdd(&tot[0], events);
  const unsigned long long t_cen = warp_sum_u(s_cen), t_sc = warp_sum_u(s_sc);
  if ((threadIdx.x & 31) == 0) {
    if (t_cen) atomicAdd(&tot[1], t_cen);
    if (t_sc) atomicAdd(&tot[2], t_sc);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long cap = blk_cnt[B_CAP], bd = tot[0] - tot[1] - tot[2];
    if (tot[0] + cap) atomicAdd(a.stats + S_EVENTS, tot[0] + cap);
    if (bd) atomicAdd(a.stats + S_BOUNDARY, bd);
    if (tot[2]) atomicAdd(a.stats + S_SCATTER, tot[2]);
    if (tot[1]) atomicAdd(a.stats + S_CENSUS, tot[1]);
    if (blk_cnt[B_FLOOR]) atomicAdd(a.stats + S_FLOOR, (unsigned long long)blk_cnt[B_FLOOR]);
    if (blk_cnt[B_REFLECT]) atomicAdd(a.stats + S_REFLECT, (unsigned long long)blk_cnt[B_REFLECT]);
    if (cap) atomicAdd(a.stats + S_CAP, cap);
    if (blk_cnt[B_ESCAPE]) atomicAdd(a.stats + S_ESCAPE, (unsigned long long)blk_cnt[B_ESCAPE]);
  }
}

// Entry-queue form: persistent warps claim runs of the flattened entry index with guided atomic
// tickets; a lane that takes entry q looks up its instance once and keeps the instance's constants
// (cell and edge bases, cell count, reflect mask, weight floor, Philox key) in registers.
// refill_min: a warp refills its idle lanes once at least that many are idle (1 = at
// every event boundary), or when all are idle.
__global__ void __launch_bounds__(256) k_btrack(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned blk_cnt[B_N];
  WarpStage* stages = reinterpret_cast<WarpStage*>(smem);
  const int nwarps = blockDim.x >> 5;
  long long* pref = reinterpret_cast<long long*>(stages + nwarps);
  if (threadIdx.x < B_N) blk_cnt[threadIdx.x] = 0u;
  load_pref(pref, a.live_pref, a.K);

  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  WarpStage* st = stages + (threadIdx.x >> 5);
  const unsigned long long n = (unsigned long long)pref[a.K];
  const BatchBank B = a.bank[*a.sel];
  const uint32_t step = *a.step;
  const float dt = (float)a.dt;
  const float c_light = (float)C_LIGHT;
  const unsigned refill_min = (unsigned)max(1, min(32, a.refill_min));

  Runs run{0u, 0u};  // every run a ticket
  bool drained = false, has = false;
  BHist h{};
  uint32_t lid = 0;
  int k = 0, cb = 0, eb = 0, nc = 0, rmask = 0;
  uint64_t seed = 0;
  float wfloor = 0.f;
  double inv_q = 0.0;  // the instance's fixed-point energy quantum, inverted
  unsigned s_cen = 0, s_sc = 0;
  // events of finished histories, summed per lane while they belong to one instance (a
  // warp's claims are contiguous runs of one instance's entries) and added to the
  // instance's ledger when the instance changes: one atomic per run, not per history
  unsigned long long ev_acc = 0ull, ev_all = 0ull;
  int ev_k = 0;

  for (;;) {
    unsigned need = __ballot_sync(FULL, !has);
    if ((unsigned)__popc(need) >= refill_min) {
      while (need && !drained) {
        if (run.next >= run.end && !next_run(a.queue, a.chunk, (uint32_t)n, 0, run)) {
          drained = true;
          break;
        }
        const uint32_t avail = run.end - run.next;
        const uint32_t rank = __popc(need & lt_mask);
        if (!has && rank < avail) {
          const long long q = (long long)(run.next + rank);
          k = find_inst(pref, a.K, q);
          lid = (uint32_t)(q - pref[k]);
          h.pid = (uint32_t)(a.slot_off[k] + lid);
          h.w = B.w[h.pid];
          h.dcen = (dt - B.t[h.pid]) * c_light;
          if (h.w > 0.f && h.dcen > 0.f) {
            h.x = B.p1[h.pid]; h.u = B.d1[h.pid]; h.ci = B.cell[h.pid];
            cb = a.cell_off[k]; nc = a.cell_off[k + 1] - cb; eb = cb + k;
            rmask = a.reflect[k]; seed = a.seed[k];
            const long long nb = a.n_bank[k];
            const double W = a.wsum[k];
            wfloor = (float)(1e-10 * W / (double)(nb > 0 ? nb : 1));
            inv_q = fx_inv_quantum(W);
            h.tab = __ldg(a.sass + cb + h.ci);
            h.ev = 0;
            h.w_in = h.w;
            has = true;
          }
        }
        run.next += min((uint32_t)__popc(need), avail);
        need = __ballot_sync(FULL, !has);
      }
    }
    if (!__any_sync(FULL, has)) break;

    BOut o{};
    int cg = 0;
    if (has) {
      cg = cb + h.ci;
      const U4 r = draw(seed, lid, h.ev, step, TAG_TRANSPORT);
      const float2 e = make_float2(__ldg(a.ef + eb + h.ci), __ldg(a.ef + eb + h.ci + 1));
      batch_event(h, o, e, r, nc, rmask, wfloor, blk_cnt, a.flags, s_cen, s_sc);
      if (o.escaped >= 0) atomicAdd(a.esc_fx + 2 * k + o.escaped, fx_units((double)o.esc_w, inv_q));
      if (o.kill > 0.f) atomicAdd(a.dep_fx + cb + h.ci, fx_units((double)o.kill, inv_q));
      if (o.finished) {
        batch_retire(B, h);
        if (k != ev_k) {
          if (ev_acc) atomicAdd(a.ledger + (size_t)ev_k * IMC_BL_N + IMC_BL_EVENTS, (double)ev_acc);
          ev_k = k;
          ev_acc = 0ull;
        }
        ev_acc += h.ev;
        ev_all += h.ev;
        has = false;
      } else if (o.flush) {
        h.tab = __ldg(a.sass + cb + h.ci);
      }
    }
    // lanes of one cell share its instance's quantum
    const unsigned long long ud = o.flush ? fx_units(o.lost, inv_q) : 0ull;
    warp_tally_fx(ud != 0ull || o.wd != 0.f, cg, ud, (double)o.wd, a.dep_fx, a.si, st);
  }
  if (ev_acc) atomicAdd(a.ledger + (size_t)ev_k * IMC_BL_N + IMC_BL_EVENTS, (double)ev_acc);
  batch_event_counts(a, blk_cnt, ev_all, s_cen, s_sc);
}

// Work-unit form, for batches whose largest instance has at most IMC_BATCH_SMEM_CELLS cells.  A
// block claims a unit of consecutive entries of the batch (instance-major: one instance, or the
// end of one and the start of the next) and tracks it instance by instance with all its warps,
// each refilling idle lanes (kUnitRefillMin at a time) from a shared-memory cursor.  For the
// instance at hand the block keeps the cell table and the edges in shared memory and sums the
// deposition there (fixed point), adding it to the instance's global tally when it moves to another
// instance; w*s, only from cells without absorption, goes to global memory.
//
// A unit is 1/kUnitShare of what is left per block, at least one entry per thread and at most
// chunk x warps.  The instances differ in cost per entry by two orders of magnitude (a few events
// per history in a thin one, several hundred at a thick wave front), so whole chunks (32 entries a
// thread at the default) leave the last blocks running long after the others; units much smaller
// than these wait too often for their longest history.  Three steps of 256 instances with 5.8 M
// source particles: 28.9 ms with whole chunks, 12.9 at a share of 16, 11.8 at 32; 0.58 M: 6.8, 3.4,
// 3.4; 58 M: 115 (before this form's other changes), 96, 97.
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_down_sync(FULL, v, o);
  return v;
}

constexpr int kUnitThreads = 256;
constexpr int kUnitShare = 32;
constexpr int kUnitRefillMin = 8;

inline size_t units_smem(int M) { return (size_t)M * (8 + 8 + 8) + sizeof(WarpStage) * (kUnitThreads / 32); }

__global__ void __launch_bounds__(kUnitThreads, 1024 / kUnitThreads) k_btrack_units(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned blk_cnt[B_N];
  __shared__ unsigned long long s_base, s_cur, s_unit;
  __shared__ __align__(16) uint32_t s_rk[20];  // Philox round keys of the staged instance's seed
  const int M = a.max_cells;
  unsigned long long* TD = reinterpret_cast<unsigned long long*>(smem);                 // [M] deposition
  float2* SS = reinterpret_cast<float2*>(TD + M);                                       // [M] cell table
  float2* EF = SS + M;                                                                  // [M] edges
  WarpStage* st = reinterpret_cast<WarpStage*>(EF + M) + (threadIdx.x >> 5);
  if (threadIdx.x < B_N) blk_cnt[threadIdx.x] = 0u;

  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const unsigned long long n = (unsigned long long)a.live_pref[a.K];
  const BatchBank B = a.bank[*a.sel];
  const uint32_t step = *a.step;
  const float dt = (float)a.dt;
  const float c_light = (float)C_LIGHT;
  const unsigned long long unit = (unsigned long long)max(a.chunk, 32) * (blockDim.x >> 5);
  unsigned s_cen = 0, s_sc = 0;
  unsigned long long ev_all = 0ull;
  int cur_k = -1, cur_nc = 0, cur_cb = 0;  // block-uniform: the instance whose tallies are staged

  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(a.queue);
      const unsigned long long left = cur < n ? n - cur : 0ull;
      const unsigned long long row = blockDim.x;
      const unsigned long long u = min(unit, max(1ull, left / (kUnitShare * (unsigned long long)gridDim.x * row)) * row);
      s_unit = u;
      s_base = atomicAdd(a.queue, u);
    }
    __syncthreads();
    const unsigned long long base = s_base;
    if (base >= n) break;  // uniform: every thread read the same claim
    const unsigned long long end = min(base + s_unit, n);
    for (unsigned long long q0 = base; q0 < end;) {
      // the instance of entry q0: the last whose prefix is not past it
      int k = -1;
      for (int q = 0; q < a.K; q += blockDim.x)
        k += __syncthreads_count(q + (int)threadIdx.x < a.K &&
                                 (unsigned long long)a.live_pref[q + threadIdx.x] <= q0);
      const unsigned long long q1 = min(end, (unsigned long long)a.live_pref[k + 1]);
      if (k != cur_k) {
        // the staged tallies to the previous instance, then this instance's tables
        for (int c = threadIdx.x; c < cur_nc; c += blockDim.x)
          if (TD[c]) atomicAdd(a.dep_fx + cur_cb + c, TD[c]);
        __syncthreads();
        cur_k = k; cur_cb = a.cell_off[k]; cur_nc = a.cell_off[k + 1] - cur_cb;
        for (int c = threadIdx.x; c < cur_nc; c += blockDim.x) {
          TD[c] = 0ull;
          SS[c] = a.sass[cur_cb + c];
          EF[c] = make_float2(a.ef[cur_cb + k + c], a.ef[cur_cb + k + c + 1]);
        }
        if (threadIdx.x == 0) philox_round_keys(a.seed[k], s_rk);
      }
      if (threadIdx.x == 0) s_cur = q0;
      __syncthreads();
      // the instance's constants (block-uniform)
      const int nc = cur_nc;
      const int rmask = a.reflect[k];
      const long long nbk = a.n_bank[k];
      const double W = a.wsum[k];
      const float wfloor = (float)(1e-10 * W / (double)(nbk > 0 ? nbk : 1));
      const double inv_q = fx_inv_quantum(W);
      const uint32_t so = (uint32_t)a.slot_off[k];
      const long long pk = a.live_pref[k];
      const uint32_t rkx = draw_step_key(s_rk, step);
      unsigned long long ev_acc = 0ull;
      bool has = false, pend = false, drained = false;
      BHist h{};
      for (;;) {
        unsigned need = __ballot_sync(FULL, !has);
        if (need == FULL || (!drained && __popc(need) >= kUnitRefillMin)) {
          if (pend) { batch_retire(B, h); ev_acc += h.ev; pend = false; }
          while (need && !drained) {
            unsigned long long b0 = 0;
            if (lane == 0) b0 = atomicAdd(&s_cur, (unsigned long long)__popc(need));
            b0 = __shfl_sync(FULL, b0, 0);
            if (b0 >= q1) { drained = true; break; }
            const unsigned rank = __popc(need & lt_mask);
            if (!has && b0 + rank < q1) {
              const uint32_t lid = (uint32_t)((long long)(b0 + rank) - pk);
              h.pid = so + lid;
              h.w = B.w[h.pid];
              h.dcen = (dt - B.t[h.pid]) * c_light;
              if (h.w > 0.f && h.dcen > 0.f) {
                h.x = B.p1[h.pid]; h.u = B.d1[h.pid]; h.ci = B.cell[h.pid];
                h.tab = SS[h.ci];
                h.key = draw_key(s_rk, lid, step, TAG_TRANSPORT);
                h.ev = 0;
                h.w_in = h.w;
                has = true;
              }
            }
            need = __ballot_sync(FULL, !has);
          }
          if (need == FULL) break;
        }
        BOut o{};
        int c0 = 0;
        if (has) {
          c0 = h.ci;
          const U4 r = draw_next4(reinterpret_cast<const uint4*>(s_rk) + 1, h.key, rkx, h.ev);
          batch_event(h, o, EF[c0], r, nc, rmask, wfloor, blk_cnt, a.flags, s_cen, s_sc);
          if (o.flush) {
            const unsigned long long ud = fx_units(o.lost, inv_q);
            if (ud) smem_add_u64(TD + c0, ud);
            if (o.escaped >= 0) atomicAdd(a.esc_fx + 2 * k + o.escaped, fx_units((double)o.esc_w, inv_q));
            if (o.kill > 0.f) smem_add_u64(TD + h.ci, fx_units((double)o.kill, inv_q));
          }
          if (o.finished) { has = false; pend = true; }
          else if (o.flush) h.tab = SS[h.ci];
        }
        warp_tally1(o.wd != 0.f, cur_cb + c0, (double)o.wd, a.si, st);
      }
      // the unit's events of this instance to its ledger, one atomic per warp
      ev_all += ev_acc;
      const unsigned long long t_ev = warp_sum_u64(ev_acc);
      if (lane == 0 && t_ev) atomicAdd(a.ledger + (size_t)k * IMC_BL_N + IMC_BL_EVENTS, (double)t_ev);
      __syncthreads();  // every warp is done with s_cur and the tables of this range
      q0 = q1;
    }
  }
  for (int c = threadIdx.x; c < cur_nc; c += blockDim.x)
    if (TD[c]) atomicAdd(a.dep_fx + cur_cb + c, TD[c]);
  batch_event_counts(a, blk_cnt, ev_all, s_cen, s_sc);
}

// ---------------------------------------------------------------- comb
// ecen[c] = sum of live weights per cell (all instances)
__global__ void __launch_bounds__(256) k_bcomb_ecen(BatchArgs a) {
  extern __shared__ long long pref[];
  __shared__ WarpStage stages[8];
  load_pref(pref, a.live_pref, a.K);
  WarpStage* st = stages + (threadIdx.x >> 5);
  const BatchBank B = a.bank[*a.sel];
  const long long total = pref[a.K];
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x; base < total; base += stride) {
    const long long q = base + threadIdx.x;
    bool live = false;
    int bin = 0;
    double w = 0.0;
    if (q < total) {
      const int k = find_inst(pref, a.K, q);
      const long long pid = a.slot_off[k] + (q - pref[k]);
      const float wf = B.w[pid];
      if (wf > 0.f) { live = true; bin = a.cell_off[k] + B.cell[pid]; w = (double)wf; }
    }
    warp_tally1(live, bin, w, a.ecen, st);
  }
}

// copies per entry n = floor(w / ew + xi), xi from Philox (entry index in its instance,
// 0, step, TAG_COMB); copies per cell, per instance and per tile of BATCH_TILE entries.
// A thread takes four consecutive entries (one or two Philox blocks instead of four), its runs of one
// cell are one add to the block's table, and a tile within one instance adds its total once.  With a
// thread per entry, an FP64 division each and two warp-grouped FP64 sums: 141 -> 93 us a launch
// (256 instances, combs of 6 to 28 M entries).
constexpr int kCombThreads = BATCH_TILE / 4;
__global__ void __launch_bounds__(kCombThreads) k_bcomb_count(BatchArgs a) {
  extern __shared__ long long pref[];
  __shared__ BlockCounts<BATCH_TILE / 2> cells;
  __shared__ unsigned sh[kCombThreads / 32];
  load_pref(pref, a.live_pref, a.K);
  const BatchBank B = a.bank[*a.sel];
  const uint32_t step = *a.step;
  const long long total = pref[a.K];
  const long long ntiles = (total + BATCH_TILE - 1) / BATCH_TILE;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    counts_init(cells);
    __syncthreads();
    const long long q0 = tile * BATCH_TILE + 4 * threadIdx.x;
    const long long tend = min(total, (tile + 1) * BATCH_TILE);
    const bool one = pref[find_inst(pref, a.K, tile * BATCH_TILE) + 1] >= tend;  // block-uniform
    unsigned sum = 0;
    if (q0 < total) {
      int k = find_inst(pref, a.K, q0);
      int n[4] = {0, 0, 0, 0};
      U4 r{0u, 0u, 0u, 0u};
      long long drawn = -1;    // the Philox block r holds
      unsigned run = 0, inst = 0;  // copies of the current run of one cell, of the current instance
      int bin = -1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long q = q0 + j;
        if (q >= total) break;
        if (q >= pref[k + 1]) {
          if (!one && inst) atomicAdd(a.copies_d + k, (double)inst);
          inst = 0; drawn = -1;
          do { ++k; } while (q >= pref[k + 1]);
        }
        const long long lid = q - pref[k];
        const long long pid = a.slot_off[k] + lid;
        const float wf = B.w[pid];
        if (!(wf > 0.f)) continue;
        const int b = a.cell_off[k] + B.cell[pid];
        const double ew = a.ew[b];
        if (!(ew > 0.0)) continue;
        if ((lid >> 2) != drawn) { drawn = lid >> 2; r = draw(a.seed[k], (uint32_t)drawn, 1, step, TAG_COMB); }
        n[j] = comb_floor(wf, ew, u4_word(r, (int)(lid & 3)));
        if (b != bin) {
          if (run) counts_add(cells, bin, run, a.ncopy);
          run = 0; bin = b;
        }
        run += (unsigned)n[j]; inst += (unsigned)n[j]; sum += (unsigned)n[j];
      }
      if (run) counts_add(cells, bin, run, a.ncopy);
      if (!one && inst) atomicAdd(a.copies_d + k, (double)inst);
      if (q0 + 3 < total) *reinterpret_cast<int4*>(a.cnt + q0) = make_int4(n[0], n[1], n[2], n[3]);
      else for (int j = 0; j < 4 && q0 + j < total; ++j) a.cnt[q0 + j] = n[j];
    }
    const unsigned ws = __reduce_add_sync(FULL, sum);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = ws;
    __syncthreads();
    if (threadIdx.x == 0) {
      long long v = 0;
      for (int w = 0; w < kCombThreads / 32; ++w) v += (long long)sh[w];
      a.blk[tile] = v;
      if (one && v) atomicAdd(a.copies_d + find_inst(pref, a.K, tile * BATCH_TILE), (double)v);
    }
    counts_flush(cells, a.ncopy);
    __syncthreads();
  }
}

// exclusive scans: tile totals (output position of each tile) and copies per instance;
// the new census of each instance, capped at what its slots hold next to a step's sources
__global__ void __launch_bounds__(1024) k_bcomb_scan(BatchArgs a) {
  __shared__ long long sh[1024];
  const int t = threadIdx.x;
  const long long total = a.live_pref[a.K];
  const long long nblk = (total + BATCH_TILE - 1) / BATCH_TILE;
  auto scan = [&](long long* x, long long m) {
    const long long per = (m + 1023) / 1024;
    const long long lo = min((long long)t * per, m), hi = min(lo + per, m);
    long long s = 0;
    for (long long q = lo; q < hi; ++q) s += x[q];
    sh[t] = s;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
      const long long v = t >= d ? sh[t - d] : 0;
      __syncthreads();
      sh[t] += v;
      __syncthreads();
    }
    long long run = sh[t] - s;
    for (long long q = lo; q < hi; ++q) { const long long v = x[q]; x[q] = run; run += v; }
    if (t == 1023) x[m] = sh[1023];
    __syncthreads();
  };
  scan(a.blk, nblk);
  for (int k = t; k < a.K; k += 1024) {
    const long long c = (long long)a.copies_d[k];
    a.inst_pref[k] = c;
    long long keep = c;
    if (c > a.census_cap[k]) { atomicOr(a.flags, (int)IMC_FLAG_COMB_OVERFLOW); keep = a.census_cap[k]; }
    a.n_census[k] = keep;
  }
  __syncthreads();
  scan(a.inst_pref, a.K);
}

// Copies written in entry order into the instance's slots of the other bank.  The tile's entries are
// staged in shared memory (a thread per four entries, only those with copies); then a thread per output
// copy writes its entry's fields, so loads and stores of a warp are contiguous however many copies an
// entry makes.  Which entry a copy belongs to: a bit marks each entry's first copy (kCombWindow copies
// at a time), and the marks up to a copy count the entries with copies up to its own: one word and its
// prefix, the same for a whole warp.  With a binary search for the entry and one for its instance, and
// its fields gathered, per copy: 434 -> 169 us a
// launch (up to 22.7 M copies of 28 M entries).
constexpr int kCombWindow = 32 * kCombThreads;
size_t scatter_bytes() {
  return BATCH_TILE * (4 * sizeof(int) + sizeof(unsigned short)) + 2 * kCombThreads * sizeof(int);
}

// inclusive scan over the block's threads; every thread gets its value and the total
__device__ __forceinline__ int comb_scan(int x, int* sh, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(FULL, x, o); if (lane >= o) x += y; }
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  total = 0;
  for (int w = 0; w < kCombThreads / 32; ++w) { const int v = sh[w]; if (w < wid) x += v; total += v; }
  return x;
}

__global__ void __launch_bounds__(kCombThreads) k_bcomb_scatter(BatchArgs a) {
  extern __shared__ long long pref[];
  __shared__ int sh[3][kCombThreads / 32];
  unsigned* mark = reinterpret_cast<unsigned*>(pref + a.K + 1);
  int* before = reinterpret_cast<int*>(mark + kCombThreads);  // marks in earlier words
  float* sP = reinterpret_cast<float*>(before + kCombThreads);
  float* sD = sP + BATCH_TILE;
  float* sW = sD + BATCH_TILE;
  int* sC = reinterpret_cast<int*>(sW + BATCH_TILE);
  unsigned short* entry = reinterpret_cast<unsigned short*>(sC + BATCH_TILE);  // those with copies
  load_pref(pref, a.live_pref, a.K);
  const int sel = *a.sel;
  const BatchBank B = a.bank[sel];
  const BatchBank O = a.bank[1 - sel];
  const int lane = threadIdx.x & 31;
  const long long total = pref[a.K];
  const long long ntiles = (total + BATCH_TILE - 1) / BATCH_TILE;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long tile0 = tile * BATCH_TILE;
    const int e0 = 4 * threadIdx.x;
    const long long q0 = tile0 + e0;
    int c[4] = {0, 0, 0, 0};
    if (q0 + 3 < total) {
      const int4 v = *reinterpret_cast<const int4*>(a.cnt + q0);
      c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
    } else {
      for (int j = 0; j < 4; ++j) if (q0 + j < total) c[j] = a.cnt[q0 + j];
    }
    const int s4 = c[0] + c[1] + c[2] + c[3];
    if (s4 > 0) {
      int k = find_inst(pref, a.K, q0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c[j] == 0) continue;
        while (q0 + j >= pref[k + 1]) ++k;
        const long long pid = a.slot_off[k] + (q0 + j - pref[k]);
        const int cell = B.cell[pid];
        sP[e0 + j] = B.p1[pid]; sD[e0 + j] = B.d1[pid]; sC[e0 + j] = cell;
        sW[e0 + j] = (float)a.ew[a.cell_off[k] + cell];
      }
    }
    const int m4 = (c[0] > 0) + (c[1] > 0) + (c[2] > 0) + (c[3] > 0);
    int tot, dummy;
    const int first = comb_scan(s4, sh[0], tot) - s4;
    int rank = comb_scan(m4, sh[1], dummy) - m4;
#pragma unroll
    for (int j = 0; j < 4; ++j) if (c[j] > 0) entry[rank++] = (unsigned short)(e0 + j);
    int k = find_inst(pref, a.K, tile0);
    const bool one = pref[k + 1] >= min(total, tile0 + BATCH_TILE);  // the tile lies in one instance
    const long long out0 = a.blk[tile];
    long long dst0 = a.slot_off[k] + out0 - a.inst_pref[k];
    long long room = a.census_cap[k] - (out0 - a.inst_pref[k]);
    int marked = 0;  // marks of earlier windows
    for (int w0 = 0; w0 < tot; w0 += kCombWindow) {
      mark[threadIdx.x] = 0u;
      __syncthreads();
      int pos = first - w0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c[j] > 0 && (unsigned)pos < (unsigned)kCombWindow) atomicOr(mark + (pos >> 5), 1u << (pos & 31));
        pos += c[j];
      }
      __syncthreads();
      int in_window;
      const int pc = __popc(mark[threadIdx.x]);
      before[threadIdx.x] = marked + comb_scan(pc, sh[2], in_window) - pc;
      marked += in_window;
      __syncthreads();
      const int n_out = min(tot - w0, kCombWindow);
      for (int o = threadIdx.x; o < n_out; o += kCombThreads) {  // o % 32 == lane
        const int e = entry[before[o >> 5] + __popc(mark[o >> 5] & (FULL >> (31 - lane))) - 1];
        if (!one) {
          k = find_inst(pref, a.K, tile0 + e);
          dst0 = a.slot_off[k] + out0 - a.inst_pref[k];
          room = a.census_cap[k] - (out0 - a.inst_pref[k]);
        }
        if (w0 + o >= room) continue;  // overflow: flagged by the scan
        const long long dst = dst0 + w0 + o;
        O.p1[dst] = sP[e]; O.d1[dst] = sD[e]; O.w[dst] = sW[e]; O.t[dst] = 0.f; O.cell[dst] = sC[e];
      }
      __syncthreads();  // marks are reused, by the next window or (with the staged entries) tile
    }
    __syncthreads();  // a tile without copies too: sh is reused
  }
}

// census energy after the comb per instance: sum over cells of copies * FP32(ew)
__global__ void __launch_bounds__(256) k_bcomb_disc(BatchArgs a) {
  __shared__ WarpStage stages[8];
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  double after = 0.0;
  int k = 0;
  if (c < a.n_cells) {
    k = a.cell_inst[c];
    after = a.ncopy[c] * (double)(float)a.ew[c];
  }
  warp_tally1(after != 0.0, k, after, a.comb_after, stages + (threadIdx.x >> 5));
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

int grid_for(long long n, int block) {
  long long g = (n + block - 1) / block;
  if (g > 148LL * 16) g = 148LL * 16;
  return (int)(g < 1 ? 1 : g);
}

size_t pref_bytes(const BatchArgs& a) { return sizeof(long long) * (size_t)(a.K + 1); }

}  // namespace

cudaError_t imc_batch_launch_fill(const BatchArgs& a, int ic, long long bound, cudaStream_t s) {
  if (bound <= 0) return cudaSuccess;
  ++g_imc_launches;
  k_bfill<<<grid_for(bound, 256), 256, pref_bytes(a), s>>>(a, ic);
  return cudaGetLastError();
}

cudaError_t imc_batch_launch_wsum(const BatchArgs& a, cudaStream_t s) {
  ++g_imc_launches;
  k_bwsum<<<grid_for(a.n_slots, 256), 256, pref_bytes(a), s>>>(a);
  return cudaGetLastError();
}

cudaError_t imc_batch_launch_track(const BatchArgs& a, int block, int grid, cudaStream_t s) {
  if (block > 256) return cudaErrorInvalidConfiguration;
  ++g_imc_launches;
  if (a.form != 2 && a.max_cells > 0 && a.max_cells <= IMC_BATCH_SMEM_CELLS) {
    const size_t sh = units_smem(a.max_cells);
    const cudaError_t e = smem_opt_in<k_btrack_units>(sh);
    if (e != cudaSuccess) return e;
    const long long blocks = std::max(1LL, (long long)grid * block / kUnitThreads);
    k_btrack_units<<<(unsigned)blocks, kUnitThreads, sh, s>>>(a);
    return cudaGetLastError();
  }
  const size_t sh = (size_t)(block / 32) * sizeof(WarpStage) + pref_bytes(a);
  const cudaError_t e = smem_opt_in<k_btrack>(sh);
  if (e != cudaSuccess) return e;
  k_btrack<<<grid, block, sh, s>>>(a);
  return cudaGetLastError();
}

cudaError_t imc_batch_launch_comb_ecen(const BatchArgs& a, cudaStream_t s) {
  ++g_imc_launches;
  k_bcomb_ecen<<<grid_for(a.n_slots, 256), 256, pref_bytes(a), s>>>(a);
  return cudaGetLastError();
}

cudaError_t imc_batch_launch_comb_copy(const BatchArgs& a, cudaStream_t s) {
  const int g = (int)std::min<long long>(std::max<long long>(a.max_tiles, 1), (long long)sm_count() * 8);
  const size_t sh = pref_bytes(a) + scatter_bytes();
  cudaError_t e = smem_opt_in<k_bcomb_scatter>(sh);
  if (e != cudaSuccess) return e;
  g_imc_launches += 4;
  k_bcomb_count<<<g, kCombThreads, pref_bytes(a), s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_bcomb_scan<<<1, 1024, 0, s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_bcomb_scatter<<<g, kCombThreads, sh, s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_bcomb_disc<<<(a.n_cells + 255) / 256, 256, 0, s>>>(a);
  return cudaGetLastError();
}

// ================================================================== C entry points
namespace {

#define BCUDA(call)                                 \
  do {                                              \
    cudaError_t e__ = (call);                       \
    if (e__ != cudaSuccess) {                       \
      imc_note_cuda_error((int)e__);                \
      (void)cudaGetLastError();                     \
      return IMC_ERR_CUDA;                          \
    }                                               \
  } while (0)

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

struct BatchLayout {
  size_t cell_inst, ef, vol, sass, cellf, emit_E, emit_n, emit_off, emit_w, tilt, ecen, ew, ncopy;
  size_t n_side, w_side, n_bank, n_new, census_cap, live_pref, new_pref, inst_pref, copies_d, wsum, esc_fx, dep_fx;
  size_t comb_after, e_side, e_emit, comb_before, cnt, blk, queue, total;
  long long max_tiles;
};

BatchLayout batch_layout(const imc_batch* b) {
  BatchLayout L{};
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t r = o; o += al256(bytes); return r; };
  const size_t nc = (size_t)b->n_cells, K = (size_t)b->n_inst, ns = (size_t)std::max<int64_t>(b->n_slots, 1);
  L.max_tiles = (long long)((ns + BATCH_TILE - 1) / BATCH_TILE);
  L.cell_inst = take(4 * nc); L.ef = take(4 * (nc + K)); L.vol = take(8 * nc);
  L.sass = take(8 * nc); L.cellf = take(16 * nc); L.emit_E = take(8 * nc); L.emit_n = take(8 * nc);
  L.emit_off = take(8 * (nc + K)); L.emit_w = take(4 * nc); L.tilt = take(8 * nc);
  L.ecen = take(8 * nc); L.ew = take(8 * nc); L.ncopy = take(8 * nc);
  L.n_side = take(8 * 2 * K); L.w_side = take(4 * 2 * K); L.n_bank = take(8 * K); L.n_new = take(8 * K);
  L.census_cap = take(8 * K); L.live_pref = take(8 * (K + 1)); L.new_pref = take(8 * (K + 1));
  L.inst_pref = take(8 * (K + 1)); L.copies_d = take(8 * K); L.wsum = take(8 * K); L.esc_fx = take(8 * 2 * K); L.dep_fx = take(8 * nc);
  L.comb_after = take(8 * K); L.e_side = take(8 * 2 * K); L.e_emit = take(8 * K); L.comb_before = take(8 * K);
  L.cnt = take(4 * ns); L.blk = take(8 * ((size_t)L.max_tiles + 1)); L.queue = take(8);
  L.total = o;
  return L;
}

template <class T>
T* wp(void* ws, size_t off) { return reinterpret_cast<T*>(static_cast<char*>(ws) + off); }

BatchArgs make_args(const imc_batch* b, const imc_batch_state* s, void* ws, const BatchLayout& L) {
  BatchArgs a{};
  a.K = b->n_inst; a.n_cells = b->n_cells; a.n_slots = b->n_slots; a.max_tiles = L.max_tiles;
  a.dt = b->dt; a.theta = b->theta;
  a.cell_off = b->cell_off; a.edges = b->edges; a.slot_off = reinterpret_cast<const long long*>(b->slot_off);
  a.seed = b->seed; a.n_target = reinterpret_cast<const long long*>(b->n_target);
  a.n_boundary = reinterpret_cast<const long long*>(b->n_boundary);
  a.n_max = reinterpret_cast<const long long*>(b->n_max);
  a.face_T = b->face_T; a.reflect = b->reflect; a.op_a = b->opacity_a; a.op_p = b->opacity_p; a.cv = b->cv;
  for (int q = 0; q < 2; ++q)
    a.bank[q] = BatchBank{s->bank[q].pos1, s->bank[q].dir1, s->bank[q].weight, s->bank[q].time, s->bank[q].cell};
  a.sel = s->sel; a.step = s->step; a.n_census = reinterpret_cast<long long*>(s->n_census);
  a.T = s->T; a.e = s->e; a.tr = s->tr; a.dep = s->dep; a.si = s->si; a.emitted = s->emitted;
  a.ledger = s->ledger; a.stats = s->stats; a.flags = s->flags;
  a.cell_inst = wp<int>(ws, L.cell_inst); a.ef = wp<float>(ws, L.ef); a.vol = wp<double>(ws, L.vol);
  a.sass = wp<float2>(ws, L.sass); a.cellf = wp<double2>(ws, L.cellf); a.emit_E = wp<double>(ws, L.emit_E);
  a.emit_n = wp<long long>(ws, L.emit_n); a.emit_off = wp<long long>(ws, L.emit_off);
  a.emit_w = wp<float>(ws, L.emit_w); a.tilt = wp<double>(ws, L.tilt);
  a.ecen = wp<double>(ws, L.ecen); a.ew = wp<double>(ws, L.ew); a.ncopy = wp<double>(ws, L.ncopy);
  a.n_side = wp<long long>(ws, L.n_side); a.w_side = wp<float>(ws, L.w_side);
  a.n_bank = wp<long long>(ws, L.n_bank); a.n_new = wp<long long>(ws, L.n_new);
  a.census_cap = wp<long long>(ws, L.census_cap); a.live_pref = wp<long long>(ws, L.live_pref);
  a.new_pref = wp<long long>(ws, L.new_pref); a.inst_pref = wp<long long>(ws, L.inst_pref);
  a.copies_d = wp<double>(ws, L.copies_d); a.wsum = wp<double>(ws, L.wsum);
  a.esc_fx = wp<unsigned long long>(ws, L.esc_fx); a.dep_fx = wp<unsigned long long>(ws, L.dep_fx);
  a.comb_after = wp<double>(ws, L.comb_after); a.e_side = wp<double>(ws, L.e_side);
  a.e_emit = wp<double>(ws, L.e_emit); a.comb_before = wp<double>(ws, L.comb_before);
  a.cnt = wp<int>(ws, L.cnt); a.blk = wp<long long>(ws, L.blk); a.queue = wp<unsigned long long>(ws, L.queue);
  a.chunk = 1024; a.refill_min = 1;
  a.max_cells = b->max_cells;
  return a;
}

constexpr int kMaxInstances = 4096;

imc_status batch_check(const imc_batch* b, const imc_batch_state* s, void* ws, size_t wsb) {
  if (!b || !s || !ws) return IMC_ERR_INVALID_ARG;
  if (b->n_inst < 1 || b->n_inst > kMaxInstances || b->n_cells < b->n_inst || b->n_slots < 1) return IMC_ERR_INVALID_ARG;
  if (b->n_slots >= (1LL << 31) || b->max_new < 0 || !(b->dt > 0.0)) return IMC_ERR_INVALID_ARG;
  if (!b->cell_off || !b->edges || !b->slot_off || !b->seed || !b->n_target || !b->n_boundary || !b->n_max ||
      !b->face_T || !b->reflect || !b->opacity_a || !b->opacity_p || !b->cv)
    return IMC_ERR_INVALID_ARG;
  for (int q = 0; q < 2; ++q) {
    const imc_bank& k = s->bank[q];
    if (!k.pos1 || !k.dir1 || !k.weight || !k.time || !k.cell || k.capacity < b->n_slots) return IMC_ERR_INVALID_ARG;
  }
  if (!s->sel || !s->step || !s->n_census || !s->T || !s->e || !s->tr || !s->dep || !s->si || !s->emitted ||
      !s->ledger || !s->stats || !s->flags)
    return IMC_ERR_INVALID_ARG;
  if (wsb < batch_layout(b).total) return IMC_ERR_WORKSPACE;
  return IMC_OK;
}

int track_grid(const imc_batch_launch* l, int* block) {
  int bs = (l && l->block_size > 0) ? l->block_size : 256;
  bs = std::max(32, std::min(256, bs / 32 * 32));
  const int bps = (l && l->blocks_per_sm > 0) ? l->blocks_per_sm : 4;
  *block = bs;
  return sm_count() * bps;
}

}  // namespace

extern "C" {

size_t imc_batch_workspace_bytes(const imc_batch* b) {
  if (!b || b->n_inst < 1 || b->n_cells < 1) return 0;
  return batch_layout(b).total;
}

imc_status imc_batch_init(const imc_batch* b, imc_batch_state* s, const double* T0, const double* Tr0,
                          void* workspace, size_t workspace_bytes, void* stream) {
  imc_status st = batch_check(b, s, workspace, workspace_bytes);
  if (st != IMC_OK) return st;
  if (!T0 || !Tr0) return IMC_ERR_INVALID_ARG;
  cudaStream_t cs = (cudaStream_t)stream;
  const BatchLayout L = batch_layout(b);
  BatchArgs a = make_args(b, s, workspace, L);
  BCUDA(cudaMemsetAsync(s->sel, 0, sizeof(int32_t), cs));
  BCUDA(cudaMemsetAsync(s->step, 0, sizeof(uint32_t), cs));
  BCUDA(cudaMemsetAsync(s->flags, 0, sizeof(int32_t), cs));
  BCUDA(cudaMemsetAsync(s->stats, 0, sizeof(unsigned long long) * IMC_STAT_N, cs));
  BCUDA(cudaMemsetAsync(s->n_census, 0, sizeof(int64_t) * b->n_inst, cs));
  BCUDA(cudaMemsetAsync(s->dep, 0, sizeof(double) * b->n_cells, cs));
  BCUDA(cudaMemsetAsync(s->si, 0, sizeof(double) * b->n_cells, cs));
  BCUDA(cudaMemsetAsync(s->emitted, 0, sizeof(double) * b->n_cells, cs));
  BCUDA(cudaMemsetAsync(s->tr, 0, sizeof(double) * b->n_cells, cs));
  BCUDA(imc_batch_launch_setup(a, T0, cs));
  BCUDA(imc_batch_launch_ic_plan(a, Tr0, cs));
  BCUDA(imc_batch_launch_prefix(a, cs));
  long long bound = 0;
  {
    // host bound of the initial census: n_target + nc per instance
    bound = b->max_new;
  }
  BCUDA(imc_batch_launch_fill(a, 1, bound, cs));
  BCUDA(imc_batch_launch_ledger(a, 1, cs));
  BCUDA(imc_batch_launch_material_fleck(a, 0, cs));
  int flags = 0;
  BCUDA(cudaMemcpyAsync(&flags, s->flags, sizeof(int), cudaMemcpyDeviceToHost, cs));
  BCUDA(cudaStreamSynchronize(cs));
  if (flags & IMC_FLAG_COMB_OVERFLOW) return IMC_ERR_BANK_OVERFLOW;
  if (flags & IMC_FLAG_NONFINITE) return IMC_ERR_NONFINITE;
  return IMC_OK;
}

imc_status imc_batch_step(const imc_batch* b, imc_batch_state* s, const imc_batch_launch* launch, void* workspace,
                          size_t workspace_bytes, void* stream) {
  imc_status st = batch_check(b, s, workspace, workspace_bytes);
  if (st != IMC_OK) return st;
  cudaStream_t cs = (cudaStream_t)stream;
  const BatchLayout L = batch_layout(b);
  BatchArgs a = make_args(b, s, workspace, L);
  if (launch && launch->chunk > 0) a.chunk = launch->chunk;
  if (launch && launch->refill_min > 0) a.refill_min = std::min(32, launch->refill_min);
  if (launch) a.form = launch->form;
  int block = 256;
  const int grid = track_grid(launch, &block);
  BCUDA(imc_batch_launch_plan(a, cs));
  BCUDA(imc_batch_launch_prefix(a, cs));
  BCUDA(imc_batch_launch_fill(a, 0, b->max_new, cs));
  BCUDA(imc_batch_launch_wsum(a, cs));
  BCUDA(imc_batch_launch_track(a, block, grid, cs));
  BCUDA(imc_batch_launch_material_fleck(a, 1, cs));
  BCUDA(imc_batch_launch_comb_ecen(a, cs));
  BCUDA(imc_batch_launch_comb_plan(a, cs));
  BCUDA(imc_batch_launch_comb_copy(a, cs));
  BCUDA(imc_batch_launch_ledger(a, 0, cs));
  return IMC_OK;
}

}  // extern "C"
