// imc_transport.cu — event-based tracking of a census/source bank to census.
//
// Reference behaviour (per event and per history):
//   slab   IMC/IMC1D.py:75-130 (move_particle), 133-200 (move_particles)
//   sphere IMC/IMC1D.py:336-436, 439-532
//   xy/rz  IMC/IMC2D.py:711-935 (events), 938-1107 (history loop)
//   multigroup  MG_IMC/MG_IMC2D.py:580-989 (xy, rz), MG_IMC/MG_IMC1D.py:276-461 (sphere)
//
// Execution model: a persistent grid of the blocks that are resident.  Each warp keeps 32
// histories in registers, from a run of bank indices: its first one is dealt to it, later ones
// are guided atomic tickets (imc_event.cuh, Runs).  An event advances every live lane (distance
// to face / effective scatter / census, implicit capture w *= exp(-sigma_a s)); lanes whose
// history ended wait until kRefillMin of the warp are idle, then are stored and refilled
// together, so warps do not carry dead lanes until the bank drains (the in-warp form of bank
// compaction between events).  Particle state is FP32; energy removed from a history is
// accounted as the exact FP64 difference of its FP32 weights while it stays in one cell, and
// flushed in fixed point when it leaves, into one of the tallies below.  Random numbers: Philox
// keyed by the run seed, counter (id_base + bank index, event number, step, TAG_TRANSPORT).
#include <algorithm>

#include "imc_event.cuh"
#include "imc_internal.h"

using namespace imcdev;

namespace {

// Block-level counters for rare events (shared-memory atomics keep them out of registers).
enum : int { B_FLOOR = 0, B_REFLECT, B_CAP, B_ESCAPE, B_CAPTURE, B_N };

// MG: group-indexed tables and tallies, escaped energy also by group.  In 2-D the rules of
// MG_IMC/MG_IMC2D.py:580-989 (no effective-scatter cap, no absorption for sigma_a <= 1e-12,
// the weight floor ends a history after its event is committed); on the 1-D sphere those of
// MG_IMC/MG_IMC1D.py:276-461, which are the gray spherical ones (cap, floor kill with local
// deposit) with the floor coefficient 1e-14.
// CF: Carter-Forest (IMC/IMC1D_CarterForest.py:63-331, 614-820; IMC/IMC2D_CarterForest.py:
// 102-508).  The table holds (0, sigma_a): the flight samples the absorption distance in the
// scatter slot (same threshold and cap) and captures nothing on the way; at an absorption the
// photon is re-emitted in the new direction the event drew after a delay ~ Exp(cf_rate) if that
// falls inside the step, else captured (its weight deposited).  Histories at or below the
// weight floor are not moved (they stay in census).
// One event of one history (distance to the cell boundary / effective scatter / census,
// implicit capture, crossing with reflection or escape, weight floor, events cap) and, when
// the history ends, its final state written back to the bank.  Shared by the persistent
// kernel k_track (the history in registers, refilled in-warp) and the event-by-event kernel
// k_event (the history in device arrays, survivors compacted between launches): both follow
// a history through the same arithmetic and the same Philox draws.
struct Hist {
  uint32_t pid, ev;
  float x, y, u, v, w, dcen, w_in;
  int ci, cj, grp;
  float2 tab;      // cell table entry of the current (group, cell)
  DrawKey key;     // the history's part of its Philox draws
};
struct EvOut {
  int cell;        // (group, cell) index of the cell the event took place in
  bool flush;      // its visit ends: deposition `lost`
  float wd;        // w*s of the flight in a cell without absorption (else 0)
  double lost;
  bool finished;   // the history ended: history_retire stores its final state
};

// EDGES: E1, E2 hold the edges in shared memory (else they are read from the FP32 copies through L1)
template <int GEOM, bool SMEM_CELLS, bool MG, bool CF, bool EDGES>
__device__ __forceinline__ void history_event(const TrackArgs& a, Hist& h, EvOut& o, const float2* E1,
                                              const float2* E2, const float2* CS, unsigned* blk_cnt,
                                              unsigned long long* blk_esc, unsigned long long* dep_t,
                                              const U4& r, float weight_floor,
                                              double inv_q, unsigned& s_cen, unsigned& s_sc) {
  constexpr bool ONED = GEOM == G_SLAB || GEOM == G_SPHERE;
  constexpr bool MG2 = MG && !ONED;  // MG_IMC2D history rules
  const float c_light = (float)C_LIGHT;
  auto table = [&](int cq) { return SMEM_CELLS ? CS[cq] : __ldg(a.sass + cq); };
  const float x = h.x, y = h.y, u = h.u, v = h.v, w = h.w;
  const int c = h.ci + a.nx * h.cj;
  const int cq = MG ? c + a.nc * h.grp : c;  // (group, cell) table / tally index
  o.cell = cq;
  const float sa = h.tab.x, ss = h.tab.y;
  bool finished = false;
  if (h.ev >= (uint32_t)a.max_events) {
    // events-per-history cap (IMC/IMC2D.py:974-977): stops, weight stays in census
    atomicAdd(&blk_cnt[B_CAP], 1u);
    if (!a.cap_is_reference) atomicOr(a.flags, (int)IMC_FLAG_EVENT_CAP);
    finished = true;
  } else {
    ++h.ev;
    const float2 e1 = cell_edges<EDGES>(E1, a.e1, h.ci);
    const float2 e2 = ONED ? make_float2(0.f, 0.f) : cell_edges<EDGES>(E2, a.e2, h.cj);
    const Flight f = next_flight<GEOM, !MG2>(e1, e2, ss, x, y, u, v, h.dcen, r);
    const float d = f.d;
    const int evt = f.evt, di = f.di, dj = f.dj;
    // implicit capture (the energy removed is counted at the flush, w_in - w)
    const float wn = (MG2 && !(sa > 1e-12f)) ? w : w * __expf(-sa * d);
    // path-length intensity: w*s is needed only in cells without absorption (table
    // entry 0: below the estimator's threshold, or Carter-Forest); elsewhere it is
    // lost / (sigma_a V dt), formed from the deposition tally when the step ends
    if (!(sa > 0.f)) o.wd = w * d;
    h.dcen -= d;
    bool captured = false;
    if (CF && evt == EV_SCATTER) {
      // absorption (IMC/IMC1D_CarterForest.py:146-194, IMC/IMC2D_CarterForest.py:189-210)
      const float rate = __ldg(a.cf_rate + c);
      const float tr = h.dcen / c_light;  // time left after the flight
      const uint32_t ub = ONED ? r.z : r.w;
      if (!(rate > 0.f)) {
        captured = !ONED;  // no re-emission: 1-D redirects, 2-D captures
      } else if (a.cf_fastpath > 0.f && tr > 1e-14f && rate * tr > a.cf_fastpath) {
        captured = u01f(ub) < __expf(-rate * tr);
      } else {
        const float delay = fdiv(neglog_u(ub), rate);
        if (ONED ? (tr > 1e-14f && delay < tr) : (delay < tr - 1e-15f)) h.dcen = fmaxf(0.f, (tr - delay) * c_light);
        else captured = true;
      }
      // a capture deposits the whole weight: w becomes 0 below, so w_in - w includes it
      if (captured) atomicAdd(&blk_cnt[B_CAPTURE], 1u);
    }
    // crossings are counted as the events that are nothing else
    s_sc += evt == EV_SCATTER && !captured ? 1u : 0u;
    s_cen += evt == EV_CENSUS ? 1u : 0u;

    if (!MG && !CF && !ONED && wn <= weight_floor) {
      // IMC/IMC2D.py:1043-1047: history stops in place keeping its weight
      atomicAdd(&blk_cnt[B_FLOOR], 1u);
      h.w = wn;
      finished = true;
    } else {
      h.w = captured ? 0.f : wn; h.x = f.x; h.y = f.y; h.u = f.u; h.v = f.v;
      if (CF && captured) finished = true;
      if ((di | dj) != 0) {
        // leaving the cell: flush the visit (before an escape zeroes w) and start the next
        o.flush = true; o.lost = (double)h.w_in - (double)h.w;
        h.w_in = h.w;
        const int ni = h.ci + di, nj = h.cj + dj;
        if ((unsigned)ni >= (unsigned)a.nx || (unsigned)nj >= (unsigned)a.ny) {
          const int side = ni < 0 ? 0 : ni >= a.nx ? 1 : nj < 0 ? 2 : 3;
          if ((a.reflect_mask >> side) & 1) {  // stays in its cell
            if (side < 2) h.u = -h.u; else h.v = -h.v;
            atomicAdd(&blk_cnt[B_REFLECT], 1u);
          } else {
            const unsigned long long uw = fx_units((double)h.w, inv_q);
            atomicAdd(&blk_esc[side], uw);
            if (MG) atomicAdd(a.esc_fx + 4 + h.grp, uw);
            atomicAdd(&blk_cnt[B_ESCAPE], 1u);
            h.w = 0.f;
            finished = true;
          }
        } else {
          h.ci = ni; h.cj = nj;
          h.tab = table(cq + di + a.nx * dj);
        }
      }
      if (ONED) {
        if (!CF && !finished && h.w < weight_floor) {
          // IMC/IMC1D.py:188-195: kill and deposit the remainder in the current cell
          // (every cell, including the two edge cells the reference skips).  Without a
          // crossing in this event the visit's flush at the history end (w_in - 0) carries
          // it; after one, the old cell holds the flush slot and the remainder is added to
          // the new cell here.  Its intensity share, lost / (sigma_a V dt), follows from the
          // deposition tally.
          atomicAdd(&blk_cnt[B_FLOOR], 1u);
          if (o.flush) {
            const int c2 = h.ci + a.nx * h.cj + (MG ? a.nc * h.grp : 0);
            atomicAdd(dep_t + c2, fx_units((double)h.w, inv_q));
          }
          h.w = 0.f;
          finished = true;
        }
      } else if (MG2 && !finished && h.dcen > 0.f && h.w <= weight_floor) {
        // MG_IMC/MG_IMC2D.py:858-860: the next event would stop at the floor (a weight
        // that underflowed to 0 included)
        atomicAdd(&blk_cnt[B_FLOOR], 1u);
        finished = true;
      } else if (!finished && !(h.w > 0.f)) {
        h.w = 0.f;
        finished = true;
      }
      if (!(h.dcen > 0.f)) finished = true;
    }
  }
  // A history that ends without leaving its cell flushes that cell's visit now.  (One
  // that ended by crossing has already queued the old cell and holds nothing new: a
  // 1-D weight-floor kill after a crossing deposits directly.)
  if (finished && !o.flush) { o.flush = true; o.lost = (double)h.w_in - (double)h.w; }
  o.finished = finished;
}

// Stores the final state of an ended history.  True when it ended alive, its weight then
// belonging to the comb's census sums in bin `cen_bin`.
template <int GEOM>
__device__ __forceinline__ bool history_retire(const TrackArgs& a, const Hist& h, int& cen_bin) {
  a.w[h.pid] = h.w;
  if (!(h.w > 0.f)) return false;
  // census, cap and frozen histories keep their (pre-event, when frozen) state
  const int c = h.ci + a.nx * h.cj;
  a.p1[h.pid] = h.x; a.d1[h.pid] = h.u;
  if (GEOM == G_XY || GEOM == G_RZ) { a.p2[h.pid] = h.y; a.d2[h.pid] = h.v; }
  a.cell[h.pid] = c;
  cen_bin = c + (a.ecen_by_group ? a.nc * h.grp : 0);
  return true;
}

// The block's event counts and escaped energy to the global ones (every thread calls it; ends
// with the block synchronised): events, scatters and census events from the threads' own
// counters, the rare ones from blk_cnt; crossings are the events that are none of those.
__device__ __forceinline__ void add_event_counts(const TrackArgs& a, const unsigned* blk_cnt,
                                                 const unsigned long long* blk_esc, unsigned s_ev, unsigned s_cen,
                                                 unsigned s_sc) {
  __shared__ unsigned long long tot[3];
  if (threadIdx.x < 3) tot[threadIdx.x] = 0ull;
  __syncthreads();
  const unsigned long long t_ev = warp_sum_u(s_ev), t_cen = warp_sum_u(s_cen), t_sc = warp_sum_u(s_sc);
  if ((threadIdx.x & 31) == 0) {
    if (t_ev) atomicAdd(&tot[0], t_ev);
    if (t_cen) atomicAdd(&tot[1], t_cen);
    if (t_sc) atomicAdd(&tot[2], t_sc);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long cap = blk_cnt[B_CAP], capt = blk_cnt[B_CAPTURE];
    const unsigned long long bd = tot[0] - tot[1] - tot[2] - capt;
    if (tot[0] + cap) atomicAdd(a.stats + S_EVENTS, tot[0] + cap);
    if (bd) atomicAdd(a.stats + S_BOUNDARY, bd);
    if (tot[2]) atomicAdd(a.stats + S_SCATTER, tot[2]);
    if (tot[1]) atomicAdd(a.stats + S_CENSUS, tot[1]);
    if (capt) atomicAdd(a.stats + S_CAPTURE, capt);
    if (blk_cnt[B_FLOOR]) atomicAdd(a.stats + S_FLOOR, (unsigned long long)blk_cnt[B_FLOOR]);
    if (blk_cnt[B_REFLECT]) atomicAdd(a.stats + S_REFLECT, (unsigned long long)blk_cnt[B_REFLECT]);
    if (cap) atomicAdd(a.stats + S_CAP, cap);
    if (blk_cnt[B_ESCAPE]) atomicAdd(a.stats + S_ESCAPE, (unsigned long long)blk_cnt[B_ESCAPE]);
  }
  if (threadIdx.x < 4 && blk_esc[threadIdx.x] != 0ull) atomicAdd(a.esc_fx + threadIdx.x, blk_esc[threadIdx.x]);
}

// Where a cell visit's deposition (fixed point) and path-length intensity (FP64) are summed:
//   T_GLOBAL  global memory, the warp's lanes grouped by cell first (one reduction per cell)
//   T_SMALL   both per block in shared memory, added to the global ones at the block's end
//   T_WIDE    one block per SM (kWideThreads at most) with the step's main tally per (group, cell)
//             in shared memory: the deposition, or with Carter-Forest the intensity (nothing is
//             deposited in flight there); the other tally, rare, goes to global memory
// Grouping lanes by cell costs a warp-wide match and a serial sum over each group's lanes at nearly
// every event; a shared-memory atomic per flushing lane does not.  T_SMALL serves meshes whose
// tallies fit beside each of several blocks an SM; T_WIDE every mesh whose one tally fits in an
// SM's shared memory once (26 thousand entries).  The ten launches of a crooked-pipe run
// (60 x 210, up to 8.7 M histories and 68 M segments a launch): 18.6 ms with T_GLOBAL at the
// default launch shape, 12.6 ms with T_WIDE.
//
// Ended histories wait until kRefillMin lanes of the warp are idle; then their final states and
// census sums are stored and the lanes refilled in one go, so this part runs once per kRefillMin
// endings instead of whenever any lane ends (at about 8 segments per history, nearly every
// event): the same ten launches 14.5 ms at 1, 13.2 at 4, 12.6 at 8, 12.6 at 12; with the flights as
// they are now 11.9, 10.8, 10.2 (and 10.3 at 16).  Eight launches of a multigroup slab, a million
// particles each: 5.9, 5.5, 5.4 (5.8 at 16); four of a sphere, a million each: 9.0, 8.9, 9.3 (10.4);
// slabs of 4 thousand to 4 million, banks of 20 thousand and larger meshes: within 1 % from 1 to 16.
constexpr int kRefillMin = 8;
constexpr int kWideThreads = 1024;
//   T_LONG    as T_GLOBAL, on a mesh so long that its edges (8 bytes a cell) in shared memory would leave
//             fewer blocks resident (edges_pay): they are read through L1.  Slabs of 14, 20 and 28 thousand
//             cells, three steps of a million particles: 23.2, 23.5 and 23.8 ms with the edges staged in
//             the one block that then fits an SM, 9.6, 9.7 and 9.8 so
enum : int { T_GLOBAL = 0, T_SMALL, T_WIDE, T_HASH, T_LONG };
constexpr bool wide_block(int tally) { return tally == T_WIDE || tally == T_HASH; }

// T_HASH, for meshes past T_WIDE: one wide block per SM keeps the sums of the (group, cell) entries
// its histories touch in an open table in shared memory (deposition, and census energy for the comb).
// An entry takes the first free of kHashProbes slots; one that finds none adds to global memory.
// With T_GLOBAL the adds of every warp meet at the few entries where the radiation is, and the L2
// slices that hold those serve one add after another, loads of other warps waiting behind them: a
// ten-group crooked pipe (126 thousand entries, 2.1 M histories of 1.2 events) spent 255 us a launch
// at 19 % of its issue slots, 56 MB of DRAM traffic.  So, an SM adds once per entry and launch:
// 16 launches 3.12 -> 1.45 ms, 2 M particles a step 9.2 -> 3.1 ms; one group, 200 x 400 cells, 2 M
// particles 21.6 -> 17.5 ms (20.6 with 4096 slots), 140 x 210 cells, 500 thousand 4.2 -> 3.2 ms.
// It takes its start and end (164 KB cleared, then read) to earn: below a history or two per lane
// T_GLOBAL's smaller blocks are as fast or faster (200 x 400 cells at 30 thousand particles a step
// 0.92 against 1.04 ms, 100 thousand 1.65 against 1.70, 200 thousand 2.61 against 2.40).
constexpr int kHashSlots = 8192, kHashProbes = 4;
constexpr uint32_t kHashPerLane = 2;  // histories per lane from which T_HASH is taken
struct HashTally {
  unsigned long long* dep;
  double* cen;
  int* key;
};
__device__ __forceinline__ HashTally hash_tally(void* p) {
  unsigned long long* d = static_cast<unsigned long long*>(p);
  double* c = reinterpret_cast<double*>(d + kHashSlots);
  return HashTally{d, c, reinterpret_cast<int*>(c + kHashSlots)};
}
__device__ __forceinline__ int hash_slot(const HashTally& t, int entry) {
  const unsigned h = ((unsigned)entry * 2654435761u) >> 8;
#pragma unroll 1
  for (int p = 0; p < kHashProbes; ++p) {
    const int q = (int)((h + (unsigned)p) & (unsigned)(kHashSlots - 1));
    int k = *(volatile int*)(t.key + q);
    if (k == entry) return q;
    if (k == -1) {
      k = atomicCAS(t.key + q, -1, entry);
      if (k == -1 || k == entry) return q;
    }
  }
  return -1;
}
// Census energy of the warp's lanes (all call it), grouped by entry first: the table's FP64 add is a
// compare-and-swap loop, which lanes of one entry would take in turn.
__device__ __forceinline__ void hash_census(const HashTally& t, bool flush, int entry, double v, double* global,
                                            WarpStage* st) {
  if (__ballot_sync(FULL, flush) == 0u) return;
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(FULL, flush ? entry : -1 - lane);
  st->a[lane] = v;
  __syncwarp();
  if (flush && (__ffs(peers) - 1) == lane) {
    double sum = 0.0;
    unsigned m = peers;
    while (m) { const int l = __ffs(m) - 1; m &= m - 1; sum += st->a[l]; }
    const int q = hash_slot(t, entry);
    if (q >= 0) atomicAdd(t.cen + q, sum);
    else atomicAdd(global + entry, sum);
  }
  __syncwarp();
}

template <int GEOM, bool SMEM_CELLS, bool MG, bool CF, int TALLY>
__global__ void __launch_bounds__(wide_block(TALLY) ? kWideThreads : 256, wide_block(TALLY) ? 1 : 4) k_track(TrackArgs a) {
  pdl_wait();     // the previous kernel of the stream has completed
  pdl_trigger();  // the next one may be scheduled
  const float dtk = a.dt_dev ? (float)*a.dt_dev : a.dt;  // graph replay: step length and Philox
  const uint32_t stepk = a.step_dev ? *a.step_dev : a.step;  // step counter from device memory
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned blk_cnt[B_N];
  __shared__ unsigned long long blk_esc[4];
  constexpr bool ONED = GEOM == G_SLAB || GEOM == G_SPHERE;
  constexpr bool MG2 = MG && !ONED;  // MG_IMC2D history rules
  constexpr bool TD_S = TALLY == T_SMALL || (TALLY == T_WIDE && !CF);  // deposition in shared memory
  constexpr bool TS_S = TALLY == T_SMALL || (TALLY == T_WIDE && CF);   // intensity in shared memory
  WarpStage* stages = reinterpret_cast<WarpStage*>(smem);
  const int nwarps = blockDim.x >> 5;
  float2* E1 = reinterpret_cast<float2*>(stages + nwarps);  // (lower, upper) edge per index
  float2* E2 = E1 + a.nx;
  float2* CS = E2 + a.ny;
  constexpr bool EDGES = TALLY != T_LONG;
  const int ncg = a.nc * a.ng;
  unsigned long long* TD = reinterpret_cast<unsigned long long*>(CS + (SMEM_CELLS ? ncg : 0));
  double* TS = reinterpret_cast<double*>(TD + (TD_S ? ncg : 0));
  unsigned long long* const dep_t = TD_S ? TD : a.dep_fx;
  if (EDGES) {
    for (int q = threadIdx.x; q < a.nx; q += blockDim.x) E1[q] = make_float2(a.e1[q], a.e1[q + 1]);
    for (int q = threadIdx.x; q < a.ny; q += blockDim.x) E2[q] = make_float2(a.e2[q], a.e2[q + 1]);
  }
  if (SMEM_CELLS)
    for (int q = threadIdx.x; q < ncg; q += blockDim.x) CS[q] = a.sass[q];
  if (TD_S) for (int q = threadIdx.x; q < ncg; q += blockDim.x) TD[q] = 0ull;
  if (TS_S) for (int q = threadIdx.x; q < ncg; q += blockDim.x) TS[q] = 0.0;
  const HashTally HT = hash_tally(TD);
  if (TALLY == T_HASH)
    for (int q = threadIdx.x; q < kHashSlots; q += blockDim.x) { HT.dep[q] = 0ull; HT.cen[q] = 0.0; HT.key[q] = -1; }
  if (threadIdx.x < B_N) blk_cnt[threadIdx.x] = 0u;
  if (threadIdx.x < 4) blk_esc[threadIdx.x] = 0ull;
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  WarpStage* st = stages + (threadIdx.x >> 5);
  const uint32_t n = (uint32_t)*a.n_dev;

  // T_SMALL: events between two looks at the idle lanes (1 in the checked build, which looks at every
  // history before every event).  Tracking with 1, these, and twice as many: twenty steps of a 4k slab
  // 4.08, 3.90, 3.84 ms, 40k 6.77, 6.59, 6.53, three of a 4M slab (short histories) 1.34, 1.43, 1.65;
  // eight of a 1M multigroup slab 5.70, 5.42, 5.28; five of a 1M 40 x 40 mesh 1.76, 1.68, 1.71.
#ifdef IMC_CHECKED
  constexpr int kEvents = 1;
#else
  constexpr int kEvents = ONED ? 4 : 2;
#endif
  Runs run = first_run(n, a.sms);  // warp-uniform
  bool drained = false;
  bool has = false, pend = false;  // pend: an ended history whose final state is not stored yet
  Hist h;
  h.pid = 0; h.ev = 0; h.x = h.y = h.u = h.v = h.w = h.dcen = h.w_in = 0.f;
  h.ci = h.cj = h.grp = 0; h.tab = make_float2(0.f, 0.f); h.key = DrawKey{0u, 0u, 0u};
  const uint32_t rkx = draw_step_key(a.rk, stepk);
  auto table = [&](int cq) { return SMEM_CELLS ? CS[cq] : __ldg(a.sass + cq); };
  unsigned s_ev = 0, s_cen = 0, s_sc = 0;  // events of ended histories, census events, scatters
  unsigned n_alive = 0;                 // entries alive at the end (census sums for the comb)
  const float c_light = (float)C_LIGHT;
  // weight floor, IMC/IMC1D.py:1007 / IMC/IMC2D.py:1771 (1e-10); MG_IMC/MG_IMC1D.py:1127 (1e-14)
  const float weight_floor = (float)(a.floor_coef * (*a.wsum) / (double)(n > 0 ? n : 1));
  const double inv_q = fx_inv_quantum(*a.wsum);  // fixed-point energy tallies
  const float inv_nx = 1.0f / (float)a.nx;  // cell -> (i, j) at refill without an integer divide

  for (;;) {
    unsigned need = __ballot_sync(FULL, !has);
    if (need == FULL || (!drained && __popc(need) >= kRefillMin)) {
      // ---------------- store the ended histories, refill from the warp's run ----------------
      bool cen = false;
      int cen_bin = 0;
      if (pend) { cen = history_retire<GEOM>(a, h, cen_bin); s_ev += h.ev; }
      if (a.ecen) {
        // (the table's entries are (group, cell): a multigroup census summed by cell alone goes past it)
        if (TALLY == T_HASH && (!MG || a.ecen_by_group)) hash_census(HT, cen, cen_bin, (double)h.w, a.ecen, st);
        else warp_tally1(cen, cen_bin, (double)h.w, a.ecen, st);
        n_alive += cen ? 1u : 0u;
      }
      pend = false;
      while (need && !drained) {
        if (run.next >= run.end && !next_run(a.queue, a.chunk, n, a.sms, run)) { drained = true; break; }
        const uint32_t avail = run.end - run.next;
        const uint32_t rank = __popc(need & lt_mask);
        if (!has && rank < avail) {
          h.pid = run.next + rank;
          h.w = a.w[h.pid];
          h.dcen = (dtk - a.t[h.pid]) * c_light;
          const bool moves = (MG2 || CF ? h.w > weight_floor : h.w > 0.f) && h.dcen > 0.f;
          if (!moves && h.w > 0.f && a.ecen) {
            // not tracked but alive: part of the census the comb sees
            const int b = a.cell[h.pid] + (a.ecen_by_group ? a.nc * a.group[h.pid] : 0);
#ifdef IMC_CHECKED
            if (b >= 0 && b < a.nc * (a.ecen_by_group ? a.ng : 1))
#endif
            { atomicAdd(a.ecen + b, (double)h.w); ++n_alive; }
          }
          if (moves) {
            h.x = a.p1[h.pid]; h.u = a.d1[h.pid];
            if (MG) h.grp = a.group[h.pid];
            if (GEOM == G_XY || GEOM == G_RZ) { h.y = a.p2[h.pid]; h.v = a.d2[h.pid]; }
            const int c = a.cell[h.pid];
#ifdef IMC_CHECKED
            // bounds-checked build: an entry outside the mesh (or group range), or with a
            // non-finite weight, is reported and left untouched
            if (c < 0 || c >= a.nc || (MG && (h.grp < 0 || h.grp >= a.ng)) || !isfinite(h.w)) {
              atomicOr(a.flags, (int)IMC_FLAG_BOUNDS);
            } else
#endif
            {
              // j from a float estimate, corrected to the exact quotient (the estimate is off
              // by at most one for any int c)
              h.cj = __float2int_rd(((float)c + 0.5f) * inv_nx);
              h.ci = c - h.cj * a.nx;
              if (h.ci < 0) { --h.cj; h.ci += a.nx; } else if (h.ci >= a.nx) { ++h.cj; h.ci -= a.nx; }
              h.tab = table(MG ? c + a.nc * h.grp : c);
              h.ev = 0;
              h.w_in = h.w;
              h.key = draw_key(a.rk, a.id_base + h.pid, stepk, TAG_TRANSPORT);
              has = true;
            }
          }
        }
        run.next += min((uint32_t)__popc(need), avail);
        need = __ballot_sync(FULL, !has);
      }
      if (need == FULL) break;
    }
#ifdef IMC_CHECKED
    if (has && (h.ci < 0 || h.ci >= a.nx || h.cj < 0 || h.cj >= a.ny || !isfinite(h.w) || !isfinite(h.x) ||
                !isfinite(h.dcen))) {
      atomicOr(a.flags, (int)IMC_FLAG_BOUNDS);
      has = false;  // nothing more is tallied at an invalid index
    }
#endif
    if (TALLY == T_SMALL) {
      // Carter-Forest adds w*s at every flight, and its absorptions keep histories where they started
      // (a warp's are neighbours in the bank): the first live lane's cell is probably several lanes'.
      // One cell, four steps of 500 thousand histories: an add per lane 1.10 ms, by groups of lanes
      // found with a match (the earlier form) 0.88, so 0.53; 50 cells 0.82, 0.68, 0.54; 1000 closed
      // cells, where few lanes share one, 5.2, 6.8, 5.5.
      int hot = -1;
      if (CF) {
        const unsigned live = __ballot_sync(FULL, has);
        if (live) hot = __shfl_sync(FULL, h.ci + a.nx * h.cj, __ffs(live) - 1);
      }
#pragma unroll 1
      for (int rep = 0; rep < kEvents; ++rep) {
        EvOut o{0, false, 0.f, 0.0, false};
        if (has) {
          history_event<GEOM, SMEM_CELLS, MG, CF, true>(a, h, o, E1, E2, CS, blk_cnt, blk_esc, dep_t,
                                                        draw_next(a.rk, h.key, rkx, h.ev), weight_floor, inv_q, s_cen,
                                                        s_sc);
          if (o.finished) { has = false; pend = true; }
        }
        __syncwarp();  // the warp together again: lanes left apart run the next event one by one
        const unsigned long long ud = o.flush ? fx_units(o.lost, inv_q) : 0ull;
        if (ud) smem_add_u64(TD + o.cell, ud);
        if (CF) smem_tally_hot(o.wd != 0.f, o.cell, (double)o.wd, TS, hot);
        else if (o.wd != 0.f) atomicAdd(TS + o.cell, (double)o.wd);
        __syncwarp();
      }
      continue;
    }
    EvOut o{0, false, 0.f, 0.0, false};
    if (has) {
      history_event<GEOM, SMEM_CELLS, MG, CF, EDGES>(a, h, o, E1, E2, CS, blk_cnt, blk_esc, dep_t,
                                                     draw_next(a.rk, h.key, rkx, h.ev), weight_floor, inv_q, s_cen,
                                                     s_sc);
      if (o.finished) { has = false; pend = true; }
    }
    // ---------------- tallies ----------------
    // deposited energy in fixed point when a cell visit ends; w*s (raw, only from cells without
    // absorption) in FP64 at every flight
    const unsigned long long ud = o.flush ? fx_units(o.lost, inv_q) : 0ull;
    const double vs = (double)o.wd;
    if (TD_S && ud) smem_add_u64(TD + o.cell, ud);
    if (TS_S && o.wd != 0.f) atomicAdd(TS + o.cell, vs);
    if (TALLY == T_HASH) {
      if (ud) {
        const int q = hash_slot(HT, o.cell);
        if (q >= 0) smem_add_u64(HT.dep + q, ud);
        else atomicAdd(a.dep_fx + o.cell, ud);
      }
      warp_tally1(o.wd != 0.f, o.cell, vs, a.si, st);
    } else if (TALLY == T_GLOBAL || TALLY == T_LONG) warp_tally_fx(ud != 0ull || o.wd != 0.f, o.cell, ud, vs, a.dep_fx, a.si, st);
    else if (!TD_S) warp_tally_fx(ud != 0ull, o.cell, ud, 0.0, a.dep_fx, a.si, st);
    else if (!TS_S) warp_tally1(o.wd != 0.f, o.cell, vs, a.si, st);
  }

  // ---------------- statistics ----------------
  if (a.ecen) {
    const unsigned long long t_alive = warp_sum_u(n_alive);
    if (lane == 0 && t_alive) atomicAdd(a.n_live, t_alive);
  }
  add_event_counts(a, blk_cnt, blk_esc, s_ev, s_cen, s_sc);
  // the block's tallies (every warp's last flush is behind the __syncthreads above)
  if (TALLY == T_HASH)
    for (int q = threadIdx.x; q < kHashSlots; q += blockDim.x) {
      const int e = HT.key[q];
      if (e < 0) continue;
      if (HT.dep[q]) atomicAdd(a.dep_fx + e, HT.dep[q]);
      if (HT.cen[q] != 0.0) atomicAdd(a.ecen + e, HT.cen[q]);
    }
  if (TD_S) for (int q = threadIdx.x; q < ncg; q += blockDim.x) if (TD[q]) atomicAdd(a.dep_fx + q, TD[q]);
  if (TS_S) for (int q = threadIdx.x; q < ncg; q += blockDim.x) if (TS[q] != 0.0) atomicAdd(a.si + q, TS[q]);
}

// dynamic shared memory of the tracking kernels: per-warp staging, edges, the cell table and
// `tallies` 8-byte block tallies per (group, cell)
inline size_t stage_smem(int block) { return (size_t)(block / 32) * sizeof(WarpStage); }
inline size_t track_smem(const TrackArgs& a, int block, bool cells, int tallies) {
  size_t sh = stage_smem(block) + sizeof(float2) * ((size_t)a.nx + a.ny);
  if (cells) sh += sizeof(float2) * a.nc * a.ng;
  return sh + 8ull * tallies * a.nc * a.ng;
}

template <auto Kernel>
cudaError_t launch_sized(const TrackArgs& a, int block, int bps, size_t sh, cudaStream_t s) {
  const cudaError_t e = smem_opt_in<Kernel>(sh);
  if (e != cudaSuccess) return e;
  IMC_LAUNCH_PDL(Kernel, a.sms * resident_blocks<Kernel>(bps, block, sh), block, sh, s, a);
  return cudaGetLastError();
}

// Whether edges in shared memory, `sh` bytes a block with the rest, leave room for `want` blocks an SM
// (228 KB, a block's own share 1 KB and its static bytes).
inline bool edges_pay(size_t sh, int want) { return (size_t)std::max(1, want) * (sh + 1280) <= 228 * 1024; }

// T_SMALL is built only with the shared-memory cell table (small meshes).  Tallies or a table that were
// asked for and fit by themselves, but not beside a long mesh's edges, are left in global memory.
template <int GEOM, bool MG, bool CF = false>
cudaError_t launch_geom(const TrackArgs& a, const TrackLaunch& l, cudaStream_t s) {
  const int block = l.block;
  const size_t edges = track_smem(a, block, false, 0) - stage_smem(block);
  auto fits = [&](bool cells, int tallies) { return track_smem(a, block, cells, tallies) <= kSmemPerBlock; };
  auto asked = [&](bool cells, int tallies) {  // (what cannot fit without the edges fails at the launch)
    return fits(cells, tallies) || track_smem(a, block, cells, tallies) - edges > kSmemPerBlock;
  };
  const bool sm = l.smem_cells, st = l.smem_tally && asked(true, 2);
  // One wide block per SM holding as many threads as the requested shape keeps resident there,
  // when its tally fits; the cell table beside it if that fits too (else it is read through L1,
  // which measured the same on the crooked pipe).
  const int wide = std::max(128, std::min(kWideThreads, block * l.blocks_per_sm)) & ~31;
  if (!st && l.wide_ok && block <= 256 && track_smem(a, wide, false, 1) <= kSmemPerBlock) {
    if (sm && track_smem(a, wide, true, 1) <= kSmemPerBlock)
      return launch_sized<k_track<GEOM, true, MG, CF, T_WIDE>>(a, wide, 1, track_smem(a, wide, true, 1), s);
    return launch_sized<k_track<GEOM, false, MG, CF, T_WIDE>>(a, wide, 1, track_smem(a, wide, false, 1), s);
  }
  if constexpr (!CF) {
    const size_t sh = track_smem(a, wide, false, 0) + 20 * (size_t)kHashSlots;
    if (!st && l.wide_ok && block <= 256 && sh <= kSmemPerBlock &&
        l.n_bound >= (long long)kHashPerLane * l.sms * wide)
      return launch_sized<k_track<GEOM, false, MG, CF, T_HASH>>(a, wide, 1, sh, s);
  }
  if (sm && st) return launch_sized<k_track<GEOM, true, MG, CF, T_SMALL>>(a, block, l.blocks_per_sm, track_smem(a, block, true, 2), s);
  if (sm && asked(true, 0))
    return launch_sized<k_track<GEOM, true, MG, CF, T_GLOBAL>>(a, block, l.blocks_per_sm, track_smem(a, block, true, 0), s);
  if (edges_pay(track_smem(a, block, false, 0), std::min(l.blocks_per_sm, 1024 / block)))
    return launch_sized<k_track<GEOM, false, MG, CF, T_GLOBAL>>(a, block, l.blocks_per_sm, track_smem(a, block, false, 0), s);
  return launch_sized<k_track<GEOM, false, MG, CF, T_LONG>>(a, block, l.blocks_per_sm, stage_smem(block), s);
}

// ---------------------------------------------------------------------------------
// Event-by-event form (the textbook event-based loop): one launch advances every live
// history by one event; the histories still alive are compacted into the next launch's list.
// The history state lives in the bank (position, direction, weight, cell) and in scratch
// arrays (event count, distance to census, weight at the visit's start, w*s); the physics is
// history_event, so a history follows exactly the path and draws it follows in k_track.
// ---------------------------------------------------------------------------------
struct EventScratch {
  uint32_t* live[2];        // lists of live bank indices
  unsigned* count;          // [2] their lengths
  uint32_t* ev; float* dcen; float* w_in; // [capacity]
};

// The histories that move (as k_track's refill decides) into list 0, with their scratch state.
template <bool MG2CF>
__global__ void k_event_init(TrackArgs a, EventScratch e) {
  const float dtk = a.dt_dev ? (float)*a.dt_dev : a.dt;
  const uint32_t n = (uint32_t)*a.n_dev;
  const float weight_floor = (float)(a.floor_coef * (*a.wsum) / (double)(n > 0 ? n : 1));
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t trips = (n + stride - 1) / stride;  // uniform: every lane reaches the ballot
  for (uint32_t it = 0; it < trips; ++it) {
    const uint32_t k = it * stride + blockIdx.x * blockDim.x + threadIdx.x;
    bool moves = false;
    if (k < n) {
      const float w = a.w[k];
      const float dc = (dtk - a.t[k]) * (float)C_LIGHT;
      moves = (MG2CF ? w > weight_floor : w > 0.f) && dc > 0.f;
      if (moves) { e.ev[k] = 0u; e.dcen[k] = dc; e.w_in[k] = w; }
    }
    const unsigned m = __ballot_sync(FULL, moves);
    unsigned base = 0;
    if (lane == 0 && m) base = atomicAdd(e.count, (unsigned)__popc(m));
    base = __shfl_sync(FULL, base, 0);
    if (moves) e.live[0][base + __popc(m & ((1u << lane) - 1u))] = k;
  }
}

// (The edges are read through L1: staged in shared memory by every launch they took from 2 % longer, at
// a hundred cells, to 3.4 times as long, at 27 thousand, where they leave one block an SM.)
template <int GEOM, bool MG, bool CF>
__global__ void __launch_bounds__(256) k_event(TrackArgs a, EventScratch e, int cur) {
  const uint32_t stepk = a.step_dev ? *a.step_dev : a.step;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned blk_cnt[B_N];
  __shared__ unsigned long long blk_esc[4];
  WarpStage* stages = reinterpret_cast<WarpStage*>(smem);
  if (threadIdx.x < B_N) blk_cnt[threadIdx.x] = 0u;
  if (threadIdx.x < 4) blk_esc[threadIdx.x] = 0ull;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  WarpStage* st = stages + (threadIdx.x >> 5);
  const uint32_t n = (uint32_t)*a.n_dev;  // the whole bank: the weight floor is k_track's
  const float weight_floor = (float)(a.floor_coef * (*a.wsum) / (double)(n > 0 ? n : 1));
  const double inv_q = fx_inv_quantum(*a.wsum);
  const uint32_t n_in = e.count[cur];
  const uint32_t* live_in = e.live[cur];
  uint32_t* live_out = e.live[cur ^ 1];
  unsigned* n_out = e.count + (cur ^ 1);
  unsigned s_ev = 0, s_cen = 0, s_sc = 0;  // events, census events, scatters
  const uint32_t rkx = draw_step_key(a.rk, stepk);
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t trips = (n_in + stride - 1) / stride;
  for (uint32_t it = 0; it < trips; ++it) {
    const uint32_t i = it * stride + blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < n_in;
    EvOut o{0, false, 0.f, 0.0, false};
    bool alive = false;
    uint32_t pid = 0;
    if (active) {
      Hist h;
      pid = live_in[i];
      h.pid = pid;
      h.x = a.p1[pid]; h.u = a.d1[pid]; h.w = a.w[pid];
      h.y = 0.f; h.v = 0.f;
      if (GEOM == G_XY || GEOM == G_RZ) { h.y = a.p2[pid]; h.v = a.d2[pid]; }
      h.grp = MG ? a.group[pid] : 0;
      const int c = a.cell[pid];
      h.ev = e.ev[pid]; h.dcen = e.dcen[pid]; h.w_in = e.w_in[pid];
#ifdef IMC_CHECKED
      // bounds-checked build: an entry outside the mesh or group range, or with a non-finite
      // weight or position, is reported and dropped from the loop untouched
      if (c < 0 || c >= a.nc || (MG && (h.grp < 0 || h.grp >= a.ng)) || !isfinite(h.w) || !isfinite(h.x) ||
          !isfinite(h.dcen)) {
        atomicOr(a.flags, (int)IMC_FLAG_BOUNDS);
        o.finished = true;
      } else
#endif
      {
        h.cj = c / a.nx; h.ci = c - h.cj * a.nx;
        h.tab = __ldg(a.sass + (MG ? c + a.nc * h.grp : c));
        h.key = draw_key(a.rk, a.id_base + pid, stepk, TAG_TRANSPORT);
        const uint32_t ev0 = h.ev;
        history_event<GEOM, false, MG, CF, false>(a, h, o, nullptr, nullptr, nullptr, blk_cnt, blk_esc, a.dep_fx,
                                                  draw_next(a.rk, h.key, rkx, h.ev), weight_floor, inv_q, s_cen, s_sc);
        s_ev += h.ev - ev0;
        int bin;
        if (o.finished) history_retire<GEOM>(a, h, bin);
      }
      if (!o.finished) {
        alive = true;
        a.p1[pid] = h.x; a.d1[pid] = h.u; a.w[pid] = h.w;
        if (GEOM == G_XY || GEOM == G_RZ) { a.p2[pid] = h.y; a.d2[pid] = h.v; }
        a.cell[pid] = h.ci + a.nx * h.cj;
        e.ev[pid] = h.ev; e.dcen[pid] = h.dcen; e.w_in[pid] = h.w_in;
      }
    }
    // survivors into the next list (warp-aggregated append)
    const unsigned m = __ballot_sync(FULL, alive);
    unsigned base = 0;
    if (lane == 0 && m) base = atomicAdd(n_out, (unsigned)__popc(m));
    base = __shfl_sync(FULL, base, 0);
    if (alive) live_out[base + __popc(m & ((1u << lane) - 1u))] = pid;
    const unsigned long long ud = o.flush ? fx_units(o.lost, inv_q) : 0ull;
    warp_tally_fx(ud != 0ull || o.wd != 0.f, o.cell, ud, (double)o.wd, a.dep_fx, a.si, st);
  }
  add_event_counts(a, blk_cnt, blk_esc, s_ev, s_cen, s_sc);
}

template <int GEOM, bool MG, bool CF>
cudaError_t launch_event(const TrackArgs& a, const EventScratch& e, int cur, int block, int grid, cudaStream_t s) {
  k_event<GEOM, MG, CF><<<grid, block, stage_smem(block), s>>>(a, e, cur);
  return cudaGetLastError();
}

cudaError_t launch_event_geom(const TrackArgs& a, int geom, const EventScratch& e, int cur, int block, int grid,
                              cudaStream_t s) {
  if (a.ng > 1) {
    switch (geom) {
      case G_SPHERE: return launch_event<G_SPHERE, true, false>(a, e, cur, block, grid, s);
      case G_XY: return launch_event<G_XY, true, false>(a, e, cur, block, grid, s);
      case G_RZ: return launch_event<G_RZ, true, false>(a, e, cur, block, grid, s);
      default: return cudaErrorInvalidValue;
    }
  }
  if (a.cf_rate) {
    switch (geom) {
      case G_SLAB: return launch_event<G_SLAB, false, true>(a, e, cur, block, grid, s);
      case G_SPHERE: return launch_event<G_SPHERE, false, true>(a, e, cur, block, grid, s);
      case G_XY: return launch_event<G_XY, false, true>(a, e, cur, block, grid, s);
      case G_RZ: return launch_event<G_RZ, false, true>(a, e, cur, block, grid, s);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (geom) {
    case G_SLAB: return launch_event<G_SLAB, false, false>(a, e, cur, block, grid, s);
    case G_SPHERE: return launch_event<G_SPHERE, false, false>(a, e, cur, block, grid, s);
    case G_XY: return launch_event<G_XY, false, false>(a, e, cur, block, grid, s);
    case G_RZ: return launch_event<G_RZ, false, false>(a, e, cur, block, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

// Fixed-point tallies to the FP64 outputs: deposition per unit volume per (group, cell),
// escaped energy per side and (MG) per group, and the path-length intensity.
// cellf[q] = (1/V, si factor): a factor > 0 is 1/(sigma_a V dt) and the cell's intensity is
// its deposited energy times it (the sum over the cell's flights of (w - w') / (sigma_a V dt));
// < 0 is -1/(V dt), the cell has no absorption and si holds the raw sum of w*s.
__global__ void k_tally_finalize(TrackArgs a) {
  pdl_wait();     // the previous kernel of the stream has completed
  pdl_trigger();  // the next one may be scheduled
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const double W = *a.wsum;
  const int ncg = a.nc * a.ng;
  if (q < ncg) {
    const double2 cf = a.cellf[q];
    const double E = fx_energy(a.dep_fx[q], W);
    a.dep[q] = E * cf.x;
    a.si[q] = cf.y > 0.0 ? E * cf.y : a.si[q] * -cf.y;
  }
  else if (q < ncg + 4) a.escaped[q - ncg] = fx_energy(a.esc_fx[q - ncg], W);
  else if (q < ncg + 4 + a.ng && a.ng > 1) a.escaped_group[q - ncg - 4] = fx_energy(a.esc_fx[q - ncg], W);
}

}  // namespace

cudaError_t imc_launch_tally_finalize(const TrackArgs& a, cudaStream_t s) {
  ++g_imc_launches;
  const int n = a.nc * a.ng + 4 + a.ng;
  IMC_LAUNCH_PDL(k_tally_finalize, (n + 255) / 256, 256, 0, s, a);
  return cudaGetLastError();
}

size_t imc_event_scratch_bytes(long long capacity) {
  const size_t cap = (size_t)(capacity > 0 ? capacity : 1);
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  return al(8) + 2 * al(4 * cap) + 3 * al(4 * cap);
}

cudaError_t imc_run_event_tracking(const TrackArgs& a, int geom, void* scratch, long long capacity,
                                   long long n_upper, int block, int sms, long long max_launches, bool* cap_hit,
                                   cudaStream_t s) {
  const size_t cap = (size_t)(capacity > 0 ? capacity : 1);
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  char* p = static_cast<char*>(scratch);
  EventScratch e;
  e.count = reinterpret_cast<unsigned*>(p); p += al(8);
  e.live[0] = reinterpret_cast<uint32_t*>(p); p += al(4 * cap);
  e.live[1] = reinterpret_cast<uint32_t*>(p); p += al(4 * cap);
  e.ev = reinterpret_cast<uint32_t*>(p); p += al(4 * cap);
  e.dcen = reinterpret_cast<float*>(p); p += al(4 * cap);
  e.w_in = reinterpret_cast<float*>(p);
  *cap_hit = false;
  cudaError_t err = cudaMemsetAsync(e.count, 0, 8, s);
  if (err != cudaSuccess) return err;
  const bool mg2cf = (a.ng > 1 && geom >= G_XY) || a.cf_rate != nullptr;
  const int init_grid = (int)std::min<long long>((n_upper + 255) / 256 + 1, (long long)sms * 16);
  ++g_imc_launches;
  if (mg2cf) k_event_init<true><<<init_grid, 256, 0, s>>>(a, e);
  else k_event_init<false><<<init_grid, 256, 0, s>>>(a, e);
  if ((err = cudaGetLastError()) != cudaSuccess) return err;
  // one launch per event; every 8 launches the live count comes back to size the grid and to
  // stop (each launch advances every live history by one event, so at most max_events + 1
  // launches are needed)
  long long bound = n_upper;
  int cur = 0;
  for (long long it = 0; bound > 0; ++it) {
    if (it > max_launches) { *cap_hit = true; break; }
    if ((err = cudaMemsetAsync(e.count + (cur ^ 1), 0, 4, s)) != cudaSuccess) return err;
    const int grid = (int)std::max<long long>(1, std::min<long long>((bound + block - 1) / block, (long long)sms * 8));
    ++g_imc_launches;
    if ((err = launch_event_geom(a, geom, e, cur, block, grid, s)) != cudaSuccess) return err;
    cur ^= 1;
    if ((it & 7) == 7) {
      unsigned live = 0;
      if ((err = cudaMemcpyAsync(&live, e.count + cur, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return err;
      if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return err;
      bound = live;
    }
  }
  return cudaSuccess;
}

cudaError_t imc_launch_track(const TrackArgs& a, int geom, const TrackLaunch& l, cudaStream_t s) {
  ++g_imc_launches;
  if (a.ng > 1) {  // multigroup: 2-D (MG_IMC/MG_IMC2D.py) and the 1-D sphere (MG_IMC/MG_IMC1D.py)
    switch (geom) {
      case G_SPHERE: return launch_geom<G_SPHERE, true>(a, l, s);
      case G_XY: return launch_geom<G_XY, true>(a, l, s);
      case G_RZ: return launch_geom<G_RZ, true>(a, l, s);
      default: return cudaErrorInvalidValue;
    }
  }
  if (a.cf_rate) {  // Carter-Forest, gray
    switch (geom) {
      case G_SLAB: return launch_geom<G_SLAB, false, true>(a, l, s);
      case G_SPHERE: return launch_geom<G_SPHERE, false, true>(a, l, s);
      case G_XY: return launch_geom<G_XY, false, true>(a, l, s);
      case G_RZ: return launch_geom<G_RZ, false, true>(a, l, s);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (geom) {
    case G_SLAB: return launch_geom<G_SLAB, false>(a, l, s);
    case G_SPHERE: return launch_geom<G_SPHERE, false>(a, l, s);
    case G_XY: return launch_geom<G_XY, false>(a, l, s);
    case G_RZ: return launch_geom<G_RZ, false>(a, l, s);
    default: return cudaErrorInvalidValue;
  }
}
