// imc_adjoint.cu — vector-Jacobian product of one step's deposition tally with respect to
// the per-cell opacity sigma, for 2-D gray steps (xy, rz; IMC/IMC2D.py:711-1107 events).
//
// Tally and its derivative.  For cotangent g, the step's score is T = sum_c g_c dep_c and
// a history contributes L = sum_i a_i d_i over its segments i (cell c_i, length s_i,
// entering weight w_i, leaving weight w_{i+1} = w_i exp(-sigma_a,c_i s_i), deposit
// d_i = w_i - w_{i+1}, a_i = g_{c_i} / V_{c_i}).  Two effects of sigma_j:
//  * implicit capture (path-length / pathwise term): holding the path fixed,
//      dL/dsigma_a,j = sum_{k in j} s_k (a_k w_{k+1} + L_{<=k} - L),
//    L_{<=k} = sum_{i<=k} a_i d_i (what the history scored before it left segment k);
//  * effective scatter (likelihood-ratio term): the path density carries
//    exp(-sigma_s,j s_k) per segment in j and a factor sigma_s,j per scatter in j, so
//      dE[L]/dsigma_s,j = E[ sum_{k in j} (L - L_{<k}) (-s_k + [scatter at k] / sigma_s,j) ],
//    with only the score accrued from segment k on (earlier scores are independent of it).
//    A cell whose scatter distance is capped (sigma_s L > 1e4) or off (sigma_s <= 1e-12)
//    samples independently of sigma_s and contributes no such term.
//  * Fleck factor: sigma_a = f sigma, f = 1 / (1 + b sigma), so dsigma_a/dsigma = f^2 and
//    dsigma_s/dsigma = 1 - f^2.
// Replay.  Each lane tracks a history twice from its Philox counter (bank index, event,
// step, TAG_TRANSPORT): pass 0 computes L, pass 1 accumulates the per-visit sums
// gp = sum s_k (a_k w_{k+1} + L_{<=k} - L) and
// gs = sum (L - L_{<k}) ([scatter at k] - sigma_s s_k),
// and adds f^2 gp + (1 - f^2) / sigma_s gs to grad[cell] when the history leaves the cell (the
// per-cell factors are tables made beforehand).  No path is stored; the bank is read, never
// written.  A flight is the forward tracking kernel's (next_flight), so each replay follows the
// forward step's path.
#include <algorithm>

#include "imc_event.cuh"
#include "imc_internal.h"

using namespace imcdev;

namespace {

constexpr int kAdjWide = 1024;    // threads of a wide block
constexpr int kAdjRefillMin = 8;  // idle lanes before they are loaded again (as in the tracking)

__global__ void k_adjoint_tables(AdjointArgs A) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= A.t.nc) return;
  const double sig = A.sig64[c];
  const double f = sig > 0.0 ? A.sa64[c] / sig : 1.0;
  const double ss = A.ss64[c];
  A.score[c] = A.cot[c] * A.t.cellf[c].x;
  A.chain[c] = make_double2(f * f, ss > 0.0 ? (1.0 - f * f) / ss : 0.0);
}

// WIDE: one block per SM with the gradient in shared memory (added to the global one at its end),
// where it fits: a shared atomic per cell visit, against a match of the warp's lanes by cell and
// a serial sum per group for the global form.  Lanes that are to start a history, or its second
// pass, are loaded kAdjRefillMin at a time.  Both passes of 4e6 histories on 128 x 128 cells:
// 3.5 ms, against 6.4 ms with the global tally, the factors formed per visit (two FP64 divisions)
// and a lane reloaded whenever it ends.
// EDGES: the edges are staged in shared memory (else, on a long mesh, read through L1).
template <int GEOM, bool WIDE, bool EDGES>
__global__ void __launch_bounds__(WIDE ? kAdjWide : 256, WIDE ? 1 : 4) k_adjoint(AdjointArgs A) {
  const TrackArgs& a = A.t;
  extern __shared__ __align__(16) unsigned char smem[];
  WarpStage* stages = reinterpret_cast<WarpStage*>(smem);  // not WIDE
  float2* E1 = reinterpret_cast<float2*>(smem + (WIDE ? 0 : sizeof(WarpStage) * (blockDim.x >> 5)));
  float2* E2 = E1 + a.nx;
  double* G = reinterpret_cast<double*>(E2 + a.ny);  // WIDE: [nc]
  if (EDGES) {
    for (int q = threadIdx.x; q < a.nx; q += blockDim.x) E1[q] = make_float2(a.e1[q], a.e1[q + 1]);
    for (int q = threadIdx.x; q < a.ny; q += blockDim.x) E2[q] = make_float2(a.e2[q], a.e2[q + 1]);
  }
  if (WIDE) for (int q = threadIdx.x; q < a.nc; q += blockDim.x) G[q] = 0.0;
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  WarpStage* st = stages + (threadIdx.x >> 5);
  const uint32_t n = (uint32_t)*a.n_dev;
  const float c_light = (float)C_LIGHT;
  const float weight_floor = (float)(1e-10 * (*a.wsum) / (double)(n > 0 ? n : 1));
  const uint32_t rkx = draw_step_key(a.rk, a.step);

  Runs run = first_run(n, a.sms);
  bool drained = false;
  bool has = false, again = false;  // again: the lane's history is to be followed a second time
  int phase = 0;
  uint32_t pid = 0, ev = 0;
  DrawKey key{0u, 0u, 0u};
  float x = 0, y = 0, u = 0, v = 0, w = 0, dcen = 0;
  float2 tab = make_float2(0.f, 0.f);
  int ci = 0, cj = 0;
  double L = 0.0, Lcum = 0.0, gp = 0.0, gs1 = 0.0, gs2 = 0.0;

  for (;;) {
    const unsigned idle = __ballot_sync(FULL, !has);
    const unsigned more = __ballot_sync(FULL, again);
    if (idle == FULL || (__popc(idle) >= kAdjRefillMin && (!drained || more))) {
      bool load = again;
      if (again) { phase = 1; again = false; }
      unsigned need = __ballot_sync(FULL, !has && !load);
      for (;;) {
        if (need && !drained && run.next >= run.end && !next_run(a.queue, a.chunk, n, a.sms, run))
          drained = true;
        if (need && !drained) {
          const uint32_t avail = run.end - run.next;
          const uint32_t rank = __popc(need & lt_mask);
          if (!has && !load && rank < avail) { pid = run.next + rank; phase = 0; L = 0.0; load = true; }
          run.next += min((uint32_t)__popc(need), avail);
        }
        if (load) {
          load = false;
          w = a.w[pid];
          dcen = (a.dt - a.t[pid]) * c_light;
          if (w > 0.f && dcen > 0.f) {
            x = a.p1[pid]; u = a.d1[pid]; y = a.p2[pid]; v = a.d2[pid];
            const int c = a.cell[pid];
            cj = c / a.nx; ci = c - cj * a.nx;
            tab = __ldg(a.sass + c);
            key = draw_key(a.rk, a.id_base + pid, a.step, TAG_TRANSPORT);
            ev = 0;
            Lcum = 0.0; gp = 0.0; gs1 = 0.0; gs2 = 0.0;
            has = true;
          }
        }
        need = __ballot_sync(FULL, !has);
        if (!need || drained) break;
      }
      if (need == FULL) break;
    }
    bool flush = false;
    int flush_cell = 0;
    double val = 0.0;
    if (has) {
      const int c = ci + a.nx * cj;
      const float sa = tab.x, ss = tab.y;
      bool finished = false, left = false;
      if (ev >= (uint32_t)a.max_events) {
        finished = true;  // cap: the history stops where it is, in both passes
      } else {
        const U4 r = draw_next(a.rk, key, rkx, ev);
        ++ev;
        const Flight f = next_flight<GEOM, true>(cell_edges<EDGES>(E1, a.e1, ci), cell_edges<EDGES>(E2, a.e2, cj), ss,
                                                 x, y, u, v, dcen, r);
        const float wn = w * __expf(-sa * f.d);
        const double dd = (double)w - (double)wn;  // exact
        const double ac = __ldg(A.score + c);
        if (phase == 0) {
          L += ac * dd;
        } else {
          const double R = L - Lcum;  // what the history scores from this flight on
          Lcum += ac * dd;
          gp += (double)f.d * (ac * (double)wn + Lcum - L);
          // sampling depends on sigma_s where the scatter slot holds it
          if (ss > 0.f) {
            gs1 += R * (double)f.d;
            if (f.evt == EV_SCATTER) gs2 += R;
          }
        }
        dcen -= f.d;
        if (wn <= weight_floor) {
          finished = true;  // IMC/IMC2D.py:1043-1047: the history stops at the floor
        } else {
          w = wn; x = f.x; y = f.y; u = f.u; v = f.v;
          if ((f.di | f.dj) != 0) {
            left = true;
            const int ni = ci + f.di, nj = cj + f.dj;
            if ((unsigned)ni >= (unsigned)a.nx || (unsigned)nj >= (unsigned)a.ny) {
              const int side = ni < 0 ? 0 : ni >= a.nx ? 1 : nj < 0 ? 2 : 3;
              if ((a.reflect_mask >> side) & 1) {  // stays in its cell
                if (side < 2) u = -u; else v = -v;
              } else {
                finished = true;
              }
            } else {
              ci = ni; cj = nj;
              tab = __ldg(a.sass + c + f.di + a.nx * f.dj);
            }
          }
          if (!(w > 0.f) || !(dcen > 0.f)) finished = true;
        }
      }
      if (phase == 1 && (left || finished)) {
        const double2 k = __ldg(A.chain + c);
        val = k.x * gp + (k.y * gs2 - (1.0 - k.x) * gs1);
        flush = val != 0.0;
        flush_cell = c;
        gp = 0.0; gs1 = 0.0; gs2 = 0.0;
      }
      if (finished) { has = false; again = phase == 0; }
    }
    if (WIDE) { if (flush) atomicAdd(G + flush_cell, val); }
    else warp_tally1(flush, flush_cell, val, A.grad, st);
  }
  if (WIDE) {
    __syncthreads();
    for (int q = threadIdx.x; q < a.nc; q += blockDim.x) if (G[q] != 0.0) atomicAdd(A.grad + q, G[q]);
  }
}

template <auto Kernel>
cudaError_t launch_replay(const AdjointArgs& a, int block, int bps, size_t sh, cudaStream_t s) {
  const cudaError_t e = smem_opt_in<Kernel>(sh);
  if (e != cudaSuccess) return e;
  Kernel<<<a.t.sms * resident_blocks<Kernel>(bps, block, sh), block, sh, s>>>(a);
  return cudaGetLastError();
}

template <int GEOM>
cudaError_t launch_adj(const AdjointArgs& a, int block, int bps, cudaStream_t s) {
  k_adjoint_tables<<<(a.t.nc + 255) / 256, 256, 0, s>>>(a);
  const size_t edges = sizeof(float2) * ((size_t)a.t.nx + a.t.ny), stages = (size_t)(block / 32) * sizeof(WarpStage);
  const size_t wide_sh = edges + sizeof(double) * (size_t)a.t.nc;
  if (block <= 256 && wide_sh <= kSmemPerBlock)
    return launch_replay<k_adjoint<GEOM, true, true>>(a, std::max(128, std::min(kAdjWide, block * bps)) & ~31, 1,
                                                      wide_sh, s);
  if (edges + stages <= kSmemPerBlock)
    return launch_replay<k_adjoint<GEOM, false, true>>(a, block, bps, edges + stages, s);
  return launch_replay<k_adjoint<GEOM, false, false>>(a, block, bps, stages, s);
}

}  // namespace

cudaError_t imc_launch_adjoint(const AdjointArgs& a, int geom, int block, int bps, cudaStream_t s) {
  g_imc_launches += 2;
  switch (geom) {
    case G_XY: return launch_adj<G_XY>(a, block, bps, s);
    case G_RZ: return launch_adj<G_RZ>(a, block, bps, s);
    default: return cudaErrorInvalidValue;
  }
}
