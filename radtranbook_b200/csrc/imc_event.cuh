// imc_event.cuh — one flight of a history in FP32: the distance to the cell's faces, the next
// effective scatter or census, and where the event leaves the photon.  Shared by the tracking
// kernels and the adjoint's replays, so that a replay follows its history bit for bit.
//
//   slab IMC/IMC1D.py:75-130; sphere IMC/IMC1D.py:336-436; xy, rz IMC/IMC2D.py:711-935
#pragma once
#include "imc_device.cuh"

namespace imcdev {

// What an event costs is its instructions: the kernel issues one in four of every five cycles, so
// the geometry is written for few and uniform ones.  Against the straightforward form (one branch
// per face and root, thresholds and caps tested per flight, all ten Philox rounds per draw, FP64
// path length carried in registers) the ten launches of a 2M crooked-pipe run take 10.4 ms
// instead of 12.6, the slab Marshak wave's twenty 7.1 instead of 8.5; every history is
// bit-identical.

// The scatter slot of a table entry (scatter_entry): > 0 the effective scatter opacity, 0 none
// (at or below the geometry's threshold), < 0 minus the opacity of a cell whose distance is
// capped (sigma_s L > 1e4 -> 1e4 / L; IMC/IMC1D.py:83-88, IMC/IMC2D.py:758-765).
template <bool CAPS>
__device__ __forceinline__ float scatter_flight(float ss, float L, uint32_t x, float s_other) {
  if (ss > 0.f) {
    if (scatter_may_win(x, ss, s_other)) return fdiv(neglog_u(x), ss);
  } else if (CAPS && ss < 0.f) {
    if (scatter_may_win(x, 10000.0f / L, s_other)) return neglog_u(x) * (L * 1e-4f);
  }
  return BIGF;
}

// The (lower, upper) edges of cell i along one direction: from a shared-memory table of pairs, or from
// the edges themselves through L1.
template <bool STAGED>
__device__ __forceinline__ float2 cell_edges(const float2* staged, const float* e, int i) {
  return STAGED ? staged[i] : make_float2(__ldg(e + i), __ldg(e + i + 1));
}

struct Flight {
  float d;           // path length
  int evt;           // EV_*
  int di, dj;        // the cell step of a boundary crossing
  float x, y, u, v;  // position and direction after the event
};

// e1, e2: the cell's (lower, upper) edges (e2 unused in 1-D); ss: its scatter slot; CAPS: the
// geometry caps optically thick scatter distances
template <int GEOM, bool CAPS>
__device__ __forceinline__ Flight next_flight(float2 e1, float2 e2, float ss, float x, float y, float u, float v,
                                              float dcen, const U4& r) {
  constexpr bool ONED = GEOM == G_SLAB || GEOM == G_SPHERE;
  float d, sb, xn, yn = y, un = u, vn = v;
  int evt, di = 0, dj = 0;
  // ---- distance to the cell boundary ----
  float s_rin = BIGF, s_rout = BIGF, st_ = 0.f, sx = BIGF, sy = BIGF;  // sy: z faces in RZ
  float din = BIGF, dout = BIGF, om = 0.f;
  if (GEOM == G_SLAB) {
    sb = slab_face(x, u, e1.x, e1.y);
  } else if (GEOM == G_SPHERE) {
    om = (1.f - u) * (1.f + u);
    const float b2 = x * x * om;
    dout = outer_root(x, u, e1.y, b2);
    din = inner_root(x, u, e1.x, b2);
    sb = fminf(dout, din);
  } else {
    if (GEOM == G_XY) {
      if (u != 0.f) sx = fdiv((u > 0.f ? e1.y : e1.x) - x, u);
      if (v != 0.f) sy = fdiv((v > 0.f ? e2.y : e2.x) - y, v);
      sx = fmaxf(sx, 0.f); sy = fmaxf(sy, 0.f);
      sb = fminf(sx, sy);
    } else {
      const float sin2 = (1.f - v) * (1.f + v);
      om = (1.f - u) * (1.f + u);
      if (sin2 >= 1e-15f) {
        // outer_root and inner_root with one quotient: moving outwards (u >= 0) only the
        // outer face is met and its root is a quotient; moving inwards the inner root is the
        // quotient, the outer one q - r u
        const float ist = frsqrt(sin2);
        st_ = sin2 * ist;
        const float b2 = x * x * om;
        const float q = sqrt_nn(fmaf(e1.y, e1.y, -b2));
        const float disc = fmaf(e1.x, e1.x, -b2);
        const bool out = u >= 0.f;
        const float R = out ? e1.y : e1.x;
        const float P = (R - x) * (R + x);
        const float den = out ? fmaxf(fmaf(x, u, q), 1e-30f) : fmaf(disc, frsqrt(disc), -(x * u));
        const float quo = fdiv(out ? P : -P, den);
        s_rout = fmaxf(out ? quo : fmaf(-x, u, q), 0.f) * ist;
        if (!out && e1.x > 0.f && disc > 0.f) s_rin = fmaxf(quo, 0.f) * ist;
      }
      if (fabsf(v) > 1e-15f) sy = fmaxf(fdiv((v > 0.f ? e2.y : e2.x) - y, v), 0.f);
      sb = fminf(fminf(s_rin, s_rout), sy);
    }
  }
  // ---- effective scatter and census ----
  float L = e1.y - e1.x;  // used by capped cells only
  if (!ONED) L = fminf(L, e2.y - e2.x);
  const float ds = scatter_flight<CAPS>(ss, L, r.x, fminf(sb, dcen));
  d = sb; evt = EV_BOUNDARY;
  if (ds < d) { d = ds; evt = EV_SCATTER; }
  if (dcen < d) { d = dcen; evt = EV_CENSUS; }
  // ---- move ----
  if (GEOM == G_SLAB) {
    xn = fmaf(u, d, x);
    if (evt == EV_BOUNDARY) { di = u > 0.f ? 1 : -1; xn = u > 0.f ? e1.y : e1.x; }
    else { if (evt == EV_SCATTER) un = fmaf(2.f, u01f(r.y), -1.f); xn = fminf(fmaxf(xn, e1.x), e1.y); }
  } else if (GEOM == G_SPHERE) {
    const float ax = fmaf(u, d, x);
    float rn = sqrt_nn(fmaf(ax, ax, d * d * om));
    float mun = rn > 1e-15f ? fmaf(x, u, d) / rn : 1.f;
    if (evt == EV_BOUNDARY) {
      di = dout <= din ? 1 : -1;
      rn = dout <= din ? e1.y : e1.x;
      mun = fmaf(x, u, d) / rn;
    } else {
      if (evt == EV_SCATTER) mun = fmaf(2.f, u01f(r.y), -1.f);
      rn = fminf(fmaxf(rn, e1.x), e1.y);
    }
    xn = rn; un = fminf(1.f, fmaxf(-1.f, mun));
  } else if (GEOM == G_XY) {
    xn = fmaf(u, d, x); yn = fmaf(v, d, y);
    if (evt == EV_BOUNDARY) {
      if (sx <= sy) di = u > 0.f ? 1 : -1;
      else dj = v > 0.f ? 1 : -1;
    } else if (evt == EV_SCATTER) {
      const float uz = fmaf(2.f, u01f(r.y), -1.f);
      const float rxy = sqrt_nn((1.f - uz) * (1.f + uz));
      float sp, cp;
      sincospif(2.f * u01f(r.z), &sp, &cp);
      un = rxy * cp; vn = rxy * sp;
    }
    xn = di > 0 ? e1.y : di < 0 ? e1.x : fminf(fmaxf(xn, e1.x), e1.y);
    yn = dj > 0 ? e2.y : dj < 0 ? e2.x : fminf(fmaxf(yn, e2.x), e2.y);
  } else {
    const float l = d * st_;
    const float ax = fmaf(u, l, x);
    const float rn = sqrt_nn(fmaf(ax, ax, l * l * om));
    yn = fmaf(d, v, y);
    if (rn > 1e-15f && l > 0.f) un = fminf(1.f, fmaxf(-1.f, fdiv(fmaf(x, u, l), rn)));
    if (evt == EV_BOUNDARY) {
      if (sb == s_rin) di = -1;
      else if (sb == s_rout) di = 1;
      else dj = v < 0.f ? -1 : 1;
    } else if (evt == EV_SCATTER) {
      vn = fmaf(2.f, u01f(r.y), -1.f);
      un = cospif(2.f * u01f(r.z));
    }
    xn = di > 0 ? e1.y : di < 0 ? e1.x : fminf(fmaxf(rn, e1.x), e1.y);
    yn = dj > 0 ? e2.y : dj < 0 ? e2.x : fminf(fmaxf(yn, e2.x), e2.y);
  }
  return Flight{d, evt, di, dj, xn, yn, un, vn};
}

// A warp's runs of bank entries.  The first is its own, without a ticket: `first` consecutive
// entries, dealt so that neighbouring runs go to different SMs and, within an SM, to different
// schedulers (warp slots go round the four schedulers, so the blocks of one SM start at different
// warps); a bank too small to give every warp a full row is spread over about four warps a
// scheduler.  (With every run a ticket, the warps that came first held the work of a small bank
// while other schedulers had none: one of 592 executed 6.5 times the average of a 4k slab step's
// instructions.  The twenty launches of a 20k crooked-pipe run 0.67 -> 0.52 ms, of a 4k slab run
// 5.5 -> 4.0.)  So the grid has no more blocks than are resident (resident_blocks): dealt to twice as many,
// half the runs of a 40k slab wave waited for the other half (256 x 8 threads an SM: 7.97 ms, now 4.48).
// Later runs are guided tickets: a share of what is left, at most `chunk`, at least 32, so
// early ones are long contiguous (coherent) runs and the drain is finely balanced.
struct Runs { uint32_t next, end; };  // the warp's current run

__device__ __forceinline__ uint32_t first_length(uint32_t n, int sms) {
  const uint32_t slots = (uint32_t)sms * 16u;
  return min(32u, max(4u, (n + slots - 1) / slots));
}
__device__ __forceinline__ Runs first_run(uint32_t n, int sms) {
  const uint32_t warps = blockDim.x >> 5, first = first_length(n, sms);
  const uint32_t w = ((threadIdx.x >> 5) + blockIdx.x / (uint32_t)sms) % warps;
  const uint32_t base = min(n, (w * gridDim.x + blockIdx.x) * first);
  return Runs{base, min(n, base + first)};
}

// The next run of a warp whose current one is used up (sms = 0: no first runs were dealt).  Every lane calls it; false when no entry is left.
__device__ __forceinline__ bool next_run(unsigned long long* queue, int chunk, uint32_t n, int sms, Runs& r) {
  unsigned long long base = 0, claim = 0;
  const unsigned long long nw = (unsigned long long)gridDim.x * (blockDim.x >> 5);
  const uint32_t dealt = sms ? (uint32_t)min((unsigned long long)n, nw * first_length(n, sms)) : 0u;
  const unsigned long long rest = n - dealt;
  if (rest == 0) return false;
  if ((threadIdx.x & 31) == 0) {
    const unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(queue);
    const unsigned long long left = cur < rest ? rest - cur : 0ull;
    claim = min((unsigned long long)chunk, max(32ull, left / (2ull * nw)));
    base = atomicAdd(queue, claim);
  }
  base = __shfl_sync(FULL, base, 0);
  claim = __shfl_sync(FULL, claim, 0);
  if (base >= rest) return false;
  r.next = dealt + (uint32_t)base;
  r.end = dealt + (uint32_t)min(base + claim, rest);
  return true;
}

}  // namespace imcdev
