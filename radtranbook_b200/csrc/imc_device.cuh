// imc_device.cuh — device building blocks of the B200 IMC engine.
//
//  * Philox-4x32-10 (Salmon et al., SC'11), keyed by the run seed, counter
//    (particle index, draw block / event number, step, stream tag).
//  * 23-bit open-interval uniforms, identical in FP32 and FP64.
//  * FP32 event geometry for slab / sphere / xy / rz (the reference's event
//    functions IMC/IMC1D.py:75-130, 336-436 and IMC/IMC2D.py:711-935, rewritten in
//    cancellation-free form; the cell index, not the position, decides the cell).
//  * Warp-aggregated FP64 tally reduction (match_any + per-warp shared staging).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace imcdev {

constexpr double C_LIGHT = 29.98;
constexpr double A_RAD = 0.01372;
constexpr float BIGF = 1e30f;
constexpr unsigned FULL = 0xffffffffu;

enum : int { G_SLAB = 0, G_SPHERE = 1, G_XY = 2, G_RZ = 3 };
enum : int { EV_CENSUS = 0, EV_BOUNDARY = 1, EV_SCATTER = 2 };
enum : int { S_EVENTS = 0, S_BOUNDARY, S_SCATTER, S_CENSUS, S_CAPTURE, S_FLOOR, S_REFLECT, S_CAP, S_ESCAPE, S_N };

enum : uint32_t {
  TAG_TRANSPORT = 0x10000000u,
  TAG_BOUNDARY = 0x20000000u,
  TAG_SOURCE = 0x30000000u,
  TAG_EMISSION = 0x40000000u,
  TAG_IC = 0x50000000u,
  TAG_COMB = 0x60000000u,
};

struct U4 { uint32_t x, y, z, w; };

// The 64-bit product of two 32-bit words as its low and high halves: one wide multiply.
__device__ __forceinline__ void mul_wide(uint32_t a, uint32_t b, uint32_t& lo, uint32_t& hi) {
  asm("{\n.reg .u64 p;\nmul.wide.u32 p, %2, %3;\nmov.b64 {%0, %1}, p;\n}" : "=r"(lo), "=r"(hi) : "r"(a), "r"(b));
}

__device__ __forceinline__ U4 philox4x32_10(U4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    if (r) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
    const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
    c = U4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
  }
  return c;
}

// ((x>>9) + 0.5) * 2^-23 = (2k+1) * 2^-24, k < 2^23: 24 significant bits, so exact in
// float and double alike, and never 0 or 1.
__device__ __forceinline__ float u01f(uint32_t x) { return __uint2float_rn(((x >> 9) << 1) | 1u) * 5.9604644775390625e-8f; }
__device__ __forceinline__ double u01d(uint32_t x) { return (double)(((x >> 9) << 1) | 1u) * 5.9604644775390625e-8; }

__device__ __forceinline__ U4 draw(uint64_t seed, uint32_t idx, uint32_t block, uint32_t step, uint32_t tag) {
  return philox4x32_10(U4{idx, block, step, tag}, (uint32_t)seed, (uint32_t)(seed >> 32));
}

// The 20 round keys of a seed (k0 + r*0x9E3779B9, k1 + r*0xBB67AE85, r = 0..9), for kernels
// that carry them in their parameter block: the rounds then read them as constant operands
// instead of stepping the key in registers.  Same outputs as draw().
__host__ __device__ inline void philox_round_keys(uint64_t seed, uint32_t* rk) {
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    rk[2 * r] = k0; rk[2 * r + 1] = k1;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
}

__device__ __forceinline__ U4 draw_rk(const uint32_t* rk, uint32_t idx, uint32_t block, uint32_t step,
                                      uint32_t tag) {
  U4 c{idx, block, step, tag};
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
    c = U4{hi1 ^ c.y ^ rk[2 * r], lo1, hi0 ^ c.w ^ rk[2 * r + 1], lo0};
  }
  return c;
}

// draw_rk for a run of blocks of one (idx, step, tag): the first two rounds' products of the
// words that do not change with the block are formed once (draw_key), and each draw starts
// after round 2 with one of its four products instead of four.  Same numbers as draw_rk.
struct DrawKey { uint32_t a, b, c; };
__device__ __forceinline__ DrawKey draw_key(const uint32_t* rk, uint32_t idx, uint32_t step, uint32_t tag) {
  const uint32_t lo0 = 0xD2511F53u * idx, hi0 = __umulhi(0xD2511F53u, idx);
  const uint32_t z1 = hi0 ^ tag ^ rk[1];  // word z after round 1
  return DrawKey{__umulhi(0xCD9E8D57u, z1) ^ (0xCD9E8D57u * step) ^ rk[2], 0xCD9E8D57u * z1, lo0 ^ rk[3]};
}
// rkx = high half of 0xCD9E8D57 * step, ^ rk[0] (the step's, the same for every history)
__device__ __forceinline__ uint32_t draw_step_key(const uint32_t* rk, uint32_t step) {
  return __umulhi(0xCD9E8D57u, step) ^ rk[0];
}
__device__ __forceinline__ U4 draw_next(const uint32_t* rk, const DrawKey& k, uint32_t rkx, uint32_t block) {
  const uint32_t x1 = rkx ^ block;  // word x after round 1
  uint32_t l, h;
  mul_wide(0xD2511F53u, x1, l, h);
  U4 c{k.a, k.b, h ^ k.c, l};
#pragma unroll
  for (int r = 2; r < 10; ++r) {
    uint32_t lo0, hi0, lo1, hi1;
    mul_wide(0xD2511F53u, c.x, lo0, hi0);
    mul_wide(0xCD9E8D57u, c.z, lo1, hi1);
    c = U4{hi1 ^ c.y ^ rk[2 * r], lo1, hi0 ^ c.w ^ rk[2 * r + 1], lo0};
  }
  return c;
}

// draw_next with the round keys of rounds 3..10 read as four 16-byte words (rk4: keys 4..19 of
// philox_round_keys, 16-byte aligned, e.g. staged in shared memory): four vector loads where
// draw_next makes sixteen scalar ones.
__device__ __forceinline__ U4 draw_next4(const uint4* rk4, const DrawKey& key, uint32_t rkx, uint32_t block) {
  const uint32_t x1 = rkx ^ block;
  uint32_t a0, b0, a1, b1;
  mul_wide(0xD2511F53u, x1, a0, b0);
  U4 c{key.a, key.b, b0 ^ key.c, a0};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 k = rk4[q];
    mul_wide(0xD2511F53u, c.x, a0, b0);
    mul_wide(0xCD9E8D57u, c.z, a1, b1);
    c = U4{b1 ^ c.y ^ k.x, a1, b0 ^ c.w ^ k.y, a0};
    mul_wide(0xD2511F53u, c.x, a0, b0);
    mul_wide(0xCD9E8D57u, c.z, a1, b1);
    c = U4{b1 ^ c.y ^ k.z, a1, b0 ^ c.w ^ k.w, a0};
  }
  return c;
}

// Word q (0..3) of a Philox block: the comb's uniform of pre-comb entry k is word k % 4 of
// block (k / 4, 1), so four consecutive entries share one block.
__device__ __forceinline__ uint32_t u4_word(const U4& r, int q) {
  return q == 0 ? r.x : q == 1 ? r.y : q == 2 ? r.z : r.w;
}

// -log(u) for u = u01: distance in mean free paths.
__device__ __forceinline__ float neglog_u(uint32_t x) { return -logf(u01f(x)); }


// Whether a scatter at -log(u)/sigma, u = u01(x), can come before s_other.  With p = 1 - u
// (exact in FP32, at least 2^-24) the scatter is at least p/sigma away, so p >= sigma s_other
// (1 + 1e-6) rules it out whatever the rounding of the logarithm and the quotient; that
// settles nearly every flight of a thin cell.  What is left is tested in FP64 with a short
// series of exp(-sigma s_other) when sigma s_other is small, so that the logarithm is
// evaluated only when it can win.
__device__ __forceinline__ bool scatter_may_win(uint32_t x, float sig, float s_other) {
  const float tf = sig * s_other;
  if (1.0f - u01f(x) >= tf * 1.000001f) return false;
  if (tf > 0.010001f) return true;  // not small, whatever the product's rounding
  const double t = (double)sig * (double)s_other;
  if (!(t < 0.01)) return true;
  const double thr = 1.0 - t * (1.0 - t * (0.5 - t * (1.0 / 6.0)));
  return u01d(x) > thr;
}

// The tracking's approximate quotient and reciprocal square root: the hardware approximations
// without the steps that widen them to subnormal operands, which no distance, direction or
// opacity here has (histories are bit-identical to __fdividef / rsqrtf; a crossing has up to
// eight of them: 12.7 -> 11.9 ms for the ten launches of a 2M crooked-pipe run).
__device__ __forceinline__ float fdiv(float a, float b) {
  float q;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(a), "f"(b));
  return q;
}
__device__ __forceinline__ float frsqrt(float x) {
  float q;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(x));
  return q;
}

// ---- 1-D slab: distance to the exit face in the direction of mu ----
__device__ __forceinline__ float slab_face(float x, float mu, float xl, float xr) {
  const float db = fdiv(mu > 0.f ? (xr - x) : (xl - x), mu);
  return fmaxf(db, 0.f);
}

// ---- sphere / cylinder: cancellation-free roots of l^2 + 2 r mu l + (r^2 - R^2) = 0 ----
// sqrt(x) = x * x^(-1/2): one hardware reciprocal square root and a multiply (a few ulp,
// against the ~10-instruction correctly rounded sqrtf); 0 for x <= 0.  Tracking is FP32
// with statistical tolerances, and every kernel that replays a history uses the same form.
__device__ __forceinline__ float sqrt_nn(float x) { return x > 0.f ? x * frsqrt(x) : 0.f; }

__device__ __forceinline__ float outer_root(float r, float mu, float R, float b2) {
  const float q = sqrt_nn(fmaf(R, R, -b2));
  float l = (mu >= 0.f) ? fdiv((R - r) * (R + r), fmaxf(fmaf(r, mu, q), 1e-30f)) : fmaf(-r, mu, q);
  return fmaxf(l, 0.f);
}
__device__ __forceinline__ float inner_root(float r, float mu, float R, float b2) {
  if (!(R > 0.f) || !(mu < 0.f)) return BIGF;
  const float disc = fmaf(R, R, -b2);
  if (!(disc > 0.f)) return BIGF;
  const float l = fdiv((r - R) * (r + R), fmaf(disc, frsqrt(disc), -(r * mu)));
  return fmaxf(l, 0.f);
}

// ---- warp-aggregated FP64 reduction into global tallies ----
// Every lane of the warp must call this (converged).  Lanes with flush=false pass any
// key.  Lanes flushing the same cell are grouped with __match_any_sync; the lowest lane
// of each group sums the group's values (staged in per-warp shared memory) and issues
// one FP64 red per tally.
struct WarpStage { double a[32]; double b[32]; };

__device__ __forceinline__ void warp_tally1(bool flush, int key, double va, double* __restrict__ ta,
                                            WarpStage* st) {
  const unsigned fm = __ballot_sync(FULL, flush);
  if (fm == 0u) return;
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(FULL, flush ? key : -1 - lane);
  if (__all_sync(FULL, !flush || __popc(peers) == 1)) {
    if (flush) atomicAdd(ta + key, va);
    return;
  }
  st->a[lane] = va;
  __syncwarp();
  if (flush && (__ffs(peers) - 1) == lane) {
    double sa = 0.0;
    unsigned m = peers;
    while (m) { const int l = __ffs(m) - 1; m &= m - 1; sa += st->a[l]; }
    atomicAdd(ta + key, sa);
  }
  __syncwarp();
}

// An add per flushing lane into a block's shared tally, the lanes of the cell `hot` (warp-uniform) as one:
// an FP64 shared-memory add is a compare-and-swap loop, which lanes of one cell take in turn.  Every
// lane of the warp calls it (converged).
__device__ __forceinline__ void smem_tally_hot(bool flush, int cell, double v, double* t, int hot) {
  const bool mine = flush && cell == hot;
  if (__popc(__ballot_sync(FULL, mine)) >= 4) {
    double s = mine ? v : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(t + hot, s);
    if (flush && !mine) atomicAdd(t + cell, v);
  } else if (flush) {
    atomicAdd(t + cell, v);
  }
}

// ---- block-aggregated per-bin sums ----
// The census of a step piles up in a few cells (the hottest radiation), so even after
// per-warp aggregation thousands of FP64 atomics land on each of those addresses and
// serialise in the L2.  A block first sums its (bin, value) pairs in a shared-memory hash
// table (per-warp groups add once), then flushes one global atomic per distinct bin.
// Probing is bounded: a bin that finds no slot in BINS_PROBES tries adds to global memory.
constexpr int BINS_PROBES = 8;
template <int S>
struct BlockBins {
  int key[S];
  double val[S];
};

template <int S>
__device__ __forceinline__ void bins_init(BlockBins<S>& t) {
  for (int i = threadIdx.x; i < S; i += blockDim.x) { t.key[i] = -1; t.val[i] = 0.0; }
}

template <int S>
__device__ __forceinline__ void bins_add(BlockBins<S>& t, int bin, double v, double* __restrict__ global) {
  const unsigned h = ((unsigned)bin * 2654435761u) >> 8;
#pragma unroll 1
  for (int p = 0; p < BINS_PROBES; ++p) {
    const int s = (int)((h + (unsigned)p) & (unsigned)(S - 1));
    const int old = atomicCAS(&t.key[s], -1, bin);
    if (old == -1 || old == bin) { atomicAdd(&t.val[s], v); return; }
  }
  atomicAdd(global + bin, v);
}

// warp_tally1 whose group sums go into the block's table (every lane calls it, converged)
template <int S>
__device__ __forceinline__ void warp_bins_add(bool flush, int key, double v, BlockBins<S>& t,
                                              double* __restrict__ global, WarpStage* st) {
  const unsigned fm = __ballot_sync(FULL, flush);
  if (fm == 0u) return;
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(FULL, flush ? key : -1 - lane);
  st->a[lane] = v;
  __syncwarp();
  if (flush && (__ffs(peers) - 1) == lane) {
    double s = 0.0;
    unsigned m = peers;
    while (m) { const int l = __ffs(m) - 1; m &= m - 1; s += st->a[l]; }
    bins_add(t, key, s, global);
  }
  __syncwarp();
}

// after a __syncthreads(): one global atomic per occupied slot
template <int S>
__device__ __forceinline__ void bins_flush(BlockBins<S>& t, double* __restrict__ global) {
  for (int i = threadIdx.x; i < S; i += blockDim.x)
    if (t.key[i] >= 0) atomicAdd(global + t.key[i], t.val[i]);
}

// The same per-block aggregation for integer counts (32-bit shared-memory adds, exact).
template <int S>
struct BlockCounts {
  int key[S];
  unsigned val[S];
};

template <int S>
__device__ __forceinline__ void counts_init(BlockCounts<S>& t) {
  for (int i = threadIdx.x; i < S; i += blockDim.x) { t.key[i] = -1; t.val[i] = 0u; }
}

template <int S, typename G>
__device__ __forceinline__ void counts_add(BlockCounts<S>& t, int bin, unsigned v, G* __restrict__ global) {
  const unsigned h = ((unsigned)bin * 2654435761u) >> 8;
#pragma unroll 1
  for (int p = 0; p < BINS_PROBES; ++p) {
    const int s = (int)((h + (unsigned)p) & (unsigned)(S - 1));
    const int old = atomicCAS(&t.key[s], -1, bin);
    if (old == -1 || old == bin) { atomicAdd(&t.val[s], v); return; }
  }
  atomicAdd(global + bin, (G)v);
}

template <int S, typename G>
__device__ __forceinline__ void counts_flush(BlockCounts<S>& t, G* __restrict__ global) {
  for (int i = threadIdx.x; i < S; i += blockDim.x)
    if (t.key[i] >= 0) atomicAdd(global + t.key[i], (G)t.val[i]);
}

// Comb copies of an entry of weight wf in a bin of comb weight ew > 0: floor(w / ew + xi), xi the
// uniform of the Philox word xw.  The quotient is formed in FP32 first; only where that leaves the
// floor open is it divided in FP64.  With ew normal in FP32 and its reciprocal too, the FP32 sum is
// off by at most 5e-7 (s + 1): ew's rounding and the sum's 2^-24 each, the quotient 2 ulp.  Outside
// that range (an FP32 subnormal keeps few digits of ew; above 2^126 the quotient is 0) every copy is
// divided in FP64.
__device__ __forceinline__ int comb_floor(float wf, double ew, uint32_t xw) {
  const float ef = (float)ew;
  const float s = __fdividef(wf, ef) + u01f(xw);
  const float fl = floorf(s), fr = s - fl, open = 1e-6f * (s + 1.f);
  if (ef > 2e-38f && ef < 8e37f && s < 4e6f && fr > open && fr < 1.f - open) return (int)fl;
  return (int)floor((double)wf / ew + u01d(xw));
}

// ---- energy tallies in 64-bit fixed point ----
// Deposited and escaped energy are summed as integers in units of q = W * 2^-60, W the
// total weight tracked in the step (an upper bound of every such sum, so no total exceeds
// 2^60 units).  Integer adds are exact and independent of order: each deposit is rounded
// once, by at most q/2, however many adds a cell receives, which keeps the step's energy
// balance far inside 1e-12 where FP64 atomics would drift with the square root of the
// number of adds.
constexpr double FX_ONE = 1152921504606846976.0;  // 2^60
__device__ __forceinline__ double fx_inv_quantum(double wsum) { return wsum > 0.0 ? FX_ONE / wsum : 0.0; }
__device__ __forceinline__ unsigned long long fx_units(double e, double inv_q) { return __double2ull_rn(e * inv_q); }
__device__ __forceinline__ double fx_energy(unsigned long long u, double wsum) { return (double)u * (wsum / FX_ONE); }

// 64-bit add to a shared-memory tally as two 32-bit adds, the low word's carry going into the
// high word: the sum is exact modulo 2^64 in any order, and both adds are native shared-memory
// atomics, where the 64-bit one is a compare-and-swap loop (the ten launches of a 2M crooked-pipe
// run: 14.0 ms with the 64-bit atomic, 12.6 ms so).
__device__ __forceinline__ void smem_add_u64(unsigned long long* t, unsigned long long v) {
  unsigned* q = reinterpret_cast<unsigned*>(t);
  const unsigned lo = (unsigned)v;
  const unsigned old = atomicAdd(q, lo);
  const unsigned hi = (unsigned)(v >> 32) + (old + lo < lo ? 1u : 0u);
  if (hi) atomicAdd(q + 1, hi);
}

// Two tallies at once, the first in fixed point (a zero value issues no reduction)
__device__ __forceinline__ void warp_tally_fx(bool flush, int key, unsigned long long ua, double vb,
                                              unsigned long long* __restrict__ ta, double* __restrict__ tb,
                                              WarpStage* st) {
  const unsigned fm = __ballot_sync(FULL, flush);
  if (fm == 0u) return;
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(FULL, flush ? key : -1 - lane);
  if (__all_sync(FULL, !flush || __popc(peers) == 1)) {
    if (flush) { if (ua) atomicAdd(ta + key, ua); if (vb != 0.0) atomicAdd(tb + key, vb); }
    return;
  }
  unsigned long long* sa_u = reinterpret_cast<unsigned long long*>(st->a);
  sa_u[lane] = ua; st->b[lane] = vb;
  __syncwarp();
  if (flush && (__ffs(peers) - 1) == lane) {
    unsigned long long su = 0ull;
    double sb = 0.0;
    unsigned m = peers;
    while (m) {
      const int l = __ffs(m) - 1;
      m &= m - 1;
      su += sa_u[l]; sb += st->b[l];
    }
    if (su) atomicAdd(ta + key, su);
    if (sb != 0.0) atomicAdd(tb + key, sb);
  }
  __syncwarp();
}

// Group of a photon sampled from the Planck spectrum at T (mixture of Gammas,
// MG_IMC/MG_IMC2D.py:202-254): n from the 1/n^4 mixture CDF, x = (four Exp(1)) / n,
// energy T*x located in the group edges.
// below_last: an energy below the lowest edge goes to the last group (MG_IMC/MG_IMC1D.py:180-186);
// otherwise to the first (MG_IMC/MG_IMC2D.py:242-243)
__device__ __forceinline__ int planck_group(double T, const double* edges, int G, const double* mixcdf, double un,
                                            double u1, double u2, double u3, double u4, bool below_last = false) {
  if (!(T > 0.0)) return 0;
  double ns = 200.0;
  for (int i = 0; i < 200; ++i) if (un <= mixcdf[i]) { ns = (double)(i + 1); break; }
  const double x = (-log(u1) - log(u2) - log(u3) - log(u4)) / ns;
  const double f = T * x;
  if (f < edges[0]) return below_last ? G - 1 : 0;
  if (f >= edges[G]) return G - 1;
  for (int g = 0; g < G; ++g) if (f >= edges[g] && f < edges[g + 1]) return g;
  return G - 1;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
__device__ __forceinline__ unsigned long long warp_sum_u(unsigned v) {
  return (unsigned long long)__reduce_add_sync(FULL, v);
}

}  // namespace imcdev
