// imc_block.cuh — single-block FP64 building blocks shared by the per-problem planning
// kernels (one 1024-thread block per problem): the canonical summation order, the count
// scan and the volume-source plan.  Files that include this are compiled without FMA
// contraction, so the numbers match the CPU oracle's (canon_sum, ceil counts) exactly.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace imcblk {

constexpr int NT = 1024;

__device__ __forceinline__ double pow4(double T) { const double t2 = T * T; return t2 * t2; }
__device__ __forceinline__ double pow3(double T) { return T * T * T; }

// The halving tree over 1024 partial sums (red[t] += red[t + h], h = 512 .. 1), by any whole number
// of warps: its last five levels are one warp's, by shuffles (the same pairs).  The result is on
// every thread; red may be used again after.
__device__ __forceinline__ double tree_1024(double* red) {
  for (int h = NT / 2; h >= 32; h >>= 1) {
    for (int t = threadIdx.x; t < h; t += blockDim.x) red[t] += red[t + h];
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    double v = red[threadIdx.x];
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) v += __shfl_down_sync(0xffffffffu, v, h);
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const double r = red[0];
  __syncthreads();
  return r;
}

// 1024 strided partial sums, then a halving tree (the oracle's canon_sum).  Each partial
// loads B of its terms at a time before adding them in order (same sum, fewer waits; B = 16
// only where the kernel has registers to spare at 1024 threads).
template <int B = 8>
__device__ inline double block_canon_sum(const double* x, long long n, double* red) {
  const int t = threadIdx.x;
  double s = 0.0;
  for (long long i0 = t; i0 < n; i0 += (long long)B * NT) {
    double v[B];
#pragma unroll
    for (int j = 0; j < B; ++j) { const long long i = i0 + (long long)j * NT; v[j] = i < n ? x[i] : 0.0; }
#pragma unroll
    for (int j = 0; j < B; ++j) if (i0 + (long long)j * NT < n) s += v[j];
  }
  red[t] = s;
  __syncthreads();
  return tree_1024(red);
}

// Exclusive offset of this thread's value over the block (1024 threads); sh needs 32 entries,
// and holds the block's total in sh[31] until the next call.
__device__ inline long long block_exclusive(long long s, long long* sh) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  long long x = s;  // inclusive scan within the warp
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) { const long long y = __shfl_up_sync(0xffffffffu, x, d); if (lane >= d) x += y; }
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  if (wid == 0) {
    long long v = lane < NT / 32 ? sh[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const long long y = __shfl_up_sync(0xffffffffu, v, d); if (lane >= d) v += y; }
    sh[lane] = v;  // inclusive over the warps
  }
  __syncthreads();
  return x - s + (wid ? sh[wid - 1] : 0);
}

// Exclusive scan of per-order-position counts n[0..m) into off[0..m]; returns the total.
// Integer sums are exact in any order: each thread sums a contiguous chunk, the chunk totals
// are scanned, and each thread writes its chunk's offsets.  sh needs 32 entries.
__device__ inline long long block_scan_counts(const long long* n, long long* off, int m, long long* sh) {
  const int t = threadIdx.x;
  const int per = (m + NT - 1) / NT;
  const int lo = min(t * per, m), hi = min(lo + per, m);
  long long s = 0;
  for (int o = lo; o < hi; ++o) s += n[o];
  long long run = block_exclusive(s, sh);
  const long long total = sh[NT / 32 - 1];
  __syncthreads();  // sh is the caller's again
  for (int o = lo; o < hi; ++o) { const long long v = n[o]; off[o] = run; run += v; }
  if (t == 0) off[m] = total;
  __syncthreads();
  return total;
}

// The same with the counts in shared memory (a bank holds fewer than 2^31 entries), scanned in
// place, so that the offsets leave in contiguous stores.
__device__ inline long long block_scan_counts(int* n, long long* off, int m, long long* sh) {
  const int t = threadIdx.x;
  const int per = (m + NT - 1) / NT;
  const int lo = min(t * per, m), hi = min(lo + per, m);
  long long s = 0;
  for (int o = lo; o < hi; ++o) s += n[o];
  long long run = block_exclusive(s, sh);
  const long long total = sh[NT / 32 - 1];
  for (int o = lo; o < hi; ++o) { const int v = n[o]; n[o] = (int)run; run += v; }
  __syncthreads();
  for (int o = t; o < m; o += NT) off[o] = n[o];
  if (t == 0) off[m] = total;
  __syncthreads();
  return total;
}

// The tracking table's scatter slot: the effective scatter opacity, 0 at or below the geometry's
// threshold, negative where the distance is capped (sigma_s L > 1e4 in FP32, L the cell's smaller
// width; L = 0: no cap), so that a flight neither compares with the threshold nor forms L.
__device__ __forceinline__ float scatter_entry(double ss64, float threshold, float L) {
  const float ss = (float)ss64;
  if (!(ss > threshold)) return 0.f;
  return ss * L > 10000.0f ? -ss : ss;
}

// order position o = i*ny + j (the reference's i-outer, j-inner source loops)
__device__ __forceinline__ int order_to_cell(int o, int nx, int ny) {
  const int i = o / ny, j = o - (o / ny) * ny;
  return i + nx * j;
}

// Volume-source counts (ceil(N QV_c / Q), in source order; min1_round: max(1, round), the
// Carter-Forest 1-D emission rule), per-cell weights and the energy actually issued per
// cell (n_c times the FP32 weight, exact in FP64), whose canonical sum goes to *total (its partial
// sums follow the cells as the counts do, so they are formed on the way).  The counts stay in
// shared memory (s_cnt, nc ints) where the caller has room, else in cnt.
__device__ inline long long plan_volume(const double* QV, long long N, int nx, int ny, int nc, int* s_cnt,
                                        long long* cnt, long long* off, float* w, double* issued, double* red,
                                        long long* sh, double* total, bool min1_round = false) {
  constexpr int B = 4;
  const double Qt = block_canon_sum(QV, nc, red);
  double s = 0.0;
  // cells in storage order (coalesced loads); the count goes to the cell's order position
  for (int c0 = threadIdx.x; c0 < nc; c0 += B * NT) {
    double q[B];
#pragma unroll
    for (int j = 0; j < B; ++j) q[j] = c0 + j * NT < nc ? QV[c0 + j * NT] : 0.0;
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int c = c0 + j * NT;
      if (c >= nc) break;
      const int cj = c / nx, o = (c - cj * nx) * ny + cj;
      long long n = 0;
      if (Qt > 0.0 && N > 0)
        n = min1_round ? max(1LL, (long long)rint((double)N * q[j] / Qt)) : (long long)ceil((double)N * q[j] / Qt);
      if (s_cnt) s_cnt[o] = (int)n; else cnt[o] = n;
      const float wc = n > 0 ? (float)(q[j] / (double)n) : 0.f;
      w[c] = wc;
      const double e = (double)n * (double)wc;
      issued[c] = e;
      s += e;
    }
  }
  red[threadIdx.x] = s;
  __syncthreads();
  *total = tree_1024(red);
  return s_cnt ? block_scan_counts(s_cnt, off, nc, sh) : block_scan_counts(cnt, off, nc, sh);
}

}  // namespace imcblk
