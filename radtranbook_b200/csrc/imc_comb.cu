// imc_comb.cu — stochastic comb of the census bank (IMC/IMC1D.py:770-828,
// IMC/IMC2D.py:1448-1511, MG_IMC/MG_IMC2D.py:1270-1378).
//
//   1. ecen[b]  = sum of live weights per bin (cell, or cell + nc*group)      k_comb_ecen
//   2. ew[b]    = ecen / max(1, rint(Nmax ecen / E))                          k_comb_plan
//   3. n_k      = floor(w_k / ew[b] + xi_k), xi word k % 4 of Philox block
//      (k / 4, 1, step, TAG_COMB); tile totals and, by the last block to finish,
//      their exclusive scan                                                   k_comb_count
//   4. copies written in bank order (tile-local scan + tile offset; entries
//      staged in shared memory, one thread per output copy), and by blocks of
//      their own disc[b] = ecen - (copies in b) * FP32(ew) and optionally that
//      energy after the comb per bin (exact: equal FP32 weights summed in FP64) k_comb_scatter
// Order of the output bank = order of the input bank, so the result is deterministic.
// Modes (MG_IMC/MG_IMC1D.py:1187-1200, 808-820): when the comb plan decides not to comb
// (Nmax = 0, or fewer live entries than a threshold) every live entry is copied once with its
// weight (disc = 0); with conserve_rad each bin's copies share its pre-comb energy equally.
#include <algorithm>

#include "imc_device.cuh"
#include "imc_internal.h"

using namespace imcdev;

namespace {

constexpr int TILE = 1024;      // entries per tile: one count total, one scatter block
constexpr int WARP_ENTRIES = 128;  // entries a warp counts at a time (four per lane)

__device__ __forceinline__ int bin_of(const CombArgs& a, long long k) {
  return a.per_group ? a.cell[k] + a.nc * a.group[k] : a.cell[k];
}

// Bounds-checked build: a bin outside [0, nb) is reported and its entry treated as dead.
__device__ __forceinline__ bool bin_ok(const CombArgs& a, int b) {
#ifdef IMC_CHECKED
  if (b >= 0 && b < a.nb) return true;
  if (a.sum) atomicOr(&a.sum->flags, (int)IMC_FLAG_BOUNDS);
  return false;
#else
  (void)a; (void)b;
  return true;
#endif
}

// weight of every copy in bin b: the comb weight, or the bin's energy shared equally
__device__ __forceinline__ float copy_weight(const CombArgs& a, int b) {
  if (!a.conserve_rad) return (float)a.ew[b];
  const double n = (double)a.ncopy[b];
  return n > 0.0 ? (float)(a.ecen[b] / n) : 0.f;
}

constexpr int ECH = 4096;       // consecutive entries per k_comb_ecen block
constexpr int EBINS = 1024;     // shared-memory bins per block

// Each block sums a contiguous run of ECH entries into its shared bins (warp groups first),
// then adds one value per distinct bin to ecen.
__global__ void __launch_bounds__(256) k_comb_ecen(CombArgs a) {
  pdl_wait();     // the previous kernel of the stream has completed
  pdl_trigger();  // the next one may be scheduled
  __shared__ BlockBins<EBINS> t;
  __shared__ WarpStage stages[8];
  WarpStage* st = stages + (threadIdx.x >> 5);
  bins_init(t);
  __syncthreads();
  const long long n_in = min((long long)*a.d_n_in, (long long)a.n_bound);  // a count above the bound is never read
  const long long base = (long long)blockIdx.x * ECH;
  // block-uniform trip count keeps every warp converged for the aggregated reduction
  unsigned n_live = 0;
  for (int i = 0; i < ECH; i += 256) {
    const long long k = base + i + threadIdx.x;
    bool live = false;
    int b = 0;
    double w = 0.0;
    if (k < n_in) {
      const float wf = a.w[k];
      if (wf > 0.f) { b = bin_of(a, k); live = bin_ok(a, b); w = live ? (double)wf : 0.0; if (!live) b = 0; }
    }
    n_live += live ? 1u : 0u;
    warp_bins_add(live, b, w, t, a.ecen, st);
  }
  n_live = __reduce_add_sync(FULL, n_live);
  if ((threadIdx.x & 31) == 0 && n_live && a.n_live) atomicAdd(a.n_live, (unsigned long long)n_live);
  __syncthreads();
  bins_flush(t, a.ecen);
}

// copies of one entry: floor(w / ew + xi), xi its comb uniform (word k % 4 of Philox block
// (k / 4, 1, step, TAG_COMB), k the pre-comb index)
__device__ __forceinline__ int comb_copies(const CombArgs& a, float wf, int bk, bool compact, uint32_t xw, int& b) {
  b = 0;
  if (!(wf > 0.f) || !bin_ok(a, bk)) return 0;
  b = bk;
  if (compact) return 1;
  const double ew = a.ew[b];
  return ew > 0.0 ? comb_floor(wf, ew, xw) : 0;
}

// Copies per entry, per tile and per bin.  A block takes `per` consecutive tiles, its warps
// WARP_ENTRIES entries at a time with 16-byte vector loads (where the bank arrays allow them).
// Copies per bin are summed in shared memory, runs of equal bins in a lane first, and added to the
// global ones once per block: in a counter per bin (DENSE: many entries, bins that fit), else in a
// hash table over the block's one tile.  The last block to finish scans the
// tile totals (a ticket; no block waits).  With a hash table of bins per 4096 entries instead, which
// a mixed bank overflows, and an FP64 division per entry this took 94 us for 8.7 M entries in 12600
// bins and 45 us for 91 thousand in 3150 (23 blocks); now 55 and 13 us.
constexpr int kCountMaxTiles = 64;  // tiles a block takes at most
constexpr int kCountSlots = TILE / 2;  // hash table of a block (a tile rarely has more bins; adds past it go to global memory)

template <bool DENSE>
__global__ void __launch_bounds__(512, 2) k_comb_count(CombArgs a, long long ntiles, int per) {
  pdl_wait();     // the previous kernel of the stream has completed
  pdl_trigger();  // the next one may be scheduled
  extern __shared__ unsigned bin_cnt[];  // DENSE: [nb]
  __shared__ unsigned long long tile_sum[kCountMaxTiles];
  __shared__ long long sh[32];
  __shared__ bool last;
  const uint32_t step = a.step_dev ? *a.step_dev : a.step;  // graph replay
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int q = threadIdx.x; q < per; q += blockDim.x) tile_sum[q] = 0ull;
  BlockCounts<kCountSlots>& hash = *reinterpret_cast<BlockCounts<kCountSlots>*>(bin_cnt);  // else
  if (DENSE) for (int q = threadIdx.x; q < a.nb; q += blockDim.x) bin_cnt[q] = 0u;
  else counts_init(hash);
  __syncthreads();
  const long long n_in = min((long long)*a.d_n_in, (long long)a.n_bound);  // the tiles cover n_bound entries
  const bool compact = *a.mode != 0;
  const long long tile0 = (long long)blockIdx.x * per;
  const int units = (int)max(0LL, min((long long)per, ntiles - tile0)) * (TILE / WARP_ENTRIES);
  for (int u = wid; u < units; u += nw) {
    const long long kj = tile0 * TILE + (long long)u * WARP_ENTRIES + 4 * lane;
    float wv[4] = {0.f, 0.f, 0.f, 0.f};
    int bv[4] = {0, 0, 0, 0};
    if (a.vec16 && kj + 3 < n_in) {  // kj % 4 == 0: the 16-byte loads are aligned
      const float4 W = *reinterpret_cast<const float4*>(a.w + kj);
      const int4 C = *reinterpret_cast<const int4*>(a.cell + kj);
      wv[0] = W.x; wv[1] = W.y; wv[2] = W.z; wv[3] = W.w;
      bv[0] = C.x; bv[1] = C.y; bv[2] = C.z; bv[3] = C.w;
      if (a.per_group) {
        const int4 g = *reinterpret_cast<const int4*>(a.group + kj);
        bv[0] += a.nc * g.x; bv[1] += a.nc * g.y; bv[2] += a.nc * g.z; bv[3] += a.nc * g.w;
      }
    } else {
      for (int q = 0; q < 4; ++q)
        if (kj + q < n_in) { wv[q] = a.w[kj + q]; bv[q] = bin_of(a, kj + q); }
    }
    // one Philox block for the four entries kj..kj+3 (kj % 4 == 0), drawn when one of them is alive
    U4 r{0u, 0u, 0u, 0u};
    if (!compact && (wv[0] > 0.f || wv[1] > 0.f || wv[2] > 0.f || wv[3] > 0.f))
      r = draw_rk(a.rk, (uint32_t)(kj >> 2), 1, step, TAG_COMB);
    int nv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) nv[q] = comb_copies(a, wv[q], bv[q], compact, u4_word(r, q), bv[q]);
    if (kj + 3 < n_in) {
      *reinterpret_cast<int4*>(a.cnt + kj) = make_int4(nv[0], nv[1], nv[2], nv[3]);  // workspace: aligned
    } else {
      for (int q = 0; q < 4; ++q) if (kj + q < n_in) a.cnt[kj + q] = nv[q];
    }
    // copies per bin: equal neighbours are one add
    unsigned run = 0, tsum = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      run += (unsigned)nv[q];
      tsum += (unsigned)nv[q];
      const bool ends = run != 0u && (q == 3 || bv[q + 1] != bv[q]);
      if (ends) { if (DENSE) atomicAdd(bin_cnt + bv[q], run); else counts_add(hash, bv[q], run, a.ncopy); }
      if (q < 3 && bv[q + 1] != bv[q]) run = 0u;
    }
    const unsigned ws = __reduce_add_sync(FULL, tsum);
    if (lane == 0 && ws) atomicAdd(&tile_sum[u / (TILE / WARP_ENTRIES)], (unsigned long long)ws);
  }
  __syncthreads();
  if (DENSE) {
    for (int q = threadIdx.x; q < a.nb; q += blockDim.x)
      if (bin_cnt[q]) atomicAdd(a.ncopy + q, (unsigned long long)bin_cnt[q]);
  } else {
    counts_flush(hash, a.ncopy);
  }
  for (int q = threadIdx.x; q < per && tile0 + q < ntiles; q += blockDim.x) a.blk[tile0 + q] = (long long)tile_sum[q];
  // ---- the last block: exclusive scan of the tile totals in place (blk[ntiles] = total) ----
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(a.ticket, 1ull) == (unsigned long long)gridDim.x - 1ull;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) *a.ticket = 0ull;  // for a comb launched again on this workspace
  const int t = threadIdx.x, nt = blockDim.x;
  const long long share = (ntiles + nt - 1) / nt;
  const long long lo = min((long long)t * share, ntiles), hi = min(lo + share, ntiles);
  long long sum = 0;
  for (long long q = lo; q < hi; ++q) sum += __ldcg(a.blk + q);
  long long x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const long long y = __shfl_up_sync(FULL, x, o); if (lane >= o) x += y; }
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  if (wid == 0) {
    long long v = lane < nw ? sh[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const long long y = __shfl_up_sync(FULL, v, o); if (lane >= o) v += y; }
    sh[lane] = v;
  }
  __syncthreads();
  long long run = x - sum + (wid ? sh[wid - 1] : 0);
  for (long long q = lo; q < hi; ++q) { const long long v = __ldcg(a.blk + q); a.blk[q] = run; run += v; }
  if (t == 0) {
    const long long total = sh[31];
    a.blk[ntiles] = total;
    a.sum->n_out = total;
    if (total > a.out_capacity) { atomicOr(&a.sum->flags, (int)IMC_FLAG_COMB_OVERFLOW); a.sum->n_census = 0; }
    else a.sum->n_census = total;  // the combed bank is the next step's census
  }
}

// Shared memory of k_comb_scatter: the tile's inclusive copy counts, then its entries' fields
// (pos1, dir1, copy weight, cell; pos2, dir2 in 2-D; group when the bank has one), TILE each, and
// the entry of each of the first SCAT_MAP output copies.
constexpr int SCAT_T = TILE / 4;
constexpr int SCAT_MAP = 2 * TILE;
__host__ __device__ inline int scatter_fields(bool two_d, bool grp) { return 4 + (two_d ? 2 : 0) + (grp ? 1 : 0); }
__host__ __device__ inline size_t scatter_smem(bool two_d, bool grp) {
  return sizeof(int) * (size_t)TILE * (1 + scatter_fields(two_d, grp)) + sizeof(unsigned short) * SCAT_MAP;
}

// One block per tile (the first ntiles blocks): its entries are staged in shared memory with
// 16-byte loads (one thread per four entries), each thread notes its entries' output positions, and
// one thread per output copy then copies its entry's fields from shared memory, so the global loads
// and the stores of a warp are both contiguous.  A tile with more than SCAT_MAP copies finds the
// entries of the others by a binary search of the scanned counts, and one with more than four times that
// those of all.  `split` blocks share a tile, each staging it and writing a stretch of its copies, where
// a small bank makes many copies an entry (scatter_split).  The remaining blocks take 256
// bins each: disc and the energy after the comb.  Against tiles of 4096 entries, a search for
// every copy, the copy weight gathered per copy and a launch of its own for the bins: 28 -> 13 us
// for 91 thousand entries, 29 -> 20 us for 1.7 M; 8.7 M take the same 88 us (0.40 GB moved, at two
// thirds of the rate of a copy).
__global__ void __launch_bounds__(SCAT_T) k_comb_scatter(CombArgs a, long long ntiles, int split) {
  pdl_wait();     // the previous kernel of the stream has completed
  pdl_trigger();  // the next one may be scheduled
  extern __shared__ __align__(16) int sm_tile[];
  __shared__ int sh[SCAT_T / 32];
  const bool compact = *a.mode != 0;
  if ((long long)blockIdx.x >= ntiles * split) {
    const long long b = ((long long)blockIdx.x - ntiles * split) * blockDim.x + threadIdx.x;
    double after = 0.0;
    if (b < a.nb) {
      // compact only: every live entry kept with its weight, nothing is lost
      after = compact ? a.ecen[b] : (double)a.ncopy[b] * (double)copy_weight(a, (int)b);
      a.disc[b] = a.ecen[b] - after;
      if (a.after) a.after[b] = after;
    }
    after = warp_sum_d(after);
    if ((threadIdx.x & 31) == 0 && after != 0.0) atomicAdd(&a.sum->comb_after, after);
    return;
  }
  const bool two_d = a.p2 != nullptr, grp = a.group != nullptr;
  int* incl = sm_tile;
  float* sP1 = reinterpret_cast<float*>(incl + TILE);
  float* sD1 = sP1 + TILE;
  float* sW = sD1 + TILE;
  int* sC = reinterpret_cast<int*>(sW + TILE);
  float* sP2 = reinterpret_cast<float*>(sC + TILE);   // 2-D only
  float* sD2 = sP2 + TILE;                            // 2-D only
  int* sG = reinterpret_cast<int*>(two_d ? sD2 + TILE : sP2);  // with a group array only
  unsigned short* entry = reinterpret_cast<unsigned short*>(sm_tile + TILE * (1 + scatter_fields(two_d, grp)));
  const long long tile = split > 1 ? blockIdx.x / split : blockIdx.x;
  const long long tile0 = tile * TILE;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long n_in = min((long long)*a.d_n_in, (long long)a.n_bound);
  const int q0 = 4 * threadIdx.x;
  const long long k0 = tile0 + q0;
  const bool full = k0 + 3 < n_in;
  int c[4] = {0, 0, 0, 0};
  if (full) {
    const int4 v = *reinterpret_cast<const int4*>(a.cnt + k0);  // 16-byte aligned: k0 % 4 == 0
    c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
  } else {
    for (int j = 0; j < 4; ++j) if (k0 + j < n_in) c[j] = a.cnt[k0 + j];
  }
  const int s4 = c[0] + c[1] + c[2] + c[3];
  // stage the fields of the four entries (only where they have copies)
  const uintptr_t al = reinterpret_cast<uintptr_t>(a.p1) | reinterpret_cast<uintptr_t>(a.d1) |
                       reinterpret_cast<uintptr_t>(a.p2) | reinterpret_cast<uintptr_t>(a.d2) |
                       (grp ? reinterpret_cast<uintptr_t>(a.group) : 0);
  if (s4 > 0) {
    int cl[4] = {0, 0, 0, 0}, gr[4] = {0, 0, 0, 0};
    if (full && a.vec16 && (al & 15u) == 0) {
      *reinterpret_cast<float4*>(sP1 + q0) = *reinterpret_cast<const float4*>(a.p1 + k0);
      *reinterpret_cast<float4*>(sD1 + q0) = *reinterpret_cast<const float4*>(a.d1 + k0);
      const int4 C = *reinterpret_cast<const int4*>(a.cell + k0);
      cl[0] = C.x; cl[1] = C.y; cl[2] = C.z; cl[3] = C.w;
      if (two_d) {
        *reinterpret_cast<float4*>(sP2 + q0) = *reinterpret_cast<const float4*>(a.p2 + k0);
        *reinterpret_cast<float4*>(sD2 + q0) = *reinterpret_cast<const float4*>(a.d2 + k0);
      }
      if (grp) {
        const int4 G = *reinterpret_cast<const int4*>(a.group + k0);
        gr[0] = G.x; gr[1] = G.y; gr[2] = G.z; gr[3] = G.w;
      }
    } else {
      for (int j = 0; j < 4; ++j) {
        if (c[j] == 0) continue;
        const long long k = k0 + j;
        sP1[q0 + j] = a.p1[k]; sD1[q0 + j] = a.d1[k]; cl[j] = a.cell[k];
        if (two_d) { sP2[q0 + j] = a.p2[k]; sD2[q0 + j] = a.d2[k]; }
        if (grp) gr[j] = a.group[k];
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (c[j] == 0) continue;
      sC[q0 + j] = cl[j];
      if (grp) sG[q0 + j] = gr[j];
      sW[q0 + j] = compact ? a.w[k0 + j] : copy_weight(a, a.per_group ? cl[j] + a.nc * gr[j] : cl[j]);
    }
  }
  // block-exclusive scan of the threads' sums, then the entries' inclusive sums
  int x = s4;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(FULL, x, o); if (lane >= o) x += y; }
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  int run = x - s4, total = 0;
  for (int q = 0; q < SCAT_T / 32; ++q) { if (q < wid) run += sh[q]; total += sh[q]; }
  const int mapped = total <= 4 * SCAT_MAP ? SCAT_MAP : 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    for (int o = run; o < run + c[j] && o < mapped; ++o) entry[o] = (unsigned short)(q0 + j);
    run += c[j];
    incl[q0 + j] = run;
  }
  __syncthreads();
  int first = 0, last = total;
  if (split > 1) {
    const int share = (total / split / SCAT_T + 1) * SCAT_T, part = (int)(blockIdx.x - tile * split);
    first = min(total, part * share);
    last = min(total, first + share);
  }
  const long long out0 = a.blk[tile];
  for (int o = first + threadIdx.x; o < last; o += blockDim.x) {
    const long long dst = out0 + o;
    if (dst >= a.out_capacity) break;  // overflow: flagged by the scan, caller regrows
    int e;
    if (o < mapped) {
      e = entry[o];
    } else {
      int lo = 0, hi = TILE - 1;  // the entry j with incl[j-1] <= o < incl[j]
      while (lo < hi) { const int mid = (lo + hi) >> 1; if (incl[mid] > o) hi = mid; else lo = mid + 1; }
      e = lo;
    }
    a.op1[dst] = sP1[e]; a.od1[dst] = sD1[e];
    if (two_d) { a.op2[dst] = sP2[e]; a.od2[dst] = sD2[e]; }
    a.ow[dst] = sW[e];
    a.ot[dst] = 0.f; a.ocell[dst] = sC[e];
    if (a.ogroup) a.ogroup[dst] = grp ? sG[e] : 0;
  }
}

}  // namespace

cudaError_t imc_launch_comb_ecen(const CombArgs& a, cudaStream_t s) {
  if (a.n_bound <= 0) return cudaSuccess;
  ++g_imc_launches;
  IMC_LAUNCH_PDL(k_comb_ecen, (unsigned)((a.n_bound + ECH - 1) / ECH), 256, 0, s, a);
  return cudaGetLastError();
}

cudaError_t imc_launch_comb_count(const CombArgs& a, cudaStream_t s) {
  ++g_imc_launches;
  const long long ntiles = (a.n_bound + TILE - 1) / TILE;
  // a counter per bin pays from about half a million entries (below, zeroing and flushing it costs
  // more than the hash table's probes), two blocks per SM while it fits
  const size_t dense = sizeof(unsigned) * (size_t)a.nb;
  if (a.n_bound >= (1LL << 19) && dense <= 100 * 1024) {
    int per = (int)std::min<long long>(kCountMaxTiles, std::max<long long>(4, (ntiles + 295) / 296));
    const cudaError_t e = smem_opt_in<k_comb_count<true>>(dense);
    if (e != cudaSuccess) return e;
    IMC_LAUNCH_PDL(k_comb_count<true>, (unsigned)((ntiles + per - 1) / per), 512, dense, s, a, ntiles, per);
  } else {
    const int per = 1, threads = 32 * (TILE / WARP_ENTRIES);
    IMC_LAUNCH_PDL(k_comb_count<false>, (unsigned)std::max<long long>(1, ntiles), threads,
                   sizeof(BlockCounts<kCountSlots>), s, a, ntiles, per);
  }
  return cudaGetLastError();
}

// Blocks a tile: one per SCAT_MAP copies that the target asks of each, as long as they all fit the chip
// (four blocks an SM).
static int scatter_split(long long n_max, long long ntiles) {
  const long long copies = n_max / std::max(1LL, ntiles);
  return (int)std::max(1LL, std::min((copies + SCAT_MAP - 1) / SCAT_MAP, 4LL * 148 / std::max(1LL, ntiles)));
}

cudaError_t imc_launch_comb_scatter(const CombArgs& a, cudaStream_t s) {
  const long long ntiles = (a.n_bound + TILE - 1) / TILE;
  ++g_imc_launches;
  const int split = scatter_split(a.n_max, ntiles);
  const size_t smem = scatter_smem(a.p2 != nullptr, a.group != nullptr);
  static_assert(sizeof(int) * TILE * 8 + 2 * SCAT_MAP <= 48 * 1024, "no opt-in for the largest layout");
  IMC_LAUNCH_PDL(k_comb_scatter, (unsigned)(ntiles * split + (a.nb + SCAT_T - 1) / SCAT_T), SCAT_T, smem, s, a, ntiles,
                 split);
  return cudaGetLastError();
}
