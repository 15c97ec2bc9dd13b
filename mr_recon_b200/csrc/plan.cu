// Plan creation and trajectory binning.
//
// A plan holds the geometry of n_slices NUFFT problems. mrn_plan_set_traj
// turns a trajectory into the per-tile sample lists the tile kernels consume:
//   interpolation: every sample belongs to the tile holding its first tap;
//   gridding     : every sample is listed once for each tile its footprint
//                  touches (1..2^d entries), so each tile owns its output.
// Both lists are sorted by tile with a stable radix sort (samples keep their
// trajectory order inside a tile) and cut into work items of at most
// max_chunk samples. This replaces the per-call locs preparation of the
// reference (prep_ungrid_shapes / prep_grid_shapes, ungrid.py:851-894,
// grid.py:508-553) and has no counterpart in its Triton launch (one program
// per point chunk, ungrid.py:127-129).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>

#include "common.cuh"
#include "internal.cuh"

using namespace mrn;

namespace mrn {

thread_local int g_last_cuda_error = 0;

int cuda_fail(cudaError_t e) {
  g_last_cuda_error = (int)e;
  return e == cudaErrorMemoryAllocation ? MRN_ERR_NOMEM : MRN_ERR_CUDA;
}

int set_dynamic_smem_fn(const void* kernel, size_t dyn) {
  struct Rec {
    size_t static_bytes;
    size_t opted;  // largest dynamic size opted into so far
  };
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, Rec> seen;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e);
  std::lock_guard<std::mutex> lock(mu);
  auto it = seen.find({kernel, dev});
  if (it == seen.end()) {
    cudaFuncAttributes a;
    e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess) return cuda_fail(e);
    it = seen.emplace(std::make_pair(kernel, dev), Rec{a.sharedSizeBytes, 0}).first;
  }
  Rec& r = it->second;
  if (dyn + r.static_bytes <= 48 * 1024 || dyn <= r.opted) return MRN_OK;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  if (e != cudaSuccess) return cuda_fail(e);
  r.opted = dyn;
  return MRN_OK;
}

__device__ __forceinline__ int find_slice_by_point(const SliceGeom* sl, int ns, int64_t p) {
  int lo = 0, hi = ns - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (sl[mid].pt_off <= p) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int find_slice_by_tile(const SliceGeom* sl, int ns, int t, int gridding) {
  int lo = 0, hi = ns - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if ((gridding ? sl[mid].gtile_base : sl[mid].tile_base) <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Distinct tiles of one dimension touched by the valid taps of a sample at
// wrapped coordinate u: taps j = lo + q, valid iff |(float)j - u| <= r (the
// float32 mask of weights1d..3d, kernels.py:268-393), cell = j mod nos. The valid
// taps are a run and tiles have at least ntaps - 1 cells (tiles_for), so they
// are those of its ends.
__device__ __forceinline__ int dim_tiles(float u, float r, int ntaps, int nos, int nt, int (&tiles)[2]) {
  const int lo = (int)ceilf(__fsub_rn(u, r));
  auto valid = [&](int q) { return fabsf(__fsub_rn((float)(lo + q), u)) <= r; };
  int q0 = 0, q1 = ntaps - 1;
  while (q0 <= q1 && !valid(q0)) ++q0;
  while (q1 > q0 && !valid(q1)) --q1;
  if (q0 > q1) return 0;
  tiles[0] = nt == 1 ? 0 : tile_of(pos_mod(lo + q0, nos), nos, nt);
  tiles[1] = nt == 1 ? 0 : tile_of(pos_mod(lo + q1, nos), nos, nt);
  return tiles[0] == tiles[1] ? 1 : 2;
}

// Per sample: scaled, wrapped coordinates (fourier.py:420-430 then
// ungrid.py:873), interpolation tile key (tile of the first candidate tap),
// and the number of gridding tiles its footprint touches.
__global__ void k_prep_points(const SliceGeom* __restrict__ sl, int ns, int ndim, KBParams kb,
                              const float* __restrict__ trj, int64_t npts,
                              float4* __restrict__ coord, unsigned* __restrict__ key_i,
                              int* __restrict__ val_i, int* __restrict__ ecnt) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npts) return;
  const int s = find_slice_by_point(sl, ns, p);
  const SliceGeom& g = sl[s];
  const int64_t lp = p - g.pt_off;
  float u[kMaxDim] = {0.f, 0.f, 0.f};
  int lin = 0;
  int ntouch = 1;
  for (int i = 0; i < ndim; ++i) {
    const float k = trj[(g.pt_off + lp) * ndim + i];
    float v = __fadd_rn(__fmul_rn(k, g.scale[i]), g.shift[i]);
    v = remainder_f32(v, (float)g.nos[i]);
    u[i] = v;
    const int lo = (int)ceilf(__fsub_rn(v, kb.radius[i]));
    const int t0 = tile_of(pos_mod(lo, g.nos[i]), g.nos[i], g.ntile[i]);
    lin = lin * g.ntile[i] + t0;
    int tiles[2];
    ntouch *= dim_tiles(v, kb.radius[i], kb.ntaps[i], g.nos[i], g.gntile[i], tiles);
  }
  coord[p] = make_float4(u[0], u[1], u[2], 0.f);
  key_i[p] = (unsigned)(g.tile_base + lin);
  val_i[p] = (int)p;
  ecnt[p] = ntouch;
}

// Start of a gridding entry's window of K - 1 cells along the last axis (tile
// `tile` of it; K: gtaps), or 10 - K where all K taps lie inside the tile: the
// order of the register-tile gridding's entries within a tile.
__device__ __forceinline__ int window_code(const SliceGeom& g, const KBParams& kb, float u, int tile, int i) {
  const int K = kb.gtaps, KW = K - 1, n = g.nos[i], org = tile_begin(tile, n, g.gntile[i]);
  const int size = tile_begin(tile + 1, n, g.gntile[i]) - org;
  const int lo = (int)ceilf(__fsub_rn(u, kb.radius[i]));
  int st = (lo < 0 ? lo + n : (lo >= n ? lo - n : lo)) - org;
  if (st >= size) st -= n;
  const bool last = fabsf(__fsub_rn((float)(lo + K - 1), u)) <= kb.radius[i];
  return last && st >= 0 && st + K <= size ? 10 - K : min(max(st, 0), size - KW);
}

// Emit (tile, point) gridding entries at the scanned offsets; with code_bits
// the key is the tile above kGPartBits zeros and the window code.
__global__ void k_emit_entries(const SliceGeom* __restrict__ sl, int ns, int ndim, KBParams kb,
                               const float4* __restrict__ coord, int64_t npts,
                               const int* __restrict__ eoff, int code_bits, unsigned* __restrict__ key,
                               int* __restrict__ val) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npts) return;
  const int s = find_slice_by_point(sl, ns, p);
  const SliceGeom& g = sl[s];
  const float4 c4 = coord[p];
  const float uu[3] = {c4.x, c4.y, c4.z};
  int tiles[kMaxDim][2] = {};
  int nt[kMaxDim] = {1, 1, 1};
  for (int i = 0; i < ndim; ++i)
    nt[i] = dim_tiles(uu[i], kb.radius[i], kb.ntaps[i], g.nos[i], g.gntile[i], tiles[i]);
  unsigned win[2] = {0u, 0u};
  for (int c = 0; code_bits > 0 && c < nt[ndim - 1]; ++c)
    win[c] = (unsigned)window_code(g, kb, uu[ndim - 1], tiles[ndim - 1][c], ndim - 1);
  int o = eoff[p];
  for (int a = 0; a < nt[0]; ++a)
    for (int b = 0; b < (ndim > 1 ? nt[1] : 1); ++b)
      for (int c = 0; c < (ndim > 2 ? nt[2] : 1); ++c) {
        int lin = tiles[0][a];
        if (ndim > 1) lin = lin * g.gntile[1] + tiles[1][b];
        if (ndim > 2) lin = lin * g.gntile[2] + tiles[2][c];
        const int w = ndim == 3 ? c : b;
        key[o] = (unsigned)(g.gtile_base + lin) << code_bits | (w == 0 ? win[0] : win[1]);
        val[o] = (int)p;
        ++o;
      }
}

// Entries per tile (192^3 kooshball, 20.6 M entries: 242 us, one atomic per entry 535).
__global__ void k_tile_hist(const unsigned* __restrict__ key, int code_bits, int64_t n, int* __restrict__ cnt) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const unsigned k = key[e] >> code_bits;
  const unsigned peers = __match_any_sync(__activemask(), k);
  if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(cnt + k, __popc(peers));
}

// Put the part of the trajectory into the keys of tiles of more entries than a
// work item of their slice takes.
__global__ void k_entry_parts(const SliceGeom* __restrict__ sl, int ns, const int* __restrict__ val,
                              const int* __restrict__ cnt, const int2* __restrict__ ent, int64_t n,
                              unsigned* __restrict__ key) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int t = (int)(key[e] >> kGCodeBits), s = find_slice_by_tile(sl, ns, t, 1);
  if (cnt[t] <= ent[s].y) return;
  const SliceGeom& g = sl[s];
  key[e] |= (unsigned)(((int64_t)val[e] - g.pt_off) * (1 << kGPartBits) / g.m) << kGWinBits;
}

__global__ void k_gather_coords(const float4* __restrict__ src, const int* __restrict__ perm,
                                int64_t n, float4* __restrict__ dst) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) dst[e] = src[perm[e]];
}

__global__ void k_tile_ranges(const unsigned* __restrict__ key, int code_bits, int64_t n, int ntiles,
                              int* __restrict__ start, int* __restrict__ end) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const unsigned k = key[e] >> code_bits;
  if ((int)k >= ntiles) return;
  if (e == 0 || key[e - 1] >> code_bits != k) start[k] = (int)e;
  if (e == n - 1 || key[e + 1] >> code_bits != k) end[k] = (int)(e + 1);
}

// Items per tile: entries / chunk, rounded up (gridding: the chunk of the
// tile's slice, and at least one item, which stores an empty tile's zeros).
__global__ void k_item_counts(const SliceGeom* __restrict__ sl, int ns, const int2* __restrict__ ent,
                              const int* __restrict__ start, const int* __restrict__ end,
                              int ntiles, int chunk, int gridding, int* __restrict__ nitems) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  const int c = end[t] - start[t];
  const int k = gridding ? ent[find_slice_by_tile(sl, ns, t, 1)].y : chunk;
  nitems[t] = max(gridding, (c + k - 1) / k);
}

// Work items of every tile at the scanned offsets. Gridding tiles with more
// than one item are split tiles: each gets a run of n partial-tile slots
// (counts[4] hands them out) and a record {tile, first slot, n} in
// split_tiles (counts[3] counts them); item q of the tile writes slot
// first + q. The order in which tiles claim slots does not matter: the
// reduction adds a tile's slots in item order.
__global__ void k_emit_items(const SliceGeom* __restrict__ sl, int ns, const int* __restrict__ start,
                             const int* __restrict__ end, const int* __restrict__ nitems,
                             const int* __restrict__ ioff, int ntiles, int chunk,
                             Item* __restrict__ items, int4* __restrict__ split_tiles,
                             int* __restrict__ counts, int count_slot, int gridding) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  const int n = nitems[t];
  const int s = find_slice_by_tile(sl, ns, t, gridding);
  const int c = end[t] - start[t];
  int base = -1;
  if (gridding && n > 1) {
    base = atomicAdd(&counts[4], n);
    const int k = atomicAdd(&counts[3], 1);
    split_tiles[k] = make_int4(t, base, n, 0);
  }
  for (int q = 0; q < n; ++q) {
    // the tile's entries spread evenly over its items (at most chunk each)
    const int b0 = (int)(((int64_t)q * c) / n), b1 = (int)(((int64_t)(q + 1) * c) / n);
    Item it;
    it.slice = s;
    it.tile = t - (gridding ? sl[s].gtile_base : sl[s].tile_base);
    it.start = start[t] + b0;
    it.count = b1 - b0;
    it.split = base >= 0 ? base + q + 1 : 0;
    it.pad[0] = it.pad[1] = it.pad[2] = 0;
    items[ioff[t] + q] = it;
  }
  if (t == ntiles - 1) counts[count_slot] = ioff[t] + n;
}

// Sort keys of the longest-first item order: count + 1 for real items, 0 for
// the padding (slice -1) past them, so a stable descending sort keeps real
// items of equal length in tile order and leaves the padding last.
__global__ void k_item_keys(const Item* __restrict__ items, int64_t n, unsigned* __restrict__ key,
                            int* __restrict__ idx) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Item it = items[i];
  key[i] = it.slice < 0 ? 0u : (unsigned)it.count + 1u;
  idx[i] = (int)i;
}

__global__ void k_gather_items(const Item* __restrict__ src, const int* __restrict__ idx, int64_t n,
                               Item* __restrict__ dst) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

// Gridding entries per work item of a slice: from its own entries alone, so that
// a cell's sums are the same whatever shares the plan. About six items per SM in
// 2D and four in 3D would share a slice's entries evenly; fewer entries leave
// the densest tiles as a tail, more split tiles cost partial tiles. 2D 96..256
// (256^2, 32 coils, 266 k entries: 64 / 128 / 192 / 256 / 512 entries 172 / 110 /
// 91 / 87 / 111 us; 128^2, 1 coil, 50 k: 64 / 96 / 128 / 256 27.5 / 28.3 / 32 / 46,
// but 16 such slices of 8 coils together 223 / 181 / 164 / 141), 3D 512..4096
// (192^3, 16 coils, 20.6 M: 2048 / 4096 / 8192 6.1 / 5.8 / 5.7 ms; the last one's
// longer partial sums near the k-space centre round more; 64^3, 8 coils, 0.7 M:
// 512 / 1024 / 2048 / 4096 238 / 206 / 219 / 349 us, four such slices 909 / 718 /
// 615 / 601).
__host__ __device__ static int grid_chunk_of(int ndim, int sm_count, int64_t entries) {
  if (ndim == 1) return 1024;
  const int64_t lo = ndim == 2 ? 96 : 512, hi = ndim == 2 ? 256 : 4096;
  const int64_t share = entries / ((ndim == 2 ? 6 : 4) * (int64_t)sm_count);
  const int64_t step = ndim == 2 ? 64 : 32, c = (share + step - 1) / step * step;
  return (int)(c < lo ? lo : (c > hi ? hi : c));
}

// Per slice {gridding entries, entries per work item} (chunk 0: grid_chunk_of).
__global__ void k_slice_entries(const SliceGeom* __restrict__ sl, int ns, const int* __restrict__ off,
                                const int* __restrict__ cnt, int64_t npts, int ndim, int sm_count, int chunk,
                                int2* __restrict__ out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ns) return;
  const int64_t p0 = sl[s].pt_off, p1 = p0 + sl[s].m;
  int e = 0;
  if (p1 > p0) e = (p1 < npts ? off[p1] : off[npts - 1] + cnt[npts - 1]) - off[p0];
  out[s] = make_int2(e, chunk > 0 ? chunk : grid_chunk_of(ndim, sm_count, e));
}

static inline unsigned blocks_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// Tiles per dimension for an edge length: at most ceil(nos / edge), and each
// tile at least K-1 cells wide so a kernel footprint touches at most two tiles
// per dimension (balanced partition, tile_begin / tile_of).
static int tiles_for(int nos, int edge, int K) {
  int nt = (nos + edge - 1) / edge;
  if (K > 1) nt = std::min(nt, std::max(1, nos / (K - 1)));
  return std::max(1, nt);
}


// Tile arrays are allocated for the larger of the two tilings.
// Kernel shape parameters: beta per dimension, and the I0 power series
// c_k = (beta^2/4)^k / (k!)^2 (in double) that the fast kernels evaluate,
// which exists only when every dimension has the same beta.
static void kb_set_beta(KBParams& kb, const double* betas, int ndim) {
  const double beta = betas[0];
  kb.beta = (float)beta;
  kb.uniform_beta = 1;
  for (int i = 0; i < kMaxDim; ++i) {
    kb.betad[i] = (float)(i < ndim ? betas[i] : beta);
    if (i < ndim && (float)betas[i] != kb.beta) kb.uniform_beta = 0;
  }
  const double q = beta * beta / 4.0;
  double c = 1.0, sum = 0.0;
  for (int k = 0; k < kKBTerms; ++k) {
    kb.coef[k] = (float)c;
    sum += c;
    c *= q / ((double)(k + 1) * (k + 1));
  }
  // c now holds the first omitted term; later terms shrink by q / (k+1)^2 each
  const double ratio = q / ((double)(kKBTerms + 1) * (kKBTerms + 1));
  const double tail = ratio < 1.0 ? c / (1.0 - ratio) : 1e300;
  kb.series = tail < 1e-9 * sum ? 1 : 0;
  // fewest terms (a multiple of 4, at least 16) whose dropped tail is below
  // 1e-9 of the sum; the tail after term n is bounded by the omitted terms
  // kept in coef plus the geometric bound above
  kb.nterms = kKBTerms;
  for (int n = 16; n < kKBTerms; n += 4) {
    double t = tail;
    for (int k = n; k < kKBTerms; ++k) t += (double)kb.coef[k];
    if (t < 1e-9 * sum) { kb.nterms = n; break; }
  }
}

static int64_t tile_capacity(const mrn_plan* P) { return std::max(P->ntiles, P->ngtiles); }

// Interpolation and gridding tilings of every slice, and their global tile ids.
void compute_tiling(mrn_plan* P) {
  int tiles = 0, gtiles = 0;
  for (int i = 0; i < kMaxDim; ++i) P->tmax_cells[i] = P->tmax_gcells[i] = 1;
  for (auto& g : P->h_slices) {
    int tc = 1, gc = 1;
    for (int i = 0; i < kMaxDim; ++i) {
      if (i >= P->ndim) {
        g.ntile[i] = g.gntile[i] = 1;
        continue;
      }
      const int K = P->kb.ntaps[i];
      const int nt = tiles_for(g.nos[i], P->tile[i], K);
      const int gt = tiles_for(g.nos[i], P->gtile[i], K);
      g.ntile[i] = nt;
      g.gntile[i] = gt;
      tc *= nt;
      gc *= gt;
      P->tmax_cells[i] = std::max(P->tmax_cells[i], (g.nos[i] + nt - 1) / nt);
      P->tmax_gcells[i] = std::max(P->tmax_gcells[i], (g.nos[i] + gt - 1) / gt);
    }
    g.tile_base = tiles;
    g.gtile_base = gtiles;
    tiles += tc;
    gtiles += gc;
  }
  P->ntiles = tiles;
  P->ngtiles = gtiles;
}

static cudaEvent_t pool_event(mrn_plan* P) {
  if (!P->ev_pool.empty()) {
    cudaEvent_t e = P->ev_pool.back();
    P->ev_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
  return e;
}

StageTimer::StageTimer(mrn_plan* p, int stage, cudaStream_t s) : P(p), st(s) {
  if (!P || !P->timing) return;
  mrn_plan::TimingRec r{stage, pool_event(P), pool_event(P)};
  if (!r.a || !r.b) return;
  cudaEventRecord(r.a, st);
  P->timing_recs.push_back(r);
  idx = (int)P->timing_recs.size() - 1;
}

StageTimer::~StageTimer() {
  if (idx >= 0) cudaEventRecord(P->timing_recs[idx].b, st);
}

// Upload the slice table and its shared-k-space twin (every ksp_off 0).
cudaError_t upload_slices(mrn_plan* P) {
  cudaError_t e = cudaMemcpy(P->d_slices, P->h_slices.data(), P->nslices * sizeof(SliceGeom),
                             cudaMemcpyHostToDevice);
  if (e != cudaSuccess || !P->d_slices_kshared) return e;
  std::vector<SliceGeom> ks(P->h_slices);
  for (auto& g : ks) g.ksp_off = g.row_off = 0;
  return cudaMemcpy(P->d_slices_kshared, ks.data(), P->nslices * sizeof(SliceGeom), cudaMemcpyHostToDevice);
}

template <class T>
static int dev_alloc(T** p, size_t n) {
  if (*p) { cudaFree(*p); *p = nullptr; }
  if (n == 0) n = 1;
  cudaError_t e = cudaMalloc((void**)p, n * sizeof(T));
  if (e != cudaSuccess) return cuda_fail(e);
  return MRN_OK;
}

// New tile edges: recompute both tilings, grow the per-tile arrays when the
// finer tiling needs more entries, refresh the device slice table. The bound
// trajectory's binning is stale afterwards (mrn_plan_set_traj again).
static int retile(mrn_plan* P) {
  P->traj_set = false;
  P->wtab_ok = false;
  compute_tiling(P);
  const int64_t need = std::max<int64_t>(tile_capacity(P), 1);
  int rc = MRN_OK;
  if (need > P->cap_tiles) {
    int** bufs[] = {&P->d_tile_start_i, &P->d_tile_end_i, &P->d_tile_start_g, &P->d_tile_end_g,
                    &P->d_tile_nitems, &P->d_tile_item_off};
    for (int** b : bufs)
      if ((rc = dev_alloc(b, (size_t)need)) != MRN_OK) {
        P->cap_tiles = 0;
        return rc;
      }
    if ((rc = dev_alloc(&P->d_split_tiles, (size_t)need)) != MRN_OK) {
      P->cap_tiles = 0;
      return rc;
    }
    P->cap_tiles = need;
  }
  cudaError_t e = cudaSetDevice(P->device);
  if (e == cudaSuccess) e = upload_slices(P);
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

static int ensure_cub(mrn_plan* P, size_t bytes) {
  if (bytes <= P->cub_tmp_bytes && P->d_cub_tmp) return MRN_OK;
  if (P->d_cub_tmp) cudaFree(P->d_cub_tmp);
  P->d_cub_tmp = nullptr;
  P->cub_tmp_bytes = 0;
  cudaError_t e = cudaMalloc(&P->d_cub_tmp, bytes);
  if (e != cudaSuccess) return cuda_fail(e);
  P->cub_tmp_bytes = bytes;
  return MRN_OK;
}

}  // namespace mrn

#define CK(x)                                   \
  do {                                          \
    cudaError_t _e = (x);                       \
    if (_e != cudaSuccess) return cuda_fail(_e); \
  } while (0)
#define RK(x)                  \
  do {                         \
    int _r = (x);              \
    if (_r != MRN_OK) return _r; \
  } while (0)

extern "C" {

const char* mrn_version(void) { return "mrnufft 0.1.0 (sm_100a)"; }

const char* mrn_error_string(int code) {
  switch (code) {
    case MRN_OK: return "ok";
    case MRN_ERR_ARG: return "invalid argument";
    case MRN_ERR_WIDTH: return "kernel width out of range (1 <= width < 16)";
    case MRN_ERR_CUDA: return "CUDA error";
    case MRN_ERR_CUFFT: return "cuFFT error";
    case MRN_ERR_NOMEM: return "device allocation failed";
    case MRN_ERR_STATE: return "trajectory not set on plan";
    case MRN_ERR_UNSUPPORTED: return "unsupported configuration";
    case MRN_ERR_SCRATCH: return "problem exceeds the 32 MiB fixed scratch of mrn_interp_noalloc";
    default: return "unknown error";
  }
}

int mrn_last_cuda_error(void) { return mrn::g_last_cuda_error; }

int mrn_plan_create(mrn_plan** out, int ndim, int n_slices, const int* im_size,
                    const int64_t* n_pts, const int* n_coil, double oversamp,
                    const double* width, double beta, int flags, const int* tile,
                    int coil_group, int max_chunk, int device) {
  if (!out || !im_size || !n_pts || !n_coil || !width) return MRN_ERR_ARG;
  *out = nullptr;
  if (ndim < 1 || ndim > kMaxDim || n_slices < 1) return MRN_ERR_ARG;
  const bool raw = (flags & MRN_PLAN_RAW) != 0;
  if (!raw && !(oversamp >= 1.0)) return MRN_ERR_ARG;
  for (int i = 0; i < ndim; ++i)
    if (!(width[i] >= 1.0) || !(width[i] < (double)kMaxTaps)) return MRN_ERR_WIDTH;
  if (tile)
    for (int i = 0; i < ndim; ++i)
      if (tile[i] < 1) return MRN_ERR_ARG;
  if (coil_group < 0 || max_chunk < 0) return MRN_ERR_ARG;

  mrn_plan* P = new mrn_plan();
  P->ndim = ndim;
  P->nslices = n_slices;
  P->flags = flags;
  P->device = device;
  P->oversamp = raw ? 1.0 : oversamp;
  int maxtaps = 0;
  for (int i = 0; i < ndim; ++i) {
    P->width[i] = width[i];
    P->kb.radius[i] = (float)width[i] / 2.0f;
    P->kb.inv_radius[i] = 1.0f / P->kb.radius[i];
    P->kb.ntaps[i] = (int)std::floor(width[i]) + 1;
    maxtaps = std::max(maxtaps, P->kb.ntaps[i]);
  }
  P->tap_max = maxtaps <= 8 ? 8 : 16;
  if (beta <= 0.0) {
    if (raw) { delete P; return MRN_ERR_ARG; }
    const double w = width[0];
    beta = M_PI * std::sqrt(std::pow(w / oversamp * (oversamp - 0.5), 2) - 0.8);
  }
  P->beta = beta;
  {
    double betas[kMaxDim];
    for (int i = 0; i < kMaxDim; ++i) betas[i] = beta;
    kb_set_beta(P->kb, betas, ndim);
  }

  int maxc = 0;
  for (int s = 0; s < n_slices; ++s) {
    if (n_coil[s] < 1 || n_pts[s] < 0) { delete P; return MRN_ERR_ARG; }
    for (int i = 0; i < ndim; ++i)
      if (im_size[s * ndim + i] < 1) { delete P; return MRN_ERR_ARG; }
    maxc = std::max(maxc, n_coil[s]);
  }
  P->max_coil = maxc;

  // Built-in interpolation tile: 10 cells per edge in 2D (tile + halo as a [cell][coil]
  // region for 32 coils: three CTAs per SM), 4 in 3D (16-coil groups), 256 in 1D.
  int deftile[kMaxDim];
  for (int i = 0; i < ndim; ++i) deftile[i] = (ndim == 1) ? 256 : (ndim == 2 ? 10 : 4);
  for (int i = 0; i < ndim; ++i) P->tile[i] = tile ? tile[i] : deftile[i];
  // gridding tiles: 8x8 in 2D (one warp owns a tile), else the interpolation tile
  for (int i = 0; i < ndim; ++i) P->gtile[i] = (ndim >= 2 && !tile) ? 8 : P->tile[i];
  P->max_chunk = max_chunk > 0 ? max_chunk : (ndim == 2 ? 256 : 1024);
  P->grid_chunk = max_chunk;  // 0: from each slice's entry count, at mrn_plan_set_traj

  // Slices
  int64_t img = 0, ksp = 0, ugrid = 0, trjo = 0, pts = 0, xo = 0;
  int64_t prow = 0, irow = 0, xrow = 0;
  int64_t maxe = 0;
  int64_t apodn = 0;
  P->h_slices.resize(n_slices);
  for (int s = 0; s < n_slices; ++s) {
    SliceGeom& g = P->h_slices[s];
    std::memset(&g, 0, sizeof(g));
    int64_t nimg = 1, gos = 1, spans = 1;
    for (int i = 0; i < kMaxDim; ++i) {
      g.n[i] = 1; g.nos[i] = 1; g.ntile[i] = 1; g.hshift[i] = 0; g.scale[i] = 1.f; g.shift[i] = 0.f;
    }
    for (int i = 0; i < ndim; ++i) {
      const int n = im_size[s * ndim + i];
      const int nos = raw ? n : (int)std::ceil(oversamp * n);
      g.n[i] = n;
      g.nos[i] = nos;
      g.hshift[i] = raw ? 0 : nos / 2;
      g.scale[i] = raw ? 1.0f : (float)((double)nos / (double)n);
      g.shift[i] = raw ? 0.0f : (float)(nos / 2);
      nimg *= n;
      gos *= nos;
      spans *= 2;
      g.apod_off[i] = (int)apodn;
      apodn += n;
    }
    g.ncoil = n_coil[s];
    g.m = n_pts[s];
    g.pt_off = pts;
    // rows start on 64 bytes (one-coil plans: the samples themselves)
    const int cbl = coil_block(g.ncoil);
    g.rs = (g.ncoil + cbl - 1) / cbl * cbl;
    g.row_off = maxc == 1 ? ksp : P->n_rows;
    P->n_rows += ((int64_t)g.rs * g.m + 7) / 8 * 8;
    g.img_off = img;
    g.ksp_off = ksp;
    g.ugrid_off = ugrid;
    g.x_off = xo;
    g.gos = gos;
    g.nimg = nimg;
    g.inv_sqrt_n = (float)(1.0 / std::sqrt((double)nimg));
    g.prow_off = prow;
    g.irow_off = irow;
    g.xrow_off = xrow;
    prow += (int64_t)g.ncoil * gos / g.nos[ndim - 1];
    irow += (int64_t)g.ncoil * nimg / g.n[ndim - 1];
    xrow += nimg / g.n[ndim - 1];
    img += (int64_t)g.ncoil * nimg;
    ksp += (int64_t)g.ncoil * g.m;
    ugrid += (int64_t)g.ncoil * gos;
    trjo += g.m * ndim;
    pts += g.m;
    xo += nimg;
    maxe += spans * g.m;
  }
  P->n_img = img;
  P->n_ksp = ksp;
  P->n_grid = ugrid;
  P->n_trj = trjo;
  P->n_pts = pts;
  P->n_x = xo;
  P->n_prow = prow;
  P->n_irow = irow;
  P->n_xrow = xrow;
  compute_tiling(P);
  if (pts >= (int64_t)INT32_MAX || maxe >= (int64_t)INT32_MAX) { delete P; return MRN_ERR_UNSUPPORTED; }

  // Coil group: all coils of the widest slice, limited by shared memory.
  P->coil_group_req = coil_group > 0 ? std::min(coil_group, 64) : 0;
  if (coil_group > 0) {
    P->coil_group = std::min(coil_group, 64);
  } else {
    int64_t cells = 1;
    for (int i = 0; i < ndim; ++i) cells *= (P->tmax_cells[i] + P->kb.ntaps[i] - 1);
    const int64_t budget = 96 * 1024;  // bytes of tile data per CTA, two CTAs per SM
    int cg = (int)std::max<int64_t>(1, budget / ((cells | 1) * 8));
    cg = std::min(cg, 64);
    cg = std::min(cg, maxc);
    // balance groups: same number of groups, fewest coils per group
    const int ngroups = (maxc + cg - 1) / cg;
    cg = (maxc + ngroups - 1) / ngroups;
    P->coil_group = std::max(1, cg);
  }

  // FFT groups (one grid size, one way to transform it) in first-seen order; the internal grid buffer is ordered by group.
  if (!raw) {
    for (int s = 0; s < n_slices; ++s) {
      const SliceGeom& g = P->h_slices[s];
      const bool native = ffx_pays(ndim, g.nos, g.ncoil);
      int found = -1;
      for (size_t q = 0; q < P->fft.size(); ++q) {
        bool same = P->fft[q].native == native;
        for (int i = 0; i < ndim; ++i) same &= (P->fft[q].nos[i] == g.nos[i]);
        if (same) { found = (int)q; break; }
      }
      if (found < 0) {
        mrn_plan::FftGroup fg{};
        for (int i = 0; i < kMaxDim; ++i) fg.nos[i] = g.nos[i];
        fg.native = native;
        fg.batch = 0;
        fg.handle = 0;
        P->fft.push_back(fg);
        found = (int)P->fft.size() - 1;
      }
      P->fft[found].slices.push_back(s);
      P->fft[found].batch += g.ncoil;
    }
  } else {
    for (int s = 0; s < n_slices; ++s) P->h_slices[s].grid_off = P->h_slices[s].ugrid_off;
  }
  for (auto& g : P->h_slices) g.cb = 1;  // ffx_refresh sets the native slices' block

  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) { delete P; return cuda_fail(e); }
  cudaDeviceGetAttribute(&P->sm_count, cudaDevAttrMultiProcessorCount, device);

  int rc = MRN_OK;
#define PK(x) do { rc = (x); if (rc != MRN_OK) { mrn_plan_destroy(P); return rc; } } while (0)
  PK(dev_alloc(&P->d_slices, n_slices));
  PK(dev_alloc(&P->d_slices_kshared, n_slices));
  e = upload_slices(P);
  if (e != cudaSuccess) { mrn_plan_destroy(P); return cuda_fail(e); }

  // Apodization tables a(x) = sqrt(beta^2 - (pi W x)^2) / sinh(.), x = (q - N//2)/Nos
  // (fourier.py:376-418), in double then rounded.
  {
    std::vector<float> ap(std::max<int64_t>(apodn, 1), 1.0f);
    if (!raw && !(flags & MRN_PLAN_NO_APOD)) {
      for (int s = 0; s < n_slices; ++s) {
        const SliceGeom& g = P->h_slices[s];
        for (int i = 0; i < ndim; ++i) {
          for (int q = 0; q < g.n[i]; ++q) {
            const double x = (double)(q - g.n[i] / 2) / (double)g.nos[i];
            const double t = M_PI * P->width[i] * x;
            const double a = std::sqrt(beta * beta - t * t);
            ap[g.apod_off[i] + q] = (float)(a / std::sinh(a));
          }
        }
      }
    }
    PK(dev_alloc(&P->d_apod, ap.size()));
    e = cudaMemcpy(P->d_apod, ap.data(), ap.size() * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { mrn_plan_destroy(P); return cuda_fail(e); }
  }

  const int64_t np = std::max<int64_t>(pts, 1);
  PK(dev_alloc(&P->d_coord_i, np));
  PK(dev_alloc(&P->d_perm_i, np));
  PK(dev_alloc(&P->d_coord_tmp, np));
  PK(dev_alloc(&P->d_entry_cnt, 2 * np));
  PK(dev_alloc(&P->d_key_a, np));
  PK(dev_alloc(&P->d_val_a, np));
  PK(dev_alloc(&P->d_key_is, np));
  {
    // sized for the finest tiling either kind may get (plan options can change them)
    const int64_t tmax = std::max<int64_t>(tile_capacity(P), 1);
    PK(dev_alloc(&P->d_tile_start_i, tmax));
    PK(dev_alloc(&P->d_tile_end_i, tmax));
    PK(dev_alloc(&P->d_tile_start_g, tmax));
    PK(dev_alloc(&P->d_tile_end_g, tmax));
    PK(dev_alloc(&P->d_tile_nitems, tmax));
    PK(dev_alloc(&P->d_tile_item_off, tmax));
    PK(dev_alloc(&P->d_split_tiles, tmax));
    P->cap_tiles = tmax;
  }
  PK(dev_alloc(&P->d_counts, 8));
  PK(dev_alloc(&P->d_slice_ent, (size_t)n_slices));
  PK(dev_alloc(&P->d_sync, 64));
  CK(cudaMemset(P->d_sync, 0, 64 * sizeof(unsigned)));
  PK(dev_alloc(&P->d_red, (size_t)n_slices * kMaxRedBlocks));
  PK(dev_alloc(&P->d_rowpart, (size_t)std::max<int64_t>(P->n_xrow, 1)));
  if (!raw) {
    PK(ffx_setup(P));
    if (dev_alloc(&P->d_grid, std::max<int64_t>(P->n_igrid, 1)) != MRN_OK) {
      // without room for whole coil blocks: blocks that the coils fill
      cudaGetLastError();
      P->d_grid = nullptr;
      P->tight_grid = true;
      PK(ffx_setup(P));
      PK(dev_alloc(&P->d_grid, std::max<int64_t>(P->n_igrid, 1)));
    }
    PK(dev_alloc(&P->d_ksp_tmp, std::max<int64_t>(P->n_ksp, 1)));
    PK(cufft_setup(P));
  }
  PK(gather_setup(P));
  if (ndim >= 2) {
    // without room for the rows the plan grids from coil rows (the tile
    // kernels in shared memory)
    e = cudaMalloc((void**)&P->d_rows, std::max<int64_t>(P->n_rows, 1) * sizeof(float2));
    if (e != cudaSuccess) {
      P->d_rows = nullptr;
      cudaGetLastError();
    }
  }
#undef PK
  *out = P;
  return MRN_OK;
}

int mrn_plan_set_beta(mrn_plan* P, const double* beta) {
  if (!P || !beta || !(P->flags & MRN_PLAN_RAW)) return MRN_ERR_ARG;
  for (int i = 0; i < P->ndim; ++i)
    if (!(beta[i] > 0.0)) return MRN_ERR_ARG;
  kb_set_beta(P->kb, beta, P->ndim);
  P->beta = beta[0];
  P->traj_set = false;
  P->wtab_ok = false;
  return MRN_OK;
}

int mrn_plan_set_option(mrn_plan* P, int option, int value) {
  if (!P) return MRN_ERR_ARG;
  switch (option) {
    case MRN_OPT_FAST_KERNELS: P->use_fast = value != 0; return MRN_OK;
    case MRN_OPT_WARP_GRIDDING: P->warp_grid = value != 0; return MRN_OK;
    case MRN_OPT_WEIGHT_TABLES: P->use_wtab = value != 0; return MRN_OK;
    case MRN_OPT_REG_GRIDDING: P->reg_grid = value != 0; return MRN_OK;
    case MRN_OPT_REG_INTERP: P->reg_interp = value != 0; return MRN_OK;
    case MRN_OPT_ENTRY_MAJOR:
      P->use_ent = value != 0;
      P->traj_set = false;  // takes effect at the next mrn_plan_set_traj
      return MRN_OK;
    case MRN_OPT_NATIVE_FFT:
      P->use_ffx = value != 0;
      {
        const int rc = ffx_refresh(P);
        return rc == MRN_OK ? cufft_setup(P) : rc;
      }
    case MRN_OPT_GRID_LANES:
      if (value != 0 && value != 8 && value != 16 && value != 32) return MRN_ERR_ARG;
      P->grid_lanes = value;
      return MRN_OK;
    case MRN_OPT_INTERP_CHUNK:
    case MRN_OPT_GRID_CHUNK:
      if (value < 1) return MRN_ERR_ARG;
      (option == MRN_OPT_INTERP_CHUNK ? P->max_chunk : P->grid_chunk) = value;
      P->traj_set = false;  // items are cut at mrn_plan_set_traj
      P->wtab_ok = false;
      return MRN_OK;
    case MRN_OPT_INTERP_TILE:
    case MRN_OPT_GRID_TILE:
      if (value < 1) return MRN_ERR_ARG;
      for (int i = 0; i < P->ndim; ++i) (option == MRN_OPT_INTERP_TILE ? P->tile : P->gtile)[i] = value;
      return retile(P);
    default: return MRN_ERR_ARG;
  }
}

int mrn_plan_enable_timing(mrn_plan* P, int on) {
  if (!P) return MRN_ERR_ARG;
  P->timing = on != 0;
  return MRN_OK;
}

int mrn_plan_timing(mrn_plan* P, double* ms, int64_t* count) {
  if (!P || !ms || !count) return MRN_ERR_ARG;
  for (int i = 0; i < kNumStages; ++i) { ms[i] = 0.0; count[i] = 0; }
  int rc = MRN_OK;
  for (auto& r : P->timing_recs) {
    cudaError_t e = cudaEventSynchronize(r.b);
    float t = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&t, r.a, r.b);
    if (e != cudaSuccess) rc = cuda_fail(e);
    else if (r.stage >= 0 && r.stage < kNumStages) { ms[r.stage] += t; count[r.stage] += 1; }
    P->ev_pool.push_back(r.a);
    P->ev_pool.push_back(r.b);
  }
  P->timing_recs.clear();
  return rc;
}

int mrn_plan_destroy(mrn_plan* P) {
  if (!P) return MRN_OK;
  for (auto& r : P->timing_recs) { P->ev_pool.push_back(r.a); P->ev_pool.push_back(r.b); }
  for (cudaEvent_t e : P->ev_pool)
    if (e) cudaEventDestroy(e);
  for (auto& fg : P->fft)
    if (fg.handle) cufftDestroy(fg.handle);
  toep_free(P);
  P->ffx.release();
  void* bufs[] = {P->d_slices, P->d_slices_kshared, P->d_apod, P->d_coord_i, P->d_perm_i, P->d_coord_g, P->d_perm_g,
                  P->d_key_a, P->d_key_b, P->d_key_is, P->d_key_g, P->d_val_a, P->d_val_b, P->d_coord_tmp,
                  P->d_entry_cnt, P->d_tile_start_i, P->d_tile_end_i, P->d_tile_start_g,
                  P->d_tile_end_g, P->d_tile_nitems, P->d_tile_item_off, P->d_items_i,
                  P->d_items_g, P->d_counts, P->d_slice_ent, P->d_split_tiles, P->d_cub_tmp, P->d_grid,
                  P->d_ksp_tmp, P->d_sync, P->d_wmeta_i, P->d_wtab_i, P->d_wmeta_g,
                  P->d_wtab_g, P->d_part, P->d_items_tmp, P->d_sort_key[0], P->d_sort_key[1],
                  P->d_sort_idx[0], P->d_sort_idx[1], P->d_red, P->d_rowpart, P->d_rows, P->d_gather};
  for (void* b : bufs)
    if (b) cudaFree(b);
  delete P;
  return MRN_OK;
}

int mrn_plan_offsets(const mrn_plan* P, int64_t* img_off, int64_t* ksp_off, int64_t* grid_off,
                     int64_t* trj_off) {
  if (!P) return MRN_ERR_ARG;
  for (int s = 0; s < P->nslices; ++s) {
    const SliceGeom& g = P->h_slices[s];
    if (img_off) img_off[s] = g.img_off;
    if (ksp_off) ksp_off[s] = g.ksp_off;
    if (grid_off) grid_off[s] = g.ugrid_off;
    if (trj_off) trj_off[s] = g.pt_off * P->ndim;
  }
  return MRN_OK;
}

int mrn_plan_sizes(const mrn_plan* P, int64_t* o) {
  if (!P || !o) return MRN_ERR_ARG;
  o[0] = P->n_img; o[1] = P->n_ksp; o[2] = P->n_grid; o[3] = P->n_trj; o[4] = P->ntiles;
  o[5] = P->h_slices[0].nos[0]; o[6] = P->h_slices[0].nos[1]; o[7] = P->h_slices[0].nos[2];
  return MRN_OK;
}

int mrn_plan_fft_kind(const mrn_plan* P) {
  if (!P) return MRN_ERR_ARG;
  if (!ffx_active(P)) return 0;
  return P->ffx.all ? 1 : 2;
}

int mrn_plan_stats(mrn_plan* P, int64_t* o) {
  if (!P || !o) return MRN_ERR_ARG;
  int hc[4] = {0, 0, 0, 0};
  if (P->traj_set) {
    cudaError_t e = cudaSetDevice(P->device);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(hc, P->d_counts, 4 * sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e);
  }
  o[0] = hc[0]; o[1] = hc[1]; o[2] = P->n_entries_grid; o[3] = hc[3];
  return MRN_OK;
}

int mrn_plan_set_traj(mrn_plan* P, const float* trj, void* stream_) {
  if (!P || (!trj && P->n_pts > 0)) return MRN_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream_;
  const int64_t M = P->n_pts;
  const int T = P->ntiles;    // interpolation tiles
  const int TG = P->ngtiles;  // gridding tiles
  const int TT = std::max(T, TG);
  if (P->cap_tiles < TT) return MRN_ERR_STATE;  // a failed retile left the tile arrays short
  const int ndim = P->ndim;
  auto bits_of = [](int n) {
    int bits = 1;
    while (bits < 31 && (1ll << bits) <= (long long)n) ++bits;
    return bits;
  };
  const int bits = bits_of(T);
  const int code_bits = code_sort_ok(P) && bits_of(TG) + kGCodeBits <= 31 ? kGCodeBits : 0;
  const int gbits = bits_of(TG) + code_bits;
  // buffers grow on demand, if need be into the room of the rows (without them
  // the plan grids from coil rows)
  auto grow = [&](auto** p, int64_t n) {
    int rc = dev_alloc(p, (size_t)n);
    if (rc == MRN_OK || !P->d_rows) return rc;
    cudaGetLastError();
    cudaFree(P->d_rows);
    P->d_rows = nullptr;
    return dev_alloc(p, (size_t)n);
  };
  P->traj_set = false;
  P->code_sorted = code_bits > 0;
  window_taps(P);

  // 1. coordinates, interpolation keys, gridding entry counts
  int* eoff = P->d_entry_cnt + std::max<int64_t>(M, 1);
  size_t need = 0, b = 0;
  const int Mi = (int)std::max<int64_t>(M, 1);
  cub::DeviceScan::ExclusiveSum(nullptr, b, P->d_entry_cnt, eoff, Mi, st);
  need = std::max(need, b);
  cub::DeviceScan::ExclusiveSum(nullptr, b, P->d_tile_nitems, P->d_tile_item_off, TT, st);
  need = std::max(need, b);
  cub::DeviceRadixSort::SortPairs(nullptr, b, P->d_key_a, P->d_key_is, P->d_val_a, P->d_perm_i,
                                  Mi, 0, bits, st);
  need = std::max(need, b);
  RK(ensure_cub(P, need));

  // gridding entries, full work items, and bounds of the split tiles and their
  // partial-tile slots, summed over the slices; the largest work item
  int64_t E = 0, full = 0, max_split = 0, max_slots = 0;
  int gchunk = 1;
  if (M > 0) {
    k_prep_points<<<blocks_for(M), 256, 0, st>>>(P->d_slices, P->nslices, ndim, P->kb, trj, M,
                                                  P->d_coord_tmp, P->d_key_a, P->d_val_a,
                                                  P->d_entry_cnt);
    CK(cudaGetLastError());
    b = P->cub_tmp_bytes;
    CK(cub::DeviceScan::ExclusiveSum(P->d_cub_tmp, b, P->d_entry_cnt, eoff, (int)M, st));
  }
  k_slice_entries<<<blocks_for(P->nslices), 256, 0, st>>>(P->d_slices, P->nslices, eoff, P->d_entry_cnt, M, ndim,
                                                          P->sm_count, P->grid_chunk, P->d_slice_ent);
  CK(cudaGetLastError());
  if (M > 0) {
    std::vector<int2> ent(P->nslices);
    CK(cudaMemcpyAsync(ent.data(), P->d_slice_ent, ent.size() * sizeof(int2), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (const int2& e : ent) {
      E += e.x;
      full += e.x / e.y;
      gchunk = std::max(gchunk, e.y);
      if (e.x > e.y) {
        max_split += e.x / e.y + 1;
        max_slots += 2 * (int64_t)(e.x / e.y) + 1;
      }
    }
  }
  max_split = std::min<int64_t>(max_split, TG);
  P->n_entries_grid = E;

  // 2. gridding entry buffers grow on demand
  const int64_t capE = std::max<int64_t>(E, 1);
  if (P->cap_entries < capE) {
    P->cap_entries = 0;  // until all of them are there
    RK(grow(&P->d_key_b, capE));
    RK(grow(&P->d_val_b, capE));
    RK(grow(&P->d_key_g, capE));
    RK(grow(&P->d_perm_g, capE));
    RK(grow(&P->d_coord_g, capE));
    P->cap_entries = capE;
  }

  // 3. emit gridding entries and sort both lists by tile (stable)
  if (M > 0) {
    k_emit_entries<<<blocks_for(M), 256, 0, st>>>(P->d_slices, P->nslices, ndim, P->kb,
                                                   P->d_coord_tmp, M, eoff, code_bits, P->d_key_b, P->d_val_b);
    if (code_bits > 0 && E > 0) {
      CK(cudaMemsetAsync(P->d_tile_end_g, 0, TG * sizeof(int), st));  // counts, until the ranges are built
      k_tile_hist<<<blocks_for(E), 256, 0, st>>>(P->d_key_b, code_bits, E, P->d_tile_end_g);
      k_entry_parts<<<blocks_for(E), 256, 0, st>>>(P->d_slices, P->nslices, P->d_val_b, P->d_tile_end_g, P->d_slice_ent, E,
                                                   P->d_key_b);
    }
    CK(cudaGetLastError());
    b = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, b, P->d_key_b, P->d_key_g, P->d_val_b, P->d_perm_g,
                                    (int)std::max<int64_t>(E, 1), 0, gbits, st);
    RK(ensure_cub(P, std::max(b, P->cub_tmp_bytes)));
    b = P->cub_tmp_bytes;
    CK(cub::DeviceRadixSort::SortPairs(P->d_cub_tmp, b, P->d_key_a, P->d_key_is, P->d_val_a,
                                       P->d_perm_i, (int)M, 0, bits, st));
    b = P->cub_tmp_bytes;
    CK(cub::DeviceRadixSort::SortPairs(P->d_cub_tmp, b, P->d_key_b, P->d_key_g, P->d_val_b,
                                       P->d_perm_g, (int)E, 0, gbits, st));
    k_gather_coords<<<blocks_for(M), 256, 0, st>>>(P->d_coord_tmp, P->d_perm_i, M, P->d_coord_i);
    if (E > 0)
      k_gather_coords<<<blocks_for(E), 256, 0, st>>>(P->d_coord_tmp, P->d_perm_g, E, P->d_coord_g);
    CK(cudaGetLastError());
  }

  // 4. per-tile ranges
  CK(cudaMemsetAsync(P->d_tile_start_i, 0, T * sizeof(int), st));
  CK(cudaMemsetAsync(P->d_tile_end_i, 0, T * sizeof(int), st));
  CK(cudaMemsetAsync(P->d_tile_start_g, 0, TG * sizeof(int), st));
  CK(cudaMemsetAsync(P->d_tile_end_g, 0, TG * sizeof(int), st));
  CK(cudaMemsetAsync(P->d_counts, 0, 8 * sizeof(int), st));
  if (M > 0) {
    k_tile_ranges<<<blocks_for(M), 256, 0, st>>>(P->d_key_is, 0, M, T, P->d_tile_start_i,
                                                 P->d_tile_end_i);
    if (E > 0)
      k_tile_ranges<<<blocks_for(E), 256, 0, st>>>(P->d_key_g, code_bits, E, TG, P->d_tile_start_g,
                                                   P->d_tile_end_g);
  }

  // 5. work items, launched at capacities known from T, M and E alone, so the
  // host needs no further read-back: a tile with c entries makes
  // ceil(c / chunk) items (gridding: at least one), hence at most
  // T + M / chunk + 1 of them; split gridding tiles of a slice of e entries
  // have more than its chunk entries each (at most e / chunk + 1 tiles) and
  // ceil(c / chunk) < 2 c / chunk items each (fewer than 2 e / chunk + 2 slots).
  const int chunk = P->max_chunk;
  const int64_t max_items_i = M > 0 ? (int64_t)T + M / chunk + 1 : 0;
  const int64_t max_items_g = (int64_t)TG + full + 1;
  if (max_items_i >= (int64_t)INT32_MAX || max_items_g >= (int64_t)INT32_MAX) return MRN_ERR_UNSUPPORTED;
  if (P->cap_items_i < max_items_i) {
    P->cap_items_i = 0;
    RK(grow(&P->d_items_i, max_items_i));
    P->cap_items_i = max_items_i;
  }
  if (P->cap_items_g < max_items_g) {
    P->cap_items_g = 0;
    RK(grow(&P->d_items_g, max_items_g));
    P->cap_items_g = max_items_g;
  }
  const int64_t max_items = std::max(max_items_i, max_items_g);
  if (P->cap_sort < max_items) {
    P->cap_sort = 0;
    RK(grow(&P->d_items_tmp, max_items));
    for (int k = 0; k < 2; ++k) {
      RK(grow(&P->d_sort_key[k], max_items));
      RK(grow(&P->d_sort_idx[k], max_items));
    }
    P->cap_sort = max_items;
  }
  const int64_t part_elems = max_slots * (int64_t)P->max_coil * grid_tile_cells(P);
  if (P->cap_part < part_elems) {
    P->cap_part = 0;
    RK(grow(&P->d_part, part_elems));
    P->cap_part = part_elems;
  }
  {
    size_t nb = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, nb, P->d_sort_key[0], P->d_sort_key[1],
                                              P->d_sort_idx[0], P->d_sort_idx[1],
                                              (int)std::max<int64_t>(max_items, 1), 0, 32, st);
    RK(ensure_cub(P, std::max(nb, P->cub_tmp_bytes)));
  }
  // Emit into the staging list (padding pre-filled with slice = -1), then
  // order longest first: CTAs start in index order, so the last wave holds
  // short items instead of a few long tiles.
  auto make_items = [&](int ntiles, int ch, int64_t cap, int count_slot, int gridding,
                        const int* tstart, const int* tend, Item* out) -> int {
    if (cap == 0) return MRN_OK;
    CK(cudaMemsetAsync(P->d_items_tmp, 0xff, (size_t)cap * sizeof(Item), st));
    k_item_counts<<<blocks_for(ntiles), 256, 0, st>>>(P->d_slices, P->nslices, P->d_slice_ent, tstart, tend, ntiles,
                                                      ch, gridding, P->d_tile_nitems);
    size_t nb = P->cub_tmp_bytes;
    CK(cub::DeviceScan::ExclusiveSum(P->d_cub_tmp, nb, P->d_tile_nitems, P->d_tile_item_off, ntiles, st));
    k_emit_items<<<blocks_for(ntiles), 256, 0, st>>>(P->d_slices, P->nslices, tstart, tend,
                                                     P->d_tile_nitems, P->d_tile_item_off, ntiles, ch,
                                                     P->d_items_tmp, P->d_split_tiles, P->d_counts,
                                                     count_slot, gridding);
    k_item_keys<<<blocks_for(cap), 256, 0, st>>>(P->d_items_tmp, cap, P->d_sort_key[0], P->d_sort_idx[0]);
    CK(cudaGetLastError());
    int kbits = 1;
    while (kbits < 32 && (1ll << kbits) <= (long long)ch + 1) ++kbits;
    nb = P->cub_tmp_bytes;
    CK(cub::DeviceRadixSort::SortPairsDescending(P->d_cub_tmp, nb, P->d_sort_key[0], P->d_sort_key[1],
                                                 P->d_sort_idx[0], P->d_sort_idx[1], (int)cap, 0, kbits,
                                                 st));
    k_gather_items<<<blocks_for(cap), 256, 0, st>>>(P->d_items_tmp, P->d_sort_idx[1], cap, out);
    CK(cudaGetLastError());
    return MRN_OK;
  };
  RK(make_items(T, chunk, max_items_i, 0, 0, P->d_tile_start_i, P->d_tile_end_i, P->d_items_i));
  RK(make_items(TG, gchunk, max_items_g, 1, 1, P->d_tile_start_g, P->d_tile_end_g, P->d_items_g));
  RK(build_wtabs(P, st));
  P->n_items_interp = max_items_i;
  P->n_items_grid = max_items_g;
  P->n_split = max_split;
  P->traj_set = true;
  return MRN_OK;
}

}  // extern "C"
