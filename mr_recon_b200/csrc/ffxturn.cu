// The turning pass of the Toeplitz normal operator (toeplitz.cu): along the
// first axis, forward FFT, product with the kernel and inverse FFT of a column
// in one kernel, so the padded spectrum never reaches global memory.
//
// The forward transform's last stage has the points u n/R + b of butterfly b
// in registers, and a transform whose first stage has the same radix R starts
// from exactly those points: the inverse runs the radices in reverse order, so
// the product needs no exchange in between. Shared memory is crossed between
// stages only (twice for a two-stage length, four times for 512 = 8 x 8 x 8).
// Rows beyond the image are neither read nor written.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "ffx_dft.cuh"
#include "internal.cuh"

namespace mrn {

namespace {

constexpr int kTurnThreads = 512;

template <int W>
struct TurnCols {
  int64_t base[W];  // row 0 of the column in the grid (-1: no column)
  int cell[W];      // cell of the later axes
};

// Lanes run across the columns, W float2 a row: two rows of W = 8 are one
// conflict-free half-warp wherever consecutive rows or blocks of an odd number
// of rows meet. Two CTAs of 512 threads an SM (64 registers): 512 points, 32
// coils, 512 columns take 75 us; with 76 registers, so one CTA, 110 us.
template <int W, bool PRIMES>
__global__ void __launch_bounds__(kTurnThreads, PRIMES ? 1 : 2)
k_ffx_turn(const SliceGeom* __restrict__ sl, const FfxTurn* __restrict__ turns, int s0,
           const float2* __restrict__ twg, const float2* __restrict__ kern, float2* __restrict__ grid) {
  constexpr int WS = W;
  extern __shared__ float2 fsm[];
  __shared__ TurnCols<W> cols;
  __shared__ FfxTurn tn;
  {
    const int* from = reinterpret_cast<const int*>(turns + s0 + blockIdx.y);
    for (int i = threadIdx.x; i < (int)(sizeof(FfxTurn) / sizeof(int)); i += blockDim.x)
      reinterpret_cast<int*>(&tn)[i] = from[i];
  }
  __syncthreads();
  const SliceGeom& g = sl[s0 + blockIdx.y];
  const int cb = g.cb, n = tn.fwd.n, tid = threadIdx.x, nt = blockDim.x;
  const int ncols = g.ncoil * tn.icells;
  const int f0 = blockIdx.x * W;
  if (f0 >= ncols) return;
  if (tid < W) {
    // columns are numbered [coil block][cell][coil of the block]
    const int f = f0 + tid;
    const int kb = f / (tn.icells * cb), nc = min(cb, g.ncoil - kb * cb);
    const int rem = f - kb * tn.icells * cb;
    const int cell = rem / max(nc, 1), cc = rem - cell * nc;
    cols.base[tid] = f < ncols ? g.grid_off + (kb * g.gos + cell) * cb + cc : (int64_t)-1;
    cols.cell[tid] = cell;
  }
  const int ns = tn.fwd.ns;
  float2* twf = fsm;
  float2* twi = twf + n;
  float2* A = twi + n;
  float2* B = A + tn.buf * WS;
  for (int i = tid; i < n - 1; i += nt) {
    twf[i] = twg[tn.fwd.tw_base + i];
    twi[i] = twg[tn.inv.tw_base + i];
  }
  const int h = tn.n_img / 2, hs = n / 2;
  const int64_t es = (int64_t)tn.icells * cb;
  __syncthreads();

  auto first = [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R, rs = ffx_block_rows(R);
    for (int idx = tid; idx < nr * W; idx += nt) {
      const int b = idx / W, w = idx - b * W;
      const int64_t base = cols.base[w];
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) {
        int j = b + t * nr + h;
        if (j >= n) j -= n;
        x[t] = make_float2(0.f, 0.f);
        if (base >= 0 && j < tn.n_img) x[t] = grid[base + j * es];
      }
      dft<R, false>(x);
      float2* d = A + b * rs * WS + w;
#pragma unroll
      for (int u = 0; u < R; ++u) d[u * WS] = x[u];
    }
  };
  auto middle = [&](auto rc, auto ic, const FfxAxis& ax, const float2* tws, const float2* a, float2* d, int s, int L,
                    int rs) {
    constexpr int R = decltype(rc)::value;
    constexpr bool INV = decltype(ic)::value;
    const int nr = n / R;
    const int tstep = nr / L * rs;  // rs: rows of a block of L points
    for (int idx = tid; idx < nr * W; idx += nt) {
      const int b = idx / W, w = idx - b * W;
      const int k = (int)__umulhi((unsigned)b, ax.mag_l[s]), j = b - k * L;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(k * rs + j + t * tstep) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<INV>(x[t], tws[j * (R - 1) + t - 1]);
      dft<R, INV>(x);
#pragma unroll
      for (int u = 0; u < R; ++u) d[(k * R * L + u * L + j) * WS + w] = x[u];
    }
  };
  // last forward stage, product, first inverse stage
  auto turn = [&](auto rc, const float2* a, float2* d) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R, rs = ffx_block_rows(R);
    const int as = ns == 2 ? ffx_block_rows(tn.fwd.radix[0]) : nr;
    const float2* tws = twf + tn.fwd.tw_off[ns - 1];
    const float2* ks = kern + tn.kern_off;
    for (int idx = tid; idx < nr * W; idx += nt) {
      const int b = idx / W, w = idx - b * W;
      const int cell = cols.cell[w];
      const bool on = cols.base[w] >= 0;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(b + t * as) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<false>(x[t], tws[b * (R - 1) + t - 1]);
      dft<R, false>(x);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        int j = u * nr + b + hs;
        if (j >= n) j -= n;
        const float2 k = on ? __ldg(ks + (int64_t)j * tn.icells + cell) : make_float2(0.f, 0.f);
        x[u] = make_float2(x[u].x * k.x - x[u].y * k.y, x[u].x * k.y + x[u].y * k.x);
      }
      dft<R, true>(x);
      float2* dp = d + b * rs * WS + w;
#pragma unroll
      for (int u = 0; u < R; ++u) dp[u * WS] = x[u];
    }
  };
  auto last = [&](auto rc, const float2* a) {
    constexpr int R = decltype(rc)::value;
    const int nr = n / R;
    const int as = ns == 2 ? ffx_block_rows(tn.inv.radix[0]) : nr;
    const float2* tws = twi + tn.inv.tw_off[ns - 1];
    for (int idx = tid; idx < nr * W; idx += nt) {
      const int b = idx / W, w = idx - b * W;
      const int64_t base = cols.base[w];
      if (base < 0) continue;
      float2 x[R];
#pragma unroll
      for (int t = 0; t < R; ++t) x[t] = a[(b + t * as) * WS + w];
#pragma unroll
      for (int t = 1; t < R; ++t) x[t] = ctw<true>(x[t], tws[b * (R - 1) + t - 1]);
      dft<R, true>(x);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        int j = u * nr + b + h;
        if (j >= n) j -= n;
        if (j < tn.n_img) grid[base + j * es] = x[u];
      }
    }
  };
#define MRN_TURN_CASE(N, CALL) case N: { std::integral_constant<int, N> rc; CALL; } break;
#define MRN_TURN_RADIX(R_, CALL)                                                              \
  switch (R_) {                                                                               \
    MRN_TURN_CASE(1, CALL) MRN_TURN_CASE(2, CALL) MRN_TURN_CASE(3, CALL) MRN_TURN_CASE(4, CALL) \
    MRN_TURN_CASE(5, CALL) MRN_TURN_CASE(6, CALL) MRN_TURN_CASE(8, CALL) MRN_TURN_CASE(9, CALL) \
    MRN_TURN_CASE(10, CALL) MRN_TURN_CASE(12, CALL) MRN_TURN_CASE(15, CALL)                   \
    MRN_TURN_CASE(16, CALL) MRN_TURN_CASE(20, CALL)                                           \
    default:                                                                                  \
      if constexpr (PRIMES) {                                                                 \
        switch (R_) {                                                                         \
          MRN_TURN_CASE(7, CALL) MRN_TURN_CASE(11, CALL) MRN_TURN_CASE(13, CALL)              \
          MRN_TURN_CASE(14, CALL) MRN_TURN_CASE(17, CALL) MRN_TURN_CASE(19, CALL)             \
          default: break;                                                                     \
        }                                                                                     \
      }                                                                                       \
  }
  // the middle stages of one direction, A -> B -> A ..
  auto middles = [&](auto ic, const FfxAxis& ax, const float2* tw) {
    int L = ax.radix[0];
#pragma unroll 1
    for (int s = 1; s + 1 < ns; ++s) {
      const int R = ax.radix[s];
      const float2* tws = tw + ax.tw_off[s];
#define MRN_TURN_MID(N) middle(std::integral_constant<int, N>(), ic, ax, tws, A, B, s, L, s == 1 ? ffx_block_rows(L) : L)
      switch (R) {
        case 2: MRN_TURN_MID(2); break;
        case 3: MRN_TURN_MID(3); break;
        case 4: MRN_TURN_MID(4); break;
        case 5: MRN_TURN_MID(5); break;
        case 6: MRN_TURN_MID(6); break;
        case 7:
          if constexpr (PRIMES) MRN_TURN_MID(7);
          break;
        case 8: MRN_TURN_MID(8); break;
        case 9: MRN_TURN_MID(9); break;
        case 10: MRN_TURN_MID(10); break;
        case 11:
          if constexpr (PRIMES) MRN_TURN_MID(11);
          break;
        default: MRN_TURN_MID(12); break;
      }
#undef MRN_TURN_MID
      __syncthreads();
      float2* t = A;
      A = B;
      B = t;
      L *= R;
    }
  };
  MRN_TURN_RADIX(tn.fwd.radix[0], first(rc))
  __syncthreads();
  middles(std::false_type(), tn.fwd, twf);
  MRN_TURN_RADIX(tn.inv.radix[0], turn(rc, A, B))
  __syncthreads();
  {
    float2* t = A;
    A = B;
    B = t;
  }
  middles(std::true_type(), tn.inv, twi);
  MRN_TURN_RADIX(tn.inv.radix[ns - 1], last(rc, A))
#undef MRN_TURN_RADIX
#undef MRN_TURN_CASE
}

template <int W, bool PRIMES>
int launch_turn(const FfxTurnSet& S, const FfxGrid& G, const float2* kern, cudaStream_t st) {
  auto k = k_ffx_turn<W, PRIMES>;
  const int rc = set_dynamic_smem(k, S.smem);
  if (rc != MRN_OK) return rc;
  const unsigned nb = (unsigned)((S.max_cols + W - 1) / W);
  for (int s0 = 0; s0 < S.nsl; s0 += 65535)
    k<<<dim3(nb, (unsigned)std::min(65535, S.nsl - s0)), S.threads, S.smem, st>>>(G.dsl, S.d_turn, s0, S.d_tw, kern,
                                                                                G.grid);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MRN_OK : cuda_fail(e);
}

}  // namespace

// Shared memory of a CTA of w columns: both tables and two buffers, each large
// enough for either direction's padded first stage.
static size_t turn_smem(const FfxTurn& t, int w) { return ((size_t)2 * t.fwd.n + (size_t)2 * t.buf * w) * sizeof(float2); }

// One turning pass per slice of direct radices (g.native_fft; the others get an
// empty one, whose blocks return). kern_off: complex offset of a slice's kernel,
// centred [n0][cells of the later axes].
int ffx_turn_build(FfxTurnSet& S, const FfxSet& F, int ndim, const std::vector<SliceGeom>& hsl,
                   const std::vector<int64_t>& kern_off, int sm_count) {
  S.release();
  std::vector<float2> tab;
  std::vector<FfxTurn> turns;
  int64_t total = 0;
  int most = 1;
  for (size_t s = 0; s < hsl.size(); ++s) {
    const SliceGeom& g = hsl[s];
    FfxTurn t{};
    if (!g.native_fft) {
      turns.push_back(t);
      continue;
    }
    for (const FfxTurn& o : turns)
      if (o.fwd.n == g.nos[0]) t = o;
    if (t.fwd.n == 0) {
      for (const FfxGroup& fg : F.grp)
        if (fg.native && fg.ax[0].n == g.nos[0]) t.fwd = fg.ax[0];
      if (t.fwd.n == 0 || t.fwd.m > 0) return MRN_ERR_UNSUPPORTED;
      t.inv = t.fwd;
      std::reverse(t.inv.radix, t.inv.radix + t.inv.ns);
      t.fwd.tw_base = (int)tab.size();
      ffx_stage_tables(t.fwd, tab);
      t.inv.tw_base = (int)tab.size();
      ffx_stage_tables(t.inv, tab);
      for (const FfxAxis* ax : {&t.fwd, &t.inv}) {
        t.buf = std::max(t.buf, ax->n / ax->radix[0] * ffx_block_rows(ax->radix[0]));
      }
    }
    t.n_img = g.n[0];
    t.icells = 1;
    for (int i = 1; i < ndim; ++i) t.icells *= g.nos[i];
    t.kern_off = kern_off[s];
    const int64_t c = (int64_t)g.ncoil * t.icells;
    S.max_cols = std::max(S.max_cols, c);
    total += c;
    for (int i = 0; i < t.fwd.ns; ++i) most = std::max(most, t.fwd.n / t.fwd.radix[i]);
    S.primes |= ffx_has_primes(t.fwd);
    turns.push_back(t);
  }
  if (S.max_cols > 0x7fffffffLL) return MRN_ERR_UNSUPPORTED;
  auto smem = [&](int w) {
    size_t m = 0;
    for (const auto& t : turns) m = std::max(m, turn_smem(t, w));
    return m;
  };
  // as the plain passes: two CTAs an SM, and a CTA for every SM
  S.w = 16;
  while (S.w > 4 && (smem(S.w) > 110 * 1024 || total / S.w < 2 * (int64_t)sm_count)) S.w /= 2;
  S.smem = smem(S.w);
  if (S.smem > 220 * 1024) return MRN_ERR_UNSUPPORTED;
  S.threads = std::min(kTurnThreads, std::max(32, (most * S.w + 31) / 32 * 32));
  S.nsl = (int)turns.size();
  cudaError_t e = cudaMalloc(&S.d_tw, tab.size() * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&S.d_turn, turns.size() * sizeof(FfxTurn));
  if (e == cudaSuccess) e = cudaMemcpy(S.d_tw, tab.data(), tab.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(S.d_turn, turns.data(), turns.size() * sizeof(FfxTurn), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    S.release();
    return MRN_ERR_CUDA;
  }
  return MRN_OK;
}

int ffx_turn(const FfxTurnSet& S, const FfxGrid& G, const float2* kern, cudaStream_t st) {
  if (S.primes) {
    if (S.w == 16) return launch_turn<16, true>(S, G, kern, st);
    if (S.w == 8) return launch_turn<8, true>(S, G, kern, st);
    return launch_turn<4, true>(S, G, kern, st);
  }
  if (S.w == 16) return launch_turn<16, false>(S, G, kern, st);
  if (S.w == 8) return launch_turn<8, false>(S, G, kern, st);
  return launch_turn<4, false>(S, G, kern, st);
}

}  // namespace mrn
