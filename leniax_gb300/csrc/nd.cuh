// Shared pieces of the general N-D engine (nd.cu, nd_rows.cu, nd_plane.cu,
// nd_conv.cu): the model table, tile geometry and the epilogue of an Euler
// step (growth, weighted field, state update, statistics moments).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "launch.cuh"
#include "line_fft.cuh"

namespace lgx {

constexpr int kNdThreads = 320;        // most threads of a transform block
constexpr int kNdBlocksPerSm = 3;      // register budget: 64 a thread ...
__host__ __device__ constexpr int nd_blocks(int kind) { return kind == LINE_WIDE ? 2 : kNdBlocksPerSm; }  // ... 96 wide
constexpr int kNdMaxN = 4096;          // longest world axis (one 4096-point line per tile)
constexpr int kBluesteinMaxN = 2048;   // longest axis with a prime factor above 7 (m <= 4096)
constexpr int kMaxPts = 4096;          // complex points of one tile buffer
constexpr int kMaxTileLines = 64;
constexpr int kNdSmemMax = 227 * 1024;
// Launches smaller than this many blocks (two on each of GB300's 152 SMs) get
// smaller tiles so that one small world still spreads over the whole GPU.
constexpr long kFillBlocks = 2 * 152;
constexpr int kRawMax = RAW_CM + kMaxChannels;

struct NdTab {  // kernel table and geometry of a model, passed by value
  int C, K, max_k, mean, state_fn, dt_mode, nd;
  int D, H, W, Wh;     // Wh = W / 2 + 1 columns of a half spectrum
  long cells, hcells;  // D H W, D H Wh
  int cin[kMaxKernels];
  int slot[kMaxKernels];
  int gf[kMaxKernels];
};

struct NdAxes {
  LineAxis x, y, z;  // along W, H and D
};

inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// threads for `items` butterflies: one each up to kNdThreads, else whole rounds
inline int nd_threads(long items) {
  const long rounds = (items + kNdThreads - 1) / kNdThreads;
  const long per = (items + rounds - 1) / std::max(1L, rounds);
  return (int)std::min<long>(kNdThreads, std::max(32L, (per + 31) / 32 * 32));
}
// butterflies of an nl-line tile's widest end stage
inline long line_items(const LineAxis& ax, int nl) {
  const int last = ax.r[ax.stages - 1];
  return (long)nl * (ax.m / std::min(ax.r[0], last > 1 ? last : ax.r[0]));
}

// Opt a kernel in to the full dynamic shared memory; the attribute belongs to
// the CUDA context, so each context gets it once (nd.cu).
cudaError_t nd_allow_smem(const void* kernel);

// ------------------------------------------------------------------ epilogue
struct EpiArgs {
  int n_worlds, n_init;
  int tiles, split, bpw;  // tiles of a world (blockIdx.x), gridDim.y = C blocks to a tile, blocks of a world
  const float* state;   // [nw, C, cells]
  float* state_out;     // [nw, C, cells]
  const float2* P;      // [nw, K, hcells] products, the last world axis inverse-transformed
  float2* S;            // [nw, C, hcells] next step's row (2D) or plane (3D) spectra, or null
  float* F;             // [nw, C, cells] weighted fields between the kernels when they do not fit shared memory
  float* pot_out;       // [nw, K, cells] or null
  const float* gf;      // [Ns, K, 2] (sol stride gf_sol_stride)
  long gf_sol_stride;
  const float* w;       // [Ns, C, K]
  long w_sol_stride;
  const float* dt;
  float* field_out;     // [nw, C, cells] or null
  float* state_copy;    // [nw, C, cells] copy of the entering state (trajectory), or null
  int* shift;           // [nw, 3] read by every block, advanced by the world's last block
  int* done;            // [nw] blocks finished this step (zero between steps)
  float* partial;       // [nw, bpw, RAWS]
  float* raw;           // the step's raw record, or null
  long raw_sol_stride, raw_init_stride;
  float scale;          // 1 / cells: the inverse transforms are unnormalised
};

// centred coordinate on one axis (statistics.py:64-81 on the world rolled by
// the carried shift): ((i - shift) mod n) - n // 2, for 0 <= i, sh < n
__device__ __forceinline__ float centred_in(int i, int sh, int n) {
  const int d = i - sh;
  return (float)((d < 0 ? d + n : d) - n / 2);
}

__device__ __forceinline__ float step_dt(const NdTab& t, const EpiArgs& a, int w, int sol) {
  if (t.dt_mode == 0) return __ldg(a.dt);
  if (t.dt_mode == 1) return __ldg(a.dt + w);
  return 1.f / __ldg(a.dt + sol);
}

// Growth of one potential: the gaussian inline, the others out of line, so that
// an unrolled butterfly's epilogue stays small.
static __device__ __noinline__ float growth_any(int id, float u, float m, float s) { return growth_fn(id, u, m, s); }
struct NdGrowth {
  int id;
  bool inl;  // the inline form holds: gaussian, its coefficient within float32's normal range
  float m, s;
  // the exponent's coefficient log2(e) / (2 s^2) as an unevaluated sum c + dc:
  // rounded to one float its error is the same in every cell of a world, and a
  // world's growth shows it where cells' roundings average out.  c lies below
  // the coefficient (four units in the last place cover the roundings of 1/q,
  // the product, s^2 and the constant), so dc > 0 and both parts of the
  // exponent of an infinite square are -inf (growth -1), not inf - inf.
  float c, dc;
  // Widths whose square, coefficient and remainder are all normal floats; for
  // the others (0, tiny, huge, infinite, NaN) c + dc is infinite or NaN and
  // growth_fn's quotient stands.
  __device__ __forceinline__ static bool regular(float s) { return fabsf(s) >= 0x1p-50f && fabsf(s) <= 0x1p50f; }
  __device__ __forceinline__ NdGrowth(int id, float m, float s)
      : id(id), inl(id == LGX_GF_GAUSSIAN && regular(s)), m(m), s(s) {
    const float q = s * s, dq = fmaf(s, s, -q), inv = 1.f / q;  // s^2 = q + dq
    c = __int_as_float(__float_as_int(kC * inv) - 4);
    dc = (fmaf(-c, q, kC) + (kDc - c * dq)) * inv;
  }
  static constexpr double kLog2E2 = 0.72134752044448170368;  // log2(e) / 2
  static constexpr float kC = (float)kLog2E2, kDc = (float)(kLog2E2 - (double)kC);
  // the gaussian's exponential at both cells
  __device__ __forceinline__ float2 gauss(float2 u) const {
    const float2 d = __fadd2_rn(u, make_float2(-m, -m));
    const float2 d2 = __fmul2_rn(d, d);
    const float2 x = __ffma2_rn(d2, make_float2(-c, -c), __fmul2_rn(d2, make_float2(-dc, -dc)));
    return make_float2(fast_exp2(x.x), fast_exp2(x.y));
  }
  // weighted growth of a pair: w (2 e - 1), for weights whose double is finite
  __device__ __forceinline__ float2 gauss_weighted(float2 u, float w) const {
    return __ffma2_rn(make_float2(2.f * w, 2.f * w), gauss(u), make_float2(-w, -w));
  }
  __device__ __forceinline__ static bool foldable(float w) { return fabsf(w) <= 0x1p126f; }
  __device__ __forceinline__ float any(float u) const { return growth_any(id, u, m, s); }
  __device__ __forceinline__ float operator()(float u) const {
    if (inl) {
      const float d = u - m, d2 = d * d;
      return fmaf(2.f, fast_exp2(fmaf(d2, -c, d2 * -dc)), -1.f);
    }
    return any(u);
  }
};

// A packed pair of rows of a tile: row0 and, when the pair is whole, row0 + 1.
struct RowPair {
  long cell;         // first cell of row0 within the channel plane
  float cz0, cy0, cz1, cy1;  // centred coordinates of the two rows
  int rows;          // 0 (past the tile), 1 or 2
  int edge;          // bit 0 / 1: the row lies on the outer layer of the un-centred world
};

__device__ __forceinline__ RowPair row_pair(const NdTab& t, int z0, int y0, int z1, int y1, int rows, int s0, int s1) {
  RowPair r;
  r.cell = ((long)z0 * t.H + y0) * t.W;
  r.rows = rows;
  const int sz = t.nd == 3 ? s0 : 0, sy = t.nd == 3 ? s1 : s0;
  r.cz0 = t.nd == 3 ? centred_in(z0, sz, t.D) : 0.f;
  r.cz1 = t.nd == 3 ? centred_in(z1, sz, t.D) : 0.f;
  r.cy0 = centred_in(y0, sy, t.H);
  r.cy1 = centred_in(y1, sy, t.H);
  const bool e0 = y0 == 0 || y0 == t.H - 1 || (t.nd == 3 && (z0 == 0 || z0 == t.D - 1));
  const bool e1 = y1 == 0 || y1 == t.H - 1 || (t.nd == 3 && (z1 == 0 || z1 == t.D - 1));
  r.edge = (e0 ? 1 : 0) | (e1 ? 2 : 0);
  return r;
}

// Per-thread statistics moments (statistics.py:64-100 in the centred frame).
struct Moments {
  float m00 = 0.f, g00 = 0.f, cpot = 0.f, cmass = 0.f, cgrow = 0.f;
  float mz = 0.f, my = 0.f, mx = 0.f, gz = 0.f, gy = 0.f, gx = 0.f, qz = 0.f, qy = 0.f, qx = 0.f;
  bool border = false;
  // one cell of both rows of a pair: entering states, positive fields, centred x
  __device__ __forceinline__ void add_cell(float2 s, float2 g, float cx) {
    const float ss = s.x + s.y;
    mx = fmaf(ss, cx, mx);
    qx = fmaf(ss * cx, cx, qx);
    gx = fmaf(g.x + g.y, cx, gx);
    cmass += (s.x > kEps ? 1.f : 0.f) + (s.y > kEps ? 1.f : 0.f);
    cgrow += (g.x > kEps ? 1.f : 0.f) + (g.y > kEps ? 1.f : 0.f);
  }
  // cells of one pair: their states' and positive fields' sums, the largest
  // state of each row, whether a cell on the x border is alive
  __device__ __forceinline__ void add_row(const RowPair& r, float2 S2, float2 G2, float2 most, bool lx) {
    border |= lx || (most.x > kEps && (r.edge & 1)) || (most.y > kEps && (r.edge & 2));
    m00 += S2.x + S2.y;
    g00 += G2.x + G2.y;
    const float y0 = S2.x * r.cy0, y1 = S2.y * r.cy1, z0 = S2.x * r.cz0, z1 = S2.y * r.cz1;
    my += y0 + y1;
    mz += z0 + z1;
    qy = fmaf(y0, r.cy0, fmaf(y1, r.cy1, qy));
    qz = fmaf(z0, r.cz0, fmaf(z1, r.cz1, qz));
    gy = fmaf(G2.x, r.cy0, fmaf(G2.y, r.cy1, gy));
    gz = fmaf(G2.x, r.cz0, fmaf(G2.y, r.cz1, gz));
  }
  __device__ __forceinline__ void count_pot(float2 u, int rows) {
    cpot += (u.x > kEps ? 1.f : 0.f) + (rows > 1 && u.y > kEps ? 1.f : 0.f);
  }
};

struct EpiShared {
  float red[kNdThreads / 32][kRawMax];
  float tot[kRawMax];
  int last;
};

// The epilogue's inputs that the launches before it write.
__device__ __forceinline__ void epi_after_wait(EpiArgs& a) {
  a.state = after_wait(a.state);
  a.P = after_wait(a.P);
  a.shift = after_wait(a.shift);
}

// The channels a block of the epilogue updates, the kernels it transforms for
// them and those whose potentials it counts (bit k: kernel k).  split: one
// channel (blockIdx.y), the kernels that feed it, counted by the first channel
// they feed; channel 0 also counts those that feed none.
struct EpiChannels {
  int lo, hi;
  unsigned long long todo, count;
};
__device__ __forceinline__ EpiChannels epi_channels(const NdTab& t, const EpiArgs& a, const float* wt) {
  const int C = t.C, K = t.K;
  static_assert(kMaxKernels <= 64, "one bit per kernel");
  const unsigned long long all = K == 64 ? ~0ull : (1ull << K) - 1ull;
  if (!a.split) return EpiChannels{0, C, all, all};
  const int lo = blockIdx.y, lane = threadIdx.x & 31;
  unsigned long long fed = 0ull, before = 0ull, any = 0ull;
  for (int h = 0; h < K; h += 32)
    for (int c = 0; c < C; ++c) {
      const float w = h + lane < K ? __ldg(wt + c * K + h + lane) : 0.f;
      const unsigned long long b = (unsigned long long)__ballot_sync(0xffffffffu, w != 0.f) << h;
      any |= b;
      if (c < lo) before |= b;
      if (c == lo) fed |= b;
    }
  const unsigned long long unfed = lo == 0 ? all & ~any : 0ull;
  return EpiChannels{lo, lo + 1, fed | unfed, (fed & ~before) | unfed};
}
// A model whose whole tiles or planes fill fewer blocks than kFillBlocks gets a
// block per channel instead of one that walks all kernels of its tile (a
// kernel that feeds several channels is then transformed for each).  12-step
// rollouts of 3 channels x 9 kernels on 100^2, us: 8 worlds 1754 -> 838, 64
// 1940 -> 1363; 10 steps of 2 x 8 on one 48^3 world 747 -> 556.
inline bool epi_split(const NdTab& t, long blocks) { return t.C > 1 && blocks < kFillBlocks; }

// The warp's total of channel c's mass, kept for epi_finish.
__device__ __forceinline__ void epi_channel_mass(EpiShared& sh, int c, float cm) {
  cm = warp_sum(cm);
  if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5][RAW_CM + c] = cm;
}

// The epilogue of the packed pairs of potentials in Z [nl][zp] (C = K = 1):
// growth, state update, stores and moments, the new cells left in Z.  `lanes`
// neighbouring threads take a row pair (epi_lanes), so the row coordinates
// multiply row sums and the cells of a pair go through the packed FP32x2 pipe.
// A rolled loop of its own rather than the middle of the row transform's
// butterflies: inlined there it was unrolled over every radix, and blocks that
// run the code once stalled on instruction fetch.
template <bool GAUSS, bool V1>
__device__ __forceinline__ void epi_pairs(const NdTab& t, const EpiArgs& a, const RowPair* rp, float2* Z, int nl,
                                          int zp, int lanes, int w, int sx, float dt, const NdGrowth& grow, float wf,
                                          Moments& mo) {
  const int W = t.W;
  const float wrap = (float)W, top = (float)(W - W / 2);
  const int x0 = threadIdx.x & (lanes - 1);
  const int per = __ffs(lanes) - 1;
  float2 S2, G2;
  for (int l = threadIdx.x >> per; l < nl; l += blockDim.x >> per) {
    const RowPair r = rp[l];
    if (r.rows == 0) continue;
    const bool two = r.rows > 1;
    const long off0 = (long)w * t.cells + r.cell;
    S2 = G2 = make_float2(0.f, 0.f);
    float2 most = make_float2(0.f, 0.f);  // largest cell of each row
    bool lx = false;
    float cx = centred_in(x0 < W ? x0 : 0, sx, W);
    float2* z = Z + l * zp;
    for (int x = x0; x < W; x += lanes) {
      const long off = off0 + x;
      const float2 s = make_float2(__ldg(a.state + off), two ? __ldg(a.state + off + W) : 0.f);
      const float2 u = __fmul2_rn(z[x], make_float2(a.scale, a.scale));
      float2 f;
      if (GAUSS) f = grow.gauss_weighted(u, wf);
      else f = make_float2(grow(u.x) * wf, grow(u.y) * wf);
      if (!two) f.y = 0.f;
      float2 n;
      if (V1) n = make_float2(__saturatef(fmaf(dt, f.x, s.x)), __saturatef(fmaf(dt, f.y, s.y)));
      else n = make_float2(state_fn(t.state_fn, s.x, f.x, dt), state_fn(t.state_fn, s.y, f.y, dt));
      z[x] = n;
      a.state_out[off] = n.x;
      if (two) a.state_out[off + W] = n.y;
      if (a.field_out) {
        a.field_out[off] = f.x;
        if (two) a.field_out[off + W] = f.y;
      }
      if (a.state_copy) {
        a.state_copy[off] = s.x;
        if (two) a.state_copy[off + W] = s.y;
      }
      if (a.pot_out) {
        a.pot_out[off] = u.x;
        if (two) a.pot_out[off + W] = u.y;
      }
      mo.count_pot(u, r.rows);
      const float2 g = make_float2(fmaxf(f.x, 0.f), fmaxf(f.y, 0.f));
      S2 = cadd(S2, s);
      G2 = cadd(G2, g);
      mo.add_cell(s, g, cx);
      most = make_float2(fmaxf(most.x, s.x), fmaxf(most.y, s.y));
      if (x == 0 || x == W - 1) lx |= fmaxf(s.x, s.y) > kEps;
      cx += (float)lanes;
      while (cx >= top) cx -= wrap;  // past the centred frame's end
    }
    mo.add_row(r, S2, G2, most, lx);
  }
}
__device__ __forceinline__ void epi_single(const NdTab& t, const EpiArgs& a, const RowPair* rp, float2* Z, int nl,
                                           int zp, int lanes, int w, int sx, float dt, Moments& mo) {
  const int sol = w / a.n_init;
  const float* gf = a.gf + sol * a.gf_sol_stride;
  const NdGrowth grow(t.gf[0], __ldg(gf), __ldg(gf + 1));
  const float wk = __ldg(a.w + sol * a.w_sol_stride);
  const float wf = t.mean ? wk / wk : wk;  // weighted_mean with one kernel: (w g) / w
  if (grow.inl && grow.foldable(wf) && t.state_fn == LGX_STATE_V1)
    epi_pairs<true, true>(t, a, rp, Z, nl, zp, lanes, w, sx, dt, grow, wf, mo);
  else
    epi_pairs<false, false>(t, a, rp, Z, nl, zp, lanes, w, sx, dt, grow, wf, mo);
}
// Several kernels: the rules at the ends of a tile's row transforms.  They take
// a butterfly's points at once: the pair's row, its addresses and the weights
// are fetched once for the R points that are inlined behind every radix (code
// that a block runs once waits for its instructions).  A step, us, cell by cell
// -> so: one world of 3 x 15 kernels on 100^2 79 -> 60, of one channel with two
// 47 -> 36; 4 worlds of 3 x 9 on 720^2 407 -> 347, on 48^3 56 -> 48.
//
// Kernel k's potentials (times scale) are stored and counted (`count`), their
// weighted growths added to the fields F [channel lo..hi-1][nl][W].
struct AddGrowth {
  const NdTab& t;
  const EpiArgs& a;
  const RowPair* rp;
  float2* F;
  const float* wt;
  NdGrowth grow;
  float* pot;  // the kernel's potential plane, or null
  int nl, k, lo, hi;
  bool count;
  Moments& mo;
  template <int R>
  __device__ __forceinline__ void operator()(int l, int at, int step, const float2 (&v)[R]) const {
    const int rows = rp[l].rows;
    if (rows == 0) return;
    float2 g[R];
#pragma unroll
    for (int q = 0; q < R; ++q) g[q] = __fmul2_rn(v[q], make_float2(a.scale, a.scale));
    if (count) {
      if (pot) {
        float* p = pot + rp[l].cell + at;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          p[q * step] = g[q].x;
          if (rows > 1) p[q * step + t.W] = g[q].y;
        }
      }
#pragma unroll
      for (int q = 0; q < R; ++q) mo.count_pot(g[q], rows);
    }
    if (grow.inl) {
#pragma unroll
      for (int q = 0; q < R; ++q) g[q] = __ffma2_rn(make_float2(2.f, 2.f), grow.gauss(g[q]), make_float2(-1.f, -1.f));
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) g[q] = make_float2(grow.any(g[q].x), grow.any(g[q].y));
    }
    for (int c = lo; c < hi; ++c) {
      const float wk = __ldg(wt + c * t.K + k);
      if (wk == 0.f) continue;
      float2* f = F + ((long)(c - lo) * nl + l) * t.W + at;
#pragma unroll
      for (int q = 0; q < R; ++q) f[q * step] = __ffma2_rn(g[q], make_float2(wk, wk), f[q * step]);
    }
  }
};
// A channel's new cells from its fields F [nl][W]: update, stores, moments.
struct UpdateCells {
  const NdTab& t;
  const EpiArgs& a;
  const RowPair* rp;
  const float2* F;
  long plane;  // the channel's first cell
  int sx;
  float dt, wsum;
  Moments& mo;
  template <int R>
  __device__ __forceinline__ void operator()(int l, int j, int nb, float2 (&v)[R]) const {
    const RowPair r = rp[l];
    const int W = t.W;
    if (r.rows == 0) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = make_float2(0.f, 0.f);
      return;
    }
    const bool two = r.rows > 1;
    const float2* f = F + (long)l * W + j;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      v[q] = f[q * nb];
      if (t.mean) v[q] = make_float2(v[q].x / wsum, v[q].y / wsum);
      if (!two) v[q].y = 0.f;
    }
    const long off = plane + r.cell + j;
    if (a.field_out) {
      float* p = a.field_out + off;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        p[q * nb] = v[q].x;
        if (two) p[q * nb + W] = v[q].y;
      }
    }
    float2 S2 = make_float2(0.f, 0.f), G2 = S2, most = S2;
    bool lx = false;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int x = j + q * nb;
      const float* p = a.state + off + q * nb;
      const float2 s = make_float2(__ldg(p), two ? __ldg(p + W) : 0.f);
      if (a.state_copy) {
        a.state_copy[off + q * nb] = s.x;
        if (two) a.state_copy[off + q * nb + W] = s.y;
      }
      const float2 g = make_float2(fmaxf(v[q].x, 0.f), fmaxf(v[q].y, 0.f));
      v[q] = make_float2(state_fn(t.state_fn, s.x, v[q].x, dt), two ? state_fn(t.state_fn, s.y, v[q].y, dt) : 0.f);
      a.state_out[off + q * nb] = v[q].x;
      if (two) a.state_out[off + q * nb + W] = v[q].y;
      S2 = cadd(S2, s);
      G2 = cadd(G2, g);
      mo.add_cell(s, g, centred_in(x, sx, W));
      most = make_float2(fmaxf(most.x, s.x), fmaxf(most.y, s.y));
      if (x == 0 || x == W - 1) lx |= fmaxf(s.x, s.y) > kEps;
    }
    mo.add_row(r, S2, G2, most, lx);
  }
};
// Channel c's update as the rule of its tile's forward transform (spectra()),
// or of nothing where no next step follows; its mass is kept for epi_finish.
template <class Spectra>
__device__ __forceinline__ void epi_channel(const NdTab& t, const EpiArgs& a, const RowPair* rp, const float2* F,
                                            int nl, int w, int c, int sx, float dt, const float* wt, Moments& mo,
                                            EpiShared& sh, const Spectra& spectra) {
  float wsum = 0.f;
  for (int k = 0; k < t.K; ++k) wsum += __ldg(wt + c * t.K + k);
  const float before = mo.m00;
  mo.m00 = 0.f;  // this channel's mass
  const UpdateCells update{t, a, rp, F, ((long)w * t.C + c) * t.cells, sx, dt, wsum, mo};
  if (a.S) {
    spectra(update);
  } else {
    for (int i = threadIdx.x; i < nl * t.W; i += blockDim.x) {
      float2 v[1];
      update(i / t.W, i % t.W, 0, v);
    }
  }
  epi_channel_mass(sh, c, mo.m00);
  mo.m00 += before;
}

// Threads per row pair: the power of two in 8..32 that leaves the fewest idle
// along a row; more where a tile has fewer pairs than its threads have warps
// (rows of thousands of cells).  A step, us, 32 -> 256 threads for a pair of
// 4096: one world of 4 x 4096 70 -> 35, of 16 x 4096 66 -> 34, 32 of 4 x 4096
// 69 -> 36.
inline int epi_lanes(int W, int nl, int threads) {
  int best = 32;
  for (int p : {16, 8})
    if ((W + p - 1) / p * p < (W + best - 1) / best * best) best = p;
  while (best >= 32 && threads % (2 * best) == 0 && 2 * best * nl <= threads && best < W) best *= 2;
  return best;
}

// Threads of an epilogue block: a world of many small tiles has its last block
// walk as many partials (epi_finish), for which it needs warps.  A step of one
// world, us, one warp -> four: 1024 x 8 x 8 85 -> 40, 4096 x 4 x 4 274 -> 113.
inline int epi_threads(int threads, int bpw) { return bpw > 256 ? std::max(threads, 128) : threads; }

// Block b of world w: reduce the threads' moments into the block's partial;
// the world's last block to finish (a ticket on the world's counter; no block
// waits) reduces all of the world's block partials in a fixed order into the
// step's raw record (with the shift s0..s2 that centred it), then advances
// the carried shift by the integer part of the centred-frame centroid
// (statistics.py:117-124).  Every thread of the block calls it, after
// epi_channel_mass of every channel.
__device__ __forceinline__ void epi_finish(const NdTab& t, const EpiArgs& a, EpiShared& sh, int w, int b,
                                           const Moments& mo, int s0, int s1, int s2) {
  const int NWARP = blockDim.x >> 5;
  const int C = t.C, nd = t.nd, bpw = a.bpw;
  const int sol = w / a.n_init, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // record order: 3D (z, y, x), 2D (y, x, 0)
  const bool d3 = nd == 3;
  float v[16] = {mo.m00, mo.g00, mo.cpot, mo.cmass, mo.cgrow,
                 d3 ? mo.mz : mo.my, d3 ? mo.my : mo.mx, d3 ? mo.mx : 0.f,
                 d3 ? mo.gz : mo.gy, d3 ? mo.gy : mo.gx, d3 ? mo.gx : 0.f,
                 d3 ? mo.qz : mo.qy, d3 ? mo.qy : mo.qx, d3 ? mo.qx : 0.f, mo.border ? 1.f : 0.f, 0.f};
  static_assert(RAW_M00 == 0 && RAW_G00 == 1 && RAW_CNT_POT == 2 && RAW_CNT_MASS == 3 && RAW_CNT_GROW == 4 &&
                    RAW_MX == 5 && RAW_GX == 8 && RAW_MX2 == 11 && RAW_BORDER == 14 && RAW_SHIFT == 15,
                "the order of v");
  const float total = warp_sum16(v);  // lane L: value L >> 1
  if ((lane & 1) == 0) sh.red[wid][lane >> 1] = total;  // slot 15 (shift) is written below
  if (lane < 2) sh.red[wid][RAW_SHIFT + 1 + lane] = 0.f;
  __syncthreads();
  const int RAWS = raw_stride(C);
  float* pw = a.partial + (long)w * bpw * RAWS;
  for (int s = threadIdx.x; s < RAWS; s += blockDim.x) {
    float acc = 0.f;
    for (int i = 0; i < NWARP; ++i) acc += sh.red[i][s];
    pw[(long)b * RAWS + s] = acc;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sh.last = atomicAdd(a.done + w, 1) == bpw - 1;
  __syncthreads();
  if (!sh.last) return;
  __threadfence();
  // A world of small tiles has many partials and this block few warps: loads in
  // flight, not one round trip to L2 a partial.  A step of one world, us, one
  // load at a time -> sixteen (and epi_threads): 100^2 31.5 -> 26.0, 144^2
  // 39.8 -> 26.2, 500^2 72 -> 52, 1031 x 64 94 -> 40, 1024 x 8 x 8 255 -> 40.
  constexpr int kLoads = 16;
  for (int s = lane; s < RAWS; s += 32) {
    float acc = 0.f;
    for (int b0 = wid; b0 < bpw; b0 += kLoads * NWARP) {
      float v[kLoads];
#pragma unroll
      for (int j = 0; j < kLoads; ++j) {
        const int bb = b0 + j * NWARP;
        v[j] = bb < bpw ? __ldcg(pw + (long)bb * RAWS + s) : 0.f;
      }
#pragma unroll
      for (int d = kLoads / 2; d > 0; d /= 2)  // by pairs: a chain of hundreds of partials rounds as often
#pragma unroll
        for (int j = 0; j < d; ++j) v[j] += v[j + d];
      acc += v[0];
    }
    sh.red[wid][s] = acc;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < RAWS; s += blockDim.x) {
    float acc = 0.f;
    for (int i = 0; i < NWARP; ++i) acc += sh.red[i][s];
    if (s == RAW_BORDER) acc = acc > 0.f ? 1.f : 0.f;
    if (s == RAW_SHIFT) acc = (float)s0;
    if (s == RAW_SHIFT + 1) acc = (float)s1;
    if (s == RAW_SHIFT + 2) acc = (float)s2;
    sh.tot[s] = acc;
    if (a.raw) a.raw[sol * a.raw_sol_stride + (w - sol * a.n_init) * a.raw_init_stride + s] = acc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int n[3] = {nd == 2 ? t.H : t.D, nd == 2 ? t.W : t.H, t.W};
    const int shf[3] = {s0, s1, s2};
    for (int i = 0; i < nd; ++i)
      a.shift[3 * w + i] = pmod(shf[i] + (int)(sh.tot[RAW_MX + i] / (sh.tot[RAW_M00] + kEps)), n[i]);
    a.done[w] = 0;
  }
}

// Point i of the packed inverse row transform: with row half spectra A and B
// at column min(i, W - i), Z = A + i B for i < W/2 and conj(A) + i conj(B) past
// it.  The real parts of the DC and Nyquist columns are what Re(IFFT) keeps.
__device__ __forceinline__ float2 pack_rows(float2 a, float2 b, int i, int W) {
  const float s = i == 0 || 2 * i == W ? 0.f : (2 * i > W ? -1.f : 1.f);
  return make_float2(fmaf(-s, b.y, a.x), fmaf(s, a.y, b.x));
}

// Half spectra of two real rows from the transform Z of row0 + i row1, at
// column k: (Z_k + conj Z_{W-k}) / 2 and (Z_k - conj Z_{W-k}) / 2i.
__device__ __forceinline__ float2 unpack_row0(float2 zk, float2 zm) {
  return make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
}
__device__ __forceinline__ float2 unpack_row1(float2 zk, float2 zm) {
  return make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
}

// ------------------------------------------------------------- launchers
// nd_rows.cu.  `rows` rows of W cells per plane, paired within the plane.
cudaError_t nd_rows_forward(const LineAxis& x, long planes, int rows, const float* src, float2* half, cudaStream_t st);
cudaError_t nd_rows_inverse(const LineAxis& x, long planes, int rows, const float2* half, float* dst, bool accumulate,
                            float scale, cudaStream_t st);
// blocks per world, and the pair-cells [bpw][nr][W] per channel of EpiArgs::F (0: the fields stay on chip)
int nd_rows_epi_blocks(const NdTab& t, const LineAxis& x, long n_worlds, long* field_pairs);
cudaError_t nd_rows_epilogue(const NdTab& t, const LineAxis& x, const EpiArgs& a, cudaStream_t st);
// nd_conv.cu.  In-place transforms along y (H points, Wh lines per z-plane).
cudaError_t nd_columns(bool inv, const NdTab& t, const LineAxis& y, long planes, float2* data, cudaStream_t st);
struct ConvArgs {
  int n_init;
  const float2* kh;    // half spectra [Ns, C, max_k, hcells] as the caller gave them
  long kh_sol_stride;
  const float2* S;     // [nw, C, hcells], the other axes transformed
  float2* P;           // forward: [nw, K, hcells] products out
  const float2* A;     // adjoint: [nw, K, hcells] spectra of a = dL/du, the other axes transformed
  float2* gk;          // adjoint: [nw, K, hcells] kernel-gradient spectra (accumulated)
  float2* Q;           // adjoint: [nw, C, hcells] correlations out
};
cudaError_t nd_convolve(bool adjoint, const NdTab& t, const LineAxis& last, long nw, const ConvArgs& a,
                        cudaStream_t st);
// nd_plane.cu.  3D worlds whose z-planes fit a tile.
bool nd_plane_ok(const NdTab& t, const NdAxes& ax);
// blocks of a world in the epilogue; *field_global: the weighted fields live in memory
int nd_plane_epi_blocks(const NdTab& t, const NdAxes& ax, long n_worlds, bool* field_global);
cudaError_t nd_plane_forward(const NdTab& t, const NdAxes& ax, long planes, const float* src, float2* half,
                             cudaStream_t st);
cudaError_t nd_plane_inverse(const NdTab& t, const NdAxes& ax, long planes, const float2* half, float* dst,
                             bool accumulate, float scale, cudaStream_t st);
cudaError_t nd_plane_epilogue(const NdTab& t, const NdAxes& ax, const EpiArgs& a, cudaStream_t st);

}  // namespace lgx
