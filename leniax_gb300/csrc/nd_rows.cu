// Row transforms of the general N-D engine and the Euler step's row epilogue.
//
// Two real rows travel as one complex row (row0 + i row1), so a pass moves and
// transforms half spectra of W/2 + 1 columns instead of full complex planes.
// The epilogue block takes a tile of row pairs of one world through the
// inverse row transform of every kernel's product, growth, the weighted field,
// the state update and its statistics moments, and the next step's forward row
// transform of the new rows: the potentials and the new rows never leave the
// block (they are stored only as the new state and as requested trajectories).
#include "nd.cuh"

namespace lgx {
namespace {

struct RowsArgs {
  const float* src;
  float* dst;
  float2* half;
  const float2* half_in;
  long pairs;       // planes * pp
  int rows, W, Wh, pp, nr;
  FastDivU ppd, whd;
  int pitch, zp;    // exchange pitch; pitch of the Z rows
  long buf;         // elements of one exchange buffer
  FastDivU nrd;
  float scale;
  int accumulate;
};

// Row pair l of the block's tile: its first row (plane * rows + row), 0, 1 or 2 rows.
__device__ __forceinline__ void tile_pair(const RowsArgs& a, int l, long* row, int* n) {
  const long g = (long)blockIdx.x * a.nr + l;
  *row = 0;
  *n = 0;
  if (g >= a.pairs) return;
  const int plane = a.ppd.div((int)g), r0 = 2 * ((int)g - plane * a.pp);
  *row = (long)plane * a.rows + r0;
  *n = min(2, a.rows - r0);
}

template <int KIND>
__global__ void __launch_bounds__(kNdThreads, nd_blocks(KIND)) nd_rows_fwd_kernel(RowsArgs a, LineAxis ax) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ long row[kMaxTileLines];
  __shared__ int cnt[kMaxTileLines];
  float2* tw = sm;
  Tile t;
  t.b[0] = tw + ax.m;
  t.b[1] = t.b[0] + a.buf;
  float2* Z = t.b[1] + a.buf;
  t.lp = a.pitch;
  t.nl = a.nr;
  t.nld = a.nrd;
  depend_wait();
  a.src = after_wait(a.src);
  t.tab = after_wait(ax.tw);
  load_line_twiddles(tw, t.tab, ax.m);
  for (int l = threadIdx.x; l < a.nr; l += blockDim.x) tile_pair(a, l, row + l, cnt + l);
  __syncthreads();
  const float* __restrict__ src = a.src;
  const int W = a.W, zp = a.zp;
  line_fft<false, false, KIND>(
      ax, tw, t,
      [&](int l, int i) {
        const float* p = src + row[l] * W + i;
        const int n = cnt[l];
        return make_float2(n > 0 ? __ldg(p) : 0.f, n > 1 ? __ldg(p + W) : 0.f);
      },
      [=](int l, int k, float2 v) { Z[l * zp + k] = v; });
  __syncthreads();
  for (int idx = threadIdx.x; idx < a.nr * a.Wh; idx += blockDim.x) {
    const int l = a.whd.div(idx), k = idx - l * a.Wh;
    const int n = cnt[l];
    if (n == 0) continue;
    const float2 zk = Z[l * zp + k], zm = Z[l * zp + (k == 0 ? 0 : W - k)];
    float2* o = a.half + row[l] * a.Wh + k;
    o[0] = unpack_row0(zk, zm);
    if (n > 1) o[a.Wh] = unpack_row1(zk, zm);
  }
}

template <int KIND>
__global__ void __launch_bounds__(kNdThreads, nd_blocks(KIND)) nd_rows_inv_kernel(RowsArgs a, LineAxis ax) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ long row[kMaxTileLines];
  __shared__ int cnt[kMaxTileLines];
  float2* tw = sm;
  Tile t;
  t.b[0] = tw + ax.m;
  t.b[1] = t.b[0] + a.buf;
  t.lp = a.pitch;
  t.nl = a.nr;
  t.nld = a.nrd;
  depend_wait();
  a.half_in = after_wait(a.half_in);
  a.dst = after_wait(a.dst);
  t.tab = after_wait(ax.tw);
  load_line_twiddles(tw, t.tab, ax.m);
  for (int l = threadIdx.x; l < a.nr; l += blockDim.x) tile_pair(a, l, row + l, cnt + l);
  __syncthreads();
  const float2* __restrict__ half = a.half_in;
  const int W = a.W, Wh = a.Wh;
  line_fft<true, false, KIND>(
      ax, tw, t,
      [&](int l, int i) {
        const bool mir = i >= Wh;
        const float2* p = half + row[l] * Wh + (mir ? W - i : i);
        const int n = cnt[l];
        const float2 z = make_float2(0.f, 0.f);
        return pack_rows(n > 0 ? __ldg(p) : z, n > 1 ? __ldg(p + Wh) : z, i, W);
      },
      [&](int l, int x, float2 v) {
        const int n = cnt[l];
        float* p = a.dst + row[l] * W + x;
        if (a.accumulate) {
          if (n > 0) p[0] = fmaf(v.x, a.scale, p[0]);
          if (n > 1) p[W] = fmaf(v.y, a.scale, p[W]);
        } else {
          if (n > 0) p[0] = v.x * a.scale;
          if (n > 1) p[W] = v.y * a.scale;
        }
      });
}

// Geometry of a row tile: nr pairs (all of `pairs` over the fill target, at
// most a buffer's worth), their exchange buffers and threads.
struct RowTile {
  int nr, pitch, zp, threads;
  long buf;
};
// Dynamic shared memory of an epilogue block that three of fit an SM: a third
// of its 228 KB, less the system's kilobyte a block and the kernel's own static
// arrays.
constexpr long kThreeBlocksSmem =
    (228 * 1024 / 3 - 1024 - (long)(sizeof(EpiShared) + kMaxTileLines * sizeof(RowPair))) / 256 * 256;
RowTile row_tile(const LineAxis& x, long pairs, long group_pairs, bool three = false) {
  RowTile r;
  // `three`: no more lines than leave room for three blocks an SM, as many as
  // the registers allow (the plain epilogue of one kernel; tiles of several
  // kernels and of wide lines measured slower when cut: 8 worlds of 360 x 480,
  // 3 x 15 kernels 4169 -> 5438 us).  12-step rollouts, us, larger tiles ->
  // these: 32 worlds of 128 x 512 771 -> 580, 512 of 80^2 782 -> 708, 128 of
  // 144^2 819 -> 792; where only the last 2.5 KB decide (two blocks at 74 KB):
  // 32 of 250^2 700 -> 568, 128 1879 -> 1695, 32 of 576^2 3067 -> 2693, 24 of
  // 480^2 1555 -> 1411, of 720^2 4968 -> 4462, 200 of 224^2 2367 -> 2142 (a
  // batch whose waves fall badly loses: 64 of 224^2 758 -> 802).
  const long pts = kThreeBlocksSmem / (long)sizeof(float2) - x.m;
  const long by_smem = three ? std::max(1L, pts / (2 * line_pitch(false, x, 1) + (x.n | 1))) : kMaxTileLines;
  const long fill = (pairs + kFillBlocks - 1) / kFillBlocks;
  // one butterfly per thread at most twice over
  const long by_items = std::max(1L, 2L * kNdThreads * std::min(x.r[0], std::max(x.r[x.stages - 1], 2)) / x.m);
  const long cap = std::max(1L, std::min<long>(std::min<long>(kMaxTileLines, by_items), kMaxPts / x.m));
  const long want = std::max(1L, std::min(std::min(cap, by_smem), std::min(fill, group_pairs)));
  const long tiles = (group_pairs + want - 1) / want;
  r.nr = (int)((group_pairs + tiles - 1) / tiles);  // even tiles over the group
  r.pitch = line_pitch(false, x, r.nr);
  r.buf = line_buf_elems(false, x, r.nr);
  r.zp = x.n | 1;
  r.threads = nd_threads(line_items(x, r.nr));
  return r;
}

cudaError_t rows_args(const LineAxis& x, long planes, int rows, RowsArgs* a, RowTile* rt) {
  a->rows = rows;
  a->W = x.n;
  a->Wh = x.n / 2 + 1;
  a->pp = (rows + 1) / 2;
  a->pairs = planes * a->pp;
  if (a->pairs >= (1L << 31)) return cudaErrorInvalidConfiguration;
  *rt = row_tile(x, a->pairs, a->pairs);
  a->nr = rt->nr;
  a->ppd = make_fastdiv((unsigned)a->pp);
  a->whd = make_fastdiv((unsigned)a->Wh);
  a->nrd = make_fastdiv((unsigned)a->nr);
  a->pitch = rt->pitch;
  a->zp = rt->zp;
  a->buf = rt->buf;
  return cudaSuccess;
}

// ------------------------------------------------------------------ epilogue
struct RowsEpi {
  int nr, pitch, zp;      // pairs per tile, pitches
  int lanes;              // threads per row pair of the epilogue
  long buf;
  FastDivU nrd, hd, whd;
  int field_smem;         // the weighted fields live in shared memory
};

// SINGLE (C = K = 1): the epilogue works on the potentials in Z and leaves the
// new cells there.  Otherwise the weighted fields of the tile accumulate over
// the kernels in F (AddGrowth, the store rule of their inverse transforms), and
// the update (UpdateCells) is the load rule of each channel's forward one.
template <bool SINGLE, int KIND>
__global__ void __launch_bounds__(kNdThreads, nd_blocks(KIND)) nd_rows_epi_kernel(NdTab t, EpiArgs a, RowsEpi g, LineAxis ax) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ RowPair rp[kMaxTileLines];
  __shared__ EpiShared sh;
  float2* tw = sm;
  Tile tl;
  tl.b[0] = tw + ax.m;
  tl.b[1] = tl.b[0] + g.buf;
  float2* Z = tl.b[1] + g.buf;
  tl.lp = g.pitch;
  tl.nl = g.nr;
  tl.nld = g.nrd;
  const int w = blockIdx.x / a.tiles, b = blockIdx.x - w * a.tiles;
  const int sol = w / a.n_init;
  const int W = t.W, Wh = t.Wh, C = t.C, K = t.K, zp = g.zp;
  load_line_twiddles(tw, ax.tw, ax.m);
  depend_wait();
  epi_after_wait(a);
  tl.tab = after_wait(ax.tw);
  const int s0 = a.shift[3 * w], s1 = a.shift[3 * w + 1], s2 = a.shift[3 * w + 2];
  const int sx = t.nd == 3 ? s2 : s1;
  const float dt = step_dt(t, a, w, sol);
  const float* gf = a.gf + sol * a.gf_sol_stride;
  const float* wt = a.w + sol * a.w_sol_stride;
  for (int l = threadIdx.x; l < g.nr; l += blockDim.x) {
    const int r0 = 2 * (b * g.nr + l), rows = max(0, min(2, t.D * t.H - r0));
    const int q0 = rows > 0 ? r0 : 0, q1 = rows > 1 ? r0 + 1 : q0;
    const int z0 = g.hd.div(q0), z1 = g.hd.div(q1);
    rp[l] = row_pair(t, z0, q0 - z0 * t.H, z1, q1 - z1 * t.H, rows, s0, s1);
  }
  __syncthreads();
  Moments mo;
  // the product rows of kernel k, packed
  auto load_rows = [&](int k) {
    const float2* __restrict__ src = a.P + ((long)w * K + k) * t.hcells + (long)2 * b * g.nr * Wh;
    return [=](int l, int i) {
      const bool mir = i >= Wh;
      const float2* p = src + (long)2 * l * Wh + (mir ? W - i : i);
      const int n = rp[l].rows;
      const float2 z = make_float2(0.f, 0.f);
      return pack_rows(n > 0 ? __ldg(p) : z, n > 1 ? __ldg(p + Wh) : z, i, W);
    };
  };
  // half spectra of the tile's new rows (in Z) into S
  auto store_spectra = [&](int c) {
    float2* o = a.S + ((long)w * C + c) * t.hcells + (long)2 * b * g.nr * Wh;
    for (int idx = threadIdx.x; idx < g.nr * Wh; idx += blockDim.x) {
      const int l = g.whd.div(idx), k = idx - l * Wh, n = rp[l].rows;
      if (n == 0) continue;
      const float2 zk = Z[l * zp + k], zm = Z[l * zp + (k == 0 ? 0 : W - k)];
      o[(long)2 * l * Wh + k] = unpack_row0(zk, zm);
      if (n > 1) o[(long)(2 * l + 1) * Wh + k] = unpack_row1(zk, zm);
    }
  };
  auto store_z = [=](int l, int k, float2 v) { Z[l * zp + k] = v; };
  if constexpr (SINGLE) {
    const auto rows0 = load_rows(0);
    line_fft<true, false, KIND>(ax, tw, tl, rows0, store_z);
    __syncthreads();
    epi_single(t, a, rp, Z, g.nr, zp, g.lanes, w, sx, dt, mo);
    const bool emit = a.S != nullptr;
    if (emit) {
      __syncthreads();
      line_fft<false, false, KIND>(
          ax, tw, tl, [=](int l, int i) { return rp[l].rows ? Z[l * zp + i] : make_float2(0.f, 0.f); }, store_z);
    }
    epi_channel_mass(sh, 0, mo.m00);
    if (emit) {
      __syncthreads();
      store_spectra(0);
    }
  } else {
    const EpiChannels ch = epi_channels(t, a, wt);
    // [channel][nr][W] pairs: fields of row0 and row1
    float2* F = g.field_smem ? Z + (long)g.nr * zp
                             : reinterpret_cast<float2*>(a.F) + ((long)(w * a.tiles + b) * C + ch.lo) * g.nr * W;
    for (int i = threadIdx.x; i < (ch.hi - ch.lo) * g.nr * W; i += blockDim.x) F[i] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int k = 0; k < K; ++k) {
      if (!((ch.todo >> k) & 1ull)) continue;
      const auto rows = load_rows(k);
      const AddGrowth add{t, a, rp, F, wt, NdGrowth(t.gf[k], __ldg(gf + 2 * k), __ldg(gf + 2 * k + 1)),
                          a.pot_out ? a.pot_out + ((long)w * K + k) * t.cells : nullptr,
                          g.nr, k, ch.lo, ch.hi, (bool)((ch.count >> k) & 1ull), mo};
      line_fft_rules<true, false, KIND>(ax, tw, tl, each_in(rows), add);
    }
    __syncthreads();
    for (int c = ch.lo; c < ch.hi; ++c)
      epi_channel(t, a, rp, F + (long)(c - ch.lo) * g.nr * W, g.nr, w, c, sx, dt, wt, mo, sh,
                  [&](const UpdateCells& update) {
                    line_fft_rules<false, false, KIND>(ax, tw, tl, update, each_out(store_z));
                    __syncthreads();
                    store_spectra(c);
                    __syncthreads();  // Z is rewritten by the next channel
                  });
    for (int c = 0; c < C; ++c)
      if (c < ch.lo || c >= ch.hi) epi_channel_mass(sh, c, 0.f);
  }
  epi_finish(t, a, sh, w, b + blockIdx.y * a.tiles, mo, s0, s1, s2);
}

struct EpiTile {
  RowTile rt;
  int tiles;
  bool split, field_smem;
  size_t smem;
};
EpiTile epi_tile(const NdTab& t, const LineAxis& x, long n_worlds) {
  EpiTile e;
  const int pp = (t.D * t.H + 1) / 2;
  const long whole = row_tile(x, kFillBlocks * (long)pp, pp).nr;
  e.split = epi_split(t, n_worlds * ((pp + whole - 1) / whole));
  e.rt = row_tile(x, n_worlds * pp * (e.split ? t.C : 1), pp, t.C == 1 && t.K == 1 && !x.wide);
  e.tiles = (pp + e.rt.nr - 1) / e.rt.nr;
  const size_t base = (size_t)(x.m + 2 * e.rt.buf + (long)e.rt.nr * e.rt.zp) * sizeof(float2);
  const size_t field = t.C == 1 && t.K == 1 ? 0 : (size_t)(e.split ? 1 : t.C) * e.rt.nr * t.W * sizeof(float2);
  // two blocks per SM keep the fields in shared memory; larger sets go through L2
  e.field_smem = base + field <= (size_t)108 * 1024;
  e.smem = base + (e.field_smem ? field : 0);
  return e;
}

}  // namespace

cudaError_t nd_rows_forward(const LineAxis& x, long planes, int rows, const float* src, float2* half,
                            cudaStream_t st) {
  RowsArgs a{};
  RowTile rt;
  cudaError_t e = rows_args(x, planes, rows, &a, &rt);
  if (e != cudaSuccess) return e;
  a.src = src;
  a.half = half;
  const size_t smem = (size_t)(x.m + 2 * rt.buf + (long)rt.nr * rt.zp) * sizeof(float2);
  auto f = for_line_kind(x, [](auto kind) { return nd_rows_fwd_kernel<decltype(kind)::value>; });
  if ((e = nd_allow_smem((const void*)f)) != cudaSuccess) return e;
  const unsigned blocks = (unsigned)((a.pairs + a.nr - 1) / a.nr);
  return launch_dependent(f, blocks, rt.threads, smem, st, a, x);
}

cudaError_t nd_rows_inverse(const LineAxis& x, long planes, int rows, const float2* half, float* dst, bool accumulate,
                            float scale, cudaStream_t st) {
  RowsArgs a{};
  RowTile rt;
  cudaError_t e = rows_args(x, planes, rows, &a, &rt);
  if (e != cudaSuccess) return e;
  a.half_in = half;
  a.dst = dst;
  a.accumulate = accumulate ? 1 : 0;
  a.scale = scale;
  const size_t smem = (size_t)(x.m + 2 * rt.buf) * sizeof(float2);
  auto f = for_line_kind(x, [](auto kind) { return nd_rows_inv_kernel<decltype(kind)::value>; });
  if ((e = nd_allow_smem((const void*)f)) != cudaSuccess) return e;
  const unsigned blocks = (unsigned)((a.pairs + a.nr - 1) / a.nr);
  return launch_dependent(f, blocks, rt.threads, smem, st, a, x);
}

int nd_rows_epi_blocks(const NdTab& t, const LineAxis& x, long n_worlds, long* field_pairs) {
  const EpiTile e = epi_tile(t, x, n_worlds);
  if (field_pairs) *field_pairs = e.field_smem ? 0 : (long)e.tiles * e.rt.nr * t.W;
  return e.tiles * (e.split ? t.C : 1);
}

cudaError_t nd_rows_epilogue(const NdTab& t, const LineAxis& x, const EpiArgs& args, cudaStream_t st) {
  EpiArgs a = args;
  const EpiTile e = epi_tile(t, x, a.n_worlds);
  a.tiles = e.tiles;
  a.split = e.split ? 1 : 0;
  a.bpw = e.tiles * (e.split ? t.C : 1);
  RowsEpi g;
  g.nr = e.rt.nr;
  g.pitch = e.rt.pitch;
  g.zp = e.rt.zp;
  const int threads = epi_threads(e.rt.threads, a.bpw);
  g.lanes = epi_lanes(t.W, e.rt.nr, threads);
  g.buf = e.rt.buf;
  g.nrd = make_fastdiv((unsigned)g.nr);
  g.hd = make_fastdiv((unsigned)t.H);
  g.whd = make_fastdiv((unsigned)t.Wh);
  g.field_smem = e.field_smem ? 1 : 0;
  const long blocks = (long)a.n_worlds * a.tiles;
  if (blocks >= (1L << 31)) return cudaErrorInvalidConfiguration;
  const bool single = t.C == 1 && t.K == 1;
  auto f = for_line_kind(x, [&](auto kind) {
    return single ? nd_rows_epi_kernel<true, decltype(kind)::value> : nd_rows_epi_kernel<false, decltype(kind)::value>;
  });
  const cudaError_t err = nd_allow_smem((const void*)f);
  if (err != cudaSuccess) return err;
  return launch_dependent(f, dim3((unsigned)blocks, e.split ? t.C : 1), threads, e.smem, st, t, a, g, x);
}

}  // namespace lgx
