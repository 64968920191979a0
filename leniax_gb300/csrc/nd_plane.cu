// z-plane passes of the general N-D engine: 3D worlds whose planes fit a tile
// take both in-plane transforms of a plane in one block, so an Euler step is
// two launches -- the convolution pass along z and nd_plane_epi_kernel, which
// takes every kernel's product plane through the inverse y and x transforms,
// growth, the weighted field, the state update and its moments, and the new
// plane through the next step's x and y transforms.  Rows travel in packed
// pairs, columns as the W/2 + 1 columns of half spectra.
#include "nd.cuh"

namespace lgx {
namespace {

struct PlaneGeo {
  int pp;             // row pairs
  int xpitch, ypitch; // exchange pitches of the row (pp lines) and column (Wh lines) transforms
  int zp, hp;         // pitch of the packed rows Z [pp][W]; of the half plane [H][Wh]
  long buf, keep;     // elements of an exchange buffer; of the Z / half-plane buffer
  FastDivU ppd, whd;
  int field_smem, lanes;  // lanes: threads per row pair of the epilogue
};

struct PlaneTile {
  float2 *twx, *twy, *keep;
  Tile t;
};

__device__ __forceinline__ PlaneTile plane_init(const PlaneGeo& g, const LineAxis& ax, const LineAxis& ay,
                                                const float2* tabx, const float2* taby, float2* sm) {
  PlaneTile p;
  p.twx = sm;
  p.twy = sm + ax.m;
  p.t.b[0] = p.twy + ay.m;
  p.t.b[1] = p.t.b[0] + g.buf;
  p.keep = p.t.b[1] + g.buf;
  load_line_twiddles(p.twx, tabx, ax.m);
  load_line_twiddles(p.twy, taby, ay.m);
  return p;
}
__device__ __forceinline__ void as_rows(Tile& t, const PlaneGeo& g) {
  t.lp = g.xpitch;
  t.nl = g.pp;
  t.nld = g.ppd;
}
__device__ __forceinline__ void as_columns(Tile& t, const PlaneGeo& g, int Wh) {
  t.lp = g.ypitch;
  t.nl = Wh;
  t.nld = g.whd;
}

// Forward y transforms of the plane whose packed row spectra are in Z, the
// half plane stored to dst.
__device__ __forceinline__ void columns_from_rows(PlaneTile& p, const PlaneGeo& g, const LineAxis& ay, int W, int Wh,
                                                  float2* __restrict__ dst) {
  const float2* Z = p.keep;
  const int zp = g.zp;
  as_columns(p.t, g, Wh);
  line_fft<false, true, LINE_PLAIN>(
      ay, p.twy, p.t,
      [=](int l, int i) {
        const float2* z = Z + (i >> 1) * zp;
        const float2 zk = z[l], zm = z[l == 0 ? 0 : W - l];
        return (i & 1) ? unpack_row1(zk, zm) : unpack_row0(zk, zm);
      },
      [=](int l, int i, float2 v) { dst[i * Wh + l] = v; });
}

// Inverse y transforms of a half plane into the kept half plane.
__device__ __forceinline__ void columns_inverse(PlaneTile& p, const PlaneGeo& g, const LineAxis& ay, int Wh,
                                                const float2* __restrict__ src) {
  float2* h = p.keep;
  const int hp = g.hp;
  as_columns(p.t, g, Wh);
  line_fft<true, true, LINE_PLAIN>(
      ay, p.twy, p.t, [=](int l, int i) { return __ldg(src + i * Wh + l); },
      [=](int l, int i, float2 v) { h[i * hp + l] = v; });
  __syncthreads();
}

// The load rule of the packed inverse rows of the kept half plane.
struct KeptRows {
  const float2* h;
  int hp, H, W, Wh;
  __device__ __forceinline__ float2 operator()(int l, int i) const {
    const bool mir = i >= Wh;
    const float2* p = h + 2 * l * hp + (mir ? W - i : i);
    return pack_rows(p[0], 2 * l + 1 < H ? p[hp] : make_float2(0.f, 0.f), i, W);
  }
};

struct PlaneArgs {
  const float* src;
  float* dst;
  const float2* half_in;
  float2* half;
  int H, W, Wh, accumulate;
  float scale;
};

__global__ void __launch_bounds__(kNdThreads, kNdBlocksPerSm) nd_plane_fwd_kernel(PlaneArgs a, PlaneGeo g, LineAxis ax,
                                                                     LineAxis ay) {
  extern __shared__ __align__(16) float2 sm[];
  depend_wait();
  a.src = after_wait(a.src);
  PlaneTile p = plane_init(g, ax, ay, after_wait(ax.tw), after_wait(ay.tw), sm);
  __syncthreads();
  const int H = a.H, W = a.W, Wh = a.Wh, zp = g.zp;
  const float* __restrict__ src = a.src + (long)blockIdx.x * H * W;
  float2* Z = p.keep;
  as_rows(p.t, g);
  line_fft<false, false, LINE_PLAIN>(
      ax, p.twx, p.t,
      [=](int l, int i) {
        const float* q = src + 2 * l * W + i;
        return make_float2(__ldg(q), 2 * l + 1 < H ? __ldg(q + W) : 0.f);
      },
      [=](int l, int k, float2 v) { Z[l * zp + k] = v; });
  __syncthreads();
  columns_from_rows(p, g, ay, W, Wh, a.half + (long)blockIdx.x * H * Wh);
}

__global__ void __launch_bounds__(kNdThreads, kNdBlocksPerSm) nd_plane_inv_kernel(PlaneArgs a, PlaneGeo g, LineAxis ax,
                                                                     LineAxis ay) {
  extern __shared__ __align__(16) float2 sm[];
  depend_wait();
  a.half_in = after_wait(a.half_in);
  a.dst = after_wait(a.dst);
  PlaneTile p = plane_init(g, ax, ay, after_wait(ax.tw), after_wait(ay.tw), sm);
  __syncthreads();
  const int H = a.H, W = a.W, Wh = a.Wh;
  columns_inverse(p, g, ay, Wh, a.half_in + (long)blockIdx.x * H * Wh);
  float* dst = a.dst + (long)blockIdx.x * H * W;
  const float scale = a.scale;
  const bool add = a.accumulate != 0;
  as_rows(p.t, g);
  line_fft<true, false, LINE_PLAIN>(ax, p.twx, p.t, KeptRows{p.keep, g.hp, H, W, Wh}, [=](int l, int x, float2 v) {
    float* q = dst + 2 * l * W + x;
    q[0] = add ? fmaf(v.x, scale, q[0]) : v.x * scale;
    if (2 * l + 1 < H) q[W] = add ? fmaf(v.y, scale, q[W]) : v.y * scale;
  });
}

// One block per (world, z-plane).  SINGLE (C = K = 1): the epilogue works on
// the potentials in Z and leaves the new cells there; otherwise the weighted
// fields accumulate in F over the kernels and the update is the load rule of
// each channel's row transform.
template <bool SINGLE>
__global__ void __launch_bounds__(kNdThreads, kNdBlocksPerSm) nd_plane_epi_kernel(NdTab t, EpiArgs a, PlaneGeo g, LineAxis ax,
                                                                     LineAxis ay) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ RowPair rp[kMaxTileLines];
  __shared__ EpiShared sh;
  PlaneTile p = plane_init(g, ax, ay, ax.tw, ay.tw, sm);
  depend_wait();
  epi_after_wait(a);
  const int w = blockIdx.x / t.D, z = blockIdx.x - w * t.D;
  const int sol = w / a.n_init;
  const int H = t.H, W = t.W, Wh = t.Wh, C = t.C, K = t.K, zp = g.zp;
  const int s0 = a.shift[3 * w], s1 = a.shift[3 * w + 1], s2 = a.shift[3 * w + 2];
  const float dt = step_dt(t, a, w, sol);
  const float* gf = a.gf + sol * a.gf_sol_stride;
  const float* wt = a.w + sol * a.w_sol_stride;
  for (int l = threadIdx.x; l < g.pp; l += blockDim.x) {
    const int y1 = min(2 * l + 1, H - 1);
    rp[l] = row_pair(t, z, 2 * l, z, y1, 2 * l + 1 < H ? 2 : 1, s0, s1);
  }
  __syncthreads();
  Moments mo;
  float2* Z = p.keep;
  auto store_z = [=](int l, int k, float2 v) { Z[l * zp + k] = v; };
  const long hplane = (long)H * Wh;
  const KeptRows kept{p.keep, g.hp, H, W, Wh};
  if constexpr (SINGLE) {
    columns_inverse(p, g, ay, Wh, a.P + (long)w * t.hcells + z * hplane);
    as_rows(p.t, g);
    line_fft<true, false, LINE_PLAIN>(ax, p.twx, p.t, kept, store_z);
    __syncthreads();
    epi_single(t, a, rp, Z, g.pp, zp, g.lanes, w, s2, dt, mo);
    if (a.S) {
      __syncthreads();
      line_fft<false, false, LINE_PLAIN>(ax, p.twx, p.t, [=](int l, int i) { return Z[l * zp + i]; }, store_z);
      __syncthreads();
      columns_from_rows(p, g, ay, W, Wh, a.S + (long)w * t.hcells + z * hplane);
    }
    epi_channel_mass(sh, 0, mo.m00);
  } else {
    const EpiChannels ch = epi_channels(t, a, wt);
    float2* F = g.field_smem ? p.keep + g.keep
                             : reinterpret_cast<float2*>(a.F) + ((long)blockIdx.x * C + ch.lo) * g.pp * W;
    for (int i = threadIdx.x; i < (ch.hi - ch.lo) * g.pp * W; i += blockDim.x) F[i] = make_float2(0.f, 0.f);
    __syncthreads();
    for (int k = 0; k < K; ++k) {
      if (!((ch.todo >> k) & 1ull)) continue;
      columns_inverse(p, g, ay, Wh, a.P + ((long)w * K + k) * t.hcells + z * hplane);
      as_rows(p.t, g);
      const AddGrowth add{t, a, rp, F, wt, NdGrowth(t.gf[k], __ldg(gf + 2 * k), __ldg(gf + 2 * k + 1)),
                          a.pot_out ? a.pot_out + ((long)w * K + k) * t.cells : nullptr,
                          g.pp, k, ch.lo, ch.hi, (bool)((ch.count >> k) & 1ull), mo};
      line_fft_rules<true, false, LINE_PLAIN>(ax, p.twx, p.t, each_in(kept), add);
      __syncthreads();  // the half plane is rewritten by the next kernel
    }
    for (int c = ch.lo; c < ch.hi; ++c)
      epi_channel(t, a, rp, F + (long)(c - ch.lo) * g.pp * W, g.pp, w, c, s2, dt, wt, mo, sh,
                  [&](const UpdateCells& update) {
                    as_rows(p.t, g);
                    line_fft_rules<false, false, LINE_PLAIN>(ax, p.twx, p.t, update, each_out(store_z));
                    __syncthreads();
                    columns_from_rows(p, g, ay, W, Wh, a.S + ((long)w * C + c) * t.hcells + z * hplane);
                    __syncthreads();  // Z is rewritten by the next channel
                  });
    for (int c = 0; c < C; ++c)
      if (c < ch.lo || c >= ch.hi) epi_channel_mass(sh, c, 0.f);
  }
  epi_finish(t, a, sh, w, z + blockIdx.y * a.tiles, mo, s0, s1, s2);
}

struct PlanePlan {
  PlaneGeo g;
  int threads;
  size_t smem;
};
PlanePlan plane_plan(const NdTab& t, const NdAxes& ax) {
  PlanePlan p;
  PlaneGeo& g = p.g;
  g.pp = (t.H + 1) / 2;
  g.xpitch = line_pitch(false, ax.x, g.pp);
  g.ypitch = line_pitch(true, ax.y, t.Wh);
  g.zp = t.W | 1;
  g.hp = t.Wh | 1;
  g.buf = std::max(line_buf_elems(false, ax.x, g.pp), line_buf_elems(true, ax.y, t.Wh));
  g.keep = std::max((long)g.pp * g.zp, (long)t.H * g.hp);
  g.ppd = make_fastdiv((unsigned)g.pp);
  g.whd = make_fastdiv((unsigned)t.Wh);
  g.field_smem = 0;
  g.lanes = 0;  // the epilogue's, by its threads
  p.threads = nd_threads(std::max(line_items(ax.x, g.pp), line_items(ax.y, t.Wh)));
  p.smem = (size_t)(t.W + t.H + 2 * g.buf + g.keep) * sizeof(float2);
  return p;
}
size_t plane_field_bytes(const NdTab& t, const PlanePlan& p, bool split) {
  return t.C == 1 && t.K == 1 ? 0 : (size_t)(split ? 1 : t.C) * p.g.pp * t.W * sizeof(float2);
}

}  // namespace

bool nd_plane_ok(const NdTab& t, const NdAxes& ax) {
  return t.D > 1 && (long)t.H * t.W <= kMaxPts && ax.x.m == t.W && ax.y.m == t.H && (t.H + 1) / 2 <= kMaxTileLines;
}

int nd_plane_epi_blocks(const NdTab& t, const NdAxes& ax, long n_worlds, bool* field_global) {
  const PlanePlan p = plane_plan(t, ax);
  const bool split = epi_split(t, n_worlds * t.D);
  if (field_global) *field_global = p.smem + plane_field_bytes(t, p, split) > (size_t)108 * 1024;
  return t.D * (split ? t.C : 1);
}

cudaError_t nd_plane_forward(const NdTab& t, const NdAxes& ax, long planes, const float* src, float2* half,
                             cudaStream_t st) {
  const PlanePlan p = plane_plan(t, ax);
  PlaneArgs a{};
  a.src = src;
  a.half = half;
  a.H = t.H;
  a.W = t.W;
  a.Wh = t.Wh;
  const long blocks = planes * t.D;
  if (blocks >= (1L << 31)) return cudaErrorInvalidConfiguration;
  const cudaError_t e = nd_allow_smem((const void*)nd_plane_fwd_kernel);
  if (e != cudaSuccess) return e;
  return launch_dependent(nd_plane_fwd_kernel, (unsigned)blocks, p.threads, p.smem, st, a, p.g, ax.x, ax.y);
}

cudaError_t nd_plane_inverse(const NdTab& t, const NdAxes& ax, long planes, const float2* half, float* dst,
                             bool accumulate, float scale, cudaStream_t st) {
  const PlanePlan p = plane_plan(t, ax);
  PlaneArgs a{};
  a.half_in = half;
  a.dst = dst;
  a.H = t.H;
  a.W = t.W;
  a.Wh = t.Wh;
  a.accumulate = accumulate ? 1 : 0;
  a.scale = scale;
  const long blocks = planes * t.D;
  if (blocks >= (1L << 31)) return cudaErrorInvalidConfiguration;
  const cudaError_t e = nd_allow_smem((const void*)nd_plane_inv_kernel);
  if (e != cudaSuccess) return e;
  return launch_dependent(nd_plane_inv_kernel, (unsigned)blocks, p.threads, p.smem, st, a, p.g, ax.x, ax.y);
}

cudaError_t nd_plane_epilogue(const NdTab& t, const NdAxes& ax, const EpiArgs& args, cudaStream_t st) {
  EpiArgs a = args;
  PlanePlan p = plane_plan(t, ax);
  bool field_global;
  a.tiles = t.D;
  a.bpw = nd_plane_epi_blocks(t, ax, a.n_worlds, &field_global);
  a.split = a.bpw > a.tiles ? 1 : 0;
  p.g.field_smem = field_global ? 0 : 1;
  const int threads = epi_threads(p.threads, a.bpw);
  p.g.lanes = epi_lanes(t.W, p.g.pp, threads);
  const size_t smem = p.smem + (p.g.field_smem ? plane_field_bytes(t, p, a.split) : 0);
  const long blocks = (long)a.n_worlds * t.D;
  if (blocks >= (1L << 31)) return cudaErrorInvalidConfiguration;
  auto f = t.C == 1 && t.K == 1 ? nd_plane_epi_kernel<true> : nd_plane_epi_kernel<false>;
  const cudaError_t e = nd_allow_smem((const void*)f);
  if (e != cudaSuccess) return e;
  return launch_dependent(f, dim3((unsigned)blocks, a.split ? t.C : 1), threads, smem, st, t, a, p.g, ax.x, ax.y);
}

}  // namespace lgx
