// Column transforms and the fused convolution pass of the general N-D engine.
//
// Along the last world axis (z in 3D, y in 2D) line i of a half-spectrum plane
// holds the points i + j I, j < L, with I = hcells / L lines per plane.  One
// block takes a tile of nl adjacent lines of one world: the forward transform
// along the axis of each channel, the spectrum products, the inverse transform
// of each product -- the last forward pass, the multiply and the first inverse
// pass in one launch.  A channel read by one kernel keeps its spectrum in
// registers between the two transforms (line_center); one read by several
// keeps it in shared memory.  The caller's half spectra are read as given (the
// 1/cells of the inverse transform is applied where the result is stored).
#include "nd.cuh"

namespace lgx {
namespace {

struct ConvTile {
  int nl, tiles, lp, sp;  // lines per tile, tiles per plane, line pitches of the exchange and of kept spectra
  long I, buf, keep;         // lines per plane; elements of an exchange buffer and of a kept spectrum tile
  FastDivU nld;
};

__device__ __forceinline__ void conv_tile_init(Tile& t, const ConvTile& g, float2* b) {
  t.b[0] = b;
  t.b[1] = b + g.buf;
  t.lp = g.lp;
  t.nl = g.nl;
  t.nld = g.nld;
}

// One channel of the tile a block (blockIdx.y): the channels share nothing.
// forward: P[w, k] = IFFT_axis(FFT_axis(S[w, c_in(k)]) * K[sol, c_in(k), slot(k)])
template <int KIND>
__global__ void __launch_bounds__(kNdThreads, nd_blocks(KIND)) nd_conv_kernel(NdTab t, ConvArgs a, ConvTile g, LineAxis ax) {
  constexpr bool BL = KIND == LINE_BLUESTEIN, WIDE = KIND == LINE_WIDE;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  Tile tl;
  conv_tile_init(tl, g, tw + ax.m);
  float2* Sc = tl.b[1] + g.buf;
  const int w = blockIdx.x / g.tiles;
  const long i0 = (long)(blockIdx.x - w * g.tiles) * g.nl;
  const int lines = (int)min((long)g.nl, g.I - i0);
  const int sol = w / a.n_init, sp = g.sp;
  const int I = (int)g.I;
  load_line_twiddles(tw, ax.tw, ax.m);
  depend_wait();
  tl.tab = after_wait(ax.tw);
  a.S = after_wait(a.S);
  __syncthreads();
  const float2 zero = make_float2(0.f, 0.f);
  const int c = blockIdx.y;
  int nk = 0, first = 0;
  for (int k = t.K - 1; k >= 0; --k)
    if (t.cin[k] == c) {
      ++nk;
      first = k;
    }
  if (nk == 0) return;
  const float2* __restrict__ S = a.S + ((long)w * t.C + c) * t.hcells + i0;
  const float2* __restrict__ Kc = a.kh + sol * a.kh_sol_stride + (long)c * t.max_k * t.hcells + i0;
  auto load = [=](int l, int i) { return l < lines ? __ldg(S + l + (long)i * I) : zero; };
  auto store_to = [=](int k) {
    float2* __restrict__ P = a.P + ((long)w * t.K + k) * t.hcells + i0;
    return [=](int l, int i, float2 v) {
      if (l < lines) P[l + (long)i * I] = v;
    };
  };
  if (!BL && nk == 1) {
    const float2* __restrict__ kk = Kc + (long)t.slot[first] * t.hcells;
    line_head<false, true, WIDE>(ax, tw, tl, each_in(load));
    line_center<false, true, WIDE>(ax, tw, tl, [=](int l, int j, int nb, auto& v) {
      constexpr int R = (int)(sizeof(v) / sizeof(float2));
      float2 s[R];
#pragma unroll
      for (int q = 0; q < R; ++q) s[q] = l < lines ? __ldg(kk + l + (long)(j + q * nb) * I) : zero;
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = cmul(v[q], s[q]);
      return true;
    });
    line_middle<true, true>(ax, tw, tl);
    const auto store = store_to(first);
    line_tail<true, true, WIDE>(ax, tw, tl, each_out(store));
  } else {
    line_fft<false, true, KIND>(ax, tw, tl, load, [=](int l, int i, float2 v) { Sc[i * sp + l] = v; });
    __syncthreads();
    for (int k = first; k < t.K; ++k) {
      if (t.cin[k] != c) continue;
      const float2* __restrict__ kk = Kc + (long)t.slot[k] * t.hcells;
      line_fft<true, true, KIND>(
          ax, tw, tl,
          [=](int l, int i) { return l < lines ? cmul(Sc[i * sp + l], __ldg(kk + l + (long)i * I)) : zero; },
          store_to(k));
    }
  }
}

// adjoint: with A_k = FFT(a_k), S_c = FFT(state_c) along the axis,
// gk[w, k] += A_k conj(S_c_in(k)) and Q[w, c] = IFFT_axis(sum_{k: c_in(k) = c}
// A_k conj(K_k)) -- the last forward passes of a and of the state, the
// spectral products and the first inverse pass of Q in one launch.
template <int KIND>
__global__ void __launch_bounds__(kNdThreads, nd_blocks(KIND)) nd_adj_conv_kernel(NdTab t, ConvArgs a, ConvTile g, LineAxis ax) {
  constexpr bool BL = KIND == LINE_BLUESTEIN, WIDE = KIND == LINE_WIDE;
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  Tile tl;
  conv_tile_init(tl, g, tw + ax.m);
  float2* Sc = tl.b[1] + g.buf;
  float2* Qc = Sc + g.keep;
  const int w = blockIdx.x / g.tiles;
  const long i0 = (long)(blockIdx.x - w * g.tiles) * g.nl;
  const int lines = (int)min((long)g.nl, g.I - i0);
  const int sol = w / a.n_init, sp = g.sp;
  const int I = (int)g.I;
  load_line_twiddles(tw, ax.tw, ax.m);
  depend_wait();
  tl.tab = after_wait(ax.tw);
  a.S = after_wait(a.S);
  a.A = after_wait(a.A);
  a.gk = after_wait(a.gk);
  __syncthreads();
  const float2 zero = make_float2(0.f, 0.f);
  const int c = blockIdx.y;
  int nk = 0, first = t.K;
  for (int k = t.K - 1; k >= 0; --k)
    if (t.cin[k] == c) {
      ++nk;
      first = k;
    }
  const float2* __restrict__ S = a.S + ((long)w * t.C + c) * t.hcells + i0;
  const float2* __restrict__ Kc = a.kh + sol * a.kh_sol_stride + (long)c * t.max_k * t.hcells + i0;
  float2* __restrict__ Q = a.Q + ((long)w * t.C + c) * t.hcells + i0;
  auto store_q = [=](int l, int i, float2 v) {
    if (l < lines) Q[l + (long)i * I] = v;
  };
  if (nk == 0) {
    for (int i = threadIdx.x; i < lines * ax.n; i += blockDim.x) {
      const int j = i / lines;
      Q[i - j * lines + (long)j * I] = zero;
    }
    return;
  }
  line_fft<false, true, KIND>(
      ax, tw, tl, [=](int l, int i) { return l < lines ? __ldg(S + l + (long)i * I) : zero; },
      [=](int l, int i, float2 v) {
        Sc[i * sp + l] = v;
        if (BL || nk > 1) Qc[i * sp + l] = zero;
      });
  __syncthreads();
  for (int k = first; k < t.K; ++k) {
    if (t.cin[k] != c) continue;
    const float2* __restrict__ A = a.A + ((long)w * t.K + k) * t.hcells + i0;
    const float2* __restrict__ kk = Kc + (long)t.slot[k] * t.hcells;
    float2* __restrict__ gk = a.gk + ((long)w * t.K + k) * t.hcells + i0;
    auto load = [=](int l, int i) { return l < lines ? __ldg(A + l + (long)i * I) : zero; };
    if (!BL && nk == 1) {
      line_head<false, true, WIDE>(ax, tw, tl, each_in(load));
      line_center<false, true, WIDE>(ax, tw, tl, [=](int l, int j, int nb, auto& v) {
        constexpr int R = (int)(sizeof(v) / sizeof(float2));
        if (l >= lines) return true;  // zeros in, zeros out
        float2 s[R], o[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          s[q] = __ldg(kk + l + (long)(j + q * nb) * I);
          o[q] = gk[l + (long)(j + q * nb) * I];
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int i = j + q * nb;
          gk[l + (long)i * I] = cadd(o[q], cmulc(v[q], Sc[i * sp + l]));
          v[q] = cmulc(v[q], s[q]);
        }
        return true;
      });
      line_middle<true, true>(ax, tw, tl);
      line_tail<true, true, WIDE>(ax, tw, tl, each_out(store_q));
    } else {
      line_fft<false, true, KIND>(ax, tw, tl, load, [=](int l, int i, float2 v) {
        if (l >= lines) return;
        float2* gp = gk + l + (long)i * I;
        *gp = cadd(*gp, cmulc(v, Sc[i * sp + l]));
        Qc[i * sp + l] = cadd(Qc[i * sp + l], cmulc(v, __ldg(kk + l + (long)i * I)));
      });
    }
  }
  __syncthreads();
  if (BL || nk > 1) {
    line_fft<true, true, KIND>(ax, tw, tl, [=](int l, int i) { return Qc[i * sp + l]; }, store_q);
  }
}

// In-place transforms along y of the half-spectrum z-planes.
struct ColArgs {
  float2* data;
  ConvTile g;
};
template <bool INV, int KIND>
__global__ void __launch_bounds__(kNdThreads, nd_blocks(KIND)) nd_columns_kernel(ColArgs a, LineAxis ax) {
  extern __shared__ __align__(16) float2 sm[];
  float2* tw = sm;
  Tile tl;
  conv_tile_init(tl, a.g, tw + ax.m);
  const long plane = blockIdx.x / a.g.tiles;
  const long i0 = (long)(blockIdx.x - plane * a.g.tiles) * a.g.nl;
  const int lines = (int)min((long)a.g.nl, a.g.I - i0);
  const int I = (int)a.g.I;
  depend_wait();
  a.data = after_wait(a.data);
  tl.tab = after_wait(ax.tw);
  load_line_twiddles(tw, tl.tab, ax.m);
  __syncthreads();
  float2* d = a.data + plane * a.g.I * ax.n + i0;
  line_fft<INV, true, KIND>(
      ax, tw, tl, [=](int l, int i) { return l < lines ? d[l + (long)i * I] : make_float2(0.f, 0.f); },
      [=](int l, int i, float2 v) {
        if (l < lines) d[l + (long)i * I] = v;
      });
}

// Tile of a strided pass over `groups` planes of I lines: at most 32 lines
// (whole 128-byte segments), as few as 4 (a 32-byte sector each) when the pass
// has too few lines to fill the GPU, evenly cut.
ConvTile conv_tile(const LineAxis& ax, long groups, long I) {
  ConvTile g;
  g.I = I;
  const long cap = std::max(1L, std::min<long>(32, kMaxPts / ax.m));
  const long fill = (groups * I + kFillBlocks - 1) / kFillBlocks;
  const long want = std::min(std::min(cap, std::max(4L, fill)), I);
  g.tiles = (int)((I + want - 1) / want);
  g.nl = (int)((I + g.tiles - 1) / g.tiles);
  g.lp = line_pitch(true, ax, g.nl);
  g.buf = line_buf_elems(true, ax, g.nl);
  g.sp = g.nl | 1;
  g.keep = (long)ax.n * g.sp;
  g.nld = make_fastdiv((unsigned)g.nl);
  return g;
}

}  // namespace

cudaError_t nd_convolve(bool adjoint, const NdTab& t, const LineAxis& ax, long nw, const ConvArgs& a,
                        cudaStream_t st) {
  const ConvTile g = conv_tile(ax, nw * t.C, t.hcells / ax.n);
  const bool bl = ax.m != ax.n;
  int per[kMaxChannels] = {0}, most = 0;
  for (int k = 0; k < t.K; ++k) most = std::max(most, ++per[t.cin[k]]);
  const int keeps = adjoint ? (bl || most > 1 ? 2 : 1) : (bl || most > 1 ? 1 : 0);
  const size_t smem = (size_t)(ax.m + 2 * g.buf + keeps * g.keep) * sizeof(float2);
  const long blocks = nw * g.tiles;
  if (blocks >= (1L << 31)) return cudaErrorInvalidConfiguration;
  auto f = for_line_kind(ax, [&](auto kind) {
    return adjoint ? nd_adj_conv_kernel<decltype(kind)::value> : nd_conv_kernel<decltype(kind)::value>;
  });
  const cudaError_t e = nd_allow_smem((const void*)f);
  if (e != cudaSuccess) return e;
  return launch_dependent(f, dim3((unsigned)blocks, (unsigned)t.C), nd_threads(line_items(ax, g.nl)), smem, st, t, a, g, ax);
}

cudaError_t nd_columns(bool inv, const NdTab& t, const LineAxis& y, long planes, float2* data, cudaStream_t st) {
  ColArgs a;
  a.data = data;
  const long groups = planes * t.D;
  a.g = conv_tile(y, groups, t.Wh);
  const size_t smem = (size_t)(y.m + 2 * a.g.buf) * sizeof(float2);
  const long blocks = groups * a.g.tiles;
  if (blocks >= (1L << 31)) return cudaErrorInvalidConfiguration;
  auto f = for_line_kind(y, [&](auto kind) {
    return inv ? nd_columns_kernel<true, decltype(kind)::value> : nd_columns_kernel<false, decltype(kind)::value>;
  });
  const cudaError_t e = nd_allow_smem((const void*)f);
  if (e != cudaSuccess) return e;
  return launch_dependent(f, (unsigned)blocks, nd_threads(line_items(y, a.g.nl)), smem, st, a, y);
}

}  // namespace lgx
