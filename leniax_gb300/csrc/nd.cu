// General N-D engine: any 2D or 3D torus with sides 2..4096 of factors 2, 3, 5
// and 7 or any side 2..2048 (odd, prime and non-square sides included, e.g.
// 48^3), any number of channels and kernels -- the forward Euler step and its
// adjoint.  leniax's get_potential_fft transforms every world axis
// (core.py:74-87); here real rows travel in packed pairs and every later axis
// works on half spectra of W/2 + 1 columns:
//
//   first step   : x (2D) or x and y (3D) transforms of the states -> S
//   Euler step   : conv   (nd_conv.cu): last axis forward, x spectrum of every
//                  kernel, last axis inverse                      -> P
//                  epilogue (nd_rows.cu, nd_plane.cu): inverse y and x
//                  transforms -> potentials u_k, growth, weighted field, state
//                  update (core.py:163-319), statistics moments
//                  (statistics.py:36-126), per-world reduction and carried
//                  shift, x (and y) transforms of the new states -> S
//   adjoint step : clip / state-function gradient, dL/df, dL/dg, growth
//                  derivative -> a_k = dL/du_k; forward transforms of a_k and
//                  of the state; kernel gradient A_k conj(S) accumulated; the
//                  correlation sum_k A_k conj(K_k) per input channel through
//                  the inverse transforms added to lambda; growth-parameter
//                  and weight gradients reduced per (world, kernel)
//
// 3D worlds whose z-planes do not fit a tile take their y transforms as a pass
// of their own (nd_columns).  An Euler step is two launches.  Measured against
// the engine this replaced (full complex planes, one radix-2..7 stage per
// block barrier, three to six launches a step): see the kernels.
//
// This engine serves the worlds the specialised engines do not (resident: 2D
// 32..128 C = K = 1; streamed: square 2D powers of two; one world per CTA: 3D
// 32^3 / 64^3 C = K = 1) and every differentiated model beyond C = K = 1.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "nd.cuh"

namespace lgx {

// (kernel, context) pairs whose dynamic shared-memory limit is already raised
cudaError_t nd_allow_smem(const void* kernel) {
  static std::mutex mu;
  static std::vector<std::pair<const void*, unsigned long long>> done;
  unsigned long long ctx = 0;
  const bool known = current_context_id(&ctx);
  const std::pair<const void*, unsigned long long> key(kernel, ctx);
  if (known) {
    std::lock_guard<std::mutex> lk(mu);
    if (std::find(done.begin(), done.end(), key) != done.end()) return cudaSuccess;
  }
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kNdSmemMax - (int)fa.sharedSizeBytes);
  if (e == cudaSuccess && known) {
    std::lock_guard<std::mutex> lk(mu);
    done.push_back(key);
  }
  return e;
}

namespace {

constexpr int kNT = 256;  // threads of the pointwise kernels

NdTab make_tab(const Model& m, int dt_mode) {
  NdTab t;
  t.C = m.C;
  t.K = m.K;
  t.max_k = m.max_k;
  t.mean = m.mean;
  t.state_fn = m.state_fn;
  t.dt_mode = dt_mode;
  t.nd = m.nb_dims;
  t.D = m.D;
  t.H = m.H;
  t.W = m.W;
  t.Wh = m.W / 2 + 1;
  t.cells = m.cells;
  t.hcells = (long)m.D * m.H * t.Wh;
  for (int k = 0; k < kMaxKernels; ++k) {
    t.cin[k] = k < m.K ? m.cin[k] : 0;
    t.slot[k] = k < m.K ? m.slot[k] : 0;
    t.gf[k] = k < m.K ? m.gf[k] : 0;
  }
  return t;
}

// ------------------------------------------------------------------ tables
// Length of an n-point line's transforms: n, or the smallest m >= 2n - 1 of
// factors 2, 3, 5, 7 (Bluestein); 0 when neither fits a tile.
int transform_len(int n) {
  int r[kLineStages];
  if (n < 2) return 0;
  if (n <= kNdMaxN && line_radices(n, r) > 0) return n;
  if (n > kBluesteinMaxN) return 0;
  for (int m = 2 * n - 1; m <= kMaxPts; ++m)
    if (line_radices(m, r) > 0 && make_plan(m).stages > 0) return m;
  return 0;
}

size_t axis_table_bytes(int n) { return al256(line_table_elems(n, transform_len(n)) * sizeof(float2)); }
size_t table_bytes(int D, int H, int W) {
  return axis_table_bytes(W) + axis_table_bytes(H) + (D > 1 ? axis_table_bytes(D) : 0);
}

// The axes of a D x H x W world with their tables at `ws`.  The x and y axes
// of 3D worlds stay plain: plane tiles hold lines of at most a few dozen.
NdAxes make_axes(int D, int H, int W, void* ws) {
  NdAxes a{};
  char* p = static_cast<char*>(ws);
  make_line_axis(W, transform_len(W), reinterpret_cast<float2*>(p), &a.x, D == 1);
  p += axis_table_bytes(W);
  make_line_axis(H, transform_len(H), reinterpret_cast<float2*>(p), &a.y, D == 1);
  p += axis_table_bytes(H);
  if (D > 1) make_line_axis(D, transform_len(D), reinterpret_cast<float2*>(p), &a.z, true);
  return a;
}

// Tables of one axis per block: the twiddles W_m^j and, for Bluestein lines,
// the chirp c_n = exp(-i pi n^2 / L) (exact reduction of n^2 mod 2L) and the
// m-point spectrum of conj(c) wrapped around.  They are made once per call
// and shared by all its launches; building them in every block of every pass
// cost each block a sincospif per point, or a whole transform.
// The twiddles of plain lines are rounded from double (an entry of tw_entry
// carries the rounding of its argument as well); a block takes a slice of them.
constexpr int kTableBlocks = 16;
__device__ __forceinline__ float2 tw_rounded(int j, int m) {
  double s, c;
  sincospi(2.0 * (double)j / (double)m, &s, &c);
  return make_float2((float)c, (float)-s);
}
struct TableArgs {
  float2* t[3];
  int n[3], m[3];
  GPlan p[3];
};
__global__ void __launch_bounds__(kNT) nd_tables_kernel(TableArgs a) {
  extern __shared__ __align__(16) float2 sm[];
  const int b = blockIdx.x, n = a.n[b], m = a.m[b];
  float2* out = a.t[b];
  if (m == n) {
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < m; j += gridDim.y * blockDim.x) out[j] = tw_rounded(j, m);
    return;
  }
  if (blockIdx.y > 0) return;
  float2 *tw = sm, *A = sm + m, *B = A + m;
  for (int j = threadIdx.x; j < m; j += blockDim.x) out[j] = tw[j] = tw_entry(j, m);
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    const int d = j < n ? j : (m - j < n ? m - j : -1);
    const float2 c = d >= 0 ? tw_entry((int)(((long)d * d) % (2L * n)), 2 * n) : make_float2(0.f, 0.f);
    if (j < n) out[m + j] = c;
    A[j] = d >= 0 ? conjf2(c) : c;
  }
  __syncthreads();
  const float2* r = fft_line<false>(A, B, a.p[b], tw);
  for (int j = threadIdx.x; j < m; j += blockDim.x) out[m + n + j] = r[j];
}

cudaError_t launch_tables(const NdAxes& ax, int D, cudaStream_t st) {
  TableArgs a{};
  const LineAxis* l[3] = {&ax.x, &ax.y, &ax.z};
  const int naxes = D > 1 ? 3 : 2;
  size_t smem = 0;
  for (int i = 0; i < naxes; ++i) {
    a.t[i] = const_cast<float2*>(l[i]->tw);
    a.n[i] = l[i]->n;
    a.m[i] = l[i]->m;
    a.p[i] = make_plan(l[i]->m);
    if (l[i]->m != l[i]->n) smem = std::max(smem, 3 * (size_t)l[i]->m * sizeof(float2));
  }
  if (smem > 0) {
    const cudaError_t e = nd_allow_smem((const void*)nd_tables_kernel);
    if (e != cudaSuccess) return e;
  }
  nd_tables_kernel<<<dim3(naxes, kTableBlocks), kNT, smem, st>>>(a);
  return cudaGetLastError();
}

inline int grid_for(long total) { return (int)std::max(1L, std::min<long>((total + kNT - 1) / kNT, 1L << 16)); }

// ------------------------------------------------------------------ transforms
const LineAxis& last_axis(const NdTab& t, const NdAxes& ax) { return t.nd == 3 ? ax.z : ax.y; }

// Every axis but the last: real planes -> half spectra, and back (the result
// times `scale` stored into dst or added to it; half is overwritten when the
// y transforms are a pass of their own).
cudaError_t forward_head(const NdTab& t, const NdAxes& ax, long planes, const float* src, float2* half,
                         cudaStream_t st) {
  if (nd_plane_ok(t, ax)) return nd_plane_forward(t, ax, planes, src, half, st);
  const cudaError_t e = nd_rows_forward(ax.x, planes, t.D * t.H, src, half, st);
  return e == cudaSuccess && t.D > 1 ? nd_columns(false, t, ax.y, planes, half, st) : e;
}
cudaError_t inverse_tail(const NdTab& t, const NdAxes& ax, long planes, float2* half, float* dst, bool accumulate,
                         float scale, cudaStream_t st) {
  if (nd_plane_ok(t, ax)) return nd_plane_inverse(t, ax, planes, half, dst, accumulate, scale, st);
  const cudaError_t e = t.D > 1 ? nd_columns(true, t, ax.y, planes, half, st) : cudaSuccess;
  return e == cudaSuccess ? nd_rows_inverse(ax.x, planes, t.D * t.H, half, dst, accumulate, scale, st) : e;
}
// The last axis on its own, in place (the z or y lines of `planes` planes).
cudaError_t last_pass(bool inv, const NdTab& t, const NdAxes& ax, long planes, float2* half, cudaStream_t st) {
  NdTab flat = t;  // the last axis of a D x (H Wh) plane is the y axis of a one-plane world of H Wh columns
  flat.D = 1;
  flat.Wh = (int)(t.hcells / last_axis(t, ax).n);
  return nd_columns(inv, flat, last_axis(t, ax), planes, half, st);
}

// ------------------------------------------------------------------ adjoint
struct AdjArgs {
  int n_worlds, n_init, clip_mask;
  const float* s;      // [nw, C, cells] state entering the step
  const float* s_next;  // [nw, C, cells] state after the step, or null
  const float* u;      // [nw, K, cells] potentials of the step
  const float* lam;    // [nw, C, cells] dL/d(state after the step)
  float* lam_out;      // [nw, C, cells] direct part of dL/d(state before the step)
  float* a;            // [nw, K, cells] dL/du_k
  float* bf;           // [nw, C, cells] dL/df_c
  float* ff;           // [nw, C, cells] f_c
  float* s_copy;       // [nw, C, cells] copy of s, stored right after a
  const float* gf;     // [Ns, K, 2]
  const float* w;      // [Ns, C, K]
  const float* T;      // [Ns]
};

// growth(u) and its derivative in u (growth_functions.py); every family but
// identity is a function of (u - m) / s, so d/dm = -d/du and
// d/ds = -d/du (u - m) / s.
__device__ __forceinline__ float growth_du(int id, float u, float m, float s, float* g) {
  if (id == LGX_GF_GAUSSIAN || id == LGX_GF_GAUSSIAN_TARGET) {
    const float d = (u - m) / s;
    const float e = expf(-(d * d) / 2.f);
    const float amp = id == LGX_GF_GAUSSIAN ? 2.f : 1.f;
    *g = id == LGX_GF_GAUSSIAN ? 2.f * e - 1.f : e;
    return -amp * e * d / s;
  }
  if (id == LGX_GF_POLY_QUAD4) {
    const float d = u - m, c = 9.f * s * s;
    const float q = 1.f - d * d / c;
    if (q > 0.f) {
      const float q3 = q * q * q;
      *g = 2.f * q3 * q - 1.f;
      return 8.f * q3 * (-2.f * d / c);
    }
    *g = -1.f;
    return 0.f;
  }
  *g = growth_fn(id, u, m, s);
  if (id == LGX_GF_IDENTITY) return 1.f;
  if (id == LGX_GF_TRIANGLE) {  // growth_functions.py:234-243: slopes 2/s and -2/s
    if (u >= m - s && u < m) return 2.f / s;
    if (u >= m && u <= m + s) return -2.f / s;
  }
  return 0.f;  // step, staircase: piecewise constant
}

// Pointwise part of the reverse step, one block per (world, chunk of cells):
// the clip / state-function gradient, dL/df per channel, dL/dg per kernel
// (the weighted merge's transpose) and the growth derivative give
// a_k = dL/du_k; the entering state is copied beside a (both are
// transformed by the same passes).  With FK > 0 the model has exactly FK
// kernels and FC channels and the block also adds its parameter partials
// (those of nd_adj_param_kernel) into its slots of pacc.
template <int FK, int FC>
__global__ void __launch_bounds__(kNT) nd_adj_point_kernel(NdTab t, AdjArgs a, int pb, float* __restrict__ pacc) {
  constexpr bool kFused = FK > 0;
  depend_wait();
  a.lam = after_wait(a.lam);
  pacc = after_wait(pacc);
  const int C = kFused ? FC : t.C, K = kFused ? FK : t.K;
  const int w = blockIdx.x / pb, b = blockIdx.x % pb;
  const long chunk = (t.cells + pb - 1) / pb;
  const long c0 = (long)b * chunk, c1 = min(t.cells, c0 + chunk);
  const int sol = w / a.n_init;
  const float dt = 1.f / __ldg(a.T + sol);
  const float* gf = a.gf + (long)sol * 2 * K;
  const float* wt = a.w + (long)sol * C * K;
  constexpr int kAcc = kFused ? FK * (2 + FC) : 1;
  float acc[kAcc];
#pragma unroll
  for (int j = 0; j < kAcc; ++j) acc[j] = 0.f;
  for (long cell = c0 + threadIdx.x; cell < c1; cell += blockDim.x) {
    float f[kMaxChannels], bb[kMaxChannels], ws[kMaxChannels];
#pragma unroll
    for (int c = 0; c < kMaxChannels; ++c) {
      f[c] = 0.f;
      ws[c] = 0.f;
      bb[c] = 0.f;
    }
    for (int k = 0; k < K; ++k) {
      const float u = __ldg(a.u + ((long)w * K + k) * t.cells + cell);
      const float g = growth_fn(t.gf[k], u, __ldg(gf + 2 * k), __ldg(gf + 2 * k + 1));
#pragma unroll
      for (int c = 0; c < kMaxChannels; ++c) {
        if (c >= C) break;
        const float wk = __ldg(wt + c * K + k);
        ws[c] += wk;
        if (wk != 0.f) f[c] = fmaf(wk, g, f[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < kMaxChannels; ++c) {
      if (c >= C) break;
      if (t.mean) f[c] = f[c] / ws[c];
      const long off = ((long)w * C + c) * t.cells + cell;
      const float lam = __ldg(a.lam + off);
      const float sv = __ldg(a.s + off);
      a.s_copy[off] = sv;
      float dsds, dsdf;  // d state' / d state and d state' / d field (core.py:245-319)
      if (t.state_fn == LGX_STATE_V1) {
        // mask: the forward's clip was inactive where its output lies strictly inside (0, 1)
        const float n = a.s_next ? __ldg(a.s_next + off) : fmaf(dt, f[c], sv);
        const float cg = a.clip_mask ? ((n > 0.f && n < 1.f) ? 1.f : 0.f) : 1.f;  // mask or straight-through
        dsds = cg;
        dsdf = dt * cg;
      } else if (t.state_fn == LGX_STATE_V2) {
        dsds = 1.f - dt;
        dsdf = dt;
      } else {
        dsds = 1.f;
        dsdf = dt;
      }
      a.lam_out[off] = lam * dsds;
      bb[c] = lam * dsdf;
      a.bf[off] = bb[c];
      a.ff[off] = f[c];
    }
    for (int k = 0; k < K; ++k) {
      const int id = t.gf[k];
      const float u = __ldg(a.u + ((long)w * K + k) * t.cells + cell);
      const float m = __ldg(gf + 2 * k), sg = __ldg(gf + 2 * k + 1);
      float g;
      const float gu = growth_du(id, u, m, sg, &g);
      float dg = 0.f;  // dL/dg_k = sum_c dL/df_c * w_ck (/ sum_j w_cj in mean mode)
#pragma unroll
      for (int c = 0; c < kMaxChannels; ++c) {
        if (c >= C) break;
        const float wk = __ldg(wt + c * K + k);
        dg = fmaf(bb[c], t.mean ? wk / ws[c] : wk, dg);
      }
      const float ak = dg * gu;
      a.a[((long)w * K + k) * t.cells + cell] = ak;
      if constexpr (kFused) {
        if (k < FK) {
          float* pk = acc + k * (2 + FC);
          if (id != LGX_GF_IDENTITY) {
            pk[0] -= ak;
            pk[1] -= ak * (u - m) / sg;
          }
#pragma unroll
          for (int c = 0; c < FC; ++c) pk[2 + c] = fmaf(bb[c], t.mean ? (g - f[c]) / ws[c] : g, pk[2 + c]);
        }
      }
    }
  }
  if constexpr (kFused) {
    __shared__ float red[kNT / 32][kAcc];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < kAcc; ++j) acc[j] = warp_sum(acc[j]);
    if (lane == 0)
#pragma unroll
      for (int j = 0; j < kAcc; ++j) red[wid][j] = acc[j];
    __syncthreads();
    if (threadIdx.x < kAcc) {
      float v = 0.f;
      for (int i = 0; i < kNT / 32; ++i) v += red[i][threadIdx.x];
      const int k = threadIdx.x / (2 + FC), j = threadIdx.x % (2 + FC);
      pacc[(((long)w * FK + k) * pb + b) * (2 + FC) + j] += v;
    }
  }
}

// Per (world, kernel, chunk of cells): dL/dm_k = -sum a_k,
// dL/ds_k = -sum a_k (u_k - m) / s, dL/dw_ck = sum dL/df_c * (g_k - f_c) /
// sum_j w_cj (mean) or dL/df_c * g_k (sum), added into the block's own slot
// pacc[w, k, b] = {dm, ds, dw_0k .. dw_(C-1)k} (each block owns its slot
// across the reverse steps, so the sums are race-free and deterministic).
__global__ void __launch_bounds__(kNT) nd_adj_param_kernel(NdTab t, int n_init, int pb, const float* __restrict__ u,
                                                           const float* __restrict__ a, const float* __restrict__ bf,
                                                           const float* __restrict__ ff, const float* __restrict__ gfp,
                                                           const float* __restrict__ wts, float* __restrict__ pacc) {
  const int C = t.C, K = t.K;
  const int w = blockIdx.x / (K * pb), k = (blockIdx.x / pb) % K, b = blockIdx.x % pb;
  const long chunk = (t.cells + pb - 1) / pb;
  const long c0 = (long)b * chunk, c1 = min(t.cells, c0 + chunk);
  const int sol = w / n_init;
  const float m = __ldg(gfp + ((long)sol * K + k) * 2), s = __ldg(gfp + ((long)sol * K + k) * 2 + 1);
  const int id = t.gf[k];
  float wsum[kMaxChannels];
#pragma unroll
  for (int c = 0; c < kMaxChannels; ++c) {
    wsum[c] = 0.f;
    if (c < C)
      for (int j = 0; j < K; ++j) wsum[c] += __ldg(wts + ((long)sol * C + c) * K + j);
  }
  float dm = 0.f, ds = 0.f, dw[kMaxChannels];
#pragma unroll
  for (int c = 0; c < kMaxChannels; ++c) dw[c] = 0.f;
  for (long cell = c0 + threadIdx.x; cell < c1; cell += blockDim.x) {
    const float uu = __ldg(u + ((long)w * K + k) * t.cells + cell);
    const float ak = __ldg(a + ((long)w * K + k) * t.cells + cell);
    if (id != LGX_GF_IDENTITY) {
      dm -= ak;
      ds -= ak * (uu - m) / s;
    }
    const float g = growth_fn(id, uu, m, s);
#pragma unroll
    for (int c = 0; c < kMaxChannels; ++c) {
      if (c >= C) break;
      const long off = ((long)w * C + c) * t.cells + cell;
      const float b = __ldg(bf + off);
      dw[c] = fmaf(b, t.mean ? (g - __ldg(ff + off)) / wsum[c] : g, dw[c]);
    }
  }
  __shared__ float red[kNT / 32][2 + kMaxChannels];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  dm = warp_sum(dm);
  ds = warp_sum(ds);
#pragma unroll
  for (int c = 0; c < kMaxChannels; ++c) dw[c] = warp_sum(dw[c]);
  if (lane == 0) {
    red[wid][0] = dm;
    red[wid][1] = ds;
    for (int c = 0; c < kMaxChannels; ++c) red[wid][2 + c] = dw[c];
  }
  __syncthreads();
  if (threadIdx.x < 2 + C) {
    float v = 0.f;
    for (int i = 0; i < kNT / 32; ++i) v += red[i][threadIdx.x];
    pacc[(((long)w * K + k) * pb + b) * (2 + C) + threadIdx.x] += v;
  }
}

// per solution: grad_gf[s, k] += sum over its inits and chunks of
// pacc[w, k, b, 0:2], grad_w[s, c, k] += sum of pacc[w, k, b, 2 + c]
__global__ void nd_param_reduce_kernel(int n_sols, int n_init, int K, int C, int pb, const float* __restrict__ pacc,
                                       float* __restrict__ grad_gf, float* __restrict__ grad_w) {
  const int per = 2 * K + C * K;
  const long total = (long)n_sols * per;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int sol = (int)(i / per), j = (int)(i % per);
    const int k = j < 2 * K ? j / 2 : (j - 2 * K) % K;
    const int slot = j < 2 * K ? j % 2 : 2 + (j - 2 * K) / K;
    float v = 0.f;
    for (int n = 0; n < n_init; ++n)
      for (int b = 0; b < pb; ++b) v += pacc[((((long)sol * n_init + n) * K + k) * pb + b) * (2 + C) + slot];
    if (j < 2 * K) grad_gf[(long)sol * 2 * K + j] += v;
    else grad_w[(long)sol * C * K + (j - 2 * K)] += v;
  }
}

// gsum[s, k] = sum over the inits of solution s of gk[w, k]
__global__ void nd_sum_inits_kernel(long per_sol, int n_sols, int n_init, const float2* __restrict__ gk,
                                    float2* __restrict__ gsum) {
  const long total = (long)n_sols * per_sol;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int sol = (int)(i / per_sol);
    const long j = i - (long)sol * per_sol;
    float2 v = make_float2(0.f, 0.f);
    for (int n = 0; n < n_init; ++n) v = cadd(v, gk[((long)sol * n_init + n) * per_sol + j]);
    gsum[i] = v;
  }
}

}  // namespace

// ---------------------------------------------------------------------- API
bool nd_side_ok(int n) { return transform_len(n) > 0; }

int nd_max_side() { return kNdMaxN; }

bool nd_supported(const Model& m) {
  if (m.nb_dims != 2 && m.nb_dims != 3) return false;
  if (m.C > kMaxChannels || m.K > kMaxKernels) return false;
  for (int i = 0; i < m.nb_dims; ++i)
    if (!nd_side_ok(m.world[i])) return false;
  return true;
}

namespace {

// chunks of cells per world of the adjoint's pointwise kernel, and per
// (world, kernel) of its parameter reduction: 16 cells per thread, or more
// blocks when the batch is too small to fill the GPU (at least one cell per
// thread, at most 256 blocks)
int nd_param_blocks(const Model& m, long n_worlds) {
  const long by_cells = (m.cells + (long)kNT * 16 - 1) / ((long)kNT * 16);
  const long fill = (kFillBlocks + n_worlds - 1) / std::max(1L, n_worlds);
  const long useful = (m.cells + kNT - 1) / kNT;
  return (int)std::max(1L, std::min<long>(256, std::min(useful, std::max(by_cells, fill))));
}

// Workspace of the steps of one call: tables, S, P, block partials, and the
// weighted fields where they do not fit shared memory.
struct StepLayout {
  size_t tables, S, P, partial, field, end;
};
StepLayout step_layout(const Model& m, int n_worlds) {
  const NdTab t = make_tab(m, 0);
  const NdAxes ax = make_axes(m.D, m.H, m.W, nullptr);
  const size_t nw = (size_t)n_worlds;
  long field = 0;
  int bpw;
  if (nd_plane_ok(t, ax)) {
    bool global;
    bpw = nd_plane_epi_blocks(t, ax, (long)nw, &global);
    if (global) field = (long)m.D * ((m.H + 1) / 2) * m.W;
  } else {
    bpw = nd_rows_epi_blocks(t, ax.x, (long)nw, &field);
  }
  StepLayout L;
  size_t off = 0;
  L.tables = off;
  off += table_bytes(m.D, m.H, m.W);
  L.S = off;
  off += al256(nw * m.C * t.hcells * sizeof(float2));
  L.P = off;
  off += al256(nw * m.K * t.hcells * sizeof(float2));
  L.partial = off;
  off += al256(nw * bpw * raw_stride(m.C) * sizeof(float));
  L.field = off;
  off += al256(nw * m.C * field * sizeof(float2));
  L.end = off;
  return L;
}

}  // namespace

size_t nd_step_workspace_bytes(const Model& m, int n_worlds) { return step_layout(m, n_worlds).end; }

cudaError_t launch_nd_begin(const Model& m, void* ws, cudaStream_t st) {
  return launch_tables(make_axes(m.D, m.H, m.W, ws), m.D, st);
}

cudaError_t launch_nd_step(const NdStep& s, cudaStream_t st) {
  const Model& m = *s.m;
  const NdTab t = make_tab(m, s.dt_mode);
  const StepLayout L = step_layout(m, s.n_worlds);
  char* base = static_cast<char*>(s.ws);
  const NdAxes ax = make_axes(m.D, m.H, m.W, base + L.tables);
  const long nw = s.n_worlds;
  float2* S = reinterpret_cast<float2*>(base + L.S);
  float2* P = reinterpret_cast<float2*>(base + L.P);
  const bool plane = nd_plane_ok(t, ax);
  cudaError_t e;
  if (!s.spec_ready && (e = forward_head(t, ax, nw * m.C, s.state, S, st)) != cudaSuccess) return e;
  ConvArgs ca{};
  ca.n_init = s.n_init;
  ca.kh = s.k_half;
  ca.kh_sol_stride = s.k_sol_stride;
  ca.S = S;
  ca.P = P;
  if ((e = nd_convolve(false, t, last_axis(t, ax), nw, ca, st)) != cudaSuccess) return e;
  const bool columns = t.D > 1 && !plane;  // the y transforms are passes of their own
  if (columns && (e = nd_columns(true, t, ax.y, nw * m.K, P, st)) != cudaSuccess) return e;
  EpiArgs a{};
  a.n_worlds = s.n_worlds;
  a.n_init = s.n_init;
  a.state = s.state;
  a.state_out = s.state_out;
  a.P = P;
  a.S = s.emit_spec ? S : nullptr;
  a.F = reinterpret_cast<float*>(base + L.field);
  a.pot_out = s.pot_out;
  a.gf = s.gf;
  a.gf_sol_stride = s.gf_sol_stride;
  a.w = s.w;
  a.w_sol_stride = s.w_sol_stride;
  a.dt = s.dt;
  a.field_out = s.field_out;
  a.state_copy = s.state_copy;
  a.shift = s.shift;
  a.done = s.done;
  a.partial = reinterpret_cast<float*>(base + L.partial);
  a.raw = s.raw;
  a.raw_sol_stride = s.raw_sol_stride;
  a.raw_init_stride = s.raw_world_stride;
  a.scale = 1.f / (float)m.cells;
  e = plane ? nd_plane_epilogue(t, ax, a, st) : nd_rows_epilogue(t, ax.x, a, st);
  if (e == cudaSuccess && columns && s.emit_spec) e = nd_columns(false, t, ax.y, nw * m.C, S, st);
  return e;
}

namespace {
struct AdjLayout {
  size_t tables, A, Q, ar, bf, ff, lam, pacc, end;
};
AdjLayout adj_layout(const Model& m, int n_sols, int n_init) {
  const NdTab t = make_tab(m, 2);
  const size_t nw = (size_t)n_sols * n_init, cells = (size_t)m.cells, KC = (size_t)(m.K + m.C);
  AdjLayout L;
  size_t off = 0;
  L.tables = off;
  off += table_bytes(m.D, m.H, m.W);
  L.A = off;  // spectra of the K planes of a, then of the C planes of the state
  off += al256(nw * KC * t.hcells * sizeof(float2));
  L.Q = off;
  off += al256(nw * m.C * t.hcells * sizeof(float2));
  L.ar = off;  // a, then the state copy: one real input for the head passes
  off += al256(nw * KC * cells * sizeof(float));
  L.bf = off;
  off += al256(nw * m.C * cells * sizeof(float));
  L.ff = off;
  off += al256(nw * m.C * cells * sizeof(float));
  L.lam = off;
  off += al256(nw * m.C * cells * sizeof(float));
  L.pacc = off;
  off += al256(nw * m.K * nd_param_blocks(m, (long)nw) * (2 + m.C) * sizeof(float));
  L.end = off;
  return L;
}
}  // namespace

size_t nd_adjoint_workspace_bytes(const Model& m, int n_sols, int n_init) { return adj_layout(m, n_sols, n_init).end; }

// A whole complex plane a (world, kernel), the size the interface has answered
// from the start; the half spectra that the adjoint accumulates fill the front.
size_t nd_kernel_grad_acc_bytes(const Model& m, int n_sols, int n_init) {
  return (size_t)n_sols * n_init * m.K * m.cells * sizeof(float2);
}

cudaError_t launch_nd_adjoint(const Model& m, const NdAdjoint& j, void* ws, cudaStream_t st) {
  const NdTab t = make_tab(m, 2);
  const AdjLayout L = adj_layout(m, j.n_sols, j.n_init);
  const int nw = j.n_sols * j.n_init;
  const size_t cells = (size_t)m.cells;
  char* base = static_cast<char*>(ws);
  const NdAxes ax = make_axes(m.D, m.H, m.W, base + L.tables);
  const size_t KC = (size_t)(m.K + m.C);
  float2* A = reinterpret_cast<float2*>(base + L.A);
  float2* S = A + (size_t)nw * m.K * t.hcells;
  float2* Q = reinterpret_cast<float2*>(base + L.Q);
  float* ar = reinterpret_cast<float*>(base + L.ar);
  float* bf = reinterpret_cast<float*>(base + L.bf);
  float* ff = reinterpret_cast<float*>(base + L.ff);
  float* lam_tmp = reinterpret_cast<float*>(base + L.lam);
  float* pacc = reinterpret_cast<float*>(base + L.pacc);
  const int pb = nd_param_blocks(m, nw);
  const bool fused = m.K == 1 && m.C == 1;  // parameter partials inside the pointwise kernel
  cudaError_t e = launch_tables(ax, m.D, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(pacc, 0, (size_t)nw * m.K * pb * (2 + m.C) * sizeof(float), st);
  if (e != cudaSuccess) return e;
  const size_t plane_c = (size_t)m.C * cells, plane_k = (size_t)m.K * cells;
  const float* lam_in = j.lambda_in;
  for (int step = j.steps - 1; step >= 0; --step) {
    float* lam_out = (step % 2 == 0) ? j.lambda_out : lam_tmp;  // step 0 lands in lambda_out
    AdjArgs a;
    a.n_worlds = nw;
    a.n_init = j.n_init;
    a.clip_mask = j.clip_mask;
    a.s = j.traj_cells + (size_t)step * nw * plane_c;
    a.s_next = step + 1 < j.steps ? a.s + (size_t)nw * plane_c : j.cells_after;
    a.u = j.traj_potential + (size_t)step * nw * plane_k;
    a.lam = lam_in;
    a.lam_out = lam_out;
    a.a = ar;
    a.bf = bf;
    a.ff = ff;
    a.gf = j.gf_params;
    a.w = j.weights;
    a.T = j.T;
    a.s_copy = ar + (size_t)nw * m.K * cells;
    if (fused) {
      e = launch_dependent(nd_adj_point_kernel<1, 1>, (unsigned)(nw * pb), kNT, 0, st, t, a, pb, pacc);
      if (e != cudaSuccess) return e;
    } else {
      e = launch_dependent(nd_adj_point_kernel<0, 0>, (unsigned)(nw * pb), kNT, 0, st, t, a, pb, pacc);
      if (e != cudaSuccess) return e;
      nd_adj_param_kernel<<<(unsigned)(nw * m.K * pb), kNT, 0, st>>>(t, j.n_init, pb, a.u, ar, bf, ff, j.gf_params,
                                                                       j.weights, pacc);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if ((e = forward_head(t, ax, (long)nw * KC, ar, A, st)) != cudaSuccess) return e;
    ConvArgs ca{};
    ca.n_init = j.n_init;
    ca.kh = j.k_half;
    ca.kh_sol_stride = (long)m.C * m.max_k * t.hcells;
    ca.S = S;
    ca.A = A;
    ca.gk = j.gk;
    ca.Q = Q;
    if ((e = nd_convolve(true, t, last_axis(t, ax), nw, ca, st)) != cudaSuccess) return e;
    if ((e = inverse_tail(t, ax, (long)nw * m.C, Q, lam_out, true, 1.f / (float)m.cells, st)) != cudaSuccess) return e;
    lam_in = lam_out;
  }
  nd_param_reduce_kernel<<<grid_for((long)j.n_sols * (2 * m.K + m.C * m.K)), kNT, 0, st>>>(
      j.n_sols, j.n_init, m.K, m.C, pb, pacc, j.grad_gf, j.grad_weights);
  return cudaGetLastError();
}

size_t nd_kernel_grad_workspace_bytes(const Model& m, int n_sols) {
  return table_bytes(m.D, m.H, m.W) + al256((size_t)n_sols * m.K * m.D * m.H * (m.W / 2 + 1) * sizeof(float2));
}

cudaError_t launch_nd_kernel_grad(const Model& m, int n_sols, int n_init, const float2* gk, float* out, void* ws,
                                  cudaStream_t st) {
  const NdTab t = make_tab(m, 2);
  const NdAxes ax = make_axes(m.D, m.H, m.W, ws);
  float2* gsum = reinterpret_cast<float2*>(static_cast<char*>(ws) + table_bytes(m.D, m.H, m.W));
  cudaError_t e = launch_tables(ax, m.D, st);
  if (e != cudaSuccess) return e;
  const long per = (long)m.K * t.hcells, planes = (long)n_sols * m.K;
  nd_sum_inits_kernel<<<grid_for((long)n_sols * per), kNT, 0, st>>>(per, n_sols, n_init, gk, gsum);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // dL/dk = Re(IFFT(sum_t A_t conj(S_t))) = unnormalised inverse / cells
  if ((e = last_pass(true, t, ax, planes, gsum, st)) != cudaSuccess) return e;
  return inverse_tail(t, ax, planes, gsum, out, false, 1.f / (float)m.cells, st);
}

size_t nd_spectrum_workspace_bytes(int nb_dims, const int* world, int planes) {
  (void)planes;
  return table_bytes(nb_dims == 3 ? world[0] : 1, world[nb_dims - 2], world[nb_dims - 1]);
}

cudaError_t launch_nd_spectrum(int nb_dims, const int* world, int planes, const float* k_real, float2* k_half,
                               void* ws, cudaStream_t st) {
  Model m;
  m.nb_dims = nb_dims;
  m.D = nb_dims == 3 ? world[0] : 1;
  m.H = world[nb_dims - 2];
  m.W = world[nb_dims - 1];
  m.cells = (long)m.D * m.H * m.W;
  m.C = m.K = m.max_k = 1;
  m.mean = 1;
  m.state_fn = 0;
  m.cin[0] = m.slot[0] = m.gf[0] = 0;
  const NdTab t = make_tab(m, 0);
  const NdAxes ax = make_axes(m.D, m.H, m.W, ws);
  cudaError_t e = launch_tables(ax, m.D, st);
  if (e == cudaSuccess) e = forward_head(t, ax, planes, k_real, k_half, st);
  return e == cudaSuccess ? last_pass(false, t, ax, planes, k_half, st) : e;
}

}  // namespace lgx
