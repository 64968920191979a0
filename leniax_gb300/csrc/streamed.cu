// Streamed Lenia step for any channel/kernel topology (2D, square power-of-two
// worlds of side 32..512): the spectra of a step travel through HBM/L2
// between its kernels.
//
//   row_fwd  : per (world, channel, packed row) N-point FFT of rows (2r, 2r+1)
//              packed as one complex row -> spec[n][c][r][.] in the
//              pair-adjacent layout (pa_pos, fft.cuh); first step only
//   col_conv : per (world, channel, block of column pairs) the block's column
//              tile arrives by TMA (2D tensor copies, 128-byte swizzle); per
//              pair: unpack + N-point FFT, then for every kernel reading that
//              channel: x prepared spectrum (column-major planes, so a
//              transform's lanes read consecutive ky; bulk-staged up to
//              N = 128), inverse FFT -> prod[n][k] (same pair-adjacent
//              layout), written back through the tile by TMA stores
//   row_inv  : per (world, block of packed rows) the block's rows of every
//              kernel's product plane arrive by bulk copies into a staging
//              ring (the next kernel's rows land while this kernel's are
//              transformed), each channel's state rows by one bulk copy;
//              inverse row FFTs -> potential, growth, weighted field in
//              registers (core.py:163-242), state update (core.py:245-319),
//              per-block raw statistics moments, and the next step's forward
//              row FFT of the new rows
//   reduce   : per world: block moments -> raw moments of the step, carried
//              torus shift update (statistics.py:117-119)
//
// This is leniax core.update with get_potential_fft (core.py:52-102), the
// true-kernel selection (tc_indices, core.py:97-98) being the (c_in, slot)
// table of the plan.
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "engine.h"
#include "fft.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace lgx {

namespace {

constexpr int kThreads = 256;  // row_fwd blocks

struct KTab {  // per-plan kernel table, passed by value
  int C, K, max_k, mean, state_fn, dt_mode;
  int cin[kMaxKernels];
  int slot[kMaxKernels];
  int gf[kMaxKernels];
};

template <int N>
struct SCfg;
template <>
struct SCfg<32> { static constexpr int G = 4; };
template <>
struct SCfg<64> { static constexpr int G = 4; };
template <>
struct SCfg<128> { static constexpr int G = 8; };
template <>
struct SCfg<256> { static constexpr int G = 16; };  // P = 16 points per lane (Q == 1 transforms)
template <>
struct SCfg<512> { static constexpr int G = 16; };

template <int N>
__device__ __forceinline__ float2* init_tw(float2* sm) {
  using GE = Geo<N, SCfg<N>::G>;
  init_twiddles<GE>(sm, sm + N, sm + 2 * N, threadIdx.x, blockDim.x);
  return sm + 3 * N;
}

// ------------------------------------------------------------------ row_fwd
template <int N>
__global__ void __launch_bounds__(kThreads) row_fwd_kernel(int n_worlds, int C, const float* __restrict__ state,
                                                           float2* __restrict__ spec) {
  constexpr int G = SCfg<N>::G;
  using GE = Geo<N, G>;
  constexpr int P = GE::P, Q = GE::Q, GPB = kThreads / G;  // groups per block
  constexpr int BPP = (N / 2 + GPB - 1) / GPB;             // blocks per plane
  extern __shared__ __align__(16) float2 sm[];
  depend_trigger();  // an ordinary launch: all before it is complete
  float2* scr = init_tw<N>(sm);
  __syncthreads();
  const int plane = blockIdx.x / BPP;  // n*C + c
  if (plane >= n_worlds * C) return;
  const int grp = threadIdx.x / G, t = threadIdx.x % G, lane = threadIdx.x & 31;
  const int r = (blockIdx.x % BPP) * GPB + grp;
  if (r >= N / 2) return;  // whole groups exit together (never used with N/2 % GPB != 0 and partial warps)
  const unsigned gmask = ((1u << G) - 1u) << (lane & ~(G - 1));
  const float* src = state + (size_t)plane * N * N;
  float2 v[P];
#pragma unroll
  for (int n2 = 0; n2 < P; ++n2)
    v[n2] = make_float2(__ldg(src + (2 * r) * N + t + G * n2), __ldg(src + (2 * r + 1) * N + t + G * n2));
  float2 u[Q][G];
  fft_standard<GE, false, false>(v, u, scr + grp * GE::SCR, sm, t, gmask);
  float2* dst = spec + ((size_t)plane * (N / 2) + r) * N;
#pragma unroll
  for (int q = 0; q < Q; ++q)
#pragma unroll
    for (int k1 = 0; k1 < G; ++k1) dst[pa_pos<N>(t + G * q + P * k1)] = u[q][k1];
}

// ----------------------------------------------------------------- col_conv
template <int N>
struct ColCfg {
  static constexpr int G = SCfg<N>::G;
  static constexpr int T = ((N / 2) * G < 128) ? (N / 2) * G : 128;  // threads per block
  static constexpr int GPB = T / G;                // column pairs per block (one per group)
  static constexpr int BPP = (N / 2) / GPB;        // blocks per plane
  static constexpr int BOXES = GPB / 8;            // TMA boxes: 8 pairs (128 bytes) x N/2 rows
  static constexpr int BOX_BYTES = (N / 2) * 128;
  static constexpr int TILE_BYTES = BOXES * BOX_BYTES;
  // kernel spectrum columns staged by bulk copy (GPB columns + the Nyquist
  // column for the block holding pair 0) up to N = 128; from N = 256 on the
  // staging buffer would cost a resident block per SM, which measured slower
  // than the (coalesced, column-major) direct loads
  static constexpr bool KSTAGE = N <= 128;
  static constexpr int KB_BYTES = KSTAGE ? (GPB + 1) * N * 8 : 0;
  static_assert(GPB % 8 == 0 && (N / 2) % GPB == 0, "column tile");
};

template <int N>
constexpr size_t col_conv_smem() {
  using CC = ColCfg<N>;
  using GE = Geo<N, CC::G>;
  // 1024 bytes of alignment slack for the swizzled tile, tile (the column
  // input, then the output staging), staged kernel columns, twiddles, group
  // scratch, DC/Nyquist mirror, two mbarriers
  return 1024 + (size_t)CC::TILE_BYTES + (size_t)CC::KB_BYTES + (size_t)3 * N * sizeof(float2) +
         (size_t)CC::GPB * GE::SCR * sizeof(float2) + (size_t)N * sizeof(float2) + 16;
}

// The n-th kernel after k (or K) reading channel ch.
__device__ __forceinline__ int next_kernel(const KTab& tab, int k, int ch, int n) {
  for (++k; k < tab.K; ++k)
    if (tab.cin[k] == ch && --n == 0) break;
  return k;
}

// One block: GPB column pairs of one (world, channel) plane.  The column tile
// arrives by TMA; per kernel reading the channel, the kernel's GPB spectrum
// columns arrive by bulk copy (issued one kernel ahead), and the product
// columns leave through the same swizzled tile by TMA stores, so the kernel's
// global traffic bypasses the load/store pipe.  gridDim.y blocks share a
// tile's kernels (block y takes every gridDim.y-th of them, each repeating the
// forward transform): see col_conv_split.
template <int N>
__global__ void __launch_bounds__(ColCfg<N>::T) col_conv_kernel(const __grid_constant__ CUtensorMap spec_map,
                                                               const __grid_constant__ CUtensorMap prod_map,
                                                               int n_worlds, int n_init, KTab tab,
                                                               const float2* __restrict__ kp, long kp_sol_stride,
                                                               int* __restrict__ status) {
  using CC = ColCfg<N>;
  constexpr int G = CC::G, GPB = CC::GPB, BPP = CC::BPP;
  using GE = Geo<N, G>;
  constexpr int P = GE::P, Q = GE::Q;
  constexpr int KPITCH = N / 2 + 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  unsigned char* tile = smraw + ((1024u - (smem_u32(smraw) & 1023u)) & 1023u);
  float2* kb = reinterpret_cast<float2*>(tile + CC::TILE_BYTES);  // [GPB + 1][N] kernel columns
  float2* sm = reinterpret_cast<float2*>(tile + CC::TILE_BYTES + CC::KB_BYTES);
  float2* scr = sm + 3 * N;
  float2* mirror = scr + GPB * GE::SCR;
  uint64_t* bar = reinterpret_cast<uint64_t*>(mirror + N);  // [0]: column tile, [1]: kernel columns
  const int plane = blockIdx.x / BPP;  // n*C + c
  if (plane >= n_worlds * tab.C) return;
  const int j0 = (blockIdx.x % BPP) * GPB;
  const int n = plane / tab.C, ch = plane % tab.C;
  const int sol = n / n_init;
  auto kplane = [&](int k) {
    return kp + sol * kp_sol_stride + ((size_t)(ch * tab.max_k + tab.slot[k]) * N) * KPITCH;
  };
  // kernel k's columns j0 .. j0 + GPB - 1 (+ column N/2 for pair 0) -> kb
  auto issue_kernel = [&](int k) {
    const unsigned main = GPB * N * sizeof(float2), nyq = j0 == 0 ? N * sizeof(float2) : 0u;
    mbar_arrive_expect_tx(&bar[1], main + nyq);
    const float2* kk = kplane(k);
    bulk_load(kb, kk + (size_t)j0 * N, main, &bar[1]);
    if (nyq) bulk_load(kb + GPB * N, kk + (size_t)(N / 2) * N, nyq, &bar[1]);
  };
  const int ks = gridDim.y;
  const int k_first = next_kernel(tab, -1, ch, blockIdx.y + 1);
  if (k_first >= tab.K) return;
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_proxy_async();
    if (CC::KSTAGE) issue_kernel(k_first);
  }
  init_twiddles<GE>(sm, sm + N, sm + 2 * N, threadIdx.x, blockDim.x);
  depend_wait();
  depend_trigger();
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(&bar[0], CC::TILE_BYTES);
    for (int b = 0; b < CC::BOXES; ++b)
      tma_load_2d(tile + b * CC::BOX_BYTES, &spec_map, (j0 + 8 * b) * 4, plane * (N / 2), &bar[0]);
  }
  __syncthreads();
  if (__syncthreads_or(!mbar_wait(&bar[0], 0))) {  // the tile never landed: record, drain, leave
    if (threadIdx.x == 0) {
      if (status) atomicExch(status, kStatusCopyTimeout);
      mbar_wait(&bar[0], 0);
      if (CC::KSTAGE) mbar_wait(&bar[1], 0);
    }
    return;
  }
  const int grp = threadIdx.x / G, t = threadIdx.x % G, lane = threadIdx.x & 31;
  const int j = j0 + grp;  // column pair (j, N-j); j == 0 carries (0, N/2)
  const unsigned gmask = ((1u << G) - 1u) << (lane & ~(G - 1));
  float2* cs = scr + grp * GE::SCR;
  unsigned char* tb = tile + (grp >> 3) * CC::BOX_BYTES;
  const int chunk = grp & 7;

  float2 v[Q][G];
  if constexpr (Q == 1) {
    // lane t carries the unpacked rows n = t + P*n2: packed row n >> 1, the
    // even row's value for even n, the odd row's for odd n (lanes 2m, 2m+1
    // read the same 16-byte pair)
#pragma unroll
    for (int n2 = 0; n2 < G; ++n2) {
      const int r = t + P * n2;
      const float4 q = *reinterpret_cast<const float4*>(tb + swz128(r >> 1, chunk));
      if (j != 0) v[0][n2] = (r & 1) ? make_float2(q.y + q.w, q.z - q.x) : make_float2(q.x + q.z, q.y - q.w);
      else v[0][n2] = (r & 1) ? make_float2(q.y, q.w) : make_float2(q.x, q.z);
    }
  } else {
#pragma unroll
    for (int jp = 0; jp < Q / 2; ++jp) {
      const int m = t + G * jp;
#pragma unroll
      for (int n2 = 0; n2 < G; ++n2) {
        const int r = m + (P / 2) * n2;
        const float4 q = *reinterpret_cast<const float4*>(tb + swz128(r, chunk));
        if (j != 0) {
          v[2 * jp][n2] = make_float2(q.x + q.z, q.y - q.w);      // 2 X[2r][j]
          v[2 * jp + 1][n2] = make_float2(q.y + q.w, q.z - q.x);  // 2 X[2r+1][j]
        } else {
          v[2 * jp][n2] = make_float2(q.x, q.z);  // X[2r][0] + i X[2r][N/2]
          v[2 * jp + 1][n2] = make_float2(q.y, q.w);
        }
      }
    }
  }
  float2 w0[P];
  fft_mirrored<GE, false, false>(v, w0, cs, sm + N, t, gmask);
  // the packed DC / Nyquist column keeps its spectrum in the block's mirror
  // buffer: Q[ky] needs A[-ky] for every kernel
  if (j == 0) {
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) mirror[t + G * k1] = w0[k1];
    __syncwarp(gmask);
  }
  int it = 0;
  for (int k = k_first; k < tab.K; k = next_kernel(tab, k, ch, ks), ++it) {
    bool ok = true;
    if constexpr (CC::KSTAGE) ok = mbar_wait(&bar[1], it & 1);
    float2 w[P];
    if (ok) {
      const float2* kc = CC::KSTAGE ? kb + grp * N : kplane(k) + (size_t)j * N;
      const float2* kn = CC::KSTAGE ? kb + GPB * N : kplane(k) + (size_t)(N / 2) * N;
      if (j != 0) {
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) w[k1] = cmul(w0[k1], kc[t + G * k1]);
      } else {
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
          const int ky = t + G * k1;
          const float2 A = kc[ky], B = kn[ky];
          w[k1] = cadd(cmul(w0[k1], A), cmul(conjf2(mirror[(N - ky) & (N - 1)]), B));
        }
      }
    }
    // past this barrier: kb is free for the next kernel, and the previous
    // product's store has read the tile
    if (threadIdx.x == 0) bulk_wait_read_all();
    if (__syncthreads_or(!ok)) {  // a kernel column copy never landed
      if (threadIdx.x == 0) {
        if (status) atomicExch(status, kStatusCopyTimeout);
        mbar_wait(&bar[1], it & 1);
        bulk_wait_all();
      }
      return;
    }
    const int k_next = next_kernel(tab, k, ch, ks);
    if (CC::KSTAGE && threadIdx.x == 0 && k_next < tab.K) issue_kernel(k_next);
    float2 u[Q][G];
    if constexpr (Q == 1) {
      // unpacked row r = t + P*k1 -> its half of pair j of packed row r >> 1
      fft_standard<GE, true, false>(w, u, cs, sm, t, gmask);
#pragma unroll
      for (int k1 = 0; k1 < G; ++k1) {
        const int r = t + P * k1;
        *reinterpret_cast<float2*>(tb + swz128(r >> 1, chunk) + (r & 1) * 8) = u[0][k1];
      }
    } else {
      fft_standard<GE, true, true>(w, u, cs, sm, t, gmask);
#pragma unroll
      for (int a = 0; a < Q / 2; ++a) {
        const int m = t + G * a;
#pragma unroll
        for (int k1 = 0; k1 < G; ++k1) {
          const int r = m + (P / 2) * k1;
          *reinterpret_cast<float4*>(tb + swz128(r, chunk)) =
              make_float4(u[2 * a][k1].x, u[2 * a][k1].y, u[2 * a + 1][k1].x, u[2 * a + 1][k1].y);
        }
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int b = 0; b < CC::BOXES; ++b)
        tma_store_2d(&prod_map, (j0 + 8 * b) * 4, (n * tab.K + k) * (N / 2), tile + b * CC::BOX_BYTES);
      bulk_commit();
    }
  }
  if (threadIdx.x == 0) bulk_wait_all();
}

// Q == 1: lane t needs Z[k], k = t + P*n2: one pair load each (k < N/2 for n2 < G/2)
template <class GE>
__device__ __forceinline__ void unpack_row_pair_q1(const float2* row, float2 (&v)[GE::Q][GE::G], int t) {
  constexpr int N = GE::N, G = GE::G, P = GE::P;
  const float4* p4 = reinterpret_cast<const float4*>(row);
#pragma unroll
  for (int n2 = 0; n2 < G; ++n2) {
    const int k = t + P * n2;
    if (n2 < G / 2) {
      const float4 q = p4[k];  // k == 0: pair 0 = (DC, Nyquist)
      v[0][n2] = k == 0 ? make_float2(q.x, q.z) : make_float2(q.x - q.w, q.y + q.z);
    } else {
      const float4 q = p4[k == N / 2 ? 0 : N - k];
      v[0][n2] = k == N / 2 ? make_float2(q.y, q.w) : make_float2(q.x + q.w, q.z - q.y);
    }
  }
}

// ------------------------------------------------------------------ row_inv
// Block = GPB groups = GPB packed rows of one world.  Work items are the
// (output channel, kernel) pairs with a nonzero weight, channel by channel,
// then the kernels that feed no channel (their potentials still count in
// potential_volume).  A warp's product rows of item i are bulk-copied into its
// buffer i & 1 (row pitch N + G) while item i-1 is transformed; after
// unpacking its row, a group reuses that row as its FFT exchange scratch.  The weighted
// field of the current channel stays in registers (2*P values per thread); a
// kernel feeding several channels is transformed once per channel, its
// potential counted (and written) at the first.
template <int N>
struct RowInvCfg {
  static constexpr int G = SCfg<N>::G;
  static constexpr int T = ((N / 2) * G < 128) ? (N / 2) * G : 128;  // threads per block
  static constexpr int GPB = T / G;
  static constexpr int BPW = (N / 2) / GPB;  // blocks per world
  static constexpr int WROWS = 32 / G;       // packed rows per warp
  static constexpr int ROWP = N + G;         // staged row pitch (float2) == Geo<N, G>::SCR
  static constexpr int BUF = WROWS * ROWP;   // float2 per warp and ring slot
  static constexpr int NBUF = 2;             // staging ring depth (items in flight: NBUF - 1)
  static constexpr int SSTP = 2 * N + 16;    // staged state rows (2r, 2r+1) pitch per group (floats)
  static constexpr int TABS = Geo<N, G>::Q == 1 ? 1 : 2;  // twiddle tables: std, rowi (the same one when Q == 1)
  // resident blocks an SM asked of the compiler: 128 registers a thread and
  // the 56 KB a block that four of them may have (a lane of 512^2 holds 32
  // points and keeps what it needs).  Issue slots were 46% busy with three
  // blocks and block barriers between the items; 8-step rollouts of 3 x 15
  // kernels, us before -> now: 256 worlds of 256^2 5628 -> 5408, 128 of 128^2
  // 1268 -> 1030, 2048 of 64^2 3744 -> 3333; one kernel, 64 of 256^2 551 -> 500.
  // Three blocks without the block barriers: 5488, 1212, 3407, 537.
  static constexpr int MINB = N == 512 ? 1 : 512 / T;
};

// item word: bit 16 = count the potential, bits 8..15 = output channel + 1 (0: none), bits 0..7 = kernel
__device__ __forceinline__ int item_k(int it) { return it & 255; }
__device__ __forceinline__ int item_co(int it) { return ((it >> 8) & 255) - 1; }
__device__ __forceinline__ bool item_count(int it) { return (it >> 16) & 1; }

template <int N>
size_t row_inv_smem(int C, int K) {
  using RC = RowInvCfg<N>;
  return (size_t)(RC::T / 32) * RC::NBUF * RC::BUF * sizeof(float2) + (size_t)RC::GPB * RC::SSTP * sizeof(float) +
         (size_t)RC::TABS * N * sizeof(float2) +
         (size_t)(RC::T / 32) * (RAW_CM + kMaxChannels) * sizeof(float) + 16 * sizeof(uint64_t) +
         (size_t)kMaxChannels * sizeof(float) + (size_t)(C * K + K + 1) * sizeof(int) +
         (size_t)(C * K + K + 1) * sizeof(float4) + (size_t)(C * K + 2 * K) * sizeof(float);
}

template <int N, int GF>
__global__ void __launch_bounds__(RowInvCfg<N>::T, RowInvCfg<N>::MINB) row_inv_kernel(
    int n_worlds, int n_init, KTab tab, const float2* __restrict__ prod, const float* __restrict__ gfp,
    long gf_sol_stride, const float* __restrict__ wts, long w_sol_stride, const float* __restrict__ dtp,
    const float* __restrict__ state, float* __restrict__ state_out, float* __restrict__ field_out,
    float* __restrict__ pot_out, const int* __restrict__ shift, float* __restrict__ partial, int* __restrict__ status,
    float2* __restrict__ spec_next) {
  using RC = RowInvCfg<N>;
  constexpr int G = RC::G, GPB = RC::GPB, BPW = RC::BPW, ROWP = RC::ROWP, NBUF = RC::NBUF;
  using GE = Geo<N, G>;
  constexpr int P = GE::P, Q = GE::Q;
  constexpr int RAWS_MAX = RAW_CM + kMaxChannels;
  constexpr int NWARPS = RC::T / 32;
  static_assert(ROWP == GE::SCR, "a staged row doubles as the group's FFT scratch");
  extern __shared__ __align__(16) float2 sm[];
  static_assert(NWARPS * (NBUF + 1) <= 16, "mbarriers reserved");
  float* sst = reinterpret_cast<float*>(sm + NWARPS * NBUF * RC::BUF);  // past the rings: [GPB][SSTP] state rows
  float2* tw = reinterpret_cast<float2*>(sst + GPB * RC::SSTP);  // twiddle tables
  float2* tw_rowi = tw + (RC::TABS - 1) * N;
  float* red = reinterpret_cast<float*>(tw + RC::TABS * N);  // [warps][RAWS_MAX]
  uint64_t* bars_all = reinterpret_cast<uint64_t*>(red + NWARPS * RAWS_MAX);  // [warps][ring, state] (16 reserved)
  float* wsum_s = reinterpret_cast<float*>(bars_all + 16);  // [kMaxChannels]
  float4* ipar = reinterpret_cast<float4*>(wsum_s + kMaxChannels);  // [C*K + K + 1] per item: weight, m, s, a
  __shared__ int s_nitems;

  const int n = blockIdx.x / BPW;
  if (n >= n_worlds) return;
  const int sol = n / n_init;
  const int grp = threadIdx.x / G, t = threadIdx.x % G, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int r0 = (blockIdx.x % BPW) * GPB;
  const int r = r0 + grp;
  const unsigned gmask = ((1u << G) - 1u) << (lane & ~(G - 1));
  float2* bufs = sm + wid * NBUF * RC::BUF;  // this warp's ring [NBUF][WROWS][ROWP]
  uint64_t* bars = bars_all + wid * (NBUF + 1);
  const int C = tab.C, K = tab.K;
  const float* gf = gfp + sol * gf_sol_stride;
  const float* wt = wts + sol * w_sol_stride;
  int* items = reinterpret_cast<int*>(ipar + (C * K + K + 1));  // [C*K + K + 1] item words
  float* wgf = reinterpret_cast<float*>(items + (C * K + K + 1));  // [C*K] weights, then [K][2] (m, s)

  // the solution's weights and growth parameters, one coalesced pass
  for (int q = threadIdx.x; q < C * K + 2 * K; q += blockDim.x)
    wgf[q] = q < C * K ? __ldg(wt + q) : __ldg(gf + (q - C * K));
  init_twiddles<GE>(tw, tw_rowi, tw_rowi, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int b = 0; b < NWARPS * (NBUF + 1); ++b) mbar_init(&bars_all[b], 1);
    fence_proxy_async();
    // work items with their growth parameters, and per-channel weight sums
    int ni = 0;
    unsigned long long seen = 0ull;
    auto param = [&](float w, int k) {
      const float m = wgf[C * K + 2 * k], sg = wgf[C * K + 2 * k + 1];
      const float a = GF == GF_FAST_GAUSSIAN ? 0.84932180028801904272f / sg
                                             : (GF == GF_FAST_POLY4 ? 1.f / (9.f * (sg * sg)) : 0.f);
      return make_float4(w, m, sg, a);
    };
    for (int co = 0; co < C; ++co) {
      float ws = 0.f;
      for (int k = 0; k < K; ++k) {
        const float w = wgf[co * K + k];
        ws += w;
        if (w == 0.f) continue;
        const bool first = !((seen >> k) & 1ull);
        seen |= 1ull << k;
        ipar[ni] = param(w, k);
        items[ni++] = (first ? (1 << 16) : 0) | ((co + 1) << 8) | k;
      }
      wsum_s[co] = ws;
    }
    for (int k = 0; k < K; ++k)
      if (!((seen >> k) & 1ull)) {
        ipar[ni] = param(0.f, k);
        items[ni++] = (1 << 16) | k;
      }
    s_nitems = ni;
  }
  __syncthreads();
  const int nit = s_nitems;
  depend_wait();
  depend_trigger();
  prod = after_wait(prod);
  state = after_wait(state);
  shift = after_wait(shift);

  // the warp stages its rows of item i into ring slot i % NBUF
  const float2* rows0 = prod + ((size_t)n * K * (N / 2) + r0 + wid * RC::WROWS) * N;
  auto issue = [&](int i) {
    const int b = i % NBUF;
    const float2* src = rows0 + (size_t)item_k(items[i]) * (N / 2) * N;
    float2* dst = bufs + b * RC::BUF;
    if (lane == 0) mbar_arrive_expect_tx(&bars[b], (unsigned)(RC::WROWS * N * sizeof(float2)));
    __syncwarp();
    if (lane < RC::WROWS) bulk_load(dst + lane * ROWP, src + (size_t)lane * N, N * sizeof(float2), &bars[b]);
  };
  // ... and channel co's state rows (2r, 2r+1) into sst
  float* sst_w = sst + wid * RC::WROWS * RC::SSTP;
  auto issue_state = [&](int co) {
    const float* src = state + (((size_t)n * C + co) * N + 2 * (r0 + wid * RC::WROWS)) * N;
    if (lane == 0) mbar_arrive_expect_tx(&bars[NBUF], (unsigned)(RC::WROWS * 2 * N * sizeof(float)));
    __syncwarp();
    if (lane < RC::WROWS)
      bulk_load(sst_w + lane * RC::SSTP, src + (size_t)lane * 2 * N, 2 * N * sizeof(float), &bars[NBUF]);
  };
  for (int q = 0; q < NBUF - 1 && q < nit; ++q) issue(q);
  int st_issued = 0, st_done = 0;  // state-row copies issued / waited for (warp-uniform)

  float dt;
  if (tab.dt_mode == 0) dt = __ldg(dtp);
  else if (tab.dt_mode == 1) dt = __ldg(dtp + n);
  else dt = 1.f / __ldg(dtp + sol);
  const int sy = shift[3 * n], sx = shift[3 * n + 1];
  float cpot = 0.f, m00 = 0.f, g00 = 0.f, cmass = 0.f, cgrow = 0.f, mxy = 0.f, mxx = 0.f, gxy = 0.f, gxx = 0.f,
        m2y = 0.f, m2x = 0.f;
  bool border = false;
  const float cya = (float)(((2 * r - sy) & (N - 1)) - N / 2);
  const float cyb = (float)(((2 * r + 1 - sy) & (N - 1)) - N / 2);
  float2 acc[P];
  bool failed = false;
  int failed_at = 0;

  // item i: wait for its rows, inverse row transform, count / write the
  // potential, accumulate the weighted growth of channel co (co >= 0).  A warp
  // stages, waits for and reuses its own rows, so no block barrier stands
  // between the items: past the warp barrier every lane is done with slot
  // (i - 1) % NBUF (item i - 1, or the fused row FFT's scratch), and the warp
  // refills that slot with item i + NBUF - 1.
  auto process = [&](int i) {
    if (__any_sync(0xffffffffu, !mbar_wait(&bars[i % NBUF], (i / NBUF) & 1))) {
      failed = true;
      failed_at = i;
      return;
    }
    const int it = items[i], k = item_k(it), co = item_co(it);
    fence_proxy_async();
    if (i + NBUF - 1 < nit) issue(i + NBUF - 1);
    // a channel's first item: its state rows start moving (the previous
    // channel's epilogue, the last reader of sst, is behind the warp barrier)
    if (co >= 0 && (i == 0 || item_co(items[i - 1]) != co)) {
      ++st_issued;
      issue_state(co);
    }
    float2* row = bufs + (i % NBUF) * RC::BUF + (lane / G) * ROWP;
    float2 v[Q][G];
    if constexpr (Q == 1) {
      unpack_row_pair_q1<GE>(row, v, t);
    } else {
      unpack_row_pair_pa<GE>(row, v, t);
    }
    __syncwarp(gmask);
    float2 w[P];
    fft_mirrored<GE, true, true>(v, w, row, tw_rowi, t, gmask);
    if (item_count(it)) {
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) cpot += (w[k1].x > kEps ? 1.f : 0.f) + (w[k1].y > kEps ? 1.f : 0.f);
      if (pot_out) {
        float* po = pot_out + ((size_t)n * K + k) * N * N;
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
          po[(2 * r) * N + t + G * k1] = w[k1].x;
          po[(2 * r + 1) * N + t + G * k1] = w[k1].y;
        }
      }
    }
    if (co >= 0) {
      const float4 ip = ipar[i];
      const float wk = ip.x;
      GrowthP g;
      g.m = ip.y;
      g.s = ip.z;
      g.a = ip.w;
      g.id = tab.gf[k];
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        if constexpr (GF == GF_GENERIC) {
          acc[k1].x = fmaf(wk, growth_cell<GF>(g, w[k1].x), acc[k1].x);
          acc[k1].y = fmaf(wk, growth_cell<GF>(g, w[k1].y), acc[k1].y);
        } else {  // w (2 e - 1) summed as 2 w e here, minus the channel's weight sum below
          acc[k1] = __ffma2_rn(make_float2(2.f * wk, 2.f * wk), growth_core2<GF>(g, w[k1]), acc[k1]);
        }
      }
    }
  };

  int i = 0;
  for (int co = 0; co < C && !failed; ++co) {
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) acc[k1] = make_float2(0.f, 0.f);
    const int i_begin = i;
    while (!failed && i < nit && item_co(items[i]) == co) process(i++);
    if (failed) break;
    if (i == i_begin) {  // a channel no kernel feeds: fetch its state rows here
      __syncwarp();
      ++st_issued;
      fence_proxy_async();
      issue_state(co);
    }
    if (__any_sync(0xffffffffu, !mbar_wait(&bars[NBUF], (st_issued - 1) & 1))) {
      failed = true;
      failed_at = i;
      break;
    }
    st_done = st_issued;
    // field (weighted_sum / weighted_mean, core.py:202-242), state update, moments
    const float wsum = wsum_s[co];
    const size_t base = ((size_t)n * C + co) * N * N;
    const float* sa_row = sst + grp * RC::SSTP;
    float* da_row = state_out + base + (size_t)(2 * r) * N;
    float* fa_row = field_out ? field_out + base + (size_t)(2 * r) * N : nullptr;
    float Sa = 0.f, Sb = 0.f, Ga = 0.f, Gb = 0.f;
    float2 nsv[P];  // the new rows (2r, 2r+1) at x = t + G*k1: the next step's row-FFT input comb
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
      const int x = t + G * k1;
      float fa = acc[k1].x, fb = acc[k1].y;
      if constexpr (GF != GF_GENERIC) {
        fa -= wsum;
        fb -= wsum;
      }
      if (tab.mean) {
        fa = fa / wsum;
        fb = fb / wsum;
      }
      const float sa = sa_row[x], sb = sa_row[N + x];
      nsv[k1] = make_float2(state_fn(tab.state_fn, sa, fa, dt), state_fn(tab.state_fn, sb, fb, dt));
      da_row[x] = nsv[k1].x;
      da_row[N + x] = nsv[k1].y;
      if (fa_row) {
        fa_row[x] = fa;
        fa_row[N + x] = fb;
      }
      const float fpa = fmaxf(fa, 0.f), fpb = fmaxf(fb, 0.f);
      const float cx = (float)(((x - sx) & (N - 1)) - N / 2);
      Sa += sa;
      Sb += sb;
      Ga += fpa;
      Gb += fpb;
      const float ss = sa + sb, gg = fpa + fpb;
      mxx = fmaf(ss, cx, mxx);
      gxx = fmaf(gg, cx, gxx);
      m2x = fmaf(ss * cx, cx, m2x);
      const bool la = sa > kEps, lb = sb > kEps;
      cmass += (la ? 1.f : 0.f) + (lb ? 1.f : 0.f);
      cgrow += (fpa > kEps ? 1.f : 0.f) + (fpb > kEps ? 1.f : 0.f);
      border |= ((x == 0 || x == N - 1) && (la || lb)) || (r == 0 && la) || (r == N / 2 - 1 && lb);
    }
    m00 += Sa + Sb;
    g00 += Ga + Gb;
    mxy += cya * Sa + cyb * Sb;
    gxy += cya * Ga + cyb * Gb;
    m2y += cya * cya * Sa + cyb * cyb * Sb;
    const float cms = warp_sum(Sa + Sb);
    if (lane == 0) red[wid * RAWS_MAX + RAW_CM + co] = cms;
    if (spec_next) {
      // the next step's row pass, fused: FFT of the packed new rows -> its
      // spectrum plane.  Exchange scratch: this group's row of ring slot
      // (i - 1) % NBUF, the one slot with no copy in flight (items i ..
      // i + NBUF - 2 are); the next process() barrier orders it before reuse.
      float2 u[Q][G];
      fft_standard<GE, false, false>(nsv, u, bufs + ((i + NBUF - 1) % NBUF) * RC::BUF + (lane / G) * ROWP, tw, t,
                                     gmask);
      float2* dst = spec_next + (((size_t)n * C + co) * (N / 2) + r) * N;
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int k1 = 0; k1 < G; ++k1) dst[pa_pos<N>(t + G * q + P * k1)] = u[q][k1];
    }
  }
  while (!failed && i < nit) process(i++);  // kernels that feed no channel
  if (failed) {
    // a staged copy never landed: record it and give the warp's copies in
    // flight a bounded time to drain; the status word marks the step's results
    if (lane == 0 && status) atomicExch(status, kStatusCopyTimeout);
    const int f = failed_at;
    for (int q = f; q < f + NBUF - 1 && q < nit; ++q) mbar_wait(&bars[q % NBUF], (q / NBUF) & 1);  // issued: <= f + NBUF - 2
    if (st_issued > st_done) mbar_wait(&bars[NBUF], (st_issued - 1) & 1);
  }
  // block reduction: warp shuffles then shared memory
  float accm[11] = {m00, g00, cpot, cmass, cgrow, mxy, mxx, gxy, gxx, m2y, m2x};
#pragma unroll
  for (int q = 0; q < 11; ++q) accm[q] = warp_sum(accm[q]);
  const bool anyb = __any_sync(0xffffffffu, border);
  if (lane == 0) {
    float* rd = red + wid * RAWS_MAX;
    rd[RAW_M00] = accm[0];
    rd[RAW_G00] = accm[1];
    rd[RAW_CNT_POT] = accm[2];
    rd[RAW_CNT_MASS] = accm[3];
    rd[RAW_CNT_GROW] = accm[4];
    rd[RAW_MX + 0] = accm[5];
    rd[RAW_MX + 1] = accm[6];
    rd[RAW_MX + 2] = 0.f;
    rd[RAW_GX + 0] = accm[7];
    rd[RAW_GX + 1] = accm[8];
    rd[RAW_GX + 2] = 0.f;
    rd[RAW_MX2 + 0] = accm[9];
    rd[RAW_MX2 + 1] = accm[10];
    rd[RAW_MX2 + 2] = 0.f;
    rd[RAW_BORDER] = anyb ? 1.f : 0.f;
    rd[RAW_SHIFT + 0] = rd[RAW_SHIFT + 1] = rd[RAW_SHIFT + 2] = 0.f;
  }
  __syncthreads();
  const int RAWS = raw_stride(C);
  if (threadIdx.x < RAWS) {
    float sum = 0.f;
    for (int w = 0; w < NWARPS; ++w) sum += red[w * RAWS_MAX + threadIdx.x];
    if (threadIdx.x == RAW_BORDER) sum = sum > 0.f ? 1.f : 0.f;
    partial[((size_t)n * BPW + (blockIdx.x % BPW)) * RAWS + threadIdx.x] = sum;
  }
}

// ------------------------------------------------------------ row_inv_split
// The row inverse for few worlds.  row_inv_kernel walks a world's C x K work
// items one after another in N/2/GPB blocks, which leaves the chip idle and
// the step as long as that chain.  Here a block owns the 32 / G packed rows of
// one warp's transforms and one output channel, its warps take the channel's
// kernels in turn (rows straight from L2 into the transform), the growths meet
// in shared memory, and the warps share the cells of the epilogue; warp 0 then
// runs the fused forward transform of the new rows while another sums the
// moments.  The growths of a cell are added in kernel order, as row_inv_kernel
// adds them, so fields, potentials and states are the same bits whatever the
// batch (the moments' sums are not: other blocks, other order).  Bound by
// instruction issue of a lone block an SM (48 blocks for one 128^2 world of
// three channels); 15 kernels of one 128^2 world: 43 us a step walking,
// 9.3 us split.
template <int N>
struct SplitCfg {
  static constexpr int G = SCfg<N>::G;
  static constexpr int RPB = 32 / G;          // packed rows per block
  static constexpr int BPC = (N / 2) / RPB;   // blocks per world and channel
  static constexpr int XCH = RPB * (N + G);   // float2 of exchange scratch per warp
  static constexpr int ACC = (N / G) * 32;    // float2: a row pair of growths per lane
};
constexpr int kSplitMinWarps = 4, kSplitMaxWarps = 8;

template <int N>
size_t row_inv_split_smem(int warps) {
  return ((size_t)3 * N + (size_t)warps * SplitCfg<N>::XCH + SplitCfg<N>::ACC) * sizeof(float2) +
         (size_t)warps * (RAW_CM + kMaxChannels) * sizeof(float);
}

template <int N, int GF>
__global__ void __launch_bounds__(32 * kSplitMaxWarps) row_inv_split_kernel(
    int n_worlds, int n_init, KTab tab, const float2* __restrict__ prod, const float* __restrict__ gfp,
    long gf_sol_stride, const float* __restrict__ wts, long w_sol_stride, const float* __restrict__ dtp,
    const float* __restrict__ state, float* __restrict__ state_out, float* __restrict__ field_out,
    float* __restrict__ pot_out, const int* __restrict__ shift, float* __restrict__ partial,
    float2* __restrict__ spec_next) {
  using SC = SplitCfg<N>;
  constexpr int G = SC::G, BPC = SC::BPC;
  using GE = Geo<N, G>;
  constexpr int P = GE::P, Q = GE::Q;
  constexpr int RAWS_MAX = RAW_CM + kMaxChannels;
  static_assert(SC::XCH >= P * 32 && SC::ACC == P * 32, "a warp's scratch holds its growths");
  __shared__ float wk_s[kSplitMaxWarps];
  extern __shared__ __align__(16) float2 sm[];
  const int warps = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float2* tw = sm;                      // 3N twiddles
  float2* xch = tw + 3 * N;             // [warps][XCH]
  float2* sum = xch + warps * SC::XCH;  // [P][32] weighted growths of the rounds before the last
  float* red = reinterpret_cast<float*>(sum + SC::ACC);  // [warps][RAWS_MAX]
  const int C = tab.C, K = tab.K;
  const int n = blockIdx.x / (BPC * C);
  if (n >= n_worlds) return;
  const int co = blockIdx.x / BPC % C;
  const int sol = n / n_init;
  const int grp = lane / G, t = lane % G;
  const int r = (blockIdx.x % BPC) * SC::RPB + grp;
  const unsigned gmask = ((1u << G) - 1u) << (lane & ~(G - 1));
  const float* gf = gfp + sol * gf_sol_stride;
  const float* wt = wts + sol * w_sol_stride;
  init_twiddles<GE>(tw, tw + N, tw + 2 * N, threadIdx.x, blockDim.x);

  // bit k: kernel k feeds this channel / an earlier one / any channel
  static_assert(kMaxKernels <= 64, "one bit per kernel");
  unsigned long long fed = 0ull, before = 0ull, any = 0ull;
  for (int h = 0; h < K; h += 32) {
    const int k = h + lane;
    for (int c = 0; c < C; ++c) {
      const float w = k < K ? __ldg(wt + c * K + k) : 0.f;
      const unsigned long long b = (unsigned long long)__ballot_sync(0xffffffffu, w != 0.f) << h;
      any |= b;
      if (c < co) before |= b;
      if (c == co) fed |= b;
    }
  }
  float wsum = 0.f;
#pragma unroll 8
  for (int k = 0; k < K; ++k) wsum += __ldg(wt + co * K + k);
  // channel 0 also takes the kernels that feed no channel (their potentials count)
  const unsigned long long all = K == 64 ? ~0ull : (1ull << K) - 1ull;
  const unsigned long long mine = fed | (co == 0 ? all & ~any : 0ull);
  float dt;
  if (tab.dt_mode == 0) dt = __ldg(dtp);
  else if (tab.dt_mode == 1) dt = __ldg(dtp + n);
  else dt = 1.f / __ldg(dtp + sol);
  // this warp's kernel among those of a round (-1: none) and its parameters,
  // fetched ahead of the rows; a kernel that feeds no channel has weight 0
  int k = -1;
  float wk = 0.f;
  GrowthP g;
  auto next_item = [&](unsigned long long todo) {
    for (int q = 0; q < wid; ++q) todo &= todo - 1;
    k = __ffsll((long long)todo) - 1;
    if (k < 0) return;
    wk = (fed >> k) & 1ull ? __ldg(wt + co * K + k) : 0.f;
    g.m = __ldg(gf + 2 * k);
    g.s = __ldg(gf + 2 * k + 1);
    g.a = GF == GF_FAST_GAUSSIAN ? 0.84932180028801904272f / g.s : (GF == GF_FAST_POLY4 ? 1.f / (9.f * (g.s * g.s)) : 0.f);
    g.id = tab.gf[k];
  };
  next_item(mine);

  depend_wait();
  depend_trigger();
  prod = after_wait(prod);
  state = after_wait(state);
  shift = after_wait(shift);
  const int sy = shift[3 * n], sx = shift[3 * n + 1];
  const size_t base = ((size_t)n * C + co) * N * N + (size_t)(2 * r) * N;
  float cpot = 0.f;
  float2* scr = xch + wid * SC::XCH;
  // A round: every warp takes one kernel and leaves its growths in its scratch,
  // then the warps add them up, cell by cell in kernel order (warp w the cells
  // k1 = w, w + warps, ...); the last round's sum is taken by the epilogue.
  auto add_round = [&](float2 f, int k1, int items) {
#pragma unroll 4
    for (int q = 0; q < items; ++q) {
      const float2 e = xch[q * SC::XCH + k1 * 32 + lane];
      const float wk = wk_s[q];
      f.x = fmaf(wk, e.x, f.x);
      f.y = fmaf(wk, e.y, f.y);
    }
    return f;
  };
  unsigned long long todo = mine;  // kernels of this and later rounds
  int left = __popcll(mine);
  const bool rounds = left > warps;  // more than one
  if (rounds)
    for (int k1 = wid; k1 < P; k1 += warps) sum[k1 * 32 + lane] = make_float2(0.f, 0.f);
  __syncthreads();
  for (;;) {
    if (k >= 0) {
      const float2* row = prod + (((size_t)n * K + k) * (N / 2) + r) * N;
      float2 v[Q][G];
      if constexpr (Q == 1) unpack_row_pair_q1<GE>(row, v, t);
      else unpack_row_pair_pa<GE>(row, v, t);
      float2 w[P];
      fft_mirrored<GE, true, true>(v, w, scr + grp * GE::SCR, tw + 2 * N, t, gmask);
      if (!((before >> k) & 1ull)) {
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) cpot += (w[k1].x > kEps ? 1.f : 0.f) + (w[k1].y > kEps ? 1.f : 0.f);
        if (pot_out) {
          float* po = pot_out + ((size_t)n * K + k) * N * N + (size_t)(2 * r) * N;
#pragma unroll
          for (int k1 = 0; k1 < P; ++k1) {
            po[t + G * k1] = w[k1].x;
            po[N + t + G * k1] = w[k1].y;
          }
        }
      }
      const bool feeds = (fed >> k) & 1ull;
      if (lane == 0) wk_s[wid] = GF == GF_GENERIC ? wk : 2.f * wk;
      __syncwarp();  // every group of the warp has read its exchange
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        float2 e = make_float2(0.f, 0.f);
        if (feeds) {
          if constexpr (GF == GF_GENERIC) e = make_float2(growth_cell<GF>(g, w[k1].x), growth_cell<GF>(g, w[k1].y));
          else e = growth_core2<GF>(g, w[k1]);  // w (2 e - 1): 2 w e here, minus the channel's weight sum below
        }
        scr[k1 * 32 + lane] = e;
      }
    }
    __syncthreads();
    if (left <= warps) break;
    for (int k1 = wid; k1 < P; k1 += warps) sum[k1 * 32 + lane] = add_round(sum[k1 * 32 + lane], k1, warps);
    for (int q = 0; q < warps; ++q) todo &= todo - 1;
    left -= warps;
    next_item(todo);
    __syncthreads();
  }

  // field (weighted_sum / weighted_mean, core.py:202-242), state update, moments
  const float cya = (float)(((2 * r - sy) & (N - 1)) - N / 2);
  const float cyb = (float)(((2 * r + 1 - sy) & (N - 1)) - N / 2);
  float Sa = 0.f, Sb = 0.f, Ga = 0.f, Gb = 0.f, cmass = 0.f, cgrow = 0.f, mxx = 0.f, gxx = 0.f, m2x = 0.f;
  bool border = false;
#pragma unroll 1
  for (int k1 = wid; k1 < P; k1 += warps) {
    const int x = t + G * k1;
    const float sa = __ldg(state + base + x), sb = __ldg(state + base + N + x);
    const float2 f = add_round(rounds ? sum[k1 * 32 + lane] : make_float2(0.f, 0.f), k1, left);
    float fa = f.x, fb = f.y;
    if constexpr (GF != GF_GENERIC) {
      fa -= wsum;
      fb -= wsum;
    }
    if (tab.mean) {
      fa = fa / wsum;
      fb = fb / wsum;
    }
    const float na = state_fn(tab.state_fn, sa, fa, dt), nb = state_fn(tab.state_fn, sb, fb, dt);
    state_out[base + x] = na;
    state_out[base + N + x] = nb;
    if (field_out) {
      field_out[base + x] = fa;
      field_out[base + N + x] = fb;
    }
    xch[k1 * 32 + lane] = make_float2(na, nb);  // read above by this thread alone
    const float fpa = fmaxf(fa, 0.f), fpb = fmaxf(fb, 0.f);
    const float cx = (float)(((x - sx) & (N - 1)) - N / 2);
    Sa += sa;
    Sb += sb;
    Ga += fpa;
    Gb += fpb;
    const float ss = sa + sb, gg = fpa + fpb;
    mxx = fmaf(ss, cx, mxx);
    gxx = fmaf(gg, cx, gxx);
    m2x = fmaf(ss * cx, cx, m2x);
    const bool la = sa > kEps, lb = sb > kEps;
    cmass += (la ? 1.f : 0.f) + (lb ? 1.f : 0.f);
    cgrow += (fpa > kEps ? 1.f : 0.f) + (fpb > kEps ? 1.f : 0.f);
    border |= ((x == 0 || x == N - 1) && (la || lb)) || (r == 0 && la) || (r == N / 2 - 1 && lb);
  }
  float accm[11] = {Sa + Sb, Ga + Gb, cpot, cmass, cgrow, cya * Sa + cyb * Sb, mxx, cya * Ga + cyb * Gb, gxx,
                    cya * cya * Sa + cyb * cyb * Sb, m2x};
#pragma unroll
  for (int q = 0; q < 11; ++q) accm[q] = warp_sum(accm[q]);
  const bool anyb = __any_sync(0xffffffffu, border);
  float* rd = red + wid * RAWS_MAX;
  if (lane == 0) {
    rd[RAW_M00] = accm[0];
    rd[RAW_G00] = accm[1];
    rd[RAW_CNT_POT] = accm[2];
    rd[RAW_CNT_MASS] = accm[3];
    rd[RAW_CNT_GROW] = accm[4];
    rd[RAW_MX + 0] = accm[5];
    rd[RAW_MX + 1] = accm[6];
    rd[RAW_MX + 2] = 0.f;
    rd[RAW_GX + 0] = accm[7];
    rd[RAW_GX + 1] = accm[8];
    rd[RAW_GX + 2] = 0.f;
    rd[RAW_MX2 + 0] = accm[9];
    rd[RAW_MX2 + 1] = accm[10];
    rd[RAW_MX2 + 2] = 0.f;
    rd[RAW_BORDER] = anyb ? 1.f : 0.f;
    rd[RAW_SHIFT + 0] = rd[RAW_SHIFT + 1] = rd[RAW_SHIFT + 2] = 0.f;
  }
  if (lane < C) rd[RAW_CM + lane] = lane == co ? accm[0] : 0.f;
  __syncthreads();
  if (wid == warps - 1) {
    const int RAWS = raw_stride(C);
    for (int q = lane; q < RAWS; q += 32) {
      float sum = 0.f;
      for (int w = 0; w < warps; ++w) sum += red[w * RAWS_MAX + q];
      if (q == RAW_BORDER) sum = sum > 0.f ? 1.f : 0.f;
      partial[(size_t)blockIdx.x * RAWS + q] = sum;
    }
  }
  if (wid == 0 && spec_next) {  // the next step's row pass: FFT of the packed new rows
    float2 nsv[P];
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) nsv[k1] = xch[k1 * 32 + lane];
    float2 u[Q][G];
    fft_standard<GE, false, false>(nsv, u, xch + SC::XCH + grp * GE::SCR, tw, t, gmask);
    float2* dst = spec_next + (((size_t)n * C + co) * (N / 2) + r) * N;
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int k1 = 0; k1 < G; ++k1) dst[pa_pos<N>(t + G * q + P * k1)] = u[q][k1];
  }
}

// ----------------------------------------------------------------- reduce
// Sum a world's block partials, write the step's raw moments, update the
// carried torus shift with trunc(centroid) (statistics.py:117-119).  WPW warps
// a world: one where a block of eight serves eight worlds, eight where one
// warp would walk a long list of partials.
constexpr int kReduceWarps = 8;

template <int WPW>
__global__ void __launch_bounds__(32 * kReduceWarps) reduce_kernel(
    int n_worlds, int n_init, int bpw, int C, int H, int W, const float* __restrict__ partial, float* __restrict__ raw,
    long raw_sol_stride, long raw_init_stride, int* __restrict__ shift) {
  constexpr int RAWS_MAX = RAW_CM + kMaxChannels;
  __shared__ float part[WPW > 1 ? WPW : 1][WPW > 1 ? RAWS_MAX : 1];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * (kReduceWarps / WPW) + wid / WPW;
  depend_wait();
  depend_trigger();
  partial = after_wait(partial);
  shift = after_wait(shift);
  if (n >= n_worlds) return;  // WPW > 1: one world a block, so whole blocks leave
  const int RAWS = raw_stride(C);
  const int sol = n / n_init, init = n - sol * n_init;
  float* rw = raw ? raw + sol * raw_sol_stride + init * raw_init_stride : nullptr;
  if constexpr (WPW > 1) {
    static_assert(WPW == kReduceWarps, "one world a block");
    for (int s = lane; s < RAWS; s += 32) {
      float v = 0.f;
#pragma unroll 4
      for (int b = wid; b < bpw; b += WPW) v += partial[((size_t)n * bpw + b) * RAWS + s];
      part[wid][s] = v;
    }
    __syncthreads();
    if (wid != 0) return;
  }
  float m00 = 0.f, mxy = 0.f, mxx = 0.f;
  const int sh0 = shift[3 * n], sh1 = shift[3 * n + 1];
  for (int s = lane; s < RAWS; s += 32) {
    float v = 0.f;
    if constexpr (WPW > 1) {
#pragma unroll
      for (int w = 0; w < WPW; ++w) v += part[w][s];
    } else {
      for (int b = 0; b < bpw; ++b) v += partial[((size_t)n * bpw + b) * RAWS + s];
    }
    if (s == RAW_BORDER) v = v > 0.f ? 1.f : 0.f;
    if (s == RAW_SHIFT) v = (float)sh0;
    if (s == RAW_SHIFT + 1) v = (float)sh1;
    if (s == RAW_SHIFT + 2) v = 0.f;
    if (rw) rw[s] = v;
    if (s == RAW_M00) m00 = v;
    if (s == RAW_MX) mxy = v;
    if (s == RAW_MX + 1) mxx = v;
  }
  __syncwarp();
  m00 = __shfl_sync(0xffffffffu, m00, RAW_M00);
  mxy = __shfl_sync(0xffffffffu, mxy, RAW_MX);
  mxx = __shfl_sync(0xffffffffu, mxx, RAW_MX + 1);
  if (lane == 0) {
    const float cy = mxy / (m00 + kEps), cx = mxx / (m00 + kEps);
    shift[3 * n] = pmod(sh0 + (int)cy, H);
    shift[3 * n + 1] = pmod(sh1 + (int)cx, W);
  }
}

template <int N>
__global__ void prepare_streamed_kernel(long n_planes, const float2* __restrict__ kh, float2* __restrict__ kp) {
  constexpr int KP = N / 2 + 2, HW = N / 2 + 1;
  const float scale = 1.f / (2.f * (float)N * (float)N);
  const long total = n_planes * N * KP;
  // column-major planes: element (ky, c) at c * N + ky, so the lanes of a
  // column transform read consecutive ky
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int ky = (int)(i % N);
    const long pc = i / N;
    const int c = (int)(pc % KP);
    const float2* src = kh + ((pc / KP) * N + ky) * HW;
    float2 o = make_float2(0.f, 0.f);
    if (c == 0) {
      float2 k0 = src[0], kn = src[N / 2];
      o = make_float2((k0.x + kn.x) * scale, (k0.y + kn.y) * scale);
    } else if (c == N / 2) {
      float2 k0 = src[0], kn = src[N / 2];
      o = make_float2((k0.x - kn.x) * scale, (k0.y - kn.y) * scale);
    } else if (c < N / 2) {
      float2 k = src[c];
      o = make_float2(k.x * scale, k.y * scale);
    }
    kp[i] = o;
  }
}

// Worlds up to which the row inverse is split over channels and kernels: as
// many as the walking kernel gives less than a block an SM.  Measured, us for
// a 16-step rollout with both kernels of 3 channels x 15 kernels (walking ->
// split; the split column includes col_conv_split): 128^2: 1 world
// 1037 -> 482, 16 1106 -> 814, 32 (128 blocks) 1143 -> 1077, 64 1383 -> 1745;
// 64^2: 64 worlds 1235 -> 864, 256 1610 -> 1880; 256^2: 4 worlds 1090 -> 868,
// 16 1406 -> 1842; one channel and kernel, 256^2: 8 worlds 535 -> 520, 16
// 577 -> 646.  At 512^2 a lane holds 32 points and the lines cross earlier:
// 3 x 9, 1 world 1198 -> 900, 2 (64 blocks) 1285 -> 1275, 4 1561 -> 2063.
template <int N>
constexpr int split_worlds() {
  return (N == 512 ? 64 : 128) / RowInvCfg<N>::BPW;
}

template <int N>
int partials_per_world(int C, int n_worlds) {
  return n_worlds <= split_worlds<N>() ? SplitCfg<N>::BPC * C : RowInvCfg<N>::BPW;
}

// Floats of row-inverse partials for up to n_worlds worlds a launch.
template <int N>
size_t partial_floats(int C, int n_worlds) {
  const size_t split = (size_t)std::min(n_worlds, split_worlds<N>()) * SplitCfg<N>::BPC * C;
  return std::max(split, (size_t)n_worlds * RowInvCfg<N>::BPW) * raw_stride(C);
}

template <int N, int GF>
cudaError_t launch_row_inv(const StreamedStep& s, const KTab& tab, cudaStream_t st) {
  float2* spec_next = s.emit_spec ? s.spec : nullptr;
  if (s.n_worlds <= split_worlds<N>()) {
    const int warps = std::min(kSplitMaxWarps, std::max(kSplitMinWarps, tab.K));
    const size_t smem = row_inv_split_smem<N>(warps);
    cudaError_t e = cudaFuncSetAttribute(row_inv_split_kernel<N, GF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)row_inv_split_smem<N>(kSplitMaxWarps));
    if (e != cudaSuccess) return e;
    return launch_dependent(row_inv_split_kernel<N, GF>, (unsigned)(s.n_worlds * tab.C * SplitCfg<N>::BPC), 32 * warps,
                            smem, st, s.n_worlds, s.n_init, tab, s.prod, s.gf, s.gf_sol_stride, s.w, s.w_sol_stride,
                            s.dt, s.state, s.state_out, s.field_out, s.pot_out, s.shift, s.partial, spec_next);
  }
  using RC = RowInvCfg<N>;
  const size_t sm_inv = row_inv_smem<N>(tab.C, tab.K);
  cudaError_t e = cudaFuncSetAttribute(row_inv_kernel<N, GF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_inv);
  if (e != cudaSuccess) return e;
  return launch_dependent(row_inv_kernel<N, GF>, (unsigned)((long)s.n_worlds * RC::BPW), RC::T, sm_inv, st, s.n_worlds,
                          s.n_init, tab, s.prod, s.gf, s.gf_sol_stride, s.w, s.w_sol_stride, s.dt, s.state,
                          s.state_out, s.field_out, s.pot_out, s.shift, s.partial, s.status, spec_next);
}

// Blocks sharing one column tile's kernels (gridDim.y): as many as there are
// kernels on a channel while the grid stays within two blocks an SM (more
// would only repeat the forward transform).  Five kernels a channel, one
// 128^2 world of three channels: 12 us on 12 blocks, 6.5 us on 60.
constexpr long kColBlocks = 304;

int col_conv_split(const Model& m, long blocks) {
  int per_channel = 0;
  for (int c = 0; c < m.C; ++c) {
    int n = 0;
    for (int k = 0; k < m.K; ++k) n += m.cin[k] == c ? 1 : 0;
    per_channel = std::max(per_channel, n);
  }
  return (int)std::max(1L, std::min((long)per_channel, kColBlocks / blocks));
}

// cuTensorMapEncodeTiled, fetched once from the driver through the runtime.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// Tensor map of the packed spectrum planes seen as rows of 2N floats:
// boxes of 32 floats (8 column pairs, 128 bytes) x N/2 packed rows,
// 128-byte swizzle.
template <int N>
bool encode_spec_map(CUtensorMap* map, const float2* spec, long planes) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)(2 * N), (cuuint64_t)(planes * (N / 2))};
  const cuuint64_t strides[1] = {(cuuint64_t)(2 * N * sizeof(float))};
  const cuuint32_t box[2] = {32, (cuuint32_t)(N / 2)};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float2*>(spec), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int N>
cudaError_t step_n(const StreamedStep& s, cudaStream_t st) {
  const Model& m = *s.m;
  constexpr int G = SCfg<N>::G;
  using GE = Geo<N, G>;
  constexpr int GPB = kThreads / G;
  constexpr int BPP = (N / 2 + GPB - 1) / GPB;
  KTab tab;
  tab.C = m.C;
  tab.K = m.K;
  tab.max_k = m.max_k;
  tab.mean = m.mean;
  tab.state_fn = m.state_fn;
  tab.dt_mode = s.dt_mode;
  for (int k = 0; k < m.K; ++k) {
    tab.cin[k] = m.cin[k];
    tab.slot[k] = m.slot[k];
    tab.gf[k] = m.gf[k];
  }
  const size_t sm_fwd = (size_t)3 * N * sizeof(float2) + (size_t)GPB * GE::SCR * sizeof(float2);
  using CC = ColCfg<N>;
  constexpr size_t sm_col = col_conv_smem<N>();
  cudaError_t e;
  e = cudaFuncSetAttribute(row_fwd_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_fwd);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(col_conv_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_col);
  if (e != cudaSuccess) return e;
  const long planes = (long)s.n_worlds * m.C;
  alignas(64) CUtensorMap spec_map, prod_map;
  if (!encode_spec_map<N>(&spec_map, s.spec, planes)) return cudaErrorInvalidValue;
  if (!encode_spec_map<N>(&prod_map, s.prod, (long)s.n_worlds * m.K)) return cudaErrorInvalidValue;
  if (!s.spec_ready)  // otherwise the previous step's row inverse already wrote this step's row spectra
    row_fwd_kernel<N><<<(unsigned)(planes * BPP), kThreads, sm_fwd, st>>>(s.n_worlds, m.C, s.state, s.spec);
  const dim3 col_grid((unsigned)(planes * CC::BPP), (unsigned)col_conv_split(m, planes * CC::BPP));
  e = launch_dependent(col_conv_kernel<N>, col_grid, CC::T, sm_col, st, spec_map, prod_map, s.n_worlds, s.n_init, tab,
                       s.kp, s.kp_sol_stride, s.status);
  if (e != cudaSuccess) return e;
  bool all_gauss = true, all_poly = true;
  for (int k = 0; k < m.K; ++k) {
    all_gauss = all_gauss && m.gf[k] == LGX_GF_GAUSSIAN;
    all_poly = all_poly && m.gf[k] == LGX_GF_POLY_QUAD4;
  }
  if (all_gauss) e = launch_row_inv<N, GF_FAST_GAUSSIAN>(s, tab, st);
  else if (all_poly) e = launch_row_inv<N, GF_FAST_POLY4>(s, tab, st);
  else e = launch_row_inv<N, GF_GENERIC>(s, tab, st);
  if (e != cudaSuccess) return e;
  return launch_streamed_reduce(s, partials_per_world<N>(m.C, s.n_worlds), st);
}

}  // namespace

bool streamed_supported(const Model& m) {
  if (m.nb_dims != 2 || m.H != m.W) return false;
  if (m.C > kMaxChannels || m.K > kMaxKernels) return false;
  if (!(m.H == 32 || m.H == 64 || m.H == 128 || m.H == 256 || m.H == 512) && !generic_size(m.H)) return false;
  return true;
}

size_t streamed_partial_floats(const Model& m, int n_worlds) {
  switch (m.H) {
    case 32: return partial_floats<32>(m.C, n_worlds);
    case 64: return partial_floats<64>(m.C, n_worlds);
    case 128: return partial_floats<128>(m.C, n_worlds);
    case 256: return partial_floats<256>(m.C, n_worlds);
    case 512: return partial_floats<512>(m.C, n_worlds);
  }
  return (size_t)n_worlds * generic_blocks_per_world(m.H) * raw_stride(m.C);  // a few packed rows per block
}

size_t streamed_workspace_bytes(const Model& m, int n_worlds, int n_sols) {
  const size_t plane = (size_t)m.H * m.W * sizeof(float);  // packed spectrum plane == state plane bytes
  size_t b = 0;
  auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
  b += al(plane * n_worlds * m.C);                                          // spec
  b += al(plane * n_worlds * m.K);                                          // prod
  b += al((size_t)n_sols * m.C * m.max_k * m.H * (m.W / 2 + 2) * sizeof(float2));  // kp
  b += al(streamed_partial_floats(m, n_worlds) * sizeof(float));  // partial
  b += al((size_t)n_worlds * 3 * sizeof(int));                              // shift
  return b;
}

cudaError_t launch_streamed_reduce(const StreamedStep& s, int bpw, cudaStream_t st) {
  const Model& m = *s.m;
  if (bpw >= 2 * kReduceWarps)
    return launch_dependent(reduce_kernel<kReduceWarps>, s.n_worlds, 32 * kReduceWarps, 0, st, s.n_worlds, s.n_init,
                            bpw, m.C, m.H, m.W, s.partial, s.raw, s.raw_sol_stride, s.raw_world_stride, s.shift);
  return launch_dependent(reduce_kernel<1>, (s.n_worlds + kReduceWarps - 1) / kReduceWarps, 32 * kReduceWarps, 0, st,
                          s.n_worlds, s.n_init, bpw, m.C, m.H, m.W, s.partial, s.raw, s.raw_sol_stride,
                          s.raw_world_stride, s.shift);
}

cudaError_t launch_streamed_step(const StreamedStep& s, cudaStream_t st) {
  // the row inverse bulk-copies state rows: the state base must be 16-byte aligned
  if ((reinterpret_cast<uintptr_t>(s.state) & 15u) != 0) return cudaErrorMisalignedAddress;
  switch (s.m->H) {
    case 32: return step_n<32>(s, st);
    case 64: return step_n<64>(s, st);
    case 128: return step_n<128>(s, st);
    case 256: return step_n<256>(s, st);
    case 512: return step_n<512>(s, st);
  }
  if (generic_size(s.m->H)) return launch_generic_step(s, st);
  return cudaErrorInvalidValue;
}

cudaError_t launch_prepare_streamed_spectrum(const Model& m, int n_sols, const float2* k_half, float2* kp,
                                             cudaStream_t st) {
  const long planes = (long)n_sols * m.C * m.max_k;
  const long total = planes * m.H * (m.W / 2 + 2);
  const int threads = 256;
  const int blocks = (int)std::min<long>((total + threads - 1) / threads, 8192);
  switch (m.H) {
    case 32: prepare_streamed_kernel<32><<<blocks, threads, 0, st>>>(planes, k_half, kp); break;
    case 64: prepare_streamed_kernel<64><<<blocks, threads, 0, st>>>(planes, k_half, kp); break;
    case 128: prepare_streamed_kernel<128><<<blocks, threads, 0, st>>>(planes, k_half, kp); break;
    case 256: prepare_streamed_kernel<256><<<blocks, threads, 0, st>>>(planes, k_half, kp); break;
    case 512: prepare_streamed_kernel<512><<<blocks, threads, 0, st>>>(planes, k_half, kp); break;
    default:
      if (generic_size(m.H)) return launch_prepare_generic_spectrum(m, n_sols, k_half, kp, st);
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace lgx
