// Line FFTs of the general N-D engine: mixed-radix Stockham transforms whose
// butterflies (radices up to 16) run in registers, with caller-supplied loads
// and stores at both ends.
//
// A 4096-point tile of lines used to be loaded into shared memory, taken
// through one radix-2/3/4/5/7 stage per block barrier (three for 48 or 100
// points, five for 1024) and read back for the store: every point crossed
// shared memory eight to twelve times.  Here a line of up to 256 points is two
// register butterflies with one shared-memory exchange between them, longer
// ones three; the first butterfly reads its points through `in` (global
// memory, or a rule such as "the packed pair of rows"), the last hands them
// to `out`.  Where a forward transform is followed by its inverse (the
// spectral product, Bluestein's filter, the Euler update between two row
// transforms) the inverse runs the radices backwards, so the last butterfly
// of one and the first of the other own the same points and the step between
// them happens in registers (center_stage).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "fft.cuh"
#include "fft_mixed.cuh"

namespace lgx {

// ------------------------------------------------------------ register DFTs
__host__ __device__ constexpr int dft_factor(int R) {
  return R % 4 == 0 ? 4 : (R % 2 == 0 ? 2 : (R % 3 == 0 ? 3 : (R % 5 == 0 ? 5 : R)));
}

// R-point DFT in registers, natural order in and out.  Odd primes pair the
// points p and R - p (cosine sums, sine differences); composite sizes are
// Cooley-Tukey over their smallest factor with compile-time twiddles.
template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
    const float2 s13 = cadd(v[1], v[3]), d13 = csub(v[1], v[3]);
    const float2 rot = INV ? make_float2(-d13.y, d13.x) : make_float2(d13.y, -d13.x);
    v[0] = cadd(s02, s13);
    v[1] = cadd(d02, rot);
    v[2] = csub(s02, s13);
    v[3] = csub(d02, rot);
  } else if constexpr (dft_factor(R) == R) {  // 3, 5, 7
    constexpr int M = (R - 1) / 2;
    float2 s[M], d[M];
    const float2 x0 = v[0];
    float2 sum = x0;
    sfor<M>([&](auto I) {
      constexpr int p = decltype(I)::value;
      s[p] = cadd(v[p + 1], v[R - 1 - p]);
      d[p] = csub(v[p + 1], v[R - 1 - p]);
      sum = cadd(sum, s[p]);
    });
    v[0] = sum;
    sfor<M>([&](auto K) {
      constexpr int k = decltype(K)::value + 1;
      float2 m = x0, n = make_float2(0.f, 0.f);
      sfor<M>([&](auto I) {
        constexpr int p = decltype(I)::value;
        constexpr float c = (float)cx_trig((long)(p + 1) * k, R, false);
        constexpr float sn = (float)(INV ? -cx_trig((long)(p + 1) * k, R, true) : cx_trig((long)(p + 1) * k, R, true));
        m = __ffma2_rn(s[p], make_float2(c, c), m);
        n = p == 0 ? __fmul2_rn(d[p], make_float2(sn, sn)) : __ffma2_rn(d[p], make_float2(sn, sn), n);
      });
      // forward: X_k = m - i n, X_{R-k} = m + i n
      v[k] = make_float2(m.x + n.y, m.y - n.x);
      v[R - k] = make_float2(m.x - n.y, m.y + n.x);
    });
  } else {
    constexpr int A = dft_factor(R), B = R / A;
    float2 y[A][B];
#pragma unroll
    for (int a = 0; a < A; ++a) {
#pragma unroll
      for (int b = 0; b < B; ++b) y[a][b] = v[a + A * b];
      dft<B, INV>(y[a]);
    }
    sfor<B>([&](auto K) {
      constexpr int k = decltype(K)::value;
      float2 t[A];
      sfor<A>([&](auto I) {
        constexpr int a = decltype(I)::value;
        t[a] = tw_mul<a * k, R, INV>(y[a][k]);
      });
      dft<A, INV>(t);
#pragma unroll
      for (int a = 0; a < A; ++a) v[k + B * a] = t[a];
    });
  }
}

// ------------------------------------------------------------------- plans
constexpr int kLineStages = 8;

// One world axis: an n-point line transform of m-point transforms (m == n, or
// the Bluestein length m >= 2n - 1).  r: radices of the forward transform, the
// inverse runs them backwards.  The ends take radices up to 10, the middle
// stages (m > 100) up to 8; a `wide` axis' ends are 8, 9, 10, 12, 14, 15 or 16.
struct LineAxis {
  int n, m, stages, wide;
  int r[kLineStages];
  int st[kLineStages], ist[kLineStages];   // twiddle step m / (Ns r) of every forward / inverse stage
  int ns[kLineStages], ins[kLineStages];   // Ns: product of the radices before the stage
  FastDivU nbd[kLineStages];               // by the stage's butterflies m / r
  FastDivU nsd[kLineStages], insd[kLineStages];
  const float2* tw;                        // W_m^j, j < m; Bluestein lines: then the chirp (n) and its filter (m)
};

inline bool wide_radix(int r) { return (r >= 8 && r <= 10) || r == 12 || (r >= 14 && r <= 16); }
inline bool line_radix(int r, bool end) {
  if (end) return r >= 2 && r <= 10;
  return r == 2 || r == 3 || r == 4 || r == 5 || r == 7 || r == 8;
}

// The fewest stages, then the smallest sum of radices.  Depth-first over the
// stage list first, last, middle...; returns the number of stages or 0.  wide:
// both ends from the wide radices, two stages at least.
inline int find_line_radices(int m, int* out, bool wide) {
  int best = 0, best_sum = 1 << 30, cur[kLineStages] = {0};
  auto end_radix = [=](int r) { return wide ? wide_radix(r) : line_radix(r, true); };
  if (!wide && m >= 2 && line_radix(m, true)) {
    out[0] = m;
    out[1] = 1;
    return 2;
  }
  auto middle = [&](auto&& self, int left, int depth, int sum, int top) -> void {
    if (left == 1) {
      if (best == 0 || depth < best || (depth == best && sum < best_sum)) {
        best = depth;
        best_sum = sum;
        out[0] = cur[0];
        out[depth - 1] = cur[1];
        for (int i = 2; i < depth; ++i) out[i - 1] = cur[i];
      }
      return;
    }
    if (depth >= kLineStages || (best && depth >= best)) return;
    for (int r = top; r >= 2; --r)
      if (left % r == 0 && line_radix(r, false)) {
        cur[depth] = r;
        self(self, left / r, depth + 1, sum + r, r);
      }
  };
  for (int a = wide ? 16 : 10; a >= 2; --a) {
    if (m % a || !end_radix(a)) continue;
    for (int b = a; b <= 16; ++b) {  // the larger radix last: the smaller one writes the exchange
      if ((m / a) % b || !end_radix(b)) continue;
      cur[0] = a;
      cur[1] = b;
      middle(middle, m / a / b, 2, a + b, 8);
    }
  }
  return best;
}

// find_line_radices, remembered by length: every step of a rollout lays out its
// axes several times over, and a search takes the host 0.1 us (48 or 100
// points) to 0.6 us (360).  One word a plan (a byte a stage; all ones: no
// plan), so threads need no lock.
inline int line_radices(int m, int* out, bool wide = false) {
  constexpr int kRemembered = 4096;
  static std::atomic<unsigned long long> plans[2][kRemembered + 1];
  if (m < 0 || m > kRemembered) return find_line_radices(m, out, wide);
  static_assert(kLineStages == 8, "a byte a stage");
  unsigned long long p = plans[wide][m].load(std::memory_order_relaxed);
  if (p == 0) {
    int r[kLineStages] = {0};
    const int stages = find_line_radices(m, r, wide);
    p = stages > 0 ? 0 : ~0ull;
    for (int s = 0; s < stages; ++s) p |= (unsigned long long)r[s] << (8 * s);
    plans[wide][m].store(p, std::memory_order_relaxed);
  }
  if (p == ~0ull) return 0;
  int stages = 0;
  for (; stages < kLineStages && (p >> (8 * stages) & 255); ++stages) out[stages] = (int)(p >> (8 * stages) & 255);
  return stages;
}

// Axis of n-point lines with m-point transforms; `tables` as laid out by
// line_table_elems.  False when m has no plan.  allow_wide: take the wide
// radices where they bring four stages down to three (1024 = 8 8 16, 768 =
// 8 12 8): one exchange and one rounding of the twiddles less, at 96 registers
// a thread and two blocks an SM instead of 64 and three.  8-step rollouts, us,
// plain -> wide: 19 worlds of 100 x 768 478 -> 451, of 768 x 100 455 -> 450;
// 14 of 100 x 1024 513 -> 478, of 1024 x 100 486 -> 468.  Bringing three
// stages down to two does not pay for the blocks: 100 x 144 431 -> 516,
// 100 x 192 426 -> 470, 100 x 256 387 -> 407, 192 x 100 426 -> 449.
inline bool make_line_axis(int n, int m, float2* tables, LineAxis* ax, bool allow_wide) {
  ax->n = n;
  ax->m = m;
  ax->stages = line_radices(m, ax->r);
  if (ax->stages == 0) return false;
  ax->wide = 0;
  int r[kLineStages];
  const int stages = allow_wide && n == m && ax->stages > 3 ? line_radices(m, r, true) : 0;
  if (stages > 0 && stages < ax->stages) {
    ax->wide = 1;
    ax->stages = stages;
    std::copy(r, r + stages, ax->r);
  }
  int ns = 1, ins = 1;
  for (int s = 0; s < ax->stages; ++s) {
    const int r = ax->r[s], ri = ax->r[ax->stages - 1 - s];
    ax->ns[s] = ns;
    ax->ins[s] = ins;
    ax->st[s] = m / (ns * r);
    ax->ist[s] = m / (ins * ri);
    ax->nbd[s] = make_fastdiv((unsigned)(m / r));
    ax->nsd[s] = make_fastdiv((unsigned)ns);
    ax->insd[s] = make_fastdiv((unsigned)ins);
    ns *= r;
    ins *= ri;
  }
  ax->tw = tables;
  return true;
}
inline size_t line_table_elems(int n, int m) { return (size_t)m + (m != n ? (size_t)n + m : 0); }

// ---------------------------------------------------------------- exchange
// Points between two stages in shared memory.  The first exchange keeps
// butterfly j's output t at [t][j] (rows of `p0` butterflies, odd), later ones
// are in point order; either way an item's R points are a constant step apart.
// LINES (a warp's lanes take neighbouring lines): the lines of a tile are
// innermost (`lp` lines, odd, per point); otherwise a line is `lp` points.
struct Tile {
  float2* b[2];  // every transform's last exchange leaves b[1] free for the next one's first
  // the axis' tables, for Bluestein lines: after_wait(LineAxis::tw), as the
  // kernel may depend on the launch that writes them
  const float2* tab;
  int lp;
  int nl;
  FastDivU nld;  // by nl
  __device__ __forceinline__ void swap() {
    float2* t = b[0];
    b[0] = b[1];
    b[1] = t;
  }
};
// points of a line in the exchange: the largest first-exchange layout (either
// direction), or m
inline int line_points(const LineAxis& ax) {
  const int a = ax.r[0], b = ax.r[ax.stages - 1];
  return std::max(ax.m, std::max(a * ((ax.m / a) | 1), b * ((ax.m / b) | 1)));
}
inline int line_pitch(bool lines, const LineAxis& ax, int nl) { return lines ? (nl | 1) : (line_points(ax) | 1); }
inline long line_buf_elems(bool lines, const LineAxis& ax, int nl) {
  return (long)line_pitch(lines, ax, nl) * (lines ? line_points(ax) : nl);
}

// ------------------------------------------------------------------ stages
// in(l, j, nb, v): v[q] = point j + q nb of line l; out(l, base, step, v):
// point base + t step is v[t].
template <bool LINES>
struct XRead {  // a stage's reads: R points of [point] or, after the first exchange, of [t][j]
  const float2* b;
  int lp, r0, p0, two;  // p0: butterflies' pitch of the first exchange (0: point order); r0: its radix
  FastDivU r0d;
  template <int R>
  __device__ __forceinline__ void operator()(int l, int j, int nb, float2 (&v)[R]) const {
    int at = j, step = nb;
    if (p0 > 0) {  // after the first exchange
      if (two) {   // the last of two stages: output j of every butterfly
        at = j * p0;
        step = 1;
      } else {  // point j + q nb is output t = j mod r0 of butterfly j / r0 + q nb / r0
        const int jj = r0d.div(j);
        at = (j - jj * r0) * p0 + jj;
        step = r0d.div(nb);
      }
    }
    const float2* p = LINES ? b + at * lp + l : b + l * lp + at;
    const int s = LINES ? step * lp : step;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = p[q * s];
  }
};
template <bool LINES>
struct XWrite {
  float2* b;
  int lp;
  template <int R>
  __device__ __forceinline__ void operator()(int l, int at, int step, const float2 (&v)[R]) const {
    float2* p = LINES ? b + at * lp + l : b + l * lp + at;
    const int s = LINES ? step * lp : step;
#pragma unroll
    for (int t = 0; t < R; ++t) p[t * s] = v[t];
  }
};

// KIND 0: first stage (no twiddles; output t of butterfly j at [t][j]), 1:
// middle, 2: last.  `items` of the tile are butterflies (l, j), neighbouring
// threads taking neighbouring lines (LINES) or butterflies.
template <int R, int KIND, bool INV, bool LINES, class In, class Out>
__device__ __forceinline__ void line_stage(int m, int Ns, int st, FastDivU div, FastDivU nsd, int nl, const float2* tw,
                                           const In& in, const Out& out) {
  const int nb = m / R, items = nl * nb;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int hi = div.div(it), lo = it - hi * (LINES ? nl : nb);
    const int l = LINES ? lo : hi, j = LINES ? hi : lo;
    const int k = KIND == 0 ? 0 : (KIND == 2 ? j : j - nsd.div(j) * Ns);
    float2 v[R];
    in(l, j, nb, v);
    if (KIND != 0) {
      const int ks = KIND == 2 ? j : k * st;
#pragma unroll
      for (int q = 1; q < R; ++q) {
        const float2 w = tw[q * ks];
        v[q] = INV ? cmulc(v[q], w) : cmul(v[q], w);
      }
    }
    dft<R, INV>(v);
    if (KIND == 0) out(l, j, nb | 1, v);
    else if (KIND == 2) out(l, j, nb, v);
    else out(l, (j - k) * R + k, Ns, v);
  }
}

// The last forward butterfly (or the last inverse one, INV), `mid` on its
// points, and the first butterfly of the opposite transform:
// mid(l, j, nb, v) sees v[t] = point j + t nb and returns false to drop the
// second half.
template <int R, bool INV, bool LINES, class In, class Mid, class Out>
__device__ __forceinline__ void center_stage(int m, FastDivU div, int nl, const float2* tw, const In& in,
                                             const Mid& mid, const Out& out) {
  const int nb = m / R, items = nl * nb;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int hi = div.div(it), lo = it - hi * (LINES ? nl : nb);
    const int l = LINES ? lo : hi, j = LINES ? hi : lo;
    float2 v[R];
    in(l, j, nb, v);
#pragma unroll
    for (int q = 1; q < R; ++q) {
      const float2 w = tw[q * j];
      v[q] = INV ? cmulc(v[q], w) : cmul(v[q], w);
    }
    dft<R, INV>(v);
    if (!mid(l, j, nb, v)) continue;
    dft<R, !INV>(v);
    out(l, j, nb | 1, v);
  }
}

#define LGX_END_RADICES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10)
#define LGX_WIDE_RADICES(X) X(8) X(9) X(10) X(12) X(14) X(15) X(16)

// Which lines a kernel is compiled for.
enum LineKind { LINE_PLAIN = 0, LINE_BLUESTEIN = 1, LINE_WIDE = 2 };
inline LineKind line_kind(const LineAxis& ax) {
  return ax.m != ax.n ? LINE_BLUESTEIN : (ax.wide ? LINE_WIDE : LINE_PLAIN);
}
// kernel<KIND...>(line_kind(ax)): f(ic<KIND>) picks the instance
template <class F>
auto for_line_kind(const LineAxis& ax, F&& f) {
  switch (line_kind(ax)) {
    case LINE_BLUESTEIN: return f(ic<LINE_BLUESTEIN>{});
    case LINE_WIDE: return f(ic<LINE_WIDE>{});
    default: return f(ic<LINE_PLAIN>{});
  }
}

// What stage s >= 1 of the INV or forward transform reads from t.b[0].
template <bool INV, bool LINES>
__device__ __forceinline__ XRead<LINES> line_reads(const LineAxis& ax, const Tile& t, int s) {
  XRead<LINES> r{t.b[0], t.lp, 0, 0, ax.stages == 2, {}};
  if (s == 1) {
    const int q = INV ? ax.stages - 1 : 0;
    r.r0 = ax.r[q];
    r.p0 = (INV ? ax.ist[0] : ax.st[0]) | 1;  // butterflies of the first stage
    r.r0d = INV ? ax.insd[1] : ax.nsd[1];     // by the first radix
  }
  return r;
}

// The middle stages 1 .. S-2 on the points of t.b[0] (after line_head's first
// butterfly, or after a line_center, the first stage of the INV transform).
template <bool INV, bool LINES>
__device__ __forceinline__ void line_middle(const LineAxis& ax, const float2* tw, Tile& t) {
  const int S = ax.stages;
  for (int s = 1; s < S - 1; ++s) {
    const XRead<LINES> rd = line_reads<INV, LINES>(ax, t, s);
    const XWrite<LINES> wr{t.b[1], t.lp};
    const int q = INV ? S - 1 - s : s;
    const int Ns = INV ? ax.ins[s] : ax.ns[s], st = INV ? ax.ist[s] : ax.st[s];
    const FastDivU nsd = INV ? ax.insd[s] : ax.nsd[s], div = LINES ? t.nld : ax.nbd[q];
    switch (ax.r[q]) {
#define LGX_CASE(R) \
  case R: line_stage<R, 1, INV, LINES>(ax.m, Ns, st, div, nsd, t.nl, tw, rd, wr); break;
      LGX_CASE(2) LGX_CASE(3) LGX_CASE(4) LGX_CASE(5) LGX_CASE(7) LGX_CASE(8)
#undef LGX_CASE
    }
    __syncthreads();
    t.swap();
  }
}

// Stages 0 .. S-2 of a transform: `in` through the first butterfly into the
// exchange, then the middle ones; ends on a barrier with the points in t.b[0].
template <bool INV, bool LINES, bool WIDE = false, class In>
__device__ __forceinline__ void line_head(const LineAxis& ax, const float2* tw, Tile& t, const In& in) {
  const int S = ax.stages;
  const XWrite<LINES> out{t.b[0], t.lp};
  const int r = INV ? ax.r[S - 1] : ax.r[0];
  const FastDivU div = LINES ? t.nld : (INV ? ax.nbd[S - 1] : ax.nbd[0]);
  if constexpr (WIDE) {
    switch (r) {
#define LGX_CASE(R) \
  case R: line_stage<R, 0, INV, LINES>(ax.m, 1, 0, div, div, t.nl, tw, in, out); break;
      LGX_WIDE_RADICES(LGX_CASE)
#undef LGX_CASE
    }
  } else {
    switch (r) {
#define LGX_CASE(R) \
  case R: line_stage<R, 0, INV, LINES>(ax.m, 1, 0, div, div, t.nl, tw, in, out); break;
      LGX_END_RADICES(LGX_CASE)
#undef LGX_CASE
    }
  }
  __syncthreads();
  line_middle<INV, LINES>(ax, tw, t);
}

// The last stage, from t.b[0] to `out`; no barrier at its end.
template <bool INV, bool LINES, bool WIDE = false, class Out>
__device__ __forceinline__ void line_tail(const LineAxis& ax, const float2* tw, Tile& t, const Out& out) {
  const int S = ax.stages;
  const XRead<LINES> rd = line_reads<INV, LINES>(ax, t, S - 1);
  const int r = INV ? ax.r[0] : ax.r[S - 1];
  const FastDivU div = LINES ? t.nld : (INV ? ax.nbd[0] : ax.nbd[S - 1]);
  if constexpr (WIDE) {
    switch (r) {
#define LGX_CASE(R) \
  case R: line_stage<R, 2, INV, LINES>(ax.m, 1, 0, div, div, t.nl, tw, rd, out); break;
      LGX_WIDE_RADICES(LGX_CASE)
#undef LGX_CASE
    }
  } else {
    switch (r) {
#define LGX_CASE(R) \
  case R: line_stage<R, 2, INV, LINES>(ax.m, 1, 0, div, div, t.nl, tw, rd, out); break;
      LGX_END_RADICES(LGX_CASE)
#undef LGX_CASE
    }
  }
  t.swap();
}

// line_tail, `mid`, then the opposite transform's first stage; ends on a
// barrier with the points of that transform in t.b[0].
template <bool INV, bool LINES, bool WIDE = false, class Mid>
__device__ __forceinline__ void line_center(const LineAxis& ax, const float2* tw, Tile& t, const Mid& mid) {
  const int S = ax.stages;
  const XRead<LINES> rd = line_reads<INV, LINES>(ax, t, S - 1);
  const XWrite<LINES> wr{t.b[1], t.lp};
  const int r = INV ? ax.r[0] : ax.r[S - 1];
  const FastDivU div = LINES ? t.nld : (INV ? ax.nbd[0] : ax.nbd[S - 1]);
  if constexpr (WIDE) {
    switch (r) {
#define LGX_CASE(R) \
  case R: center_stage<R, INV, LINES>(ax.m, div, t.nl, tw, rd, mid, wr); break;
      LGX_WIDE_RADICES(LGX_CASE)
#undef LGX_CASE
    }
  } else {
    switch (r) {
#define LGX_CASE(R) \
  case R: center_stage<R, INV, LINES>(ax.m, div, t.nl, tw, rd, mid, wr); break;
      LGX_END_RADICES(LGX_CASE)
#undef LGX_CASE
    }
  }
  __syncthreads();
  t.swap();
}

// The whole transform of the tile's lines, unnormalised, from in(l, j, nb, v)
// to out(l, base, step, v).  BL: Bluestein's chirp-z transform (L. Bluestein,
// "A linear filtering approach to the computation of discrete Fourier
// transform", 1970) for lengths with a prime factor above 7: with c_n =
// exp(-i pi n^2 / L), X_k = c_k sum_n (x_n c_n) conj(c_{k-n}), a cyclic
// convolution of length m >= 2n - 1; `bhat` is the m-point spectrum of conj(c)
// wrapped around, which is even, so the inverse transform takes the
// conjugates of all of them.  Its lines go point by point: in1(l, i) and
// out1(l, i, x) below.
template <bool INV, bool LINES, class In, class Out>
__device__ __forceinline__ void line_bluestein(const LineAxis& ax, const float2* tw, Tile& t, const In& in1,
                                               const Out& out1) {
  const int n = ax.n;
  const float2 *chirp = t.tab + ax.m, *bhat = chirp + n;
  const float inv_m = 1.f / (float)ax.m;
  line_head<false, LINES>(ax, tw, t, [&](int l, int j, int nb, auto& v) {
    constexpr int R = (int)(sizeof(v) / sizeof(float2));
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = j + q * nb;
      v[q] = make_float2(0.f, 0.f);
      if (i < n) {
        const float2 x = in1(l, i), c = __ldg(chirp + i);
        v[q] = INV ? cmulc(x, c) : cmul(x, c);
      }
    }
  });
  line_center<false, LINES>(ax, tw, t, [=](int l, int j, int nb, auto& v) {
    constexpr int R = (int)(sizeof(v) / sizeof(float2));
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const float2 h = __ldg(bhat + j + q * nb);
      v[q] = INV ? cmulc(v[q], h) : cmul(v[q], h);
    }
    return true;
  });
  line_middle<true, LINES>(ax, tw, t);
  line_tail<true, LINES>(ax, tw, t, [&](int l, int j, int nb, const auto& v) {
    constexpr int R = (int)(sizeof(v) / sizeof(float2));
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int k = j + q * nb;
      if (k < n) {
        const float2 c = __ldg(chirp + k);
        const float2 x = INV ? cmulc(v[q], c) : cmul(v[q], c);
        out1(l, k, make_float2(x.x * inv_m, x.y * inv_m));
      }
    }
  });
}

// Point-by-point rules as a stage's loads and stores.
template <class F>
struct EachIn {
  const F& f;
  template <int R>
  __device__ __forceinline__ void operator()(int l, int j, int nb, float2 (&v)[R]) const {
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = f(l, j + q * nb);
  }
};
template <class F>
struct EachOut {
  const F& f;
  template <int R>
  __device__ __forceinline__ void operator()(int l, int at, int step, const float2 (&v)[R]) const {
#pragma unroll
    for (int t = 0; t < R; ++t) f(l, at + t * step, v[t]);
  }
};
template <class F>
__device__ __forceinline__ EachIn<F> each_in(const F& f) { return EachIn<F>{f}; }
template <class F>
__device__ __forceinline__ EachOut<F> each_out(const F& f) { return EachOut<F>{f}; }

// in1(l, i) -> out1(l, k, X_k) point by point, any kind of line.
template <bool INV, bool LINES, int KIND, class In, class Out>
__device__ __forceinline__ void line_fft(const LineAxis& ax, const float2* tw, Tile& t, const In& in1,
                                         const Out& out1) {
  if constexpr (KIND == LINE_BLUESTEIN) {
    line_bluestein<INV, LINES>(ax, tw, t, in1, out1);
  } else {
    line_head<INV, LINES, KIND == LINE_WIDE>(ax, tw, t, each_in(in1));
    line_tail<INV, LINES, KIND == LINE_WIDE>(ax, tw, t, each_out(out1));
  }
}

// The same with rules that take a butterfly's points at once, as the stages do
// (Bluestein lines: one point).
template <bool INV, bool LINES, int KIND, class In, class Out>
__device__ __forceinline__ void line_fft_rules(const LineAxis& ax, const float2* tw, Tile& t, const In& in,
                                               const Out& out) {
  if constexpr (KIND == LINE_BLUESTEIN) {
    line_bluestein<INV, LINES>(
        ax, tw, t,
        [&](int l, int i) {
          float2 v[1];
          in(l, i, 0, v);
          return v[0];
        },
        [&](int l, int i, float2 x) {
          const float2 v[1] = {x};
          out(l, i, 0, v);
        });
  } else {
    line_head<INV, LINES, KIND == LINE_WIDE>(ax, tw, t, in);
    line_tail<INV, LINES, KIND == LINE_WIDE>(ax, tw, t, out);
  }
}

// An axis' twiddles into shared memory (m entries), without a barrier.  The
// table is a parameter of its own: a kernel that writes to its LineAxis, whose
// radices are indexed, keeps all of it in local memory.
__device__ __forceinline__ void load_line_twiddles(float2* tw, const float2* table, int m) {
  for (int i = threadIdx.x; i < m; i += blockDim.x) tw[i] = __ldg(table + i);
}

}  // namespace lgx
