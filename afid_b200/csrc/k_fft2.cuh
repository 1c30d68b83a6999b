// Two-pass transforms along y and z (the r2c, c2c and c2r steps of
// SolvePressureCorrection.F90:97-148) for lines of N = R1 R2 points with both
// radices at most 32.
//
// A line is two Stockham passes: R2 butterflies of radix R1, one exchange
// through shared memory, R1 butterflies of radix R2.  A thread holds one
// butterfly in registers with all its inputs in flight at once.  z reads and writes
// HBM in the butterflies: a tile costs one load latency, one exchange and two
// barriers.  y forward reads so and goes through shared memory once more, to part
// the two rows of a line; y inverse stages its lines there first, from
// coefficients read once (f2_lines_in); both take four barriers.  The four blocks
// of an SM (three with a radix above 16, two at 960 and 1024 points, whose buffers
// take 77 and 82 KB; a launch sizes them for its longest lines) are in different phases and
// cover each other's loads.  HBM traffic bounds the transforms (32 bytes per complex
// value); below that, what a tile waits for: loads, exchange, barriers.
//
// The tile kernels of k_fft.cuh, which these replace for such lines, make a pass per
// radix <= 16 over a staged tile with two barriers each.  Per step, y forward, z twice
// and y inverse, tile kernels against these: 75x150x135 0.41 and 0.21 ms, 192x384x384
// 2.11 and 1.46, 384x768x768 14.7 and 12.1, 16x1024x1024 1.69 and 1.17; and against
// warp-per-line kernels with 8 or 12 values a lane (three passes at 128 points),
// 64-box ensemble 1.86 and 1.53, 32x32x32 0.123 and 0.103, but 48 boxes of 64^3
// 0.73 and 0.82 and of 32^3 0.22 and 0.27: their 33 and 17 ky fill a z tile of 16
// badly.
//
// The exchange stores value r of butterfly j at row r, column j of a
// R1 x (R2 | 1) array per line: the writes of a pass run along a row, the reads
// down columns whose pitch is odd, so neither meets bank conflicts.  The
// twiddles exp(-2 pi i r j / N) are kept in the order pass two reads them.
#pragma once
#include "k_fft.cuh"

namespace afid {

// cos and sin of 2 pi p / q at compile time, rounded once: the series on at most
// pi/4 runs in pairs of doubles (Dekker's sums and products), since in doubles a
// third of the roots came out up to 1.1 units in the last place off.
struct F2Pair { double hi, lo; };
constexpr F2Pair f2_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
constexpr F2Pair f2_prod(double a, double b) {
  const double S = 134217729.0;                  // 2^27 + 1
  const double p = a * b, ca = S * a, cb = S * b;
  const double ah = ca - (ca - a), al = a - ah, bh = cb - (cb - b), bl = b - bh;
  return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr F2Pair f2_add(F2Pair a, F2Pair b) {
  const F2Pair s = f2_sum(a.hi, b.hi);
  return f2_sum(s.hi, s.lo + (a.lo + b.lo));
}
constexpr F2Pair f2_mul(F2Pair a, F2Pair b) {
  const F2Pair p = f2_prod(a.hi, b.hi);
  return f2_sum(p.hi, p.lo + (a.hi * b.lo + a.lo * b.hi));
}
constexpr F2Pair f2_div(F2Pair a, double n) {
  const double q = a.hi / n;
  const F2Pair p = f2_prod(q, n);
  return f2_sum(q, ((a.hi - p.hi) - p.lo + a.lo) / n);
}
constexpr double f2_series(F2Pair x, bool sine) {
  F2Pair term = sine ? x : F2Pair{1.0, 0.0}, sum = term;
  const F2Pair x2 = f2_mul(x, x);
  for (int n = 0; n < 13; ++n) {
    const int a = 2 * n + (sine ? 2 : 1);
    term = f2_div(f2_mul(term, x2), -(double)a * (double)(a + 1));
    sum = f2_add(sum, term);
  }
  return sum.hi;
}
// 2 pi p / q
constexpr F2Pair f2_angle(int p, int q) {
  return f2_div(f2_mul(F2Pair{6.283185307179586, 2.4492935982947064e-16}, F2Pair{(double)p, 0.0}), (double)q);
}
constexpr double f2_cos(int p, int q) {
  p %= q;
  if (2 * p > q) p = q - p;
  if (4 * p > q) return -f2_cos(q - 2 * p, 2 * q);
  if (8 * p > q) return f2_series(f2_angle(q - 4 * p, 4 * q), true);
  return f2_series(f2_angle(p, q), false);
}
constexpr double f2_sin(int p, int q) { return f2_cos((p % q) * 4 + 3 * q, 4 * q); }   // cos(t - pi/2)
// the worst of a series in doubles
static_assert(f2_cos(4, 15) == -0.10452846326765347 && f2_cos(7, 25) == -0.18738131458572463 && f2_sin(1, 15) == 0.4067366430758002 &&
              f2_cos(7, 30) == 0.10452846326765347 && f2_cos(1, 9) == 0.766044443118978 && f2_cos(8, 27) == -0.28680323271109026 &&
              f2_sin(1, 32) == 0.19509032201612828, "roots of unity");

template <int R>
struct F2Roots {
  double c[R], s[R];
  constexpr F2Roots() : c(), s() {
    for (int m = 0; m < R; ++m) {
      c[m] = f2_cos(m, R);
      s[m] = f2_sin(m, R);
    }
  }
};

// a (wr + i wi)
__device__ __forceinline__ double2 f2_mulc(double2 a, double wr, double wi) {
  return make_double2(__fma_rn(a.x, wr, -(a.y * wi)), __fma_rn(a.x, wi, a.y * wr));
}

// R-point DFT in registers, natural order in and out: the small radices of
// k_fft.cuh, composites as A x B (B-point DFTs over v[n1 + A n2], roots
// W_R^(n1 k2), A-point DFTs over n1 giving X[k2 + B k1]).
template <int R, int SGN>
__device__ __forceinline__ void f2_dft(double2 (&v)[R]);

template <int A, int B, int SGN>
__device__ __forceinline__ void f2_comp(double2 (&v)[A * B]) {
  constexpr F2Roots<A * B> w{};
  double2 y[A * B];
#pragma unroll
  for (int n1 = 0; n1 < A; ++n1) {
    double2 u[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) u[n2] = v[n1 + A * n2];
    f2_dft<B, SGN>(u);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2)
      y[n1 * B + k2] = n1 * k2 ? f2_mulc(u[k2], w.c[n1 * k2 % (A * B)], SGN * w.s[n1 * k2 % (A * B)]) : u[k2];
  }
#pragma unroll
  for (int k2 = 0; k2 < B; ++k2) {
    double2 u[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) u[n1] = y[n1 * B + k2];
    f2_dft<A, SGN>(u);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) v[k2 + B * k1] = u[k1];
  }
}

template <int R, int SGN>
__device__ __forceinline__ void f2_dft(double2 (&v)[R]) {
  if constexpr (R == 9) f2_comp<3, 3, SGN>(v);
  else if constexpr (R == 10) f2_comp<2, 5, SGN>(v);
  else if constexpr (R == 15) f2_comp<3, 5, SGN>(v);
  else if constexpr (R == 18) f2_comp<3, 6, SGN>(v);
  else if constexpr (R == 20) f2_comp<4, 5, SGN>(v);
  else if constexpr (R == 24) f2_comp<3, 8, SGN>(v);
  else if constexpr (R == 25) f2_comp<5, 5, SGN>(v);
  else if constexpr (R == 27) f2_comp<3, 9, SGN>(v);
  else if constexpr (R == 30) f2_comp<5, 6, SGN>(v);
  else if constexpr (R == 32) f2_comp<4, 8, SGN>(v);
  else dft_small<R, SGN>(v, nullptr, R);   // 2..6, 8, 12, 16
}

constexpr int F2_T = 128;            // threads per block
// Radices by class: 0 has both at most 16 (four blocks per SM, 128 registers a
// thread), 1 the larger one above 16 (at most three blocks, 168 registers).
__host__ __device__ constexpr int f2_blocks(int cls) { return cls ? 3 : 4; }
// lines per tile: z takes a power of two of neighbouring ky, y any number
__host__ __device__ __forceinline__ int f2_lines(int r1, int r2, bool z) {
  const int l = F2_T / (r1 > r2 ? r1 : r2);
  if (!z) return l;
  int p = 1;
  while (2 * p <= l && p < 16) p *= 2;
  return p;
}
__host__ __device__ __forceinline__ int f2_exchange(int r1, int r2, int lines) { return lines * r1 * (r2 | 1); }

enum { F2_YF = 0, F2_YI = 1, F2_Z = 2 };

// the tile a block works on
struct F2Tile {
  int N, r1, r2, pitch, L, lgL, nh, nzm, row0, nrow;   // y: first row and rows of the tile; z: first ky in row0
  double *phi;        // plane k of dph
  double2 *spec;      // plane k of the spectrum
};

template <int KIND>
__device__ __forceinline__ void f2_split(const F2Tile &T, int per, int t, int &l, int &j) {
  if constexpr (KIND == F2_Z) {
    l = t & (T.L - 1);
    j = t >> T.lgL;
  } else {
    l = t / per;
    j = t - l * per;
  }
}
template <int KIND>
__device__ __forceinline__ bool f2_active(const F2Tile &T, int per, int l, int j) {
  return KIND == F2_Z ? j < per : l < T.L;
}
// exchange index of row r, column c of line l
template <int KIND>
__device__ __forceinline__ int f2_idx(const F2Tile &T, int l, int r, int c) {
  return KIND == F2_Z ? ((r * T.pitch + c) << T.lgL) + l : (l * T.r1 + r) * T.pitch + c;
}

// The walk of the block's threads over the values q < nh of the tile's lines
// with rows in the box (the half spectra of the y transforms).
struct F2Walk {
  int l, q;
  __device__ __forceinline__ explicit F2Walk(const F2Tile &T) : l(0), q(threadIdx.x) { wrap(T); }
  __device__ __forceinline__ void wrap(const F2Tile &T) {
    while (q >= T.nh) { q -= T.nh; ++l; }
  }
  __device__ __forceinline__ void next(const F2Tile &T) { q += F2_T; wrap(T); }
  __device__ __forceinline__ bool in(const F2Tile &T) const { return 2 * l < T.nrow; }
};

// Inverse y: the complex lines Z = A + i B of the half-spectrum rows A and B of
// each line, with the Hermitian extension (imaginary parts at ky = 0 and
// ky = N/2 ignored as in a c2r transform), value n of line l to ex[l N + n].
// Each coefficient is read once; read by the butterflies themselves (twice,
// for n and N - n), the transform of 384 points took 0.58 ms against 0.36.
template <int CLS>
__device__ __forceinline__ void f2_lines_in(const F2Tile &T, double2 *ex) {
  constexpr int U = CLS ? 2 : 4;      // rows' values in flight a thread (4 spill beside the large radices)
  F2Walk w(T);
  bool first = true;
  while (first || w.in(T)) {
    double2 a[U], b[U];
    int at[U], mirror[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      at[u] = -1;
      if (w.in(T)) {
        const double2 *row = T.spec + (long long)(T.row0 + 2 * w.l) * T.nh + w.q;
        a[u] = __ldcg(row);
        b[u] = 2 * w.l + 1 < T.nrow ? __ldcg(row + T.nh) : make_double2(0.0, 0.0);
        at[u] = w.l * T.N + w.q;
        mirror[u] = w.q == 0 || 2 * w.q == T.N ? -1 : w.l * T.N + T.N - w.q;
      }
      w.next(T);
    }
    if (first) __syncthreads();          // the previous tile's exchange has been read
    first = false;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) {
        if (mirror[u] < 0) a[u].y = b[u].y = 0.0;
        ex[at[u]] = make_double2(a[u].x - b[u].y, a[u].y + b[u].x);
        if (mirror[u] >= 0) ex[mirror[u]] = make_double2(a[u].x + b[u].y, b[u].x - a[u].y);
      }
  }
  __syncthreads();
}

template <int R, int KIND, int SGN>
__device__ __forceinline__ void f2_first(const F2Tile &T, double2 *ex) {
  int l, j;
  f2_split<KIND>(T, T.r2, threadIdx.x, l, j);
  const bool act = f2_active<KIND>(T, T.r2, l, j);
  double2 v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = make_double2(0.0, 0.0);
  if (act) {
    if constexpr (KIND == F2_Z) {
      const double2 *src = T.spec + (long long)j * T.nh + T.row0 + l;
      const long long st = (long long)T.r2 * T.nh;
      if (T.row0 + l < T.nh) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = __ldcg(src + r * st);
      }
    } else if constexpr (KIND == F2_YF) {
      const double *a = T.phi + (long long)(T.row0 + 2 * l) * T.N + j;
      if (2 * l < T.nrow) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r].x = __ldcg(a + r * T.r2);
      }
      if (2 * l + 1 < T.nrow) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r].y = __ldcg(a + T.N + r * T.r2);
      }
    } else {
      if (2 * l < T.nrow) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ex[l * T.N + j + r * T.r2];
      }
    }
    f2_dft<R, SGN>(v);
  }
  __syncthreads();          // the previous tile's exchange (inverse y: this tile's lines) has been read
  if (act) {
#pragma unroll
    for (int r = 0; r < R; ++r) ex[f2_idx<KIND>(T, l, r, j)] = v[r];
  }
}

template <int R, int KIND, int SGN>
__device__ __forceinline__ void f2_second(const F2Tile &T, double2 *ex, const double2 *tws) {
  int l, j;
  f2_split<KIND>(T, T.r1, threadIdx.x, l, j);
  const bool act = f2_active<KIND>(T, T.r1, l, j);
  double2 v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = make_double2(0.0, 0.0);
  if (act) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ex[f2_idx<KIND>(T, l, j, r)];
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const double2 w = tws[r * T.r1 + j];
      v[r] = f2_mulc(v[r], w.x, SGN > 0 ? -w.y : w.y);
    }
    f2_dft<R, SGN>(v);
    if constexpr (KIND == F2_Z) {
      double2 *dst = T.spec + (long long)j * T.nh + T.row0 + l;
      const long long st = (long long)T.r1 * T.nh;
      if (T.row0 + l < T.nh) {
#pragma unroll
        for (int r = 0; r < R; ++r) __stcg(dst + r * st, v[r]);
      }
    } else if constexpr (KIND == F2_YI) {
      double *a = T.phi + (long long)(T.row0 + 2 * l) * T.N + j;
      if (2 * l < T.nrow) {
#pragma unroll
        for (int r = 0; r < R; ++r) __stcg(a + r * T.r1, v[r].x);
      }
      if (2 * l + 1 < T.nrow) {
#pragma unroll
        for (int r = 0; r < R; ++r) __stcg(a + T.N + r * T.r1, v[r].y);
      }
    }
  }
  if constexpr (KIND == F2_YF) {
    // value q of line l to ex[l N + q], then the two half spectra of each
    // line: A = (Z_q + conj Z_{N-q}) / 2, B = (Z_q - conj Z_{N-q}) / (2i)
    __syncthreads();
    if (act) {
#pragma unroll
      for (int r = 0; r < R; ++r) ex[l * T.N + j + r * T.r1] = v[r];
    }
    __syncthreads();
    for (F2Walk w(T); w.in(T); w.next(T)) {
      const double2 *z = ex + w.l * T.N;
      const double2 zq = z[w.q], zn = z[w.q ? T.N - w.q : 0];
      double2 *a = T.spec + (long long)(T.row0 + 2 * w.l) * T.nh + w.q;
      __stcg(a, make_double2((zq.x + zn.x) * 0.5, (zq.y - zn.y) * 0.5));
      if (2 * w.l + 1 < T.nrow) __stcg(a + T.nh, make_double2((zq.y + zn.y) * 0.5, (zn.x - zq.x) * 0.5));
    }
  }
}

// Tiles a block takes in a row.  z: one, so that neighbouring blocks work on
// neighbouring ky of the same rows at the same time.
__device__ __forceinline__ int f2_run_log2(int kind, int total) {
  return kind == F2_Z ? 0 : run_log2(total, (int)gridDim.x);
}

#define F2_RADICES_A(X) X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16)
#define F2_RADICES_B(X) X(18) X(20) X(24) X(25) X(27) X(30) X(32)

// Transforms of class CLS (radices r1 <= r2; see f2_blocks) of the launch's
// tiles; ``ex_len``: complex values of the exchange buffer (the twiddles
// follow it).
template <int KIND, int SGN, int CLS>
__global__ void __launch_bounds__(F2_T, f2_blocks(CLS)) k_fft2(BatchDev bt, int ns, int ex_len, int total) {
  extern __shared__ double2 f2sm[];
  double2 *const ex = f2sm, *const tws = f2sm + ex_len;
  const int lgr = f2_run_log2(KIND, total);
  const TileRange rg(total, lgr);
  if (rg.first() >= total) return;
  TileWalk wk(bt, rg.first());
  int loaded = -1, groups = 1;
  bool run = false;
  F2Tile T;
  double *phi = nullptr;
  double2 *spec = nullptr;
  long long plane = 0;
  for (int t = rg.first(); t < total; t = rg.next(t)) {
    const int lt = wk.to(bt, t);
    if (wk.b != loaded) {
      const BoxDev *B = bt.boxes + wk.b;
      loaded = wk.b;
      T.nzm = __ldg(&B->nzm);
      T.nh = __ldg(&B->nymh);
      T.N = KIND == F2_Z ? T.nzm : __ldg(&B->nym);
      T.r1 = __ldg(KIND == F2_Z ? &B->fz2[0] : &B->fy2[0]);
      T.r2 = __ldg(KIND == F2_Z ? &B->fz2[1] : &B->fy2[1]);
      T.pitch = T.r2 | 1;
      T.L = f2_lines(T.r1, T.r2, KIND == F2_Z);
      T.lgL = ilog2(T.L);
      groups = KIND == F2_Z ? (T.nh + T.L - 1) / T.L : (T.nzm + 2 * T.L - 1) / (2 * T.L);
      phi = (double *)__ldg((const unsigned long long *)&B->phi);
      spec = (double2 *)__ldg((const unsigned long long *)&B->spec);
      plane = __ldg(&B->plane);
      const double2 *tw = (const double2 *)__ldg((const unsigned long long *)(KIND == F2_Z ? &B->twz : &B->twy));
      __syncthreads();     // the previous box's twiddles have been read
      for (int q = threadIdx.x; q < T.N; q += F2_T) {
        const int r = q / T.r1, j = q - r * T.r1;
        tws[q] = __ldg(tw + r * j);
      }
      run = __syncthreads_and(__ldg(&B->active) && ns < __ldg(&B->nsst) &&
                              *(volatile int *)&((BoxScalars *)__ldg((const unsigned long long *)&B->sc))->status == 0);
    }
    if (!run) continue;
    const int k = lt / groups, g = lt - k * groups;
    T.phi = phi + (long long)k * plane;
    T.spec = spec + (long long)k * T.nzm * T.nh;
    T.row0 = g * T.L * (KIND == F2_Z ? 1 : 2);
    T.nrow = min(2 * T.L, T.nzm - T.row0);
#define F2_FIRST(R) case R: f2_first<R, KIND, SGN>(T, ex); break;
#define F2_SECOND(R) case R: f2_second<R, KIND, SGN>(T, ex, tws); break;
    if constexpr (KIND == F2_YI) f2_lines_in<CLS>(T, ex);
    if constexpr (CLS == 0) {
      switch (T.r1) { F2_RADICES_A(F2_FIRST) }
      __syncthreads();
      switch (T.r2) { F2_RADICES_A(F2_SECOND) }
    } else {
      switch (T.r1) { F2_RADICES_A(F2_FIRST) F2_RADICES_B(F2_FIRST) }
      __syncthreads();
      switch (T.r2) { F2_RADICES_B(F2_SECOND) }
    }
  }
}

}  // namespace afid
