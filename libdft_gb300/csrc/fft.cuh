// 3-D FFT building blocks for sm_103a (header-only templates).
//
// A 3-D transform of an [nx][ny][nz] grid runs as three line passes:
//   z pass  rows (x,y) are contiguous in real space; the output is written
//           transposed into the spectral layout [kz][x][y]
//   y pass  lines along y are contiguous in [kz][x][y]
//   x pass  pencils along x (stride ny); B consecutive y per CTA, so every
//           global access is a contiguous run of B complex values.
// Real fields use the half spectrum (kz = 0..nz/2) produced by packing a real
// row of length nz into nz/2 complex values (even + i odd), one FFT of length
// nz/2 and a twiddle post-processing step; the inverse does the reverse.
//
// The generic line pass (any 2^a 3^b 5^c length, and all of FP64) runs a
// Stockham autosort FFT over a tile of B lines with the butterflies in
// registers (radices 16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2): the first stage
// loads from global memory, the last one stores to it, and shared memory
// carries the line between stages.  Loads and
// stores go through functors, which is where pointwise producers (|psi|^2,
// products of fields, phase factors) and consumers (accumulate into the
// potential) are fused.  Twiddles come from per-length tables computed in
// FP64 on the host and rounded once to the bulk precision.
#pragma once

#include <string.h>

#include <type_traits>

#include <atomic>

#include "common.cuh"
#include "fast_fft.cuh"

namespace dftgpu {

constexpr int FFT_THREADS = 256;
constexpr int FFT_MAX_STAGES = 16;
constexpr int FFT_MAX_N = 1024;      // grid dimension (3-D grids)
constexpr int FFT_MAX_LINE = 4096;   // z of a 1-D grid (nx = ny = 1); transform lengths up to this

template <typename T> struct FftPlan {
  int n;                       // transform length
  int nst;                     // number of stages
  int radix[FFT_MAX_STAGES];
  const typename cplx_t<T>::type *tw;   // tw[t] = exp(-2 pi i t / n), t < n; FP64: tw[n + t] = its (cos, tan)
};
// entries of a plan's table
template <typename T> constexpr size_t plan_table(size_t n) { return sizeof(T) == 8 ? 2 * n : n; }
// The tangent of a table entry.  A cosine that rounds to zero gets a tiny one
// in its place, so that cos * tan is still the sine.
__host__ __device__ __forceinline__ double2 cos_tan(double c, double s) {
  if (c == 0.0) c = 1e-30;
  double2 r; r.x = c; r.y = s / c;
  return r;
}

// Radices of a 2^a 3^b 5^c length (DFTGPU_ERR_SIZE otherwise).
int fft_radices(int n, int prec, bool small, int *radix, int *nst);
// Host: build (and cache) the plan for length n in precision T.  small: the
// FP64 variant with radices up to 5.
template <typename T> int get_plan(int n, FftPlan<T> *plan, bool small = false);
// FP64 passes of up to 2^19 values run with the small radices: their kernels
// are over in microseconds and mostly wait for their straight-line code to
// arrive, and four radix-4 stages take 22 operations an element where two of
// radix 16 take 21.  Measured on full potentials, radices up to 5 against up
// to 16 (us): 32^3 291 / 365, 64^3 517 / 541, 96 x 90 x 80 1452 / 1493, 128^3
// (2^20 values a pass) 3259 / 3230, 160 x 150 x 144 7971 / 7295.
inline bool small_pass(int n, int na, int nb) { return (size_t) n * na * nb <= (size_t) 1 << 19; }

// ------------------------------------------------------------ butterflies
template <typename C, typename T>
__device__ __forceinline__ void dft2(C &a, C &b) { C t = a; a = t + b; b = t - b; }

// v * exp(s i 2 pi m / R) given (cos, sin) of 2 pi m / R
template <typename C, typename T> __device__ __forceinline__ C rot_cs(C v, T c, T sn, T s) {
  const T si = s * sn;
  C r; r.x = v.x * c - v.y * si; r.y = v.x * si + v.y * c;
  return r;
}

template <int R, typename C, typename T> __device__ __forceinline__ void small_dft(C *u, T s);

// Prime-factor radix R = R1 R2 (gcd 1, Good-Thomas): input n = (A1 n1 + A2 n2)
// mod R, output k = (K1 k1 + K2 k2) mod R with K1 = 1 (mod R1), 0 (mod R2)
// and K2 = 0 (mod R1), 1 (mod R2); no twiddles between the two layers.
template <int R1, int R2, int A1, int A2, int K1, int K2, typename C, typename T>
__device__ __forceinline__ void pfa_dft(C *u, T s) {
  constexpr int R = R1 * R2;
  C y[R2][R1];
#pragma unroll
  for (int n2 = 0; n2 < R2; n2++) {
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) y[n2][n1] = u[(A1 * n1 + A2 * n2) % R];
    small_dft<R1, C, T>(y[n2], s);
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) {
    C z[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) z[n2] = y[n2][k1];
    small_dft<R2, C, T>(z, s);
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) u[(K1 * k1 + K2 * k2) % R] = z[k2];
  }
}

// R-point DFT in place, natural order; s = -1 forward, +1 inverse.  Radices 2,
// 3, 4, 5 directly, 9 as 3 x 3 with its internal twiddles, 6, 10, 12, 15 as
// prime-factor pairs; a stage of radix 2, 4, 8 or 16 is poly_eval() below.
template <int R, typename C, typename T>
__device__ __forceinline__ void small_dft(C *u, T s) {
  if constexpr (R == 2) {
    dft2<C, T>(u[0], u[1]);
  } else if constexpr (R == 3) {
    const T s3 = (T) 0.86602540378443864676;
    C a = u[0], b = u[1], c = u[2];
    C m = a - (b + c) * (T) 0.5;
    C d = (b - c) * s3;
    u[0] = a + b + c;
    u[1] = m + imul<C, T>(d, s);
    u[2] = m - imul<C, T>(d, s);
  } else if constexpr (R == 4) {
    C t0 = u[0] + u[2], t1 = u[0] - u[2], t2 = u[1] + u[3], t3 = u[1] - u[3];
    u[0] = t0 + t2;
    u[2] = t0 - t2;
    u[1] = t1 + imul<C, T>(t3, s);
    u[3] = t1 - imul<C, T>(t3, s);
  } else if constexpr (R == 5) {
    const T c1 = (T) 0.30901699437494742410, c2 = (T) -0.80901699437494742410;
    const T s1 = (T) 0.95105651629515357212, s2 = (T) 0.58778525229247312917;
    C a = u[0];
    C t1 = u[1] + u[4], t2 = u[2] + u[3], t3 = u[1] - u[4], t4 = u[2] - u[3];
    C m1 = a + t1 * c1 + t2 * c2;
    C m2 = a + t1 * c2 + t2 * c1;
    C n1 = t3 * s1 + t4 * s2;
    C n2 = t3 * s2 - t4 * s1;
    u[0] = a + t1 + t2;
    u[1] = m1 + imul<C, T>(n1, s);
    u[4] = m1 - imul<C, T>(n1, s);
    u[2] = m2 + imul<C, T>(n2, s);
    u[3] = m2 - imul<C, T>(n2, s);
  } else if constexpr (R == 9) {
    // 3 x 3 with twiddles W9^(n2 k1): (n2, k1) = (1,1), (1,2), (2,1): m = 1, 2; (2,2): m = 4
    const T ca = (T) 0.766044443118978035202, sa = (T) 0.642787609686539326323;
    const T cb = (T) 0.173648177666930348852, sb = (T) 0.984807753012208059367;
    const T cd = (T) -0.939692620785908384054, sd = (T) 0.342020143325668733044;
    C y[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < 3; n1++) y[n2][n1] = u[3 * n1 + n2];
      small_dft<3, C, T>(y[n2], s);
    }
    y[1][1] = rot_cs<C, T>(y[1][1], ca, sa, s); y[1][2] = rot_cs<C, T>(y[1][2], cb, sb, s);
    y[2][1] = rot_cs<C, T>(y[2][1], cb, sb, s); y[2][2] = rot_cs<C, T>(y[2][2], cd, sd, s);
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++) {
      C z[3] = { y[0][k1], y[1][k1], y[2][k1] };
      small_dft<3, C, T>(z, s);
#pragma unroll
      for (int k2 = 0; k2 < 3; k2++) u[k1 + 3 * k2] = z[k2];
    }
  } else if constexpr (R == 6) {
    pfa_dft<2, 3, 3, 2, 3, 4, C, T>(u, s);
  } else if constexpr (R == 10) {
    pfa_dft<2, 5, 5, 2, 5, 6, C, T>(u, s);
  } else if constexpr (R == 12) {
    pfa_dft<4, 3, 3, 4, 9, 4, C, T>(u, s);
  } else if constexpr (R == 15) {
    pfa_dft<3, 5, 5, 3, 10, 6, C, T>(u, s);
  }
}

// A radix-R butterfly of power-of-two R as polynomial evaluation: the R outputs
// are P(z_j) = sum_q u_q z_j^q at z_j = w omega_R^j, and by even / odd halves
//   P(z_j), P(z_{j+M/2}) = E(z_j^2) +- z_j O(z_j^2),
// so each level is one complex a +- z b and the stage twiddle w is part of z.
// The table values read are 1 + 1 + 2 + 4 for R = 16 (z_{j+M/4} = -i z_j):
// w^{R/M} omega_M^j, j < M/4, for M = 2, 4, 8, 16.
// FP64: z = c (1 + i r) with c = cos, r = tan of its angle, so that
// t = (b.x - r b.y, b.y + r b.x) and a +- c t take six operations where a
// product by the twiddle followed by the sums takes eight, with two roundings
// on the way to each output instead of three (t.x c is Re(z b) to one
// rounding whatever the size of r).  FP32 keeps (cos, sin) pairs rounded to the
// unit circle and forms z b before the sums: eight operations like two FMAs on
// each sum, but one rounding instead of two at the size of a, which is the
// larger one in a smooth field's line (round trip of one at n = 128 1.08e-7
// against 1.13e-7).  Its untwiddled constants
// scale the norm by a fixed amount a transform (1/sqrt(2) and the pair of
// pi/8 are below the circle, radix 5 above it): with every c1 as it rounds
// radix 16 lowers it by 2.7e-8, with one of the four rounded up by 2.0e-8,
// which brings lengths 240, 160 and 80 from -2.1e-8, -9.1e-9 and -5.3e-9 to
// -1.4e-8, -2.3e-9 and below 1e-9 (all four up: 80 and 160 at +2e-8).
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

__device__ __forceinline__ void bf_z(float2 &a, float2 &b, float2 z) {   // (a + z b, a - z b)
  const float2 t = a, v = b;
  const float px = fmaf(z.x, v.x, -(z.y * v.y)), py = fmaf(z.x, v.y, z.y * v.x);
  a.x = t.x + px; a.y = t.y + py;
  b.x = t.x - px; b.y = t.y - py;
}
__device__ __forceinline__ void bf_miz(float2 &a, float2 &b, float2 z) {   // with -i z for z
  bf_z(a, b, make_float2(z.y, -z.x));
}
__device__ __forceinline__ void bf_z(double2 &a, double2 &b, double2 z) {   // z = z.x (1 + i z.y)
  const double tx = fma(-z.y, b.y, b.x), ty = fma(z.y, b.x, b.y);
  b.x = fma(-z.x, tx, a.x);
  b.y = fma(-z.x, ty, a.y);
  a.x = fma(z.x, tx, a.x);
  a.y = fma(z.x, ty, a.y);
}
__device__ __forceinline__ void bf_miz(double2 &a, double2 &b, double2 z) {
  const double tx = fma(-z.y, b.y, b.x), ty = fma(z.y, b.x, b.y);
  b.x = fma(-z.x, ty, a.x);
  b.y = fma(z.x, tx, a.y);
  a.x = fma(z.x, ty, a.x);
  a.y = fma(-z.x, tx, a.y);
}
template <typename C> __device__ __forceinline__ void bf_1(C &a, C &b) { const C t = a; a = t + b; b = t - b; }
template <typename C> __device__ __forceinline__ void bf_mi(C &a, C &b) {          // z = -i
  const C t = a, v = b;
  a.x = t.x + v.y; a.y = t.y - v.x;
  b.x = t.x - v.y; b.y = t.y + v.x;
}
// z = exp(-i pi/4) (Q = 0) or -i times it (Q = 1)
template <int Q, typename C> __device__ __forceinline__ void bf_8th(C &a, C &b) {
  typedef decltype(a.x) T;
  const T h = (T) 0.70710678118654752440;
  const C t = a;
  const T s = b.x + b.y, d = b.y - b.x;
  if (Q == 0) {            // z b = h (b.x + b.y, b.y - b.x)
    a.x = fma_t(h, s, t.x); a.y = fma_t(h, d, t.y);
    b.x = fma_t(-h, s, t.x); b.y = fma_t(-h, d, t.y);
  } else {                 // -i z b = h (b.y - b.x, -(b.x + b.y))
    a.x = fma_t(h, d, t.x); a.y = fma_t(-h, s, t.y);
    b.x = fma_t(-h, d, t.x); b.y = fma_t(h, s, t.y);
  }
}

// level tables of a twiddled butterfly: z2; z4; z8[0..1]; z16[0..3]
template <int R, typename C> struct PolyTw {
  C z[R == 2 ? 1 : R == 4 ? 2 : R == 8 ? 4 : 8];
};

// x[q S], q < M, in place of a register array u; result order j in y[0..M-1]
template <int M, int S, bool TW, int R, typename C>
__device__ __forceinline__ void poly_eval(const C *u, C *y, const PolyTw<R, C> &w) {
  if constexpr (M == 1) {
    y[0] = u[0];
  } else {
    C e[M / 2], o[M / 2];
    poly_eval<M / 2, 2 * S, TW, R, C>(u, e, w);
    poly_eval<M / 2, 2 * S, TW, R, C>(u + S, o, w);
#pragma unroll
    for (int j = 0; j < M / 2; j++) {
      if constexpr (TW) {
        constexpr int off = M == 2 ? 0 : M == 4 ? 1 : M == 8 ? 2 : 4, Q = M / 4;
        if (M == 2 || j < Q) bf_z(e[j], o[j], w.z[off + (M == 2 ? 0 : j)]);
        else bf_miz(e[j], o[j], w.z[off + j - Q]);
      } else {
        if (j == 0) bf_1(e[j], o[j]);
        else if (4 * j == M) bf_mi(e[j], o[j]);
        else if (8 * j == M) bf_8th<0>(e[j], o[j]);
        else if (8 * j == 3 * M) bf_8th<1>(e[j], o[j]);
        else {             // M = 16, odd j: exp(-2 pi i j / 16)
          C z;
          if constexpr (sizeof(e[0].x) == 4) {   // (cos, sin); one of the four c1 rounded up (below)
            if (j == 1 || j == 5) { z.x = j == 1 ? ff::FF_C1B : ff::FF_C1; z.y = -ff::FF_S1; } else { z.x = ff::FF_S1; z.y = -ff::FF_C1; }
          } else {                               // (cos, tan) of -pi/8 and -3 pi/8: tan(pi/8) = sqrt(2) - 1
            if (j == 1 || j == 5) { z.x = 0.923879532511286756128; z.y = -0.414213562373095048802; }
            else { z.x = 0.382683432365089771728; z.y = -2.414213562373095048802; }
          }
          if (j < 4) bf_z(e[j], o[j], z); else bf_miz(e[j], o[j], z);
        }
      }
      y[j] = e[j];
      y[j + M / 2] = o[j];
    }
  }
}

__host__ __device__ constexpr bool is_pow2(int r) { return (r & (r - 1)) == 0; }

// Forward R-point DFT of u_q w^q, w = exp(-2 pi i kt / n), in natural order;
// TW = false: w = 1.  tw: the plan's table of 2n (FP64) or n (FP32) entries.
template <int R, bool TW, typename T>
__device__ __forceinline__ void stage_dft(typename cplx_t<T>::type (&u)[R], int kt, int n,
                                          const typename cplx_t<T>::type *__restrict__ tw) {
  typedef typename cplx_t<T>::type C;
  if constexpr (is_pow2(R)) {
    PolyTw<R, C> w;
    if constexpr (TW) {
      if constexpr (sizeof(T) == 8) tw += n;   // the (cos, tan) half
      w.z[0] = __ldg(&tw[kt * (R / 2)]);
      if constexpr (R >= 4) w.z[1] = __ldg(&tw[kt * (R / 4)]);
      if constexpr (R >= 8) { w.z[2] = __ldg(&tw[kt * (R / 8)]); w.z[3] = __ldg(&tw[kt * (R / 8) + n / 8]); }
      if constexpr (R >= 16)
#pragma unroll
        for (int j = 0; j < 4; j++) w.z[4 + j] = __ldg(&tw[kt + j * (n / 16)]);
    }
    C y[R];
    poly_eval<R, 1, TW, R, C>(u, y, w);
#pragma unroll
    for (int q = 0; q < R; q++) u[q] = y[q];
  } else {
    if constexpr (TW) {
#pragma unroll
      for (int q = 1; q < R; q++) u[q] = cmul(u[q], __ldg(&tw[q * kt]));
    }
    small_dft<R, C, T>(u, (T) -1);
  }
}

// i / d and i % d for i < 65536 by one multiplication (m = ceil(2^32 / d))
struct FastDiv {
  unsigned d, m;
  __device__ __forceinline__ FastDiv(int d_) : d(d_), m(d_ > 1 ? 0xffffffffu / (unsigned) d_ + 1u : 0u) {}
  __device__ __forceinline__ void divmod(int i, int &q, int &r) const {
    q = d > 1 ? (int) __umulhi((unsigned) i, m) : i;
    r = i - q * (int) d;
  }
};

// Tile geometry of the line kernels: nl lines of length n, line l at l * LP,
// element e at e + e/16 (the odd line pitch and the skew keep line-fast and
// element-fast accesses off each other's banks).
struct Tile {
  int n, B, logB, nl, LP;
  __host__ __device__ static constexpr int pitch(int n) { return (n + (n >> 4)) | 1; }
  __device__ __forceinline__ int at(int l, int e) const { return l * LP + e + (e >> 4); }
};

// One stage over the tile: butterfly i of line l takes rd(l, i + q n/R) and
// gives wr(l, j + q p), j = (i - k) R + k, k = i mod p.  EF: consecutive
// threads take consecutive butterflies of a line, else consecutive lines.
// FIRST: p = 1, no twiddles.
template <int R, bool FIRST, typename T, class Rd, class Wr>
__device__ __forceinline__ void tile_stage(const Tile &g, int ef, int p, const typename cplx_t<T>::type *__restrict__ tw,
                                           const Rd &rd, const Wr &wr) {
  typedef typename cplx_t<T>::type C;
  const int nR = g.n / R, twstep = FIRST ? 0 : g.n / (p * R);
  const FastDiv byn(nR), byp(FIRST ? 1 : p);
  for (int idx = threadIdx.x; idx < g.B * nR; idx += blockDim.x) {
    int l, i;
    if (ef) byn.divmod(idx, l, i);
    else { l = idx & (g.B - 1); i = idx >> g.logB; }
    if (l >= g.nl) continue;
    C u[R];
#pragma unroll
    for (int q = 0; q < R; q++) u[q] = rd(l, i + q * nR);
    int k = 0, quo;
    if (!FIRST) byp.divmod(i, quo, k);
    (void) quo;
    stage_dft<R, !FIRST, T>(u, k * twstep, g.n, tw);
    const int j = (i - k) * R + k;
#pragma unroll
    for (int q = 0; q < R; q++) wr(l, j + q * p, u[q]);
  }
}
template <bool FIRST, typename T, class Rd, class Wr>
__device__ __forceinline__ void run_stage(int R, const Tile &g, int ef, int p,
                                          const typename cplx_t<T>::type *__restrict__ tw, const Rd &rd, const Wr &wr) {
  switch (R) {
    case 16: tile_stage<16, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 8: tile_stage<8, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 4: tile_stage<4, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 2: tile_stage<2, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 3: tile_stage<3, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 5: tile_stage<5, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 6: tile_stage<6, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 9: tile_stage<9, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 10: tile_stage<10, FIRST, T>(g, ef, p, tw, rd, wr); break;
    case 12: tile_stage<12, FIRST, T>(g, ef, p, tw, rd, wr); break;
    default: tile_stage<15, FIRST, T>(g, ef, p, tw, rd, wr); break;
  }
}

// Forward FFT of the tile: first stage from rd (ef0), the others from shared
// memory, the last one into wr (efl) when DIRECT (two stages or more), else
// the result stays in shared memory and its buffer is returned.  Writes
// alternate between b0 (first) and b1.  TRIG: the next kernel may start before
// the last stage (launch_pdl()).
template <bool DIRECT, typename T, bool TRIG = false, class Rd, class Wr>
__device__ __forceinline__ typename cplx_t<T>::type *tile_fft(const FftPlan<T> &pl, const Tile &g, int ef0, int efl,
                                                              typename cplx_t<T>::type *b0,
                                                              typename cplx_t<T>::type *b1, const Rd &rd, const Wr &wr) {
  typedef typename cplx_t<T>::type C;
  C *in = b0, *out = b1;
  if (pl.nst == 0) {       // length 1
    for (int l = threadIdx.x; l < g.nl; l += blockDim.x) b0[g.at(l, 0)] = rd(l, 0);
  } else {
    run_stage<true, T>(pl.radix[0], g, ef0, 1, pl.tw, rd, [&](int l, int e, C v) { b0[g.at(l, e)] = v; });
  }
  __syncthreads();
  int p = pl.nst ? pl.radix[0] : 1;
  for (int st = 1; st < pl.nst; st++) {
    const int R = pl.radix[st];
    const bool direct = DIRECT && st == pl.nst - 1;
    if (TRIG && direct) pdl_trigger();
    run_stage<false, T>(R, g, direct ? efl : ef0, p, pl.tw, [&](int l, int e) { return in[g.at(l, e)]; },
                        [&](int l, int e, C v) { if (direct) wr(l, e, v); else out[g.at(l, e)] = v; });
    if (!direct) __syncthreads();
    p *= R;
    C *t = in; in = out; out = t;
  }
  return in;
}

template <typename C> __device__ __forceinline__ C swap_ri(C v) { C r; r.x = v.y; r.y = v.x; return r; }
template <typename C> __device__ __forceinline__ C swap_if(C v, bool s) {
  C r; r.x = s ? v.y : v.x; r.y = s ? v.x : v.y; return r;
}

// The pair steps of the real transforms, sum = (sx, sy) and dif = (dx, dy) of the
// elements k and n - k: X[k], X[n-k] = sum / 2 +- t (the second one conjugated),
// t = -i w dif / 2, and (im, re) of Z[k], Z[n-k] = sum +- t, t = i w* dif.
// FP32 forms t first and both elements from it (14 and 12 operations): added
// into chains of FMAs on the sums, and the second element from the first, the
// small high-k element of a smooth field's line takes the rounding errors of the
// large low-k one.  FP64, bound by its operations, runs the chains (12 and 10).
// The Nyquist element, k = 0's partner, is stored by itself in both (its value
// by pair_r2c() is not used).  Error of the high-k half of a smooth line, chains
// throughout / so: FP32 n = 16 8.9e-5 / 6.1e-5, 128 8.6e-5 / 8.1e-5, FP64 n = 32
// 1.55e-13 / 1.29e-13, 128 1.71e-13 / 1.51e-13.  (FP64 with t first everywhere is
// as accurate, and 1 % of a 128^3 step slower.)
template <typename C> struct CPair { C a, b; };
template <typename T>
__device__ __forceinline__ CPair<typename cplx_t<T>::type> pair_r2c(T sx, T sy, T dx, T dy, typename cplx_t<T>::type w) {
  if (sizeof(T) == 4) {
    const T hx = (T) 0.5 * w.x, hy = (T) 0.5 * w.y;
    const T tx = fma_t(dx, hy, dy * hx), ty = fma_t(dy, hy, -(dx * hx));
    return { mk<T>(fma_t((T) 0.5, sx, tx), fma_t((T) 0.5, sy, ty)), mk<T>(fma_t((T) 0.5, sx, -tx), fma_t((T) -0.5, sy, ty)) };
  }
  const T px = fma_t(dx, w.y, fma_t(dy, w.x, sx)), py = fma_t(-dx, w.x, fma_t(dy, w.y, sy));
  return { mk<T>((T) 0.5 * px, (T) 0.5 * py), mk<T>(fma_t((T) -0.5, px, sx), fma_t((T) 0.5, py, -sy)) };
}
template <typename T>
__device__ __forceinline__ CPair<typename cplx_t<T>::type> pair_c2r(T sx, T sy, T dx, T dy, typename cplx_t<T>::type w) {
  if (sizeof(T) == 4) {
    const T tx = fma_t(dx, w.y, -(dy * w.x)), ty = fma_t(dx, w.x, dy * w.y);
    return { mk<T>(sy + ty, sx + tx), mk<T>(ty - sy, sx - tx) };
  }
  const T zx = fma_t(dx, w.y, fma_t(-dy, w.x, sx)), zy = fma_t(dx, w.x, fma_t(dy, w.y, sy));
  return { mk<T>(zy, zx), mk<T>(fma_t((T) -2, sy, zy), fma_t((T) 2, sx, -zx)) };
}

// ------------------------------------------------------------ line pass
enum { LINE_C2C = 0, LINE_R2C = 1, LINE_C2R = 2 };

template <typename T> struct LineArgs {
  FftPlan<T> plan;       // length of the complex FFT actually run
  int B, logB;           // lines per CTA (a power of two)
  int nb;                // extent of the fast line index b
  int inverse;           // LINE_C2C: 0 forward, 1 inverse
  const typename cplx_t<T>::type *tw2;  // R2C/C2R: table of length 2n
  int e_fast;            // 1: the load functor's fast address index is the element
  int e_fast_store;      // 1: the store functor's fast address index is the element
};

// Line (a, b) = (blockIdx.y, blockIdx.x * B + l), element e.
//   LINE_C2C: X = FFT(ld(a,b,e)), st(a,b,e,X[e]) for e < n
//   LINE_R2C: z = ld(a,b,e) (packed even/odd reals), st(a,b,k,X[k]) for k <= n
//   LINE_C2R: X[k] = ld(a,b,k) for k <= n, st(a,b,e, (x[2e], x[2e+1]))
// The first stage's butterflies load straight from global memory and the last
// one's store straight to it, a line crosses shared memory only between
// stages (n <= 256: once; the staged form it replaces wrote and read it once
// more at either end and twice per stage).  Inverse transforms run the
// forward stages on (im, re).  The R2C / C2R steps take k and n - k together.
// The last tile may be partial.
// FP64 is bound by its issue rate of 2 operations per clock and SM, whatever
// the occupancy, so what counts is operations per element: 22 at n = 128 with
// radices 8, 8, 2 and separate twiddle products, 18 as 16, 8 with the
// products inside the butterflies.
template <typename T, int MODE, int NB, class Ld, class St>
__global__ void __launch_bounds__(FFT_THREADS, sizeof(T) == 4 ? 3 : 2)
    line_fft_kernel(const __grid_constant__ LineArgs<T> args, const __grid_constant__ Batch<Ld, NB> lds,
                    const __grid_constant__ Batch<St, NB> sts) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Ld &ld = lds.f[NB > 1 ? blockIdx.z : 0];
  const St &st = sts.f[NB > 1 ? blockIdx.z : 0];
  const int a = blockIdx.y, b0 = blockIdx.x * args.B, n = args.plan.n;
  Tile g;
  g.n = n; g.B = args.B; g.logB = args.logB; g.LP = Tile::pitch(n);
  g.nl = args.nb - b0 < args.B ? args.nb - b0 : args.B;
  C *buf0 = reinterpret_cast<C *>(smem_raw), *buf1 = buf0 + args.B * g.LP;
  const FftPlan<T> &pl = args.plan;
  auto none = [](int, int, C) {};
  if (MODE == LINE_C2C) pdl_trigger();
  pdl_wait();

  if constexpr (MODE == LINE_C2R) {
    // Z[k] and Z[n-k], as (im, re) for the inverse, from sum, dif = X[k] +- X*[n-k]
    const int np = n / 2 + 1;
    const FastDiv byp(np);
    for (int idx = threadIdx.x; idx < np * args.B; idx += blockDim.x) {
      int l, k;
      if (args.e_fast) byp.divmod(idx, l, k);
      else { l = idx & (args.B - 1); k = idx >> args.logB; }
      if (l >= g.nl) continue;
      C xk = ld(a, b0 + l, k), xm = ld(a, b0 + l, n - k);
      if (k == 0) { xk.y = (T) 0; xm.y = (T) 0; }   // DC / Nyquist are real
      const C w = __ldg(&args.tw2[k]);
      const T sx = xk.x + xm.x, sy = xk.y - xm.y, dx = xk.x - xm.x, dy = xk.y + xm.y;
      const CPair<C> z = pair_c2r<T>(sx, sy, dx, dy, w);
      buf0[g.at(l, k)] = z.a;
      if (k > 0 && 2 * k != n) buf0[g.at(l, n - k)] = z.b;
    }
    __syncthreads();
    auto wr = [&](int l, int e, C v) { st(a, b0 + l, e, swap_ri(v)); };
    C *r = tile_fft<true, T, true>(pl, g, args.e_fast, args.e_fast_store, buf1, buf0,
                                   [&](int l, int e) { return buf0[g.at(l, e)]; }, wr);
    if (pl.nst > 1) return;
    const FastDiv byn(n);
    for (int idx = threadIdx.x; idx < n * args.B; idx += blockDim.x) {
      int l, e;
      byn.divmod(idx, l, e);
      if (l < g.nl) wr(l, e, r[g.at(l, e)]);
    }
  } else if constexpr (MODE == LINE_R2C) {
    C *r = tile_fft<false, T>(pl, g, args.e_fast, 0, buf0, buf1, [&](int l, int e) { return ld(a, b0 + l, e); }, none);
    pdl_trigger();
    // X[k] and X[n-k], k = 0..n/2, from sum, dif = Z[k] +- Z*[n-k], w = exp(-2 pi i k / 2n)
    const int np = n / 2 + 1;
    const FastDiv byp(np);
    for (int idx = threadIdx.x; idx < np * args.B; idx += blockDim.x) {
      int l, k;
      if (args.e_fast_store) byp.divmod(idx, l, k);
      else { l = idx & (args.B - 1); k = idx >> args.logB; }
      if (l >= g.nl) continue;
      const C zk = r[g.at(l, k)], zm = r[g.at(l, k == 0 ? 0 : n - k)], w = __ldg(&args.tw2[k]);
      const T sx = zk.x + zm.x, sy = zk.y - zm.y, dx = zk.x - zm.x, dy = zk.y + zm.y;
      const CPair<C> x = pair_r2c<T>(sx, sy, dx, dy, w);
      st(a, b0 + l, k, x.a);
      if (k > 0 && 2 * k != n) st(a, b0 + l, n - k, x.b);
    }
    for (int l = threadIdx.x; l < g.nl; l += blockDim.x) {   // the Nyquist element
      const C z = r[g.at(l, 0)];
      st(a, b0 + l, n, mk<T>(z.x - z.y, (T) 0));
    }
  } else {
    const bool inv = args.inverse;
    auto rd = [&](int l, int e) { return swap_if(ld(a, b0 + l, e), inv); };
    auto wr = [&](int l, int e, C v) { st(a, b0 + l, e, swap_if(v, inv)); };
    C *r = tile_fft<true, T>(pl, g, args.e_fast, args.e_fast_store, buf0, buf1, rd, wr);
    if (pl.nst > 1) return;
    const FastDiv byn(n);
    for (int idx = threadIdx.x; idx < n * args.B; idx += blockDim.x) {
      int l, e;
      if (args.e_fast_store) byn.divmod(idx, l, e);
      else { l = idx & (args.B - 1); e = idx >> args.logB; }
      if (l < g.nl) wr(l, e, r[g.at(l, e)]);
    }
  }
}

// ------------------------------------------------------------ x-pencil convolution
// Kernel spectra are stored for the non-negative octant only, in layout
// [kz][kx][ky] with extents (nz/2+1, nx/2+1, ny/2+1), already multiplied by the
// centring phase (-1)^(kx+ky+kz) and the convolution normalisation step^3/N.
enum { KER_EVEN = 0, KER_ODD_X = 1, KER_ODD_Y = 2, KER_ODD_Z = 3, KER_UNIT = 4 };

constexpr int XC_MAX_IN = 8;
constexpr int XC_MAX_OUT = 8;
constexpr int XC_MAX_TERMS = 16;

template <typename T> struct XTerm {
  const T *ker;   // octant spectrum (real part for KER_EVEN, imaginary part for KER_ODD_*)
  int kind;
  int in;         // input index
  T coef;
};

template <typename T> struct XOut {
  typename cplx_t<T>::type *dst;   // spectral buffer [kz][x][y]
  int t0, nt;                      // terms [t0, t0+nt)
  int accumulate;                  // 1: dst += result
};

template <typename T> struct XConvArgs {
  FftPlan<T> plan;                 // length nx
  int B, logB, nx, ny, nkz;        // tile width, grid dims, number of kz planes
  int acc_buf;                     // some output sums several terms
  int split;                       // blockIdx.z selects the output (each of one term)
  int kxh, kyh;                    // octant extents nx/2+1, ny/2+1
  int nin, nout;
  const typename cplx_t<T>::type *src[XC_MAX_IN];
  XOut<T> out[XC_MAX_OUT];
  XTerm<T> term[XC_MAX_TERMS];
};

template <typename T>
__device__ __forceinline__ typename cplx_t<T>::type apply_kernel(const XTerm<T> &t, typename cplx_t<T>::type v,
                                                                 int kx, int ky, int kz, const XConvArgs<T> &A) {
  typedef typename cplx_t<T>::type C;
  if (t.kind == KER_UNIT) return v * t.coef;
  const int ix = kx <= A.nx / 2 ? kx : A.nx - kx;
  const int iy = ky <= A.ny / 2 ? ky : A.ny - ky;
  const T kv = __ldg(&t.ker[((size_t) kz * A.kxh + ix) * A.kyh + iy]) * t.coef;
  if (t.kind == KER_EVEN) return v * kv;
  T sgn = (T) 1;
  if (t.kind == KER_ODD_X && kx > A.nx / 2) sgn = (T) -1;
  if (t.kind == KER_ODD_Y && ky > A.ny / 2) sgn = (T) -1;
  C r; r.x = -sgn * kv * v.y; r.y = sgn * kv * v.x;   // (i sgn kv) v
  return r;
}

// Shared memory tiles of the generic x passes: the spectrum and a work tile,
// one more for three stages or more, one for the sum of a multi-term output.
inline int xconv_bufs(int nst, bool multi) { return 2 + (nst >= 3) + (multi ? 1 : 0); }

// grid (ceil(ny / B), nkz); one CTA = B consecutive y pencils of one kz plane
// (the last tile may be partial: odd ny).  An input's spectrum is left in
// shared memory and every output's inverse transform reads it there, times its
// kernel, in its first stage, and stores from its last stage; an output that
// sums several terms adds them up in a tile first.
template <typename T>
__global__ void __launch_bounds__(FFT_THREADS, sizeof(T) == 4 ? 3 : 2) xconv_kernel(const __grid_constant__ XConvArgs<T> A) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tile g;
  const int kz = blockIdx.y, y0 = blockIdx.x * A.B;
  g.n = A.plan.n; g.B = A.B; g.logB = A.logB; g.LP = Tile::pitch(g.n);
  g.nl = A.ny - y0 < A.B ? A.ny - y0 : A.B;
  const int tile = A.B * g.LP, ns = A.plan.nst;
  C *X = reinterpret_cast<C *>(smem_raw), *W = X + tile, *V = W + (ns >= 3 ? tile : 0), *ACC = V + tile;
  const size_t off = (size_t) kz * A.nx * A.ny + y0;
  pdl_wait();
  const bool odd = (ns & 1) || ns == 0;   // the number of stage writes: the forward result ends in X
  auto none = [](int, int, C) {};
  int cur = -1;
  auto forward = [&](int in) {
    if (in == cur) return;
    cur = in;
    const C *src = A.src[in] + off;
    tile_fft<false, T>(A.plan, g, 0, 0, odd ? X : W, odd ? W : X,
                       [&](int l, int e) { return src[(size_t) e * A.ny + l]; }, none);
  };
  auto emit = [&](const XOut<T> &out, auto rd) {
    C *dst = out.dst + off;
    const bool add = out.accumulate;
    auto wr = [&](int l, int e, C v) {
      const size_t i = (size_t) e * A.ny + l;
      v = swap_ri(v);
      dst[i] = add ? dst[i] + v : v;
    };
    C *r = tile_fft<true, T>(A.plan, g, 0, 0, W, V, [&](int l, int e) { return swap_ri(rd(l, e)); }, wr);
    if (ns <= 1)
      for (int idx = threadIdx.x; idx < g.n * g.B; idx += blockDim.x) {
        const int l = idx & (g.B - 1), e = idx >> g.logB;
        if (l < g.nl) wr(l, e, r[g.at(l, e)]);
      }
    __syncthreads();   // the work tiles are free again
  };
  for (int o = A.split ? blockIdx.z : 0; o < (A.split ? (int) blockIdx.z + 1 : A.nout); o++) {
    const XOut<T> &out = A.out[o];
    if (A.split || o == A.nout - 1) pdl_trigger();
    if (out.nt == 1) {
      const XTerm<T> &tm = A.term[out.t0];
      forward(tm.in);
      emit(out, [&](int l, int e) { return apply_kernel<T>(tm, X[g.at(l, e)], e, y0 + l, kz, A); });
      continue;
    }
    for (int t = out.t0; t < out.t0 + out.nt || t == out.t0; t++) {   // no term: a zero output
      if (out.nt) forward(A.term[t].in);
      for (int idx = threadIdx.x; idx < g.n * g.B; idx += blockDim.x) {
        const int l = idx & (g.B - 1), e = idx >> g.logB;
        if (l >= g.nl) continue;
        const int i = g.at(l, e);
        C v = out.nt ? apply_kernel<T>(A.term[t], X[i], e, y0 + l, kz, A) : mk<T>((T) 0, (T) 0);
        ACC[i] = t == out.t0 ? v : ACC[i] + v;
      }
      __syncthreads();   // the spectrum's tile is free for the next term's input
    }
    emit(out, [&](int l, int e) { return ACC[g.at(l, e)]; });
  }
}

// nx = 1: the x transforms are the identity
template <typename T> __global__ void xconv_point_kernel(const __grid_constant__ XConvArgs<T> A) {
  typedef typename cplx_t<T>::type C;
  pdl_begin();
  const size_t n = (size_t) A.nkz * A.ny;
  for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x) {
    const int kz = (int) (i / A.ny), y = (int) (i - (size_t) kz * A.ny);
    C in[XC_MAX_IN];
#pragma unroll
    for (int k = 0; k < XC_MAX_IN; k++)
      if (k < A.nin) in[k] = A.src[k][i];
    for (int o = 0; o < A.nout; o++) {
      const XOut<T> &out = A.out[o];
      C v = mk<T>((T) 0, (T) 0);
      for (int t = out.t0; t < out.t0 + out.nt; t++) {
        C x = in[0];
#pragma unroll
        for (int k = 1; k < XC_MAX_IN; k++)
          if (A.term[t].in == k) x = in[k];
        v = v + apply_kernel<T>(A.term[t], x, 0, y, kz, A);
      }
      out.dst[i] = out.accumulate ? out.dst[i] + v : v;
    }
  }
}

// ------------------------------------------------------------ kinetic x pass
// psi(k) *= exp(-i hbar |k - k0|^2 dt / 2m) / N in the middle of an x-pencil
// FFT pair; k0 is the moving-background momentum of the wave function's grid.
// The factor separates, exp(c |k - k0|^2) = (1 + fx(kx)) (1 + fyz(ky, kz)),
// so each CTA tabulates fx for its line length and fyz for its lines (two
// transcendental evaluations per thread instead of one per element) and
// applies psi + psi ((1 + fx)(1 + fyz) - 1), which keeps |factor| = 1 to the
// rounding of the exponent in real time.  With cn set the factor is the
// Crank-Nicolson one of the finite-difference kinetic operator, one per axis
// (cn_m1), and separates the same way: (1 + fx)(1 + fy)(1 + fz).
template <typename T> struct KinArgs {
  FftPlan<T> plan;
  int B, logB, nx, ny, nz;
  int kz0i, nkz;        // planes kz0i .. kz0i + nkz - 1 of the spectrum, data at the first
  double2 cdt;          // -i dt / (2 m): factor = exp(cdt |k - k0|^2)
  double inv_n;
  double dkx, dky, dkz; // 2 pi / (n step)
  double kx0, ky0, kz0; // moving-background momentum
  double h;             // grid step
  int cn;               // Crank-Nicolson factors instead of exp(cdt |k - k0|^2)
  typename cplx_t<T>::type *data;
};

template <typename T>
inline void kin_args(KinArgs<T> &K, int nx, int ny, int nz, double step, double2 cdt, double kx0, double ky0,
                     double kz0, typename cplx_t<T>::type *data) {
  K.nx = nx; K.ny = ny; K.nz = nz;
  K.kz0i = 0; K.nkz = nz;
  K.data = data;
  K.cdt = cdt;
  K.inv_n = 1.0 / ((double) nx * ny * nz);
  K.dkx = 2.0 * M_PI / (nx * step);
  K.dky = 2.0 * M_PI / (ny * step);
  K.dkz = 2.0 * M_PI / (nz * step);
  K.kx0 = kx0; K.ky0 = ky0; K.kz0 = kz0;
  K.h = step;
  K.cn = 0;
}

__device__ __forceinline__ double kfreq(int i, int n, double dk) {
  return (double) (i < (n + 1) / 2 ? i : i - n) * dk;
}

template <typename T>
__global__ void __launch_bounds__(FFT_THREADS, sizeof(T) == 4 ? 3 : 2) xkinetic_kernel(const __grid_constant__ KinArgs<T> A) {
  typedef typename cplx_t<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tile g;
  const int kz = blockIdx.y, y0 = blockIdx.x * A.B;
  g.n = A.plan.n; g.B = A.B; g.logB = A.logB; g.LP = Tile::pitch(g.n);
  g.nl = A.ny - y0 < A.B ? A.ny - y0 : A.B;
  const int n = g.n, B = g.B, tile = B * g.LP;
  C *X = reinterpret_cast<C *>(smem_raw), *W = X + tile, *fx = W + tile, *fyz = fx + n;
  C *base = A.data + (size_t) kz * A.nx * A.ny + y0;
  const C c = mk<T>((T) A.cdt.x, (T) A.cdt.y);
  pdl_trigger();
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const double k = kfreq(e, A.nx, A.dkx) - A.kx0, q = k * k;
    fx[e] = A.cn ? cn_m1(c, (T) k, (T) A.h) : cexpm1(mk<T>((T) (A.cdt.x * q), (T) (A.cdt.y * q)));
  }
  const double kzv = kfreq(A.kz0i + kz, A.nz, A.dkz) - A.kz0;
  for (int l = threadIdx.x; l < B; l += blockDim.x) {
    const double k = kfreq(y0 + l, A.ny, A.dky) - A.ky0, q = k * k + kzv * kzv;
    fyz[l] = A.cn ? cprod1p(cn_m1(c, (T) k, (T) A.h), cn_m1(c, (T) kzv, (T) A.h))
                  : cexpm1(mk<T>((T) (A.cdt.x * q), (T) (A.cdt.y * q)));
  }
  const int ns = A.plan.nst;
  const bool odd = (ns & 1) || ns == 0;
  auto none = [](int, int, C) {};
  pdl_wait();
  tile_fft<false, T>(A.plan, g, 0, 0, odd ? X : W, odd ? W : X,
                     [&](int l, int e) { return base[(size_t) e * A.ny + l]; }, none);   // its barriers cover the tables
  const T inv_n = (T) A.inv_n;
  auto factor = [&](int l, int e) {
    const C v = X[g.at(l, e)];
    return swap_ri(mul_1p(mk<T>(v.x * inv_n, v.y * inv_n), cprod1p(fx[e], fyz[l])));
  };
  auto wr = [&](int l, int e, C v) { base[(size_t) e * A.ny + l] = swap_ri(v); };
  C *r = tile_fft<true, T>(A.plan, g, 0, 0, W, X, factor, wr);
  if (ns <= 1)
    for (int idx = threadIdx.x; idx < n * B; idx += blockDim.x) {
      const int l = idx & (B - 1), e = idx >> g.logB;
      if (l < g.nl) wr(l, e, r[g.at(l, e)]);
    }
}

// ------------------------------------------------------------ launch helpers
// Tile of the generic line kernels for lines of length n (largest radix big), nb
// adjacent lines in each of na planes: lines per CTA, threads and shared memory.  strided: one
// side's fast index is the line; ctas: CTAs that fit into an SM together, while
// the tile can be cut.
struct TileShape { int B, logB, threads; size_t smem; };
template <typename T> inline int max_radix(const FftPlan<T> &p) {
  int r = 1;
  for (int i = 0; i < p.nst; i++) r = p.radix[i] > r ? p.radix[i] : r;
  return r;
}
// Limits of the current device, looked up once for each: the allocation-free
// step serves whichever device is current, also without dftgpu_init.  id -1: none.
struct DevLimits { int id, sms; size_t smem; };   // smem: opt-in shared memory of a CTA
const DevLimits &dev_limits();
int choose_tile(int n, int big, int na, int nb, size_t cplx_bytes, int nbufs, bool strided, size_t table, int ctas, TileShape *t);
inline int line_bufs(int mode, int nst) { return mode == LINE_C2C ? (nst >= 3 ? 2 : 1) : 2; }

// FP32 spectra up to this size stay in L2 between the passes of a convolution
// (less than half of it): above it the x pass takes its inputs one after the
// other (launch_xconv) and the planes run in two halves (convolve).
constexpr double kBatchBytes = 48e6;

// One launch of the generic line kernel on a given plan and stream.
template <typename T, int MODE, int NB, class Ld, class St>
int launch_generic_lines(const FftPlan<T> &plan, const typename cplx_t<T>::type *tw2, int na, int nb, int nf, T sign,
                         int ef, int efs, const Batch<Ld, NB> &ld, const Batch<St, NB> &st, cudaStream_t stream);

// "Opt-in shared memory already requested" per kernel instantiation, one bit a
// device (the attribute belongs to the device's copy of the kernel).
// It lives in an anonymous namespace so that every translation unit keeps its
// own flag: without relocatable device code each translation unit registers
// its own copy of a template kernel, and the attribute must be set on each.
namespace {
template <class Kernel> struct SmemOptIn { static std::atomic<unsigned long long> done; };
template <class Kernel> std::atomic<unsigned long long> SmemOptIn<Kernel>::done{0};
template <class Flag, class K> int smem_opt_in(K kernel) {
  const DevLimits &d = dev_limits();
  if (d.id >= 0 && !(Flag::done.load() >> d.id & 1)) {
    DFT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) d.smem));
    Flag::done |= 1ull << d.id;
  }
  return DFTGPU_OK;
}
}  // namespace

bool generic_fft_only();   // DFTGPU_GENERIC_FFT=1 disables the register kernels
bool prefetch_ahead_on();  // DFTGPU_PREFETCH_AHEAD=0 disables the one-wave-ahead L2 prefetch
bool factorised_propagation();  // DFTGPU_FACTORISED_PROP=1: FP32 propagation by one kinetic pass per axis
bool march_on();  // DFTGPU_MARCH=0: the second OT pointwise pass one CTA per row instead of x-marching

// CTAs of a 256-thread kernel resident on the whole GPU at once (the distance
// of the line kernels' one-wave-ahead prefetch); 0 when prefetching is off.
template <class K> int resident_ctas(K kernel) {
  static int n = -1;
  if (n < 0) {
    int per_sm = 0;
    if (!prefetch_ahead_on() || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess)
      per_sm = 0;
    n = per_sm * rt().num_sms;
  }
  return n;
}

// TMA for the transposed side of the z passes (DFTGPU_TMA=0 turns it off)
bool tma_on();
void tma_disable();
// Tensor map over a spectral buffer [rows][nx][ny] of complex FP32 values
// (8-byte elements) with boxes {16 y, 1 x, rows} and the 128-byte swizzle.
int encode_spec_map(CUtensorMap *map, const void *spec, int nx, int ny, int rows);
// Device flag set by a kernel whose bounded wait on an asynchronous copy gave
// up (read and cleared by dftgpu_synchronize and the device-to-host copies).
int *async_fault_flag();

// Functors of the spectral layout [kz][x][y] used by z passes (kSpecZ: members
// spec, nx, ny), whose staged side may move by TMA.
template <class F> __host__ __device__ constexpr auto spec_z_of(int) -> decltype(F::kSpecZ, bool()) { return F::kSpecZ; }
template <class F> __host__ __device__ constexpr bool spec_z_of(long) { return false; }

template <int N, int MODE, int MAP, int LDS, int STS, int TMA, int NB, class Ld, class St>
void launch_line_kernel(int na, int nb, int nf, const float2 *tw, const float2 *tw2, float sign, const Batch<Ld, NB> &ld,
                        const Batch<St, NB> &st, const Batch<ff::TmaMaps, TMA ? NB : 1> &tm, int *fault) {
  constexpr int B = ff::Shape<N>::B;
  const dim3 grid(nb / B, na, nf);
  if constexpr (LDS == 0 && ff::split_of<Ld>(0)) {
    auto k = ff::line_kernel_split<N, MODE, MAP, LDS, STS, TMA, NB, Ld, St>;
    launch_pdl(k, grid, 256, 0, rt().stream, tw, tw2, sign, ld, st, resident_ctas(k), tm, fault);
  } else if constexpr (STS == 0 && ff::bounded_store_of<St>(0)) {
    auto k = ff::line_kernel_stsplit<N, MODE, MAP, LDS, STS, TMA, NB, Ld, St>;
    launch_pdl(k, grid, 256, 0, rt().stream, tw, tw2, sign, ld, st, resident_ctas(k), tm, fault);
  } else {
    auto k = ff::line_kernel<N, MODE, MAP, LDS, STS, TMA, NB, Ld, St>;
    launch_pdl(k, grid, 256, 0, rt().stream, tw, tw2, sign, ld, st, resident_ctas(k), tm, fault);
  }
}

// FP32 power-of-two lengths: register-resident kernel.  EF / EFS: the fast
// address index of the load / store side is the element (1) or the line (0).
// nf fields in one launch.  Returns -1 when the shape does not fit the kernel
// (caller falls back).
template <int N, int MODE, int EF, int EFS, int NB, class Ld, class St>
int launch_fast_lines(int na, int nb, int nf, float sign, const Batch<Ld, NB> &ld, const Batch<St, NB> &st) {
  static_assert(MODE != LINE_R2C || (EF == 1 && EFS == 0), "r2c z pass: element-fast load, line-fast store");
  static_assert(MODE != LINE_C2R || (EF == 0 && EFS == 1), "c2r z pass: line-fast load, element-fast store");
  constexpr int MAP = (EF == 0 && EFS == 0) ? ff::MAP_L : ff::MAP_E;
  constexpr int LDS = (EF == 0 && EFS == 1) ? 1 : 0;
  constexpr int STS = (EF == 1 && EFS == 0) ? 1 : 0;
  constexpr int B = ff::Shape<N>::B;
  if (nb % B) return -1;
  FftPlan<float> p1, p2;
  DFT_TRY(get_plan<float>(N, &p1));
  p2.tw = nullptr;
  if (MODE != LINE_C2C) DFT_TRY(get_plan<float>(2 * N, &p2));
  // TMA on the spectral side of the z passes: loads of the c2r / c2c passes,
  // stores of the c2c passes.  The r2c passes keep their store loop: with a
  // TMA store the 256^3 step ran at the same rate (235.4 against 236.6 steps/s).
  constexpr bool TMA_LD = LDS && spec_z_of<Ld>(0) && ff::TmaTile<N, MODE>::OK;
  constexpr bool TMA_ST = STS && MODE == LINE_C2C && spec_z_of<St>(0) && ff::TmaTile<N, MODE>::OK;
  if constexpr (TMA_LD || TMA_ST) {
    if (tma_on()) {
      constexpr int ROWS = ff::TmaTile<N, MODE>::ROWS;
      Batch<ff::TmaMaps, NB> tm;
      memset(&tm, 0, sizeof(tm));
      int rc = DFTGPU_OK;
      for (int i = 0; i < nf && !rc; i++) {
        if constexpr (TMA_LD) rc = encode_spec_map(&tm.f[i].load, ld.f[i].spec, ld.f[i].nx, ld.f[i].ny, ROWS);
        if constexpr (TMA_ST) if (!rc) rc = encode_spec_map(&tm.f[i].store, st.f[i].spec, st.f[i].nx, st.f[i].ny, ROWS);
      }
      int *fault = rc ? nullptr : async_fault_flag();
      if (fault) {
        launch_line_kernel<N, MODE, MAP, LDS, STS, 1, NB>(na, nb, nf, p1.tw, p2.tw, sign, ld, st, tm, fault);
        DFT_CHECK_LAUNCH();
        return DFTGPU_OK;
      }
      tma_disable();   // no tensor maps here: the load / store loops from now on
      g_last_error = 0;   // the encode failure is not the caller's error
    }
  }
  Batch<ff::TmaMaps, 1> none;
  memset(&none, 0, sizeof(none));
  launch_line_kernel<N, MODE, MAP, LDS, STS, 0, NB>(na, nb, nf, p1.tw, p2.tw, sign, ld, st, none, nullptr);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// One factorised kinetic pass (ff::line_kin_kernel) over na x nb lines of
// length N: line-fast (MAP_L) when the lines are strided with consecutive
// lines adjacent, element-fast (MAP_E) for contiguous rows.  Returns -1 when
// the shape does not fit (nb not a multiple of the CTA's line count).
template <int N, int MAP, class Ld, class St>
int launch_kin_lines(int na, int nb, float2 cdt, float inv_n, float dk, float k0, const Ld &ld, const St &st) {
  constexpr int B = ff::Shape<N>::B;
  if (nb % B) return -1;
  FftPlan<float> p;
  DFT_TRY(get_plan<float>(N, &p));
  // two transforms and the factor table: rows bounded to 80 registers (3 CTAs
  // per SM); strided lines keep a runtime-stride address per element and get
  // 128 (2 CTAs per SM) so that they do not spill
  auto k = ff::line_kin_kernel<N, MAP, (MAP == ff::MAP_E || !ff::bounded_store_of<St>(0)) ? 3 : 2, Ld, St>;
  k<<<dim3(nb / B, na), 256, 0, rt().stream>>>(p.tw, cdt, inv_n, dk, k0, Batch<Ld, 1>{ { ld } }, st, resident_ctas(k));
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

template <int MAP, class Ld, class St>
int launch_kin_pass(int n, int na, int nb, float2 cdt, float dk, float k0, const Ld &ld, const St &st, const char *name,
                    double bytes) {
  if (generic_fft_only()) return -1;
  if (n != 64 && n != 128 && n != 256 && n != 512) return -1;
  ProfScope prof(name, bytes);
  const float inv_n = 1.f / (float) n;
  switch (n) {
    case 64: return launch_kin_lines<64, MAP>(na, nb, cdt, inv_n, dk, k0, ld, st);
    case 128: return launch_kin_lines<128, MAP>(na, nb, cdt, inv_n, dk, k0, ld, st);
    case 256: return launch_kin_lines<256, MAP>(na, nb, cdt, inv_n, dk, k0, ld, st);
    default: return launch_kin_lines<512, MAP>(na, nb, cdt, inv_n, dk, k0, ld, st);
  }
}

template <typename T, int MODE, int NB, class Ld, class St>
int launch_generic_lines(const FftPlan<T> &plan, const typename cplx_t<T>::type *tw2, int na, int nb, int nf, T sign,
                         int ef, int efs, const Batch<Ld, NB> &ld, const Batch<St, NB> &st, cudaStream_t stream) {
  typedef typename cplx_t<T>::type C;
  LineArgs<T> args;
  args.plan = plan;
  args.nb = nb;
  args.inverse = sign > (T) 0;
  args.tw2 = tw2;
  args.e_fast = ef;
  args.e_fast_store = efs;
  TileShape t;
  DFT_TRY(choose_tile(plan.n, max_radix(plan), na * nf, nb, sizeof(C), line_bufs(MODE, plan.nst), !ef || !efs, 0, 3, &t));
  args.B = t.B;
  args.logB = t.logB;
  auto kfn = line_fft_kernel<T, MODE, NB, Ld, St>;
  typedef SmemOptIn<LineArgs<T> (*)(Ld *, St *, int (*)[MODE + 1], int (*)[NB])> Flag;
  if (t.smem > 48 * 1024) DFT_TRY(smem_opt_in<Flag>(kfn));
  launch_pdl(kfn, dim3((nb + t.B - 1) / t.B, na, nf), t.threads, t.smem, stream, args, ld, st);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// ------------------------------------------------------------ split lines
// A long FP64 line is bound by one SM's FP64 pipe (n = 2048: 2048 x 30
// operations at 2 per clock, 15 us, where the whole chip takes 0.1), and a 1-D
// grid has one line a field.  So a single line of n = n1 n2 >= kSplitLine
// values runs as two passes of short lines over many CTAs, through scratch of
// its own length that follows the spectrum:
//   pass 1: for every j2 the n1-point DFT over j1 of x[j1 n2 + j2], times
//           exp(-2 pi i j2 k1 / n), to A[k1 n2 + j2]
//   pass 2: for every k1 the n2-point DFT over j2, to X[k1 + n1 k2];
// C2R forms its Z[k] in the loads of pass 1, R2C its X[k] in a third launch.
// Inverse transforms run on (im, re).  A full real-time step of a 1-D grid, us,
// one CTA a line / split: 4096 points 779 / 369, 2048 521 / 307, 1024 (real
// transforms of 512) 316 / 270, propagation alone of 512 points 51 / 34; 256
// points stay in one launch (29).
constexpr int kSplitLine = 512;

template <class F> struct SplitLoad {       // x[j1 n2 + j2] of line functor F
  F ld; int n2, inverse;
  __device__ auto operator()(int, int j2, int j1) const { return swap_if(ld(0, 0, j1 * n2 + j2), inverse); }
};
template <typename T, class F> struct SplitPre {   // Z[k] of the C2R transform of length n, as (im, re)
  typedef typename cplx_t<T>::type C;
  F ld; const C *tw2; int n, n2;
  __device__ C operator()(int, int j2, int j1) const {
    const int k = j1 * n2 + j2;
    C xk = ld(0, 0, k), xm = ld(0, 0, n - k);
    if (k == 0) { xk.y = (T) 0; xm.y = (T) 0; }
    const C w = __ldg(&tw2[k]);
    const T sx = xk.x + xm.x, sy = xk.y - xm.y, dx = xk.x - xm.x, dy = xk.y + xm.y;
    return pair_c2r<T>(sx, sy, dx, dy, w).a;
  }
};
template <typename T> struct SplitMid {     // A[k1 n2 + j2]: pass 1 stores (line j2, element k1), pass 2 loads (line k1, element j2)
  typedef typename cplx_t<T>::type C;
  C *A; const C *tw; int n2;
  __device__ void operator()(int, int j2, int k1, C v) const { A[k1 * n2 + j2] = cmul(v, __ldg(&tw[j2 * k1])); }
  __device__ C operator()(int, int k1, int j2) const { return A[k1 * n2 + j2]; }
};
template <class F> struct SplitStore {      // X[k1 + n1 k2] of line functor F
  F st; int n1, inverse;
  template <typename C> __device__ void operator()(int, int k1, int k2, C v) const {
    st(0, 0, k1 + n1 * k2, swap_if(v, inverse));
  }
};
template <typename T> struct SplitPlain {   // R2C: Z into a plain array
  typename cplx_t<T>::type *B;
  __device__ void operator()(int, int, int k, typename cplx_t<T>::type v) const { B[k] = v; }
};
template <typename T, int NB, class St>
__global__ void split_post_kernel(int n, const typename cplx_t<T>::type *__restrict__ tw2,
                                  const __grid_constant__ Batch<SplitPlain<T>, NB> zs,
                                  const __grid_constant__ Batch<St, NB> sts) {
  typedef typename cplx_t<T>::type C;
  pdl_begin();
  const C *Z = zs.f[NB > 1 ? blockIdx.z : 0].B;
  const St &st = sts.f[NB > 1 ? blockIdx.z : 0];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (2 * k > n) return;
  const C zk = Z[k], zm = Z[k == 0 ? 0 : n - k], w = __ldg(&tw2[k]);
  const T sx = zk.x + zm.x, sy = zk.y - zm.y, dx = zk.x - zm.x, dy = zk.y + zm.y;
  const CPair<C> x = pair_r2c<T>(sx, sy, dx, dy, w);
  st(0, 0, k, x.a);
  if (k == 0) st(0, 0, n, mk<T>(zk.x - zk.y, (T) 0));
  else if (2 * k != n) st(0, 0, n - k, x.b);
}

// Functors of the potential's and the propagation's z passes, which split lines
// serve (kLine1D), and those with the scratch (SpecStoreZ, SpecLoadZ)
template <class F> __host__ __device__ constexpr auto line_1d_of(int) -> decltype(F::kLine1D, bool()) { return F::kLine1D; }
template <class F> __host__ __device__ constexpr bool line_1d_of(long) { return false; }
template <class F> auto scratch_of(const F &f, int) -> decltype(f.scratch) { return f.scratch; }
template <class F> std::nullptr_t scratch_of(const F &, long) { return nullptr; }

// Returns -1 when the line is not split: more than one line, FP32 (not bound by
// its operations: one launch is faster than two), shorter than kSplitLine, or
// no scratch.
template <typename T, int MODE, int NB, class Ld, class St>
int split_lines(int n, int na, int nb, int nf, T sign, const Batch<Ld, NB> &ld, const Batch<St, NB> &st) {
  typedef typename cplx_t<T>::type C;
  if constexpr (std::is_same<T, double>::value) {
    if (na * nb != 1 || n < kSplitLine) return -1;
    C *scr[NB];
    for (int i = 0; i < nf; i++) {
      C *a = (C *) scratch_of(ld.f[i], 0), *b = (C *) scratch_of(st.f[i], 0);
      scr[i] = a ? a : b;
      if (!scr[i]) return -1;
    }
    int n1 = 1;
    for (int d = 2; d * d <= n; d++)
      if (n % d == 0) n1 = d;
    if (n1 < 16) return -1;
    const int n2 = n / n1;
    FftPlan<T> p1, p2, pn, pr;
    DFT_TRY(get_plan<T>(n1, &p1, true));
    DFT_TRY(get_plan<T>(n2, &p2, true));
    DFT_TRY(get_plan<T>(n, &pn));
    if (MODE != LINE_C2C) DFT_TRY(get_plan<T>(2 * n, &pr));
    const int inv = sign > (T) 0;
    Batch<SplitMid<T>, NB> mid;
    memset(&mid, 0, sizeof(mid));
    // R2C: pass 1 goes to the spectrum's place, pass 2 to the scratch, the third launch back
    for (int i = 0; i < nf; i++) {
      C *A = scr[i];
      if constexpr (MODE == LINE_R2C) A = st.f[i].spec;
      mid.f[i] = SplitMid<T>{A, pn.tw, n2};
    }
    if constexpr (MODE == LINE_C2R) {
      Batch<SplitPre<T, Ld>, NB> l1;
      memset(&l1, 0, sizeof(l1));
      for (int i = 0; i < nf; i++) l1.f[i] = SplitPre<T, Ld>{ld.f[i], pr.tw, n, n2};
      DFT_TRY((launch_generic_lines<T, LINE_C2C, NB>(p1, nullptr, 1, n2, nf, (T) -1, 0, 0, l1, mid, rt().stream)));
    } else {
      Batch<SplitLoad<Ld>, NB> l1;
      memset(&l1, 0, sizeof(l1));
      for (int i = 0; i < nf; i++) l1.f[i] = SplitLoad<Ld>{ld.f[i], n2, inv};
      DFT_TRY((launch_generic_lines<T, LINE_C2C, NB>(p1, nullptr, 1, n2, nf, (T) -1, 0, 0, l1, mid, rt().stream)));
    }
    if constexpr (MODE == LINE_R2C) {
      Batch<SplitPlain<T>, NB> z;
      Batch<SplitStore<SplitPlain<T>>, NB> s2;
      memset(&z, 0, sizeof(z));
      memset(&s2, 0, sizeof(s2));
      for (int i = 0; i < nf; i++) {
        z.f[i] = SplitPlain<T>{scr[i]};
        s2.f[i] = SplitStore<SplitPlain<T>>{z.f[i], n1, 0};
      }
      DFT_TRY((launch_generic_lines<T, LINE_C2C, NB>(p2, nullptr, 1, n1, nf, (T) -1, 1, 0, mid, s2, rt().stream)));
      launch_pdl(split_post_kernel<T, NB, St>, dim3((n / 2 + 64) / 64, 1, nf), 64, 0, rt().stream, n, pr.tw, z, st);
      DFT_CHECK_LAUNCH();
    } else {
      Batch<SplitStore<St>, NB> s2;
      memset(&s2, 0, sizeof(s2));
      for (int i = 0; i < nf; i++) s2.f[i] = SplitStore<St>{st.f[i], n1, inv};
      DFT_TRY((launch_generic_lines<T, LINE_C2C, NB>(p2, nullptr, 1, n1, nf, (T) -1, 1, 0, mid, s2, rt().stream)));
    }
    return DFTGPU_OK;
  }
  return -1;
}

// Line passes of nf fields (at most NB) of one shape in one launch.
// extra_bytes: algorithmic bytes read / written by the fused functors beyond
// the transformed line data itself (e.g. the potential read by a phase load).
template <typename T, int MODE, int EF, int EFS, int NB, class Ld, class St>
int launch_lines_batch(int n_fft, int na, int nb, int nf, T sign, const Batch<Ld, NB> &ld, const Batch<St, NB> &st,
                       double extra_bytes = 0.0) {
  typedef typename cplx_t<T>::type C;
  const double lines = (double) na * nb * nf;
  const double data = MODE == LINE_C2C ? 2.0 * n_fft : (2.0 * n_fft + 1.0);
  ProfScope prof(MODE == LINE_C2C ? "fft_line_c2c" : (MODE == LINE_R2C ? "fft_line_r2c" : "fft_line_c2r"),
                 lines * data * sizeof(C) + extra_bytes);
  if constexpr (std::is_same<T, float>::value) {
    if (!generic_fft_only()) {
      int rc = -1;
      switch (n_fft) {
        case 64: rc = launch_fast_lines<64, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        case 128: rc = launch_fast_lines<128, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        case 256: rc = launch_fast_lines<256, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        case 512: rc = launch_fast_lines<512, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        case 96: rc = launch_fast_lines<96, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        case 192: rc = launch_fast_lines<192, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        case 384: rc = launch_fast_lines<384, MODE, EF, EFS, NB>(na, nb, nf, sign, ld, st); break;
        default: break;
      }
      if (rc >= 0) return rc;
    }
  }
  // only the functor pairs of the transforms with scratch instantiate the split form
  if constexpr (line_1d_of<Ld>(0) || line_1d_of<St>(0)) {
    const int rc = split_lines<T, MODE, NB>(n_fft, na, nb, nf, sign, ld, st);
    if (rc >= 0) return rc;
  }
  FftPlan<T> p1, p2;
  DFT_TRY(get_plan<T>(n_fft, &p1, small_pass(n_fft, na * nf, nb)));
  p2.tw = nullptr;
  if (MODE != LINE_C2C) DFT_TRY(get_plan<T>(2 * n_fft, &p2));
  return launch_generic_lines<T, MODE, NB>(p1, p2.tw, na, nb, nf, sign, EF, EFS, ld, st, rt().stream);
}

template <typename T, int MODE, int EF, int EFS, class Ld, class St>
int launch_lines(int n_fft, int na, int nb, T sign, const Ld &ld, const St &st, double extra_bytes = 0.0) {
  constexpr int NB = batch_of<Ld>(0) && batch_of<St>(0) ? LINE_BATCH : 1;   // one instantiation per functor pair
  Batch<Ld, NB> l;
  Batch<St, NB> t;
  memset(&l, 0, sizeof(l));
  memset(&t, 0, sizeof(t));
  l.f[0] = ld;
  t.f[0] = st;
  return launch_lines_batch<T, MODE, EF, EFS, NB>(n_fft, na, nb, 1, sign, l, t, extra_bytes);
}

template <typename T> int launch_xconv(XConvArgs<T> &A);
template <typename T> int launch_xkinetic(KinArgs<T> &A);

// the generic kinetic pass on A.plan and a given stream
template <typename T> int launch_generic_xkinetic(KinArgs<T> &A, cudaStream_t stream) {
  typedef typename cplx_t<T>::type C;
  TileShape t;
  DFT_TRY(choose_tile(A.nx, max_radix(A.plan), A.nkz, A.ny, sizeof(C), 2, true, (size_t) A.nx * sizeof(C), 2, &t));
  A.B = t.B;
  A.logB = t.logB;
  auto kfn = xkinetic_kernel<T>;
  if (t.smem > 48 * 1024) DFT_TRY(smem_opt_in<SmemOptIn<KinArgs<T> (*)()>>(kfn));
  launch_pdl(kfn, dim3((A.ny + t.B - 1) / t.B, A.nkz), t.threads, t.smem, stream, A);
  DFT_CHECK_LAUNCH();
  return DFTGPU_OK;
}

// ------------------------------------------------------------ fused z + y passes
// The fused z + y plane passes (cluster kernels, fast_fft.cuh) are selected
// with DFTGPU_FUSED_ZY=1; by default the separate passes run (measured
// faster at 256^3: 60-64 us against 73-83 us per real transform).
bool fused_zy_off();

}  // namespace dftgpu
