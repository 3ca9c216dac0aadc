// pf_gfft.cuh -- pencil passes for any transform length, one shared-memory buffer per tile.
//
// Serves every pass that has no paired power-of-two kernel (pf_pairfft.cuh): all FP64 passes
// and the FP32 passes of round, odd and prime lengths.
//
// Values.  A slot of shared memory is 16 bytes for both precisions: one complex double, or the
// complex floats of TWO pencils in the pair layout (Re A, Re B, Im A, Im B), so that FP32
// butterflies run on the packed FADD2/FFMA2 and every index, twiddle load and shared-memory
// access serves two pencils.
//
// Transform.  Decimation in frequency with a mixed-radix schedule N = R1 R2 .. RS (radices 2..8,
// 11, 13; Gentleman and Sande, AFIPS 1966), every stage in place: stage s reads the R
// elements t + r M_s of its block, and writes its outputs, times W^(q t), to the same places, so
// one buffer and one barrier per stage suffice.  The first stage takes its inputs straight from
// the loader and the last one hands its outputs, whose index follows from the block's digits,
// straight to the store: 2 (S - 1) shared-memory accesses per element.  With threads ordered by
// the first digit the last stage's outputs are consecutive.
//
// Forward and backward in one pass (the matvec's fused pass, and the convolution inside
// Bluestein's algorithm): the last forward stage, the pointwise factor and the first stage of
// the backward transform act on the same registers, and the backward transform runs the stages
// in reverse as decimation in time from the digit-reversed order, so nothing is reordered.
// Backward transforms are forward ones with real and imaginary parts swapped on the way in and
// out.
//
// Lengths L with a prime factor above 13 use Bluestein's algorithm (L. Bluestein, "A linear
// filtering approach to the computation of the discrete Fourier transform", 1970): with
// w_j = exp(-pi i j^2 / L), X_k = w_k sum_j (x_j w_j) conj(w_(k-j)), a circular convolution of
// the cheapest smooth length N >= 2 L - 1.
//
// What bounds it: latency -- of loads, barriers and instruction fetch -- at 25-30 warps per SM; the
// issue slots are 29-45% busy in FP64 strided passes, rows and covariance rows (100^3 field, 128 x 120
// x 96 spectrum; FP64 pipe 13-22%), 59% in the FP32 fused pass (128^3) and 69% in the FP64 noise pass
// (100^3; FP64 pipe 39%), which issue bounds most.  The loaders' long scoreboard is the first
// stall of all others; covariance rows add spills (868 bytes stored, 64 registers).  Measured on one B200 against the passes it replaced
// (two ping-pong buffers, runtime divisions per element, 2 CTAs per SM; compile-time schedules
// for 11 lengths; radix-2 Bluestein), us: 100^3 FP64 realization, passes of 200, 200 and 100
// points, 116 / 44 / 34 -> 67 / 21 / 17; FP64 product on 128^3 (256 points) 287 -> 193, its fused
// pass 148 -> 85; FP32 product on 150 x 100 x 75 279 -> 80; 32 uneven 2D fields, mostly
// Bluestein lengths, 1330 -> 638; FP64 covariance rows of a 256^3 DCT spectrum 1277 -> 546.
//
// Layout of a tile of B slots: strided passes keep the B adjacent pencils together (element n of
// slot b at n B + b); row passes keep rows together (b * pitch + n), the R1 sub-blocks of a row
// padded to an odd distance, which keeps the last stage's reads free of bank conflicts.
#pragma once

#include "pf_kernels.cuh"
#include "pf_pairfft.cuh"

namespace pf {

// most threads of a block, and what the register allocation (64) holds per SM.  80 registers and
// radices up to 10 (768 threads) ran slower: FP64 fused passes of 256 points on
// 129 x 256 pencils 98 against 84 us, FP64 noise passes of 200 points 87 against 75 us.
constexpr int kGThreads = 1024;
constexpr int kGStages = 8;

// complex value of real type R: double, or float2 (pencils A and B)
template <class R>
struct alignas(16) CV {
  R re, im;
};

template <typename T>
struct GT;
template <>
struct GT<double> {
  using R = double;
  using W = double2;  // table entry
  static constexpr int PAIR = 1;
};
template <>
struct GT<float> {
  using R = float2;
  using W = float4;  // table entry broadcast as (x, x, y, y)
  static constexpr int PAIR = 2;
};
template <typename T>
using GV = CV<typename GT<T>::R>;

__device__ __forceinline__ double g_add(double a, double b) { return a + b; }
__device__ __forceinline__ double g_sub(double a, double b) { return a - b; }
__device__ __forceinline__ double g_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double g_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double g_neg(double a) { return -a; }
__device__ __forceinline__ float2 g_add(float2 a, float2 b) { return f2add(a, b); }
__device__ __forceinline__ float2 g_sub(float2 a, float2 b) { return f2sub(a, b); }
__device__ __forceinline__ float2 g_mul(float2 a, float2 b) { return f2mul(a, b); }
__device__ __forceinline__ float2 g_fma(float2 a, float2 b, float2 c) { return f2fma(a, b, c); }
__device__ __forceinline__ float2 g_neg(float2 a) { return make_float2(-a.x, -a.y); }
template <class R>
__device__ __forceinline__ R g_const(double c);
template <>
__device__ __forceinline__ double g_const<double>(double c) {
  return c;
}
template <>
__device__ __forceinline__ float2 g_const<float2>(double c) {
  return make_float2((float)c, (float)c);
}

template <class R>
__device__ __forceinline__ CV<R> v_add(const CV<R>& a, const CV<R>& b) {
  return {g_add(a.re, b.re), g_add(a.im, b.im)};
}
template <class R>
__device__ __forceinline__ CV<R> v_sub(const CV<R>& a, const CV<R>& b) {
  return {g_sub(a.re, b.re), g_sub(a.im, b.im)};
}
template <class R>
__device__ __forceinline__ CV<R> v_swap(const CV<R>& a) {
  return {a.im, a.re};
}
// a + (-i) b and a - (-i) b
template <class R>
__device__ __forceinline__ CV<R> v_addmi(const CV<R>& a, const CV<R>& b) {
  return {g_add(a.re, b.im), g_sub(a.im, b.re)};
}
template <class R>
__device__ __forceinline__ CV<R> v_submi(const CV<R>& a, const CV<R>& b) {
  return {g_sub(a.re, b.im), g_add(a.im, b.re)};
}
__device__ __forceinline__ double w_re(double2 w) { return w.x; }
__device__ __forceinline__ double w_im(double2 w) { return w.y; }
__device__ __forceinline__ float2 w_re(float4 w) { return make_float2(w.x, w.y); }
__device__ __forceinline__ float2 w_im(float4 w) { return make_float2(w.z, w.w); }
// a * w and a * conj(w)
template <class R, class W>
__device__ __forceinline__ CV<R> v_mul(const CV<R>& a, W w) {
  return {g_sub(g_mul(a.re, w_re(w)), g_mul(a.im, w_im(w))), g_fma(a.re, w_im(w), g_mul(a.im, w_re(w)))};
}
template <class R, class W>
__device__ __forceinline__ CV<R> v_mulc(const CV<R>& a, W w) {
  return {g_fma(a.re, w_re(w), g_mul(a.im, w_im(w))), g_sub(g_mul(a.im, w_re(w)), g_mul(a.re, w_im(w)))};
}
// ---------------------------------------------------------------------------
// in-register forward transforms: v[q] = sum_r v[r] exp(-2 pi i r q / N)
// ---------------------------------------------------------------------------
template <class R>
__device__ __forceinline__ void g_dft3(CV<R>& a, CV<R>& b, CV<R>& c) {
  const CV<R> s = v_add(b, c), d = v_sub(b, c);
  const R h = g_const<R>(-0.5), k = g_const<R>(0.86602540378443864676372317075293618347),
          nk = g_const<R>(-0.86602540378443864676372317075293618347);
  const CV<R> m = {g_fma(h, s.re, a.re), g_fma(h, s.im, a.im)};
  a = v_add(a, s);
  b = {g_fma(k, d.im, m.re), g_fma(nk, d.re, m.im)};
  c = {g_fma(nk, d.im, m.re), g_fma(k, d.re, m.im)};
}
template <class R>
__device__ __forceinline__ void g_dft4(CV<R>& v0, CV<R>& v1, CV<R>& v2, CV<R>& v3) {
  const CV<R> a = v_add(v0, v2), b = v_sub(v0, v2), c = v_add(v1, v3), d = v_sub(v1, v3);
  v0 = v_add(a, c);
  v2 = v_sub(a, c);
  v1 = v_addmi(b, d);
  v3 = v_submi(b, d);
}
template <class R>
__device__ __forceinline__ void g_dft5(CV<R>& v0, CV<R>& v1, CV<R>& v2, CV<R>& v3, CV<R>& v4) {
  const R c1 = g_const<R>(0.30901699437494742410229341718281905886),
          c2 = g_const<R>(-0.80901699437494742410229341718281905886),
          s1 = g_const<R>(0.95105651629515357211643933337938214340),
          s2 = g_const<R>(0.58778525229247312916870595463907276860),
          ns1 = g_const<R>(-0.95105651629515357211643933337938214340);
  const CV<R> p1 = v_add(v1, v4), m1 = v_sub(v1, v4), p2 = v_add(v2, v3), m2 = v_sub(v2, v3);
  const CV<R> r1 = {g_fma(c2, p2.re, g_fma(c1, p1.re, v0.re)), g_fma(c2, p2.im, g_fma(c1, p1.im, v0.im))};
  const CV<R> r2 = {g_fma(c1, p2.re, g_fma(c2, p1.re, v0.re)), g_fma(c1, p2.im, g_fma(c2, p1.im, v0.im))};
  const CV<R> i1 = {g_fma(s2, m2.re, g_mul(s1, m1.re)), g_fma(s2, m2.im, g_mul(s1, m1.im))};
  const CV<R> i2 = {g_fma(ns1, m2.re, g_mul(s2, m1.re)), g_fma(ns1, m2.im, g_mul(s2, m1.im))};
  v0 = v_add(v0, v_add(p1, p2));
  v1 = v_addmi(r1, i1);
  v4 = v_submi(r1, i1);
  v2 = v_addmi(r2, i2);
  v3 = v_submi(r2, i2);
}

// cos and sin of 2 pi k / N for the prime radices (Taylor series in range-reduced arguments,
// evaluated by the compiler)
constexpr double g_pi = 3.14159265358979323846264338327950288;
constexpr double g_sin_series(double x) {
  double t = x, s = x;
  for (int k = 1; k < 14; k++) {
    t *= -x * x / ((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
constexpr double g_cos_series(double x) {
  double t = 1., s = 1.;
  for (int k = 1; k < 14; k++) {
    t *= -x * x / ((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
// k in [0, n): argument 2 pi k / n reduced to [0, pi/2]
constexpr double g_cos2pi(int k, int n) {
  if (2 * k > n) k = n - k;
  return 4 * k <= n ? g_cos_series(2. * g_pi * k / n) : -g_cos_series(g_pi * (n - 2 * k) / n);
}
constexpr double g_sin2pi(int k, int n) {
  if (2 * k > n) return -g_sin2pi(n - k, n);
  return 4 * k <= n ? g_sin_series(2. * g_pi * k / n) : g_sin_series(g_pi * (n - 2 * k) / n);
}
template <int N>
struct GTrig {
  double c[N], s[N];
  constexpr GTrig() : c(), s() {
    for (int k = 0; k < N; k++) {
      c[k] = g_cos2pi(k, N);
      s[k] = g_sin2pi(k, N);
    }
  }
};

// odd prime N: sums and differences of the elements r and N - r
template <int N, class R>
__device__ __forceinline__ void g_dft_prime(CV<R>* v) {
  constexpr int H = N / 2;
  constexpr GTrig<N> tr;
  CV<R> p[H], m[H];
  CV<R> s = v[0];
#pragma unroll
  for (int r = 1; r <= H; r++) {
    p[r - 1] = v_add(v[r], v[N - r]);
    m[r - 1] = v_sub(v[r], v[N - r]);
    s = v_add(s, p[r - 1]);
  }
  const CV<R> v0 = v[0];
  v[0] = s;
#pragma unroll
  for (int q = 1; q <= H; q++) {
    CV<R> a = v0, b = {g_mul(g_const<R>(tr.s[q]), m[0].re), g_mul(g_const<R>(tr.s[q]), m[0].im)};
#pragma unroll
    for (int r = 1; r <= H; r++) {
      const int k = (r * q) % N;
      a = {g_fma(g_const<R>(tr.c[k]), p[r - 1].re, a.re), g_fma(g_const<R>(tr.c[k]), p[r - 1].im, a.im)};
      if (r > 1)
        b = {g_fma(g_const<R>(tr.s[k]), m[r - 1].re, b.re), g_fma(g_const<R>(tr.s[k]), m[r - 1].im, b.im)};
    }
    v[q] = v_addmi(a, b);
    v[N - q] = v_submi(a, b);
  }
}

template <int N, class R>
__device__ __forceinline__ void g_dft(CV<R>* v) {
  if constexpr (N == 2) {
    const CV<R> a = v[0];
    v[0] = v_add(a, v[1]);
    v[1] = v_sub(a, v[1]);
  } else if constexpr (N == 3) {
    g_dft3(v[0], v[1], v[2]);
  } else if constexpr (N == 4) {
    g_dft4(v[0], v[1], v[2], v[3]);
  } else if constexpr (N == 5) {
    g_dft5(v[0], v[1], v[2], v[3], v[4]);
  } else if constexpr (N == 6) {  // 2 x 3: n = 3 n1 + 2 n2, k = 3 k1 + 4 k2 mod 6
    CV<R> a0 = v[0], a1 = v[2], a2 = v[4], b0 = v[3], b1 = v[5], b2 = v[1];
    g_dft3(a0, a1, a2);
    g_dft3(b0, b1, b2);
    v[0] = v_add(a0, b0);
    v[3] = v_sub(a0, b0);
    v[4] = v_add(a1, b1);
    v[1] = v_sub(a1, b1);
    v[2] = v_add(a2, b2);
    v[5] = v_sub(a2, b2);
  } else if constexpr (N == 8) {
    CV<R> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    g_dft4(e0, e1, e2, e3);
    g_dft4(o0, o1, o2, o3);
    const R h = g_const<R>(0.70710678118654752440084436210484903928),
            nh = g_const<R>(-0.70710678118654752440084436210484903928);
    v[0] = v_add(e0, o0);
    v[4] = v_sub(e0, o0);
    v[2] = v_addmi(e2, o2);
    v[6] = v_submi(e2, o2);
    const R ar = g_add(o1.re, o1.im), ai = g_sub(o1.im, o1.re);  // sqrt(2) o1 W8
    v[1] = {g_fma(h, ar, e1.re), g_fma(h, ai, e1.im)};
    v[5] = {g_fma(nh, ar, e1.re), g_fma(nh, ai, e1.im)};
    const R br = g_sub(o3.re, o3.im), bi = g_add(o3.im, o3.re);  // -sqrt(2) o3 W8^3
    v[3] = {g_fma(nh, br, e3.re), g_fma(nh, bi, e3.im)};
    v[7] = {g_fma(h, br, e3.re), g_fma(h, bi, e3.im)};
  } else if constexpr (N == 7 || N == 11 || N == 13) {
    g_dft_prime<N>(v);
  } else {
    static_assert(N == 1, "radix not built");
  }
}

// radices of the kernels with fused ends; of the shared stages, those that would make the common
// ones spill registers apart (with the error words' address in constant memory: 32 uneven 2D fields, mostly Bluestein
// lengths, 715 -> 664 us)
#define PF_G_COMMON_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(8)
#define PF_G_RARE_RADICES(X) X(1) X(7) X(11) X(13)
#define PF_G_FUSED_RADICES(X) PF_G_COMMON_RADICES(X) X(7)

// ---------------------------------------------------------------------------
// pass descriptor
// ---------------------------------------------------------------------------
// quotient of n by a divisor d: floor(n * m / 2^32) with m = ceil(2^32 / d), exact for
// n d < 2^32; m = 0 stands for d = 1
__host__ __device__ __forceinline__ int g_div(int n, unsigned m) {
  return m ? (int)(((unsigned long long)(unsigned)n * m) >> 32) : n;
}

struct GStage {
  int R;         // radix
  int M;         // distance of a butterfly's elements: N / (R1 .. Rs)
  int nb;        // butterflies of the stage, N / R
  int rest;      // blocks per first digit, R2 .. R(s-1)
  int block;     // distance of two blocks of one first digit (M of the stage before)
  int tw;        // offset of the stage's twiddles: W^(q t) at tw + (q - 1) M + t
  unsigned mM, mnb, mrest, mR;  // divisors M, nb, rest, R
};

template <typename T>
struct GArgs {
  using W = typename GT<T>::W;
  int N, S;            // transform length, stages
  int L;               // pencil length (N, or the length Bluestein's algorithm serves)
  int Lout;            // outputs stored
  int B, lgB;          // slots per tile (a power of two for strided passes)
  int M1p;             // padded distance of the first stage's sub-blocks
  int pitch;           // slots of one row
  int np, tpo;         // pencils (per outer block), tiles per outer block
  int args_at;         // slot of shared memory that holds a copy of these for the shared stages; 0: none
  unsigned mL, mLout;  // divisors L, outputs per row of the post-processing
  const W* tw;         // stage twiddles
  const W* twT;        // real rows: exp(-2 pi i m / 2L), m < L
  const W* chirp;      // Bluestein: w_j, j < L
  const W* bhat;       // Bluestein: transform of conj(w) over N, divided by N
  GStage st[kGStages];
};

// loaders whose values cost arithmetic go through shared memory before the first stage
template <class Ld>
struct g_direct : std::true_type {};
template <>
struct g_direct<R2CNoise> : std::false_type {};
template <>
struct g_direct<DFTNoise> : std::false_type {};
template <>
struct g_direct<DctDstNoise> : std::false_type {};
template <>
struct g_direct<CovRowLoad> : std::false_type {};

// ---- functor adaptors: slot values of pencil p (and p + 1) ----------------------------
template <class Ld>
__device__ __forceinline__ CV<double> g_load(const Ld& ld, int p, int np, int j, int io, double) {
  if (p >= np) return {0., 0.};
  const double2 a = ld.template load<double>(p, j, io);
  return {a.x, a.y};
}
template <class Ld>
__device__ __forceinline__ CV<float2> g_load(const Ld& ld, int p, int np, int j, int io, float) {
  float2 a = make_float2(0.f, 0.f), b = a;
  if (p < np) a = ld.template load<float>(p, j, io);
  if (p + 1 < np) b = ld.template load<float>(p + 1, j, io);
  return {make_float2(a.x, b.x), make_float2(a.y, b.y)};
}
// adjacent pencils of a work array in one 16-byte load
__device__ __forceinline__ CV<float2> g_load(const ArrLoad<float2>& ld, int p, int np, int j, int io, float) {
  if (ld.vec && p + 1 < np) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < ld.Lin) {
      const unsigned i = (unsigned)p + (unsigned)j * ld.jstride + (unsigned)io * ld.ostride;
      if (in_bounds32(i + 1, ld.n)) s = *reinterpret_cast<const float4*>(ld.ptr + i);
    }
    return {make_float2(s.x, s.z), make_float2(s.y, s.w)};
  }
  float2 a = make_float2(0.f, 0.f), b = a;
  if (p < np) a = ld.load<float>(p, j, io);
  if (p + 1 < np) b = ld.load<float>(p + 1, j, io);
  return {make_float2(a.x, b.x), make_float2(a.y, b.y)};
}
// reals 2m and 2m + 1 of a row as one complex
template <class Ld>
__device__ __forceinline__ CV<double> g_real(const Ld& ld, int p, int np, int m, double) {
  if (p >= np) return {0., 0.};
  double a, b;
  ld.template real2<double>(p, m, a, b);
  return {a, b};
}
template <class Ld>
__device__ __forceinline__ CV<float2> g_real(const Ld& ld, int p, int np, int m, float) {
  float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
  if (p < np) ld.template real2<float>(p, m, a, b);
  if (p + 1 < np) ld.template real2<float>(p + 1, m, c, d);
  return {make_float2(a, c), make_float2(b, d)};
}

template <class St>
__device__ __forceinline__ void g_store(const St& st, int p, int np, int j, int io, const CV<double>& v) {
  if (p < np) st.template store<double>(p, j, io, make_double2(v.re, v.im));
}
template <class St>
__device__ __forceinline__ void g_store(const St& st, int p, int np, int j, int io, const CV<float2>& v) {
  if (p < np) st.template store<float>(p, j, io, make_float2(v.re.x, v.im.x));
  if (p + 1 < np) st.template store<float>(p + 1, j, io, make_float2(v.re.y, v.im.y));
}
__device__ __forceinline__ void g_store(const ArrStore<float2>& st, int p, int np, int j, int io,
                                        const CV<float2>& v) {
  if (st.vec && p + 1 < np) {
    const unsigned i = (unsigned)p + (unsigned)j * st.jstride + (unsigned)io * st.ostride;
    if (in_bounds32(i + 1, st.n))
      *reinterpret_cast<float4*>(st.ptr + i) = make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
    return;
  }
  if (p < np) st.store<float>(p, j, io, make_float2(v.re.x, v.im.x));
  if (p + 1 < np) st.store<float>(p + 1, j, io, make_float2(v.re.y, v.im.y));
}
// reals 2m and 2m + 1 of a row (those below Lout)
template <class St>
__device__ __forceinline__ void g_store_real(const St& st, int p, int np, int m, int Lout, const CV<double>& v) {
  if (p < np) st.template real2<double>(p, m, v.re, v.im, 2 * m + 1 < Lout);
}
template <class St>
__device__ __forceinline__ void g_store_real(const St& st, int p, int np, int m, int Lout, const CV<float2>& v) {
  if (p < np) st.template real2<float>(p, m, v.re.x, v.im.x, 2 * m + 1 < Lout);
  if (p + 1 < np) st.template real2<float>(p + 1, m, v.re.y, v.im.y, 2 * m + 1 < Lout);
}

template <class Mid>
__device__ __forceinline__ CV<double> g_mid(const Mid& mid, int p, int np, int j, int io, const CV<double>& v) {
  if (p >= np) return v;
  const double2 r = mid.template operator()<double>(p, j, io, make_double2(v.re, v.im));
  return {r.x, r.y};
}
template <class Mid>
__device__ __forceinline__ CV<float2> g_mid(const Mid& mid, int p, int np, int j, int io, const CV<float2>& v) {
  float2 a = make_float2(v.re.x, v.im.x), b = make_float2(v.re.y, v.im.y);
  if (p < np) a = mid.template operator()<float>(p, j, io, a);
  if (p + 1 < np) b = mid.template operator()<float>(p + 1, j, io, b);
  return {make_float2(a.x, b.x), make_float2(a.y, b.y)};
}

// ---------------------------------------------------------------------------
// geometry of a tile in shared memory
// ---------------------------------------------------------------------------
template <typename T, bool ROWS>
struct GTile {
  const GArgs<T>& a;
  __host__ __device__ __forceinline__ int sj() const { return ROWS ? 1 : a.B; }
  __host__ __device__ __forceinline__ int m1s() const { return ROWS ? a.M1p : a.M1p * a.B; }
  // work item u of a stage with nb butterflies per slot: slot b, butterfly w
  __host__ __device__ __forceinline__ void split(int u, int nb, unsigned mnb, int& b, int& w) const {
    if constexpr (ROWS) {
      b = g_div(u, mnb);
      w = u - b * nb;
    } else {
      b = u & (a.B - 1);
      w = u >> a.lgB;
    }
  }
  __host__ __device__ __forceinline__ int slot0(int b) const { return ROWS ? b * a.pitch : b; }
  // place of element n in the order of the first stage's inputs
  __host__ __device__ __forceinline__ int place(int n) const {
    const int r = g_div(n, a.st[0].mM);
    return r * m1s() + (n - r * a.st[0].M) * sj();
  }
  // place of output j of a forward transform: its digits, first one fastest
  __host__ __device__ __forceinline__ int place_out(int j) const {
    int rem = g_div(j, a.st[0].mR);
    int at = (j - rem * a.st[0].R) * m1s();
    for (int s = 1; s < a.S; s++) {
      const int nx = g_div(rem, a.st[s].mR);
      at += (rem - nx * a.st[s].R) * a.st[s].M * sj();
      rem = nx;
    }
    return at;
  }
  // place of butterfly w of middle stage g (t: its index within its block)
  __host__ __device__ __forceinline__ int base_of(const GStage& g, int w, int& t) const {
    const int blk = g_div(w, g.mM);
    t = w - blk * g.M;
    const int q1 = g_div(blk, g.mrest);
    return q1 * m1s() + ((blk - q1 * g.rest) * g.block + t) * sj();
  }
  // place of the last stage's butterfly whose outputs are j = w + q N/R
  __host__ __device__ __forceinline__ int base_last(int w) const {
    if (a.S == 1) return 0;
    int rem = g_div(w, a.st[0].mR);
    int at = (w - rem * a.st[0].R) * m1s();
    for (int s = 1; s < a.S - 1; s++) {
      const int nx = g_div(rem, a.st[s].mR);
      at += (rem - nx * a.st[s].R) * a.st[s].M * sj();
      rem = nx;
    }
    return at;
  }
  __host__ __device__ __forceinline__ int last_step() const { return a.S == 1 ? m1s() : sj(); }
};

// Stages in place in shared memory, the same code for every loader and store (not inlined: one
// copy per precision and layout).  KIND: 0 first, 1 middle, 2 last stage of a forward transform;
// 3 middle, 4 final stage of a backward one; 5 last stage of a Bluestein convolution's forward
// transform, times the kernel, and first stage of its backward one.
template <typename T, bool ROWS, int KIND, int R>
__device__ __forceinline__ void g_stage_r(const GArgs<T>& a, const GStage& g) {
  using V = GV<T>;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* const sm = reinterpret_cast<V*>(g_smem);
  const GTile<T, ROWS> ti{a};
  constexpr bool ENDS = KIND == 0 || KIND == 4;
  constexpr bool LAST = KIND == 2 || KIND == 5;
  const int step = ENDS ? ti.m1s() : (LAST ? ti.last_step() : g.M * ti.sj());
  const int nb = g.nb;
  const V zero = {g_const<typename GT<T>::R>(0.), g_const<typename GT<T>::R>(0.)};
  const typename GT<T>::W* const tw = a.tw + g.tw;
  for (int u = threadIdx.x; u < a.B * nb; u += blockDim.x) {
    int b, w, t;
    ti.split(u, nb, g.mnb, b, w);
    int at = ti.slot0(b);
    if constexpr (ENDS) {
      t = w;
      at += w * ti.sj();
    } else if constexpr (LAST) {
      t = 0;
      at += ti.base_last(w);
    } else {
      at += ti.base_of(g, w, t);
    }
    V* const x = sm + at;
    V v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = (KIND != 0 || t + r * g.M < a.L) ? x[r * step] : zero;
      if ((KIND == 3 || KIND == 4) && r > 0) v[r] = v_mul(v[r], __ldg(tw + (r - 1) * g.M + t));
    }
    g_dft<R>(v);
    if constexpr (KIND == 5) {
#pragma unroll
      for (int q = 0; q < R; q++) v[q] = v_swap(v_mul(v[q], __ldg(a.bhat + w + q * nb)));
      g_dft<R>(v);
    }
#pragma unroll
    for (int q = 0; q < R; q++) {
      if ((KIND == 0 || KIND == 1) && q > 0) v[q] = v_mul(v[q], __ldg(tw + (q - 1) * g.M + t));
      x[q * step] = v[q];
    }
  }
  __syncthreads();
}
template <typename T, bool ROWS, int KIND>
__device__ __noinline__ void g_stage_rare(const GArgs<T>& a, int s) {
  const GStage& g = a.st[s];
  switch (g.R) {
#define PF_G_CASE(RR) \
  case RR: g_stage_r<T, ROWS, KIND, RR>(a, g); break;
    PF_G_RARE_RADICES(PF_G_CASE)
#undef PF_G_CASE
    default: break;
  }
}
template <typename T, bool ROWS, int KIND>
__device__ __noinline__ void g_stage(const GArgs<T>& a, int s) {
  const GStage& g = a.st[s];
  switch (g.R) {
#define PF_G_CASE(RR) \
  case RR: g_stage_r<T, ROWS, KIND, RR>(a, g); break;
    PF_G_COMMON_RADICES(PF_G_CASE)
#undef PF_G_CASE
    default: g_stage_rare<T, ROWS, KIND>(a, s);
  }
}

// ---------------------------------------------------------------------------
// loads and stores of the kernels with fused ends.  These kernels run for 5-30 us, of which
// fetching their instructions is a visible part, so the code per element is kept short: one
// bounds check per tile (`fits`, over the tile's last pencil; a tile that fails it is skipped by
// the whole block), slots beyond the last pencil load the last one's values and store nothing.
// ---------------------------------------------------------------------------
// FP32 pencil pairs are loaded and stored as 16 bytes, the pair of the last odd pencil and its
// neighbour in the row padding included (the host checks that the padding is there)
__device__ __forceinline__ CV<double> g_cv(double2 s) { return {s.x, s.y}; }
__device__ __forceinline__ CV<float2> g_cv(float4 s) { return {make_float2(s.x, s.z), make_float2(s.y, s.w)}; }
__device__ __forceinline__ double2 g_raw(const CV<double>& v) { return make_double2(v.re, v.im); }
__device__ __forceinline__ float4 g_raw(const CV<float2>& v) {
  return make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
}
typedef unsigned long long g_u64;

// elements t + r M1 of a slot's pencils p, p + 1 (or rows), r = 0, 1, ..; last: the last pencil
template <typename T, int MODE, class Ld>
struct GIn {  // loaders that go through shared memory
  static __device__ __forceinline__ bool fits(const GArgs<T>&, const Ld&, int, int) { return true; }
};
template <typename T, class S>
struct GIn<T, 0, ArrLoad<S>> {
  using W = typename GT<T>::W;
  const S* x;
  unsigned step;
  int n, M1, lim;
  static __device__ __forceinline__ bool fits(const GArgs<T>& a, const ArrLoad<S>& ld, int last, int io) {
    const int lim = a.L < ld.Lin ? a.L : ld.Lin;
    // an FP32 pair is read whole: up to the odd neighbour of its first pencil
    const unsigned top = sizeof(T) == 8 ? (unsigned)last : (unsigned)last | 1u;
    return lim >= 1 && (g_u64)top + (g_u64)io * ld.ostride + (g_u64)(lim - 1) * ld.jstride < (g_u64)ld.n;
  }
  __device__ __forceinline__ GIn(const GArgs<T>& a, const ArrLoad<S>& ld, int p, int last, int io, int t) {
    constexpr int PAIR = GT<T>::PAIR;
    p = p <= last ? p : last / PAIR * PAIR;
    lim = ld.Lin;
    M1 = a.st[0].M;
    n = t;
    x = ld.ptr + ((unsigned)p + (unsigned)io * ld.ostride + (unsigned)t * ld.jstride);
    step = (unsigned)M1 * ld.jstride;
  }
  __device__ __forceinline__ GV<T> next() {
    W s{};
    if (n < lim) s = *reinterpret_cast<const W*>(x);
    x += step;
    n += M1;
    return g_cv(s);
  }
};
template <typename T, class S>
struct GIn<T, 0, MirrorLoad<S>> {
  const S* x;
  unsigned js;
  int n, M1, len;
  static __device__ __forceinline__ bool fits(const GArgs<T>&, const MirrorLoad<S>& ld, int last, int io) {
    static_assert(sizeof(T) == 8, "the mirrored passes are FP64");
    return (g_u64)(unsigned)last + (g_u64)io * ld.ostride + (g_u64)(ld.T / 2) * ld.jstride < (g_u64)ld.n;
  }
  __device__ __forceinline__ GIn(const GArgs<T>& a, const MirrorLoad<S>& ld, int p, int last, int io, int t) {
    p = p <= last ? p : last;
    js = ld.jstride;
    len = ld.T;
    M1 = a.st[0].M;
    n = t;
    x = ld.ptr + ((unsigned)p + (unsigned)io * ld.ostride);
  }
  __device__ __forceinline__ GV<T> next() {
    const int m = n <= len - n ? n : len - n;
    n += M1;
    return g_cv(x[(unsigned)m * js]);
  }
};
// rows of the half spectrum, pre-processed for the half-length backward transform
template <typename T, class S>
struct GIn<T, 2, ArrLoad<S>> {
  using R_ = typename GT<T>::R;
  const S *xa, *xb;
  const typename GT<T>::W* tw;
  int n, M1, L;
  static __device__ __forceinline__ bool fits(const GArgs<T>& a, const ArrLoad<S>& ld, int last, int) {
    return a.L < ld.Lin && (g_u64)(unsigned)last * ld.rowstride + (unsigned)a.L < (g_u64)ld.n;
  }
  __device__ __forceinline__ GIn(const GArgs<T>& a, const ArrLoad<S>& ld, int p, int last, int, int t) {
    xa = ld.ptr + (unsigned)(p <= last ? p : last) * ld.rowstride;
    xb = ld.ptr + (unsigned)(p < last ? p + 1 : last) * ld.rowstride;
    L = a.L;
    tw = a.twT;
    M1 = a.st[0].M;
    n = t;
  }
  __device__ __forceinline__ CV<double> at(int k, double) const { return {xa[k].x, xa[k].y}; }
  __device__ __forceinline__ CV<float2> at(int k, float2) const {
    const float2 u = xa[k], v = xb[k];
    return {make_float2(u.x, v.x), make_float2(u.y, v.y)};
  }
  __device__ __forceinline__ GV<T> next() {
    GV<T> xk = at(n, R_()), xm = at(L - n, R_());
    if (n == 0) xk.im = xm.im = g_const<R_>(0.);
    // s = X_k + conj X_(L-k), d = X_k - conj X_(L-k), Z_k = s + i d exp(+2 pi i k / 2L)
    const GV<T> s = {g_add(xk.re, xm.re), g_sub(xk.im, xm.im)}, d = {g_sub(xk.re, xm.re), g_add(xk.im, xm.im)};
    const GV<T> u = v_mulc(d, __ldg(tw + n));
    n += M1;
    return {g_sub(s.re, u.im), g_add(s.im, u.re)};
  }
};
// rows of n0 reals (even, aligned for pairs), (x_2n, x_2n+1)
template <typename T, class X>
struct GIn<T, 1, FieldRowLoad<X>> {
  using X2 = typename FieldRowLoad<X>::S2;
  const X2 *xa, *xb;
  int n, M1, lim;
  static __device__ __forceinline__ bool fits(const GArgs<T>&, const FieldRowLoad<X>& ld, int last, int) {
    return (g_u64)((unsigned)last + 1u) * (unsigned)ld.n0 <= (g_u64)ld.n;
  }
  __device__ __forceinline__ GIn(const GArgs<T>& a, const FieldRowLoad<X>& ld, int p, int last, int, int t) {
    lim = ld.n0 / 2;
    xa = reinterpret_cast<const X2*>(ld.x + (unsigned)(p <= last ? p : last) * (unsigned)ld.n0);
    xb = reinterpret_cast<const X2*>(ld.x + (unsigned)(p < last ? p + 1 : last) * (unsigned)ld.n0);
    M1 = a.st[0].M;
    n = t;
  }
  __device__ __forceinline__ GV<T> next() {
    X2 u{}, v{};
    if (n < lim) {
      u = xa[n];
      if constexpr (sizeof(T) == 4) v = xb[n];
    }
    n += M1;
    if constexpr (sizeof(T) == 8)
      return {(T)u.x, (T)u.y};
    else
      return {make_float2((float)u.x, (float)v.x), make_float2((float)u.y, (float)v.y)};
  }
};

// Noise of the R2C half spectrum (R2CNoise) for elements n and n + L/2 of a slot's pencils, L even
// the last torus extent: stored indices and eigenvalue indices linear in n, the self-conjugate
// rule reduced to a flag of the pencil and n == 0.  Pencil p + 1 follows p in every layout.
template <typename T>
struct GNoise {
  unsigned si, ss, li, ls, second;  // first index and stride: stored frequency, eigenvalue
  int h;
  bool mirror, selfA, selfB;
  const R2CNoise& z;
  __device__ __forceinline__ GNoise(const GArgs<T>& a, const R2CNoise& nz, int p, int last, int io) : z(nz) {
    const int k1 = z.dim == 3 ? io : 0;
    second = p < last ? 1u : 0u;
    p = p <= last ? p : last;
    h = a.L / 2;
    const unsigned c0 = (unsigned)z.T0c;
    si = (unsigned)p;
    ss = c0;
    if (z.dim == 3) {
      if (z.transposed) {
        si += c0 * (unsigned)z.ext[2] * (unsigned)k1;
      } else {
        si += c0 * (unsigned)k1;
        ss = c0 * (unsigned)z.ext[1];
      }
    }
    mirror = z.dct == 1;
    const unsigned d0 = z.dct == 1 ? (unsigned)z.D0 : (z.dct == 2 ? (unsigned)z.ext[0] : c0);
    li = (unsigned)p;
    ls = d0;
    if (z.dim == 3) {
      const int m1 = mirror && k1 > z.ext[1] / 2 ? z.ext[1] - k1 : k1;
      li += d0 * (unsigned)m1;
      ls = d0 * (unsigned)(mirror ? z.D1 : z.ext[1]);
    }
    const bool self1 = z.dim < 3 || k1 == 0 || 2 * k1 == z.ext[1];
    selfA = self1 && (p == 0 || 2 * p == z.ext[0]);
    selfB = self1 && 2 * (p + 1) == z.ext[0];
  }
  __device__ __forceinline__ bool fits(const GArgs<T>& a) const {  // for the tile's last pencil
    return (g_u64)li + (g_u64)ls * (unsigned)(mirror ? h : a.L - 1) < (g_u64)z.nsq &&
           (!z.noise || 2 * ((g_u64)si + (g_u64)ss * (unsigned)(a.L - 1)) + 1 < (g_u64)z.nnoise);
  }
  // value of the normals (r1, r2) at an eigenvalue index
  __device__ __forceinline__ cx<T> value(unsigned l, bool self, T r1, T r2) const {
    const T lam = ((const T*)z.sq)[l];
    T s;
    if constexpr (sizeof(T) == 8)
      // lambda / sqrt(2) (r2cfieldbackend.hh:322-323) as a product with 1/sqrt(2) held in two
      // doubles, whose result is the rounded quotient but for rare last digits (N. Brisebarre and
      // J.-M. Muller, "Correctly rounded multiplication by arbitrary precision constants", IEEE
      // Trans. Comput. 57, 2008)
      s = fma(lam, 0x1.6a09e667f3bcdp-1, lam * -0x1.bdd3413b26456p-55);
    else
      s = lam * (T)0.70710678118654752440084436210484903928;
    return self ? mk<T>(lam * r1, (T)0) : mk<T>(s * r1, s * r2);
  }
  __device__ __forceinline__ void one(unsigned i, unsigned l0, unsigned l1, int n, bool self, cx<T>& x0,
                                      cx<T>& x1) const {
    T r1, r2, r3, r4;
    const uint4 c = pair_bits(z.seed, i, z.epoch ? __ldg(z.epoch) : 0u);
    box_muller(c.x, c.y, r1, r2);
    box_muller(c.z, c.w, r3, r4);
    x0 = value(l0, self && n == 0, r1, r2);
    x1 = value(l1, self && n == 0, r3, r4);
  }
  __device__ __forceinline__ void pair(int n, GV<T>& x0, GV<T>& x1) const {
    const unsigned i = si + ss * (unsigned)n;
    const unsigned l0 = li + ls * (unsigned)n, l1 = li + ls * (unsigned)(mirror ? h - n : h + n);
    cx<T> u0, u1;
    one(i, l0, l1, n, selfA, u0, u1);
    if constexpr (sizeof(T) == 8) {
      x0 = {u0.x, u0.y};
      x1 = {u1.x, u1.y};
    } else {
      cx<T> v0, v1;
      one(i + second, l0 + second, l1 + second, n, selfB, v0, v1);
      x0 = {make_float2(u0.x, v0.x), make_float2(u0.y, v0.y)};
      x1 = {make_float2(u1.x, v1.x), make_float2(u1.y, v1.y)};
    }
  }
};

// noise of a buffer in the reference's draw order
template <typename T>
struct GIn<T, 0, R2CNoiseBuf> {
  GNoise<T> g;
  int n, M1, L;
  static __device__ __forceinline__ bool fits(const GArgs<T>& a, const R2CNoiseBuf& ld, int last, int io) {
    return GNoise<T>(a, ld, last, last, io).fits(a);
  }
  __device__ __forceinline__ GIn(const GArgs<T>& a, const R2CNoiseBuf& ld, int p, int last, int io, int t)
      : g(a, ld, p, last, io), n(t), M1(a.st[0].M), L(a.L) {}
  __device__ __forceinline__ cx<T> one(unsigned i, unsigned l, bool self) const {
    const double* const u = g.z.noise + 2 * (size_t)i;
    return g.value(l, self, (T)u[0], (T)u[1]);
  }
  __device__ __forceinline__ GV<T> next() {
    const unsigned i = g.si + g.ss * (unsigned)n;
    const unsigned l = g.li + g.ls * (unsigned)(g.mirror && 2 * n > L ? L - n : n);
    const bool end = n == 0 || 2 * n == L;
    n += M1;
    const cx<T> u = one(i, l, end && g.selfA);
    if constexpr (sizeof(T) == 8) {
      return {u.x, u.y};
    } else {
      const cx<T> v = one(i + g.second, l + g.second, end && g.selfB);
      return {make_float2(u.x, v.x), make_float2(u.y, v.y)};
    }
  }
};

// outputs j < Lout of a slot's pencils (or rows)
template <typename T, int MODE, class St>
struct GOut;
template <typename T, int MODE, class S>
struct GOut<T, MODE, ArrStore<S>> {
  using W = typename GT<T>::W;
  S* x;
  unsigned js;
  int lim;
  static __device__ __forceinline__ bool fits(const GArgs<T>& a, const ArrStore<S>& st, int last, int io) {
    if (MODE != 0) return true;  // rows: the split phase checks each store
    const unsigned top = sizeof(T) == 8 ? (unsigned)last : (unsigned)last | 1u;
    return (g_u64)top + (g_u64)io * st.ostride + (g_u64)(a.Lout - 1) * st.jstride < (g_u64)st.n;
  }
  __device__ __forceinline__ GOut(const GArgs<T>& a, const ArrStore<S>& st, int p, int last, int io) {
    js = st.jstride;
    lim = p <= last ? a.Lout : 0;
    x = st.ptr + ((unsigned)p + (unsigned)io * st.ostride);
  }
  __device__ __forceinline__ void put(int j, const GV<T>& v) const {
    if (j < lim) *reinterpret_cast<W*>(x + (unsigned)j * js) = g_raw(v);
  }
};
template <typename T>
__device__ __noinline__ T g_mutate(int kind, T lam, T v) {
  return apply_mutator<T>(kind, lam, v);
}
// rows of n0 reals (even, aligned for pairs)
template <typename T, class X>
struct GOut<T, 2, FieldRowStore<X>> {
  using X2 = typename FieldRowStore<X>::S2;
  X2 *xa, *xb;
  int lim, lim2, kind;
  T lam;
  static __device__ __forceinline__ bool fits(const GArgs<T>&, const FieldRowStore<X>& st, int last, int) {
    return (g_u64)((unsigned)last + 1u) * (unsigned)st.n0 <= (g_u64)st.n;
  }
  __device__ __forceinline__ GOut(const GArgs<T>& a, const FieldRowStore<X>& st, int p, int last, int) {
    lim = p <= last ? a.Lout / 2 : 0;
    lim2 = p < last ? a.Lout / 2 : 0;
    xa = reinterpret_cast<X2*>(st.out + (unsigned)p * (unsigned)st.n0);
    xb = reinterpret_cast<X2*>(st.out + (unsigned)(p + 1) * (unsigned)st.n0);
    kind = st.transform;
    lam = (T)st.boxcox;
  }
  __device__ __forceinline__ void pair(X2* y, int m, T u, T v) const {
    if (kind) {
      u = g_mutate<T>(kind, lam, u);
      v = g_mutate<T>(kind, lam, v);
    }
    X2 s;
    s.x = (X)u;
    s.y = (X)v;
    y[m] = s;
  }
  __device__ __forceinline__ void put(int m, const GV<T>& w) const {
    if constexpr (sizeof(T) == 8) {
      if (m < lim) pair(xa, m, w.re, w.im);
    } else {
      if (m < lim) pair(xa, m, w.re.x, w.im.x);
      if (m < lim2) pair(xb, m, w.re.y, w.im.y);
    }
  }
};

// eigenvalue factors of a slot's pencils: linear in the pass index, mirrored for the DCT layout
template <typename T>
struct GFac {
  const T* f;
  unsigned stride, second;
  int ext;  // index j > ext / 2 reads ext - j
  static __device__ __forceinline__ unsigned first(const MultMid& m, int p, int io, unsigned& stride) {
    const int k1 = m.dim == 3 ? io : 0;
    if (m.layout == 0) {
      const int m1 = k1 <= m.ext[1] / 2 ? k1 : m.ext[1] - k1;
      stride = m.dim == 3 ? (unsigned)m.D0 * (unsigned)m.D1 : (unsigned)m.D0;
      return (unsigned)p + (m.dim == 3 ? (unsigned)m.D0 * (unsigned)m1 : 0u);
    }
    stride = m.dim == 3 ? (unsigned)m.LC0 * (unsigned)m.ext[1] : (unsigned)m.LC0;
    return (unsigned)p + (m.dim == 3 ? (unsigned)m.LC0 * (unsigned)k1 : 0u);
  }
  static __device__ __forceinline__ bool fits(const GArgs<T>& a, const MultMid& m, int last, int io) {
    unsigned s;
    const unsigned i = first(m, last, io, s);
    return (g_u64)i + (g_u64)s * (unsigned)(m.layout == 0 ? a.L / 2 : a.L - 1) < (g_u64)m.nfac;
  }
  static __device__ __forceinline__ bool fits(const GArgs<T>&, const NoMid&, int, int) { return true; }
  __device__ __forceinline__ GFac(const GArgs<T>& a, const MultMid& m, int p, int last, int io) {
    f = (const T*)m.fac + first(m, p <= last ? p : last, io, stride);
    second = p < last ? 1u : 0u;
    ext = m.layout == 0 ? a.L : 2 * a.L;
  }
  __device__ __forceinline__ typename GT<T>::R at(int j) const {
    const T* const g = f + stride * (unsigned)(2 * j > ext ? ext - j : j);
    if constexpr (sizeof(T) == 8)
      return g[0];
    else
      return make_float2(g[0], g[second]);
  }
};

// ---------------------------------------------------------------------------
// the pass.  ROWS: pencils are rows, else B * PAIR adjacent pencils of outer block io.
// MODE 0: complex pencils; 1: rows of 2L reals to L + 1 complex; 2: the reverse (FFTW c2r
// semantics, see k_c2r).  SIGN: direction of a pass without Mid (with Mid: forward, factor,
// backward).  FUSED: the end stages load and store themselves (at least two stages, radices up
// to 8); otherwise the inputs and outputs go through shared memory, for any length.
// ---------------------------------------------------------------------------
template <typename T, bool ROWS, int MODE, int SIGN, bool FUSED, class Ld, class Mid, class St>
__global__ void __launch_bounds__(kGThreads, 1)
    k_g(const __grid_constant__ GArgs<T> a, const __grid_constant__ Ld ld, const __grid_constant__ Mid mid,
        const __grid_constant__ St st) {
  chain_start();
  using R_ = typename GT<T>::R;
  using V = CV<R_>;
  constexpr int PAIR = GT<T>::PAIR;
  constexpr bool DIRECT = FUSED && g_direct<Ld>::value;
  static_assert(!Mid::active || (MODE == 0 && SIGN < 0), "the fused pass is forward, factor, backward");
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* const sm = reinterpret_cast<V*>(g_smem);
  // the shared stages take their arguments by reference: from shared memory, the kernel's
  // parameters being slow to read through a pointer
  const GArgs<T>* sa = &a;
  if (!FUSED && a.args_at) {
    int* const d = reinterpret_cast<int*>(sm + a.args_at);
    for (int i = threadIdx.x; i < (int)(sizeof(a) / 4); i += blockDim.x) d[i] = reinterpret_cast<const int*>(&a)[i];
    sa = reinterpret_cast<const GArgs<T>*>(sm + a.args_at);
    __syncthreads();
  }
  chain_wait();
  const GTile<T, ROWS> ti{a};
  const int nt = blockDim.x;
  const int B = a.B, np = a.np;
  int io = 0, p0;
  if constexpr (ROWS) {
    p0 = (int)blockIdx.x * B * PAIR;
  } else {
    io = (int)((unsigned)blockIdx.x / (unsigned)a.tpo);
    p0 = ((int)blockIdx.x - io * a.tpo) * B * PAIR;
  }
  const int sj = ti.sj(), M1 = a.st[0].M, M1s = ti.m1s();
  const int S = a.S;
  const bool blue = !FUSED && a.chirp != nullptr;
  const V zero = {g_const<R_>(0.), g_const<R_>(0.)};
  // last pencil of the tile
  const int last = (p0 + B * PAIR < np ? p0 + B * PAIR : np) - 1;
  if constexpr (FUSED) {
    if (!(GIn<T, MODE, Ld>::fits(a, ld, last, io) && GOut<T, MODE, St>::fits(a, st, last, io) &&
          GFac<T>::fits(a, mid, last, io))) {  // the same for all threads of the block
      if (threadIdx.x == 0) report_error(1u);
      return;
    }
  }

  // ---- inputs and outputs of a slot's pencils ----------------------------------------
  auto fetch = [&](int p, int n) -> V {  // element n < L
    V x;
    if constexpr (MODE == 1) {
      x = g_real(ld, p, np, n, T());
    } else if constexpr (MODE == 2) {
      V xk = g_load(ld, p, np, n, 0, T()), xm = g_load(ld, p, np, a.L - n, 0, T());
      if (n == 0) xk.im = xm.im = g_const<R_>(0.);
      // s = X_k + conj X_(L-k), d = X_k - conj X_(L-k), Z_k = s + i d exp(+2 pi i k / 2L)
      const V s = {g_add(xk.re, xm.re), g_sub(xk.im, xm.im)}, d = {g_sub(xk.re, xm.re), g_add(xk.im, xm.im)};
      const V t = v_mulc(d, __ldg(a.twT + n));
      x = {g_sub(s.re, t.im), g_add(s.im, t.re)};
    } else {
      x = g_load(ld, p, np, n, io, T());
    }
    return SIGN > 0 ? v_swap(x) : x;
  };
  auto enter = [&](int n, const V& x) -> V { return blue ? v_mul(x, __ldg(a.chirp + n)) : x; };
  auto put = [&](int p, int j, V v) {  // output j of the (backward, with Mid) transform
    if constexpr (SIGN > 0) v = v_swap(v);
    if constexpr (MODE == 2) {
      if (2 * j < a.Lout) g_store_real(st, p, np, j, a.Lout, v);
    } else {
      if (j < a.Lout) g_store(st, p, np, j, io, v);
    }
  };

  // ---- load phase ----------------------------------------------------------------------
  if constexpr (!DIRECT) {
    bool done = false;
    if constexpr (MODE == 1 && !g_direct<Ld>::value) {
      if (ld.mirror) {  // a row even about T0/2 = L: evaluate reals 0..L, mirror the rest
        static_assert(PAIR == 1, "covariance rows are FP64");
        double* const rs = reinterpret_cast<double*>(sm);
        const int cnt = a.L + 1;
        for (int u = threadIdx.x; u < B * cnt; u += nt) {
          const int b = u / cnt, j = u - b * cnt;
          const double v = p0 + b < np ? ld.template real<double>(p0 + b, j) : 0.;
          rs[2 * (ti.slot0(b) + ti.place(j >> 1)) + (j & 1)] = v;
          const int k = 2 * a.L - j;
          if (j > 0 && j < a.L) rs[2 * (ti.slot0(b) + ti.place(k >> 1)) + (k & 1)] = v;
        }
        if (blue) {
          __syncthreads();
          for (int u = threadIdx.x; u < B * a.L; u += nt) {
            int b, n;
            ti.split(u, a.L, a.mL, b, n);
            V* const x = sm + ti.slot0(b) + ti.place(n);
            *x = enter(n, *x);
          }
        }
        done = true;
      }
    }
    if constexpr (std::is_same<Ld, R2CNoise>::value) {
      if (a.L % 2 == 0) {  // one generator call for elements n and n + L/2
        static_assert(!ROWS, "noise pencils are strided");
        // the block size is a multiple of B: a thread keeps its slot
        const int b = threadIdx.x & (B - 1), dn = nt >> a.lgB, h = a.L / 2;
        if (!GNoise<T>(a, ld, last, last, io).fits(a)) {  // the same for all threads of the block
          if (threadIdx.x == 0) report_error(1u);
          return;
        }
        const GNoise<T> g(a, ld, p0 + PAIR * b, last, io);
        V* const row = sm + b;
        for (int n = (int)threadIdx.x >> a.lgB; n < h; n += dn) {
          V x0, x1;
          g.pair(n, x0, x1);
          row[ti.place(n)] = enter(n, v_swap(x0));
          row[ti.place(n + h)] = enter(n + h, v_swap(x1));
        }
        done = true;
      }
    }
    if (!done)
      for (int u = threadIdx.x; u < B * a.L; u += nt) {
        int b, n;
        ti.split(u, a.L, a.mL, b, n);
        sm[ti.slot0(b) + ti.place(n)] = enter(n, fetch(p0 + PAIR * b, n));
      }
    __syncthreads();
    g_stage<T, ROWS, 0>(*sa, 0);
  } else {
    auto stage_first = [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int u = threadIdx.x; u < B * M1; u += nt) {
        int b, t;
        ti.split(u, M1, a.st[0].mM, b, t);
        V* const x = sm + ti.slot0(b) + t * sj;
        GIn<T, MODE, Ld> in(a, ld, p0 + PAIR * b, last, io, t);
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
          v[r] = in.next();
          if (SIGN > 0) v[r] = v_swap(v[r]);
        }
        g_dft<R>(v);
        x[0] = v[0];
#pragma unroll
        for (int q = 1; q < R; q++) x[q * M1s] = v_mul(v[q], __ldg(a.tw + (q - 1) * M1 + t));
      }
    };
    switch (a.st[0].R) {
#define PF_G_CASE(RR) \
  case RR: stage_first(std::integral_constant<int, RR>()); break;
      PF_G_FUSED_RADICES(PF_G_CASE)
#undef PF_G_CASE
      default: break;
    }
    __syncthreads();
  }

  // ---- any length ------------------------------------------------------------------------
  if constexpr (!FUSED) {
    auto forward = [&]() {  // the forward transform, and for Bluestein the convolution
      for (int s = 1; s < S - 1; s++) g_stage<T, ROWS, 1>(*sa, s);
      if (blue) {
        g_stage<T, ROWS, 5>(*sa, S - 1);
        for (int s = S - 2; s >= 1; s--) g_stage<T, ROWS, 3>(*sa, s);
        g_stage<T, ROWS, 4>(*sa, 0);
      } else if (S > 1) {
        g_stage<T, ROWS, 2>(*sa, S - 1);
      }
    };
    // output j < L of forward(): with Bluestein's algorithm in the order of the inputs
    auto result = [&](int b, int j) -> V {
      const int at = ti.slot0(b) + (blue ? ti.place(j) : ti.place_out(j));
      const V v = sm[at];
      return blue ? v_mul(v_swap(v), __ldg(a.chirp + j)) : v;
    };
    forward();
    if constexpr (Mid::active) {
      for (int u = threadIdx.x; u < B * a.L; u += nt) {
        int b, j;
        ti.split(u, a.L, a.mL, b, j);
        const V y = v_swap(g_mid(mid, p0 + PAIR * b, np, j, io, result(b, j)));
        sm[ti.slot0(b) + (blue ? ti.place(j) : ti.place_out(j))] = enter(j, y);
      }
      __syncthreads();
      if (blue) {  // the backward transform is a second convolution
        g_stage<T, ROWS, 0>(*sa, 0);
        forward();
      } else {
        if (S > 1) g_stage<T, ROWS, 2>(*sa, S - 1);
        for (int s = S - 2; s >= 1; s--) g_stage<T, ROWS, 3>(*sa, s);
        g_stage<T, ROWS, 4>(*sa, 0);
      }
      const int n1 = a.Lout < a.L ? a.Lout : a.L;
      for (int u = threadIdx.x; u < B * n1; u += nt) {
        int b, j;
        ti.split(u, n1, a.mLout, b, j);
        const V v = blue ? result(b, j) : sm[ti.slot0(b) + ti.place(j)];
        put(p0 + PAIR * b, j, v_swap(v));
      }
    } else if constexpr (MODE != 1) {
      const int n1 = MODE == 2 ? (a.Lout + 1) / 2 : a.Lout;
      for (int u = threadIdx.x; u < B * n1; u += nt) {
        int b, j;
        ti.split(u, n1, a.mLout, b, j);
        put(p0 + PAIR * b, j, result(b, j));
      }
    }
  } else {
    // ---- fused ends ----------------------------------------------------------------------
#pragma unroll 1
    for (int s = 1; s < S - 1; s++) {
      switch (a.st[s].R) {
#define PF_G_CASE(RR) \
  case RR: g_stage_r<T, ROWS, 1, RR>(a, a.st[s]); break;
        PF_G_FUSED_RADICES(PF_G_CASE)
#undef PF_G_CASE
        default: break;
      }
    }
    if constexpr (MODE == 1) {
      switch (a.st[S - 1].R) {
#define PF_G_CASE(RR) \
  case RR: g_stage_r<T, ROWS, 2, RR>(a, a.st[S - 1]); break;
        PF_G_FUSED_RADICES(PF_G_CASE)
#undef PF_G_CASE
        default: break;
      }
    } else {
      // last stage: outputs to the store, or through the factor and the first stage of the
      // backward transform
      auto stage_last = [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const GStage& g = a.st[S - 1];
        for (int u = threadIdx.x; u < B * g.nb; u += nt) {
          int b, w;
          ti.split(u, g.nb, g.mnb, b, w);
          V* const x = sm + ti.slot0(b) + ti.base_last(w);
          V v[R];
#pragma unroll
          for (int r = 0; r < R; r++) v[r] = x[r * sj];
          g_dft<R>(v);
          if constexpr (Mid::active) {
            const GFac<T> fac(a, mid, p0 + PAIR * b, last, io);
#pragma unroll
            for (int q = 0; q < R; q++) {
              const R_ f = fac.at(w + q * g.nb);
              v[q] = {g_mul(v[q].im, f), g_mul(v[q].re, f)};
            }
            g_dft<R>(v);
#pragma unroll
            for (int r = 0; r < R; r++) x[r * sj] = v[r];
          } else {
            const GOut<T, MODE, St> out(a, st, p0 + PAIR * b, last, io);
#pragma unroll
            for (int q = 0; q < R; q++) out.put(w + q * g.nb, SIGN > 0 ? v_swap(v[q]) : v[q]);
          }
        }
      };
      switch (a.st[S - 1].R) {
#define PF_G_CASE(RR) \
  case RR: stage_last(std::integral_constant<int, RR>()); break;
        PF_G_FUSED_RADICES(PF_G_CASE)
#undef PF_G_CASE
        default: break;
      }
      if constexpr (Mid::active) {
        __syncthreads();
#pragma unroll 1
        for (int s = S - 2; s >= 1; s--) {
          switch (a.st[s].R) {
#define PF_G_CASE(RR) \
  case RR: g_stage_r<T, ROWS, 3, RR>(a, a.st[s]); break;
            PF_G_FUSED_RADICES(PF_G_CASE)
#undef PF_G_CASE
            default: break;
          }
        }
        auto stage_final = [&](auto rc) {
          constexpr int R = decltype(rc)::value;
          for (int u = threadIdx.x; u < B * M1; u += nt) {
            int b, t;
            ti.split(u, M1, a.st[0].mM, b, t);
            V* const x = sm + ti.slot0(b) + t * sj;
            V v[R];
            v[0] = x[0];
#pragma unroll
            for (int q = 1; q < R; q++) v[q] = v_mul(x[q * M1s], __ldg(a.tw + (q - 1) * M1 + t));
            g_dft<R>(v);
            const GOut<T, MODE, St> out(a, st, p0 + PAIR * b, last, io);
#pragma unroll
            for (int r = 0; r < R; r++) out.put(t + r * M1, v_swap(v[r]));
          }
        };
        switch (a.st[0].R) {
#define PF_G_CASE(RR) \
  case RR: stage_final(std::integral_constant<int, RR>()); break;
          PF_G_FUSED_RADICES(PF_G_CASE)
#undef PF_G_CASE
          default: break;
        }
      }
    }
  }

  if constexpr (MODE == 1) {  // split of the half-length transform: X_k and X_(L-k) from Z_k and Z_(L-k)
    const R_ half = g_const<R_>(0.5);
    const int n1 = a.L / 2 + 1;
    auto z = [&](int b, int k) -> V {
      const int at = ti.slot0(b) + (blue ? ti.place(k) : ti.place_out(k));
      return blue ? v_mul(v_swap(sm[at]), __ldg(a.chirp + k)) : sm[at];
    };
    for (int u = threadIdx.x; u < B * n1; u += nt) {
      int b, k;
      ti.split(u, n1, a.mLout, b, k);
      const V zk = z(b, k), zm = z(b, k == 0 ? 0 : a.L - k);
      // e = (Z_k + conj Z_(L-k)) / 2, o = (Z_k - conj Z_(L-k)) / 2, t = -i o exp(-pi i k / L):
      // X_k = e + t, X_(L-k) = conj(e - t)
      const V e = {g_mul(half, g_add(zk.re, zm.re)), g_mul(half, g_sub(zk.im, zm.im))};
      const V o = {g_mul(half, g_sub(zk.re, zm.re)), g_mul(half, g_add(zk.im, zm.im))};
      const V t = v_mul(V{o.im, g_neg(o.re)}, __ldg(a.twT + k));
      const int p = p0 + PAIR * b;
      g_store(st, p, np, k, 0, v_add(e, t));
      if (2 * k != a.L) g_store(st, p, np, a.L - k, 0, V{g_sub(e.re, t.re), g_sub(t.im, e.im)});
    }
  }
}

}  // namespace pf
