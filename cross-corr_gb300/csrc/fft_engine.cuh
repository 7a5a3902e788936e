// fft_engine.cuh -- device code of the fused FFT correlation (sm_103a):
// in-register small transforms, the shared-memory passes built from them, and
// the three kernels of the pipeline
//
//   row_forward   real rows -> half spectra of the rows (zero padding implied)
//   col_pairs     column transforms of left and right, product, inverse
//   row_inverse   half spectra of the output rows -> scaled, cropped output
//
// and col_forward, which transforms the columns of matrices whose spectra
// several outputs share.  fft_engine.cu plans and launches them.
//
// Transforms are decimation-in-frequency over two to four radix passes
// N = R1 [Ra [Rb]] R3.  A pass reads and writes the same places, so a pass
// costs one shared-memory round trip and one barrier.  The column kernel
// never leaves digit-reversed order: left and right spectra are in the same
// order, and the inverse (decimation in time) starts from it, so its
// innermost forward pass, the product and the first inverse pass happen in
// registers.  The row kernels transform two real rows as one complex row; a
// thread owns the passes' items k and N - k together, so the two rows'
// spectra are separated (and joined) in registers too.
//
// What bounds it.  FP32: a scalar form took 57-63% of the issue slots at 25-40%
// of the FMA pipe and under 20% of memory, so a thread works on two transforms
// in packed pairs (add, mul and fma .f32x2: the same rate per value in half
// the instructions): two adjacent columns or two row pairs.  With that the
// instructions fell by a third to two fifths and the kernels wait for their
// loads and for shared memory (50 to 65% of its wavefronts), 16 to 24 warps
// per SM: 64 outputs of 511x511 take 73 us, 113 in the scalar form.  Of the
// column kernel's time at 4096 points, the passes themselves are 57%, the left
// spectra's loads 14%, the stores 12%, the twiddles' loads 10%, the rows' 1%
// (each left out in turn, before the twiddles were halved and half of the left
// spectra loaded ahead).
// FP64 is bound by its pipe (82 to 84% busy in col_pairs and row_inverse, 69 to
// 77% in the forward kernels, whose launches are short; 1.0 TFLOP/s measured).
#pragma once

#include <cstdint>

#include "xc_common.cuh"

namespace xc {
namespace fe {

// ---------------------------------------------------------------------------
// Scalars of the transforms: f2 (two FP32 values, one of each transform) or
// double.
// ---------------------------------------------------------------------------
struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return x;
}
__device__ __forceinline__ float hi(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return y;
}
__device__ __forceinline__ f2 add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 neg(f2 a) {
  a.v ^= 0x8000000080000000ull;
  return a;
}
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double fma(double a, double b, double c) { return ::fma(a, b, c); }
__device__ __forceinline__ double neg(double a) { return -a; }

template <typename S>
struct Sc;
template <>
struct Sc<f2> {
  using real = float;
  static constexpr int NV = 2;  // transforms per thread
  using Tw = float2;  // a twiddle, the same for both transforms
  static __device__ __forceinline__ f2 bc(double c) { return pack((float)c, (float)c); }
};
template <>
struct Sc<double> {
  using real = double;
  static constexpr int NV = 1;
  using Tw = double2;
  static __device__ __forceinline__ double bc(double c) { return c; }
};

// A complex value of each transform: 16 bytes for either scalar.
template <typename S>
struct alignas(16) Cp {
  S x, y;
};
template <typename S>
__device__ __forceinline__ Cp<S> cadd(Cp<S> a, Cp<S> b) {
  return {add(a.x, b.x), add(a.y, b.y)};
}
template <typename S>
__device__ __forceinline__ Cp<S> csub(Cp<S> a, Cp<S> b) {
  return {sub(a.x, b.x), sub(a.y, b.y)};
}
// a + (D i) b, D = +-1
template <int D, typename S>
__device__ __forceinline__ Cp<S> cadd_i(Cp<S> a, Cp<S> b) {
  if (D > 0) return {sub(a.x, b.y), add(a.y, b.x)};
  return {add(a.x, b.y), sub(a.y, b.x)};
}
// a + c b for a real constant
template <typename S>
__device__ __forceinline__ Cp<S> cfma(S c, Cp<S> b, Cp<S> a) {
  return {fma(c, b.x, a.x), fma(c, b.y, a.y)};
}
// a + (D i c) b
template <int D, typename S>
__device__ __forceinline__ Cp<S> cfma_i(S c, S nc, Cp<S> b, Cp<S> a) {
  if (D > 0) return {fma(nc, b.y, a.x), fma(c, b.x, a.y)};
  return {fma(c, b.y, a.x), fma(nc, b.x, a.y)};
}
// a * b, or a * conj(b)
template <bool CONJ, typename S>
__device__ __forceinline__ Cp<S> cmul(Cp<S> a, Cp<S> b) {
  const S nby = neg(b.y);
  if (CONJ) return {fma(a.y, b.y, mul(a.x, b.x)), fma(a.x, nby, mul(a.y, b.x))};
  return {fma(a.y, nby, mul(a.x, b.x)), fma(a.x, b.y, mul(a.y, b.x))};
}
template <bool CONJ>
__device__ __forceinline__ Cp<f2> cmul(Cp<f2> a, float2 w) {
  return cmul<CONJ>(a, Cp<f2>{pack(w.x, w.x), pack(w.y, w.y)});
}
template <bool CONJ>
__device__ __forceinline__ Cp<double> cmul(Cp<double> a, double2 w) {
  return cmul<CONJ>(a, Cp<double>{w.x, w.y});
}
template <typename S>
__device__ __forceinline__ Cp<S> czero() {
  return {Sc<S>::bc(0.0), Sc<S>::bc(0.0)};
}
template <typename S>
__device__ __forceinline__ Cp<S> csel(bool p, Cp<S> a, Cp<S> b) {
  return p ? a : b;
}

// ---------------------------------------------------------------------------
// In-register transforms of R values, natural order in and out,
// X[k] = sum_n x[n] exp(D 2 pi i n k / R), D = -1 forward, +1 inverse.
// ---------------------------------------------------------------------------
template <typename S, int D, int R>
struct Dft;

template <typename S, int D>
struct Dft<S, D, 2> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    const Cp<S> a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
  }
};

template <typename S, int D>
struct Dft<S, D, 4> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    const Cp<S> a = cadd(x[0], x[2]), b = csub(x[0], x[2]);
    const Cp<S> c = cadd(x[1], x[3]), d = csub(x[1], x[3]);
    x[0] = cadd(a, c);
    x[1] = cadd_i<D>(b, d);
    x[2] = csub(a, c);
    x[3] = cadd_i<-D>(b, d);
  }
};

template <typename S, int D>
struct Dft<S, D, 3> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    constexpr double h = 0.8660254037844386467637231707529362;  // sin(2 pi / 3)
    const S ch = Sc<S>::bc(h), nh = Sc<S>::bc(-h);
    const Cp<S> s = cadd(x[1], x[2]), d = csub(x[1], x[2]);
    const Cp<S> m = cfma(Sc<S>::bc(-0.5), s, x[0]);
    x[0] = cadd(x[0], s);
    x[1] = cfma_i<D>(ch, nh, d, m);
    x[2] = cfma_i<-D>(ch, nh, d, m);
  }
};

// Odd primes by symmetry: sums and differences of x[n], x[R-n].
template <typename S, int D>
struct Dft<S, D, 5> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    constexpr double k1 = 0.3090169943749474241022934171828191, k2 = -0.8090169943749474241022934171828191;
    constexpr double l1 = 0.9510565162951535721164393333793821, l2 = 0.5877852522924731291687059546390728;
    const S c1 = Sc<S>::bc(k1), c2 = Sc<S>::bc(k2), s1 = Sc<S>::bc(l1), s2 = Sc<S>::bc(l2), n1 = Sc<S>::bc(-l1);
    const Cp<S> a1 = cadd(x[1], x[4]), b1 = csub(x[1], x[4]);
    const Cp<S> a2 = cadd(x[2], x[3]), b2 = csub(x[2], x[3]);
    const Cp<S> m1 = cfma(c2, a2, cfma(c1, a1, x[0]));
    const Cp<S> m2 = cfma(c1, a2, cfma(c2, a1, x[0]));
    const Cp<S> r1 = {fma(s2, b2.x, mul(s1, b1.x)), fma(s2, b2.y, mul(s1, b1.y))};
    const Cp<S> r2 = {fma(n1, b2.x, mul(s2, b1.x)), fma(n1, b2.y, mul(s2, b1.y))};
    x[0] = cadd(x[0], cadd(a1, a2));
    x[1] = cadd_i<D>(m1, r1);
    x[4] = cadd_i<-D>(m1, r1);
    x[2] = cadd_i<D>(m2, r2);
    x[3] = cadd_i<-D>(m2, r2);
  }
};

template <typename S, int D>
struct Dft<S, D, 7> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    constexpr double k1 = 0.6234898018587335305250048840042398, k2 = -0.2225209339563144042889025644967948,
                     k3 = -0.9009688679024191262361023195074451;
    constexpr double l1 = 0.7818314824680298087084445266740578, l2 = 0.9749279121818236070181316829939312,
                     l3 = 0.4338837391175581204757683328483587;
    const S c1 = Sc<S>::bc(k1), c2 = Sc<S>::bc(k2), c3 = Sc<S>::bc(k3);
    const S s1 = Sc<S>::bc(l1), s2 = Sc<S>::bc(l2), s3 = Sc<S>::bc(l3), n1 = Sc<S>::bc(-l1), n3 = Sc<S>::bc(-l3);
    const Cp<S> a1 = cadd(x[1], x[6]), b1 = csub(x[1], x[6]);
    const Cp<S> a2 = cadd(x[2], x[5]), b2 = csub(x[2], x[5]);
    const Cp<S> a3 = cadd(x[3], x[4]), b3 = csub(x[3], x[4]);
    const Cp<S> m1 = cfma(c3, a3, cfma(c2, a2, cfma(c1, a1, x[0])));
    const Cp<S> m2 = cfma(c1, a3, cfma(c3, a2, cfma(c2, a1, x[0])));
    const Cp<S> m3 = cfma(c2, a3, cfma(c1, a2, cfma(c3, a1, x[0])));
    const Cp<S> r1 = {fma(s3, b3.x, fma(s2, b2.x, mul(s1, b1.x))), fma(s3, b3.y, fma(s2, b2.y, mul(s1, b1.y)))};
    const Cp<S> r2 = {fma(n1, b3.x, fma(n3, b2.x, mul(s2, b1.x))), fma(n1, b3.y, fma(n3, b2.y, mul(s2, b1.y)))};
    const Cp<S> r3 = {fma(s2, b3.x, fma(n1, b2.x, mul(s3, b1.x))), fma(s2, b3.y, fma(n1, b2.y, mul(s3, b1.y)))};
    x[0] = cadd(x[0], cadd(a1, cadd(a2, a3)));
    x[1] = cadd_i<D>(m1, r1);
    x[6] = cadd_i<-D>(m1, r1);
    x[2] = cadd_i<D>(m2, r2);
    x[5] = cadd_i<-D>(m2, r2);
    x[3] = cadd_i<D>(m3, r3);
    x[4] = cadd_i<-D>(m3, r3);
  }
};

template <typename S, int D>
struct Dft<S, D, 8> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    constexpr double k = 0.7071067811865475244008443621048490;
    const S h = Sc<S>::bc(k), nh = Sc<S>::bc(-k);
    Cp<S> e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    Dft<S, D, 4>::run(e);
    Dft<S, D, 4>::run(o);
    // o[n] exp(D 2 pi i n / 8): n = 1: h (1 + D i) o, n = 2: D i o, n = 3: -h (1 - D i) o
    const Cp<S> u1 = cadd_i<D>(o[1], o[1]), u3 = cadd_i<-D>(o[3], o[3]);
    x[0] = cadd(e[0], o[0]);
    x[4] = csub(e[0], o[0]);
    x[1] = cfma(h, u1, e[1]);
    x[5] = cfma(nh, u1, e[1]);
    x[2] = cadd_i<D>(e[2], o[2]);
    x[6] = cadd_i<-D>(e[2], o[2]);
    x[3] = cfma(nh, u3, e[3]);
    x[7] = cfma(h, u3, e[3]);
  }
};

template <typename S, int D>
struct Dft<S, D, 16> {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    constexpr double kh = 0.7071067811865475244008443621048490;
    constexpr double kc = 0.9238795325112867561281831893967882, ks = 0.3826834323650897717284599840303988;
    const S h = Sc<S>::bc(kh), nh = Sc<S>::bc(-kh);
    Cp<S> y[4][4];  // [n2][k1]
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) y[n2][n1] = x[4 * n1 + n2];
      Dft<S, D, 4>::run(y[n2]);
    }
    // y[n2][k1] *= exp(D 2 pi i n2 k1 / 16)
    constexpr double sg = D > 0 ? 1.0 : -1.0;
    const auto rot = [](Cp<S> a, double wx, double wy) {
      const S cx = Sc<S>::bc(wx), cy = Sc<S>::bc(wy), ny = Sc<S>::bc(-wy);
      return Cp<S>{fma(a.y, ny, mul(a.x, cx)), fma(a.x, cy, mul(a.y, cx))};
    };
    y[1][1] = rot(y[1][1], kc, sg * ks);
    y[1][3] = rot(y[1][3], ks, sg * kc);
    y[3][1] = rot(y[3][1], ks, sg * kc);
    y[3][3] = rot(y[3][3], -kc, -sg * ks);
    // the eighths, left unscaled: u = (1 + D i) y or (1 - D i) y, times +-h below
    const Cp<S> u12 = cadd_i<D>(y[1][2], y[1][2]), u32 = cadd_i<-D>(y[3][2], y[3][2]);
    const Cp<S> u21 = cadd_i<D>(y[2][1], y[2][1]), u23 = cadd_i<-D>(y[2][3], y[2][3]);
    {  // k1 = 0
      Cp<S> z[4] = {y[0][0], y[1][0], y[2][0], y[3][0]};
      Dft<S, D, 4>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) x[4 * k2] = z[k2];
    }
    {  // k1 = 1: second input h u21
      const Cp<S> a = cfma(h, u21, y[0][1]), b = cfma(nh, u21, y[0][1]);
      const Cp<S> c = cadd(y[1][1], y[3][1]), d = csub(y[1][1], y[3][1]);
      x[1] = cadd(a, c);
      x[5] = cadd_i<D>(b, d);
      x[9] = csub(a, c);
      x[13] = cadd_i<-D>(b, d);
    }
    {  // k1 = 2: inputs y02, h u12, D i y22, -h u32
      const Cp<S> a = cadd_i<D>(y[0][2], y[2][2]), b = cadd_i<-D>(y[0][2], y[2][2]);
      const Cp<S> c = csub(u12, u32), d = cadd(u12, u32);
      x[2] = cfma(h, c, a);
      x[6] = cfma_i<D>(h, nh, d, b);
      x[10] = cfma(nh, c, a);
      x[14] = cfma_i<-D>(h, nh, d, b);
    }
    {  // k1 = 3: third input -h u23
      const Cp<S> a = cfma(nh, u23, y[0][3]), b = cfma(h, u23, y[0][3]);
      const Cp<S> c = cadd(y[1][3], y[3][3]), d = csub(y[1][3], y[3][3]);
      x[3] = cadd(a, c);
      x[7] = cadd_i<D>(b, d);
      x[11] = csub(a, c);
      x[15] = cadd_i<-D>(b, d);
    }
  }
};

// R = A B with coprime factors (Good's prime-factor algorithm, no twiddles):
// n = (B n1 + A n2) mod R, k with k = k1 mod A and k = k2 mod B.
constexpr int crt(int A, int B, int k1, int k2) {
  for (int k = 0; k < A * B; ++k)
    if (k % A == k1 && k % B == k2) return k;
  return 0;
}
template <typename S, int D, int A, int B>
struct DftPfa {
  static __device__ __forceinline__ void run(Cp<S>* x) {
    constexpr int R = A * B;
    Cp<S> y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = x[(B * n1 + A * n2) % R];
      Dft<S, D, A>::run(y[n2]);  // n k / R = n1 k / A + n2 k / B (mod 1)
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      Cp<S> z[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
      Dft<S, D, B>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) x[crt(A, B, k1, k2)] = z[k2];
    }
  }
};
template <typename S, int D>
struct Dft<S, D, 6> : DftPfa<S, D, 2, 3> {};
template <typename S, int D>
struct Dft<S, D, 10> : DftPfa<S, D, 2, 5> {};
template <typename S, int D>
struct Dft<S, D, 12> : DftPfa<S, D, 4, 3> {};
template <typename S, int D>
struct Dft<S, D, 14> : DftPfa<S, D, 2, 7> {};

// ---------------------------------------------------------------------------
// Lengths and their passes.  All lengths are multiples of 16, at most 25%
// apart (33% below 64).  Columns: X(N, R1, Ra, R3), R1 >= Ra >= R3, as few
// passes as 16 registers' worth allows.  Rows: X(N, R1, Ra, Rb, R3), with R1
// and R3 small, because a row thread holds two items of its first (inverse) or
// last (forward) pass, and alike, so that neither pass leaves threads idle.
// ---------------------------------------------------------------------------
#define XC_FFT_COLS_SHORT(X)                                                                              \
  X(16, 4, 1, 4) X(32, 8, 1, 4) X(48, 8, 1, 6) X(64, 8, 1, 8) X(80, 10, 1, 8) X(96, 12, 1, 8)              \
  X(112, 14, 1, 8) X(128, 16, 1, 8) X(160, 16, 1, 10) X(192, 16, 1, 12) X(224, 16, 1, 14) X(256, 16, 1, 16) \
  X(320, 8, 8, 5) X(384, 8, 8, 6) X(448, 8, 8, 7) X(512, 8, 8, 8)
#define XC_FFT_COLS_LONG(X)                                                                               \
  X(640, 10, 8, 8) X(768, 12, 8, 8) X(896, 14, 8, 8) X(1024, 16, 8, 8) X(1280, 16, 10, 8)                   \
  X(1536, 16, 12, 8) X(1792, 16, 14, 8) X(2048, 16, 16, 8) X(2560, 16, 16, 10) X(3072, 16, 16, 12)           \
  X(3584, 16, 16, 14) X(4096, 16, 16, 16)
#define XC_FFT_COLS(X) XC_FFT_COLS_SHORT(X) XC_FFT_COLS_LONG(X)
#define XC_FFT_ROWS(X)                                                                                     \
  X(16, 4, 1, 1, 4) X(32, 8, 1, 1, 4) X(48, 8, 1, 1, 6) X(64, 8, 1, 1, 8) X(80, 10, 1, 1, 8)                 \
  X(96, 12, 1, 1, 8) X(112, 8, 1, 1, 14) X(128, 4, 8, 1, 4) X(160, 4, 10, 1, 4) X(192, 8, 3, 1, 8)           \
  X(224, 4, 14, 1, 4) X(256, 8, 4, 1, 8) X(320, 8, 5, 1, 8) X(384, 8, 6, 1, 8) X(448, 8, 7, 1, 8)            \
  X(512, 8, 8, 1, 8) X(640, 8, 10, 1, 8) X(768, 8, 12, 1, 8) X(896, 8, 14, 1, 8) X(1024, 8, 16, 1, 8)         \
  X(1280, 8, 5, 4, 8) X(1536, 8, 6, 4, 8) X(1792, 8, 7, 4, 8) X(2048, 8, 8, 4, 8) X(2560, 8, 8, 5, 8)         \
  X(3072, 8, 8, 6, 8) X(3584, 8, 8, 7, 8) X(4096, 8, 8, 8, 8)

// Geometry of a pass structure.  Element (q1, qa, qb, m) -- index q1 S1 +
// qa Sa + qb R3 + m -- lies at q1 P1 + qa Pa + qb PR + m in shared memory:
// odd strides, so that passes that walk a digit across lanes hit different
// banks.
template <int N_, int R1_, int Ra_, int Rb_, int R3_>
struct Passes {
  static constexpr int N = N_, R1 = R1_, Ra = Ra_, Rb = Rb_, R3 = R3_;
  static_assert(R1 * Ra * Rb * R3 == N, "factors of the length");
  static constexpr int S1 = N / R1, Sa = S1 / Ra;
  static constexpr int TF = N / R3;  // items of the last pass
  static constexpr int PR = R3 | 1;
  static constexpr int Pa = Rb > 1 ? (Rb * PR) | 1 : PR;
  static constexpr int P1 = Ra > 1 ? (Ra * Pa) | 1 : Pa;
  static constexpr int rows = R1 * P1;        // padded length
  static constexpr int tw_a = (R1 - 1) * S1;  // twiddles: [q - 1][o] of each pass but the last
  static constexpr int tw_b = tw_a + (Ra - 1) * Sa;
  static constexpr int n_tw = tw_b + (Rb - 1) * R3;
  // place of offset o < S1 within the first digit's block
  static __device__ __forceinline__ int in_block(int o) {
    if (Ra == 1) return o;
    const int qa = o / Sa, r = o - qa * Sa;
    if (Rb == 1) return qa * Pa + r;
    const int qb = r / R3;
    return qa * Pa + qb * PR + (r - qb * R3);
  }
  // place of the last pass's item i, whose outputs are k = i + q TF
  static __device__ __forceinline__ int last_item(int i) {
    if (Ra == 1) return i * P1;
    const int q1 = i % R1, r = i / R1;
    if (Rb == 1) return q1 * P1 + r * Pa;
    return q1 * P1 + (r % Ra) * Pa + (r / Ra) * PR;
  }
};
template <int N>
struct RowPasses;
template <int N>
struct ColPasses;
#define XC_DEF(N_, A_, B_, C_, D_) \
  template <>                      \
  struct RowPasses<N_> : Passes<N_, A_, B_, C_, D_> {};
XC_FFT_ROWS(XC_DEF)
#undef XC_DEF
#define XC_DEF(N_, A_, B_, D_) \
  template <>                  \
  struct ColPasses<N_> : Passes<N_, A_, B_, 1, D_> {};
XC_FFT_COLS(XC_DEF)
#undef XC_DEF

// A pass between the first and the last, in place: radix R, items of `LEN`
// elements' blocks with offsets o < ST; block b of the pass starts at
// place(b), its elements PS apart.  Forward and row-inverse passes are
// decimation in frequency (twiddles after), column-inverse ones decimation in
// time (twiddles before).
template <typename S, int D, bool DIT, int R, int PS, int STEP>
__device__ __forceinline__ void butterfly(Cp<S>* base, const typename Sc<S>::Tw* __restrict__ tw, int tw_step) {
  Cp<S> x[R];
  if (!DIT) {
#pragma unroll
    for (int m = 0; m < R; ++m) x[m] = base[m * PS * STEP];
    Dft<S, D, R>::run(x);
    base[0] = x[0];
#pragma unroll
    for (int q = 1; q < R; ++q) base[q * PS * STEP] = cmul<(D > 0)>(x[q], tw[(q - 1) * tw_step]);
  } else {
    x[0] = base[0];
#pragma unroll
    for (int q = 1; q < R; ++q) x[q] = cmul<(D > 0)>(base[q * PS * STEP], tw[(q - 1) * tw_step]);
    Dft<S, D, R>::run(x);
#pragma unroll
    for (int m = 0; m < R; ++m) base[m * PS * STEP] = x[m];
  }
}
template <typename S, int D, bool DIT, typename L, int STEP>
__device__ __forceinline__ void mid_passes(Cp<S>* z, int it0, int step, const typename Sc<S>::Tw* __restrict__ tw) {
  if constexpr (L::Ra > 1) {
    for (int it = it0; it < L::N / L::Ra; it += step) {
      const int b = it / L::Sa, o = it - b * L::Sa;
      const int at = b * L::P1 + (L::Rb > 1 ? (o / L::R3) * L::PR + o % L::R3 : o);
      butterfly<S, D, DIT, L::Ra, L::Pa, STEP>(z + at * STEP, tw + L::tw_a + o, L::Sa);
    }
    __syncthreads();
  }
  if constexpr (L::Rb > 1) {
    static_assert(!DIT, "four passes: rows only");
    for (int it = it0; it < L::N / L::Rb; it += step) {
      const int b = it / L::R3, o = it - b * L::R3;
      const int at = (b / L::Ra) * L::P1 + (b % L::Ra) * L::Pa + o;
      butterfly<S, D, DIT, L::Rb, L::PR, STEP>(z + at * STEP, tw + L::tw_b + o, L::R3);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Layout of the half spectra between the kernels: matrix by matrix, blocks of
// CB = 2^lgcb columns, [block][row / RQ][column in block][row % RQ] of complex
// values, rows rounded up to whole groups of RQ and columns 0..N/2 to whole
// blocks (the columns beyond N/2 are never written by the row kernels nor read
// by them).  A whole block is contiguous (column kernels).  RQ is 4 for FP32
// blocks of two columns (lengths over 2048): a thread of the row kernels moves
// its four rows of a column as 32 contiguous bytes instead of four times 8,
// each of those instructions in 16 lines (2048x2048 x 16: 1.64 ms, 1.80 with
// RQ = 1).  Blocks of four columns keep RQ = 1: their lines are half as many,
// and the column kernels' two 8-byte accesses in the place of one of 16 cost
// more than the row kernels gain (511x511 x 64: row kernels 43 us against 49,
// column kernel 39 against 31); so do ragged batches, whose row launches mix
// both kinds of blocks.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int spectrum_rows(int H, int rq) { return (H + rq - 1) / rq * rq; }
// element offset of row y in a block of CB columns (columns RQ apart)
template <int CB, int RQ>
__device__ __forceinline__ int row_at(int y) {
  return y / RQ * (RQ * CB) + y % RQ;
}
template <typename T>
struct Cx {
  T x, y;
};
template <typename T>
struct RowSide {
  const T* src;  // matrices, H x W each
  Cx<T>* dst;    // half spectra of their rows
  int H, W;
  int groups;    // CTAs per matrix
  T scale;       // of the spectra (times the 1/2 of the separation)
};
// Ragged batches: one record per matrix (or pair), and for every CTA (column
// kernel: every unit) the record it works on and its place in it.
template <typename T>
struct RagRow {
  const T* src;
  Cx<T>* dst;
  int H, W, lgcb;
  T scale;
};
template <typename T>
struct RagCol {
  const Cx<T>* left;
  const Cx<T>* right;
  Cx<T>* out;
  int Hl, Hr, Sy, nblk;
};
template <typename T>
struct RagInv {
  const Cx<T>* src;
  T* out;
  int Sy, Sx, Wr, lgcb;
  T scale_hi, scale_lo;
};
template <typename T>
struct RowFwdArgs {
  RowSide<T> a, b;    // blocks [0, a_blocks) on side a, the rest on side b
  unsigned a_blocks;
  int nblk, lgcb;
  const void* tw;     // Sc<S>::Tw entries
  const T* zeros;     // a row of zeros, read in the place of rows past the last
  const RagRow<T>* items;  // ragged: records, and per CTA (record, row group)
  const int2* ctas;
};

template <typename T>
struct ColArgs {
  const void* left;   // row spectra of the lefts, or (LPRE) their full spectra
  const void* right;  // the same of the rights (RPRE)
  Cx<T>* out;         // column-inverted products, Sy rows in output order
  int Hl, Hr, Sy;
  int nblk;
  int n_left;         // lefts l0 .. l0 + n_left - 1 of this launch
  int l0, k0, k1;     // partners k0 .. k1 - 1 of each
  int n_kg, kc;       // partner groups of kc partners
  long long r_l, r_k, r_off;  // right(l, k) = l r_l + k r_k - r_off within `right`
  const void* tw;
  const RagCol<T>* items;  // ragged: records, and per unit (record, block)
  const int2* units;
  int n_units;
};
template <typename T>
struct ColFwdSide {
  const Cx<T>* src;   // row spectra, H rows
  void* dst;          // full spectra: Cp<S> in pass order
  int H;
};
template <typename T>
struct ColFwdArgs {
  ColFwdSide<T> a, b;       // units [0, a_units) are side a's, the rest side b's
  long long a_units, units;  // matrices x blocks
  const void* tw;
};
template <typename T>
struct RowInvArgs {
  const Cx<T>* src;   // [output of this launch][block], Sy rows
  T* out;
  int Sy, Sx, Wr;
  int groups;         // CTAs per output
  int nblk, lgcb;
  int l0, k0, nk;     // output index t of the launch: l = l0 + t / nk, k = k0 + t % nk
  long long o_l, o_k;
  T scale_hi, scale_lo;
  const void* tw;
  const RagInv<T>* items;  // ragged: records, and per CTA (record, row group)
  const int2* ctas;
};

// Row kernels: a transform (NV row pairs) on TP threads, Q of them per CTA
// (fewer in short launches, see per_cta).
template <int N>
struct RowCfg {
  using L = RowPasses<N>;
  static constexpr int TP = L::TF / 2;
  // 64 to 128 threads, the count that leaves the fewest lanes of the last
  // warp idle (small CTAs overlap one's loads with another's passes: 64
  // threads measured 34 us against 47 with 256 at 64 outputs of 511x511)
  static constexpr int idle(int q) { return ((q * TP + 31) / 32 * 32 - q * TP) * 128 / (q * TP); }
  static constexpr int pick() {
    int best = 0;
    for (int q = 1; q == 1 || q * TP <= 128; ++q)
      if (best == 0 || best * TP < 64 || idle(q) < idle(best))
        if (best == 0 || best * TP < 64 || q * TP <= 128) best = q;
    return best;
  }
  static constexpr int Q = pick();
  static constexpr int threads = Q * TP;
  static constexpr int min_ctas = 512 / threads;  // up to 128 registers a thread
  static constexpr int FS = L::rows | 1;
  static constexpr int smem = Q * FS * 16;
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Loads of what an earlier kernel of the chain wrote.  Not __ldg: the compiler
// may move a non-coherent load above the wait for that kernel; volatile
// assembly stays below it.
__device__ __forceinline__ float ld(const float* g) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(g));
  return v;
}
__device__ __forceinline__ double ld(const double* g) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(g));
  return v;
}
__device__ __forceinline__ float2 ld(const float2* g) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(g));
  return v;
}
__device__ __forceinline__ float4 ld(const float4* g) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(g));
  return v;
}
__device__ __forceinline__ double2 ld(const double2* g) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(g));
  return v;
}
// 32 bytes: a column's RQ = 4 rows
struct alignas(32) Col4 {
  float2 r[4];
};
__device__ __forceinline__ Col4 ld(const Col4* g) {
  Col4 v;
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v.r[0].x), "=f"(v.r[0].y), "=f"(v.r[1].x), "=f"(v.r[1].y), "=f"(v.r[2].x), "=f"(v.r[2].y),
                 "=f"(v.r[3].x), "=f"(v.r[3].y)
               : "l"(g));
  return v;
}
__device__ __forceinline__ void st(Col4* g, float2 r0, float2 r1, float2 r2, float2 r3) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(g), "f"(r0.x), "f"(r0.y), "f"(r1.x),
               "f"(r1.y), "f"(r2.x), "f"(r2.y), "f"(r3.x), "f"(r3.y)
               : "memory");
}
__device__ __forceinline__ Cp<f2> ld(const Cp<f2>* g) {
  Cp<f2> v;
  asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x.v), "=l"(v.y.v) : "l"(g));
  return v;
}
__device__ __forceinline__ Cp<double> ld(const Cp<double>* g) {
  const double2 v = ld(reinterpret_cast<const double2*>(g));
  return {v.x, v.y};
}

__device__ __forceinline__ Cp<f2> gather(const float* v) { return {pack(v[0], v[2]), pack(v[1], v[3])}; }
__device__ __forceinline__ Cp<double> gather(const double* v) { return {v[0], v[1]}; }

template <typename S, int N, bool RAG, int RQ>
__global__ void __launch_bounds__(RowCfg<N>::threads, RowCfg<N>::min_ctas) row_forward(const RowFwdArgs<typename Sc<S>::real> p) {
  using L = RowPasses<N>;
  using C = Cp<S>;
  using T = typename Sc<S>::real;
  constexpr int TP = RowCfg<N>::TP, NV = Sc<S>::NV;
  const int Q = blockDim.x / TP;  // at most RowCfg<N>::Q
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_launch();
  const auto* __restrict__ tw = static_cast<const typename Sc<S>::Tw*>(p.tw);
  int H, W, group, lgcb;
  const T* __restrict__ src;
  Cx<T>* dst;
  T scale;
  if constexpr (RAG) {
    const int2 e = p.ctas[blockIdx.x];
    const RagRow<T>& it = p.items[e.x];
    H = it.H;
    W = it.W;
    lgcb = it.lgcb;
    src = it.src;
    dst = it.dst;
    scale = it.scale;
    group = e.y;
  } else {
    const bool first = blockIdx.x < p.a_blocks;
    const unsigned b = first ? blockIdx.x : blockIdx.x - p.a_blocks;
    const unsigned groups = (unsigned)(first ? p.a.groups : p.b.groups);
    const unsigned mat = b / groups;
    H = first ? p.a.H : p.b.H;
    W = first ? p.a.W : p.b.W;
    lgcb = p.lgcb;
    src = (first ? p.a.src : p.b.src) + (long long)mat * H * W;
    dst = (first ? p.a.dst : p.b.dst) + (((long long)mat * p.nblk * spectrum_rows(H, RQ)) << lgcb);
    scale = first ? p.a.scale : p.b.scale;
    group = (int)(b - mat * groups);
  }
  const int f = threadIdx.x / TP, i = threadIdx.x - f * TP;
  const int row0 = (group * Q + f) * (2 * NV);
  C* z = reinterpret_cast<C*>(smem_raw) + f * RowCfg<N>::FS;
  const T* r[2 * NV];
#pragma unroll
  for (int j = 0; j < 2 * NV; ++j) r[j] = row0 + j < H ? src + (long long)(row0 + j) * W : p.zeros;
  pdl_wait();
  for (int o = i; o < L::S1; o += TP) {
    C x[L::R1];
#pragma unroll
    for (int m = 0; m < L::R1; ++m) {
      const int k = o + m * L::S1;
      T v[2 * NV];
#pragma unroll
      for (int j = 0; j < 2 * NV; ++j) v[j] = k < W ? ld(r[j] + k) : T(0);
      x[m] = gather(v);
    }
    Dft<S, -1, L::R1>::run(x);
    C* base = z + L::in_block(o);
    base[0] = x[0];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) base[q * L::P1] = cmul<false>(x[q], tw[(q - 1) * L::S1 + o]);
  }
  __syncthreads();
  mid_passes<S, -1, false, L, 1>(z, i, TP, tw);
  if (row0 >= H) return;
  // Last pass of items i and TF - i (thread 0: items 0 and TF / 2), whose
  // outputs pair up as k and N - k: for thread 0 within each item.
  const bool t0 = i == 0;
  const int iy = t0 ? L::TF / 2 : L::TF - i;
  C x[L::R3], y[L::R3];
  {
    const C* bx = z + L::last_item(i);
    const C* by = z + L::last_item(iy);
#pragma unroll
    for (int m = 0; m < L::R3; ++m) {
      x[m] = bx[m];
      y[m] = by[m];
    }
  }
  Dft<S, -1, L::R3>::run(x);
  Dft<S, -1, L::R3>::run(y);
  // The two rows' spectra: A = (Z[k] + conj Z[-k]) / 2, B = (Z[k] - conj Z[-k]) / 2i,
  // with the side's scale in the same product.
  S hs;
  if constexpr (NV == 2) hs = pack(0.5f * scale, 0.5f * scale);
  else hs = T(0.5) * scale;
  const int cb = 1 << lgcb, HP = spectrum_rows(H, RQ);
  dst += (long long)row0 * cb;
  const auto put = [&](int k, C zk, C zn) {
    const C a = {mul(hs, add(zk.x, zn.x)), mul(hs, sub(zk.y, zn.y))};
    const C bb = {mul(hs, add(zk.y, zn.y)), mul(hs, sub(zn.x, zk.x))};
    Cx<T>* d = dst + (long long)(k >> lgcb) * HP * cb + (k & (cb - 1)) * RQ;
    if constexpr (RQ == 4) {
      st(reinterpret_cast<Col4*>(d), make_float2(lo(a.x), lo(a.y)), make_float2(lo(bb.x), lo(bb.y)),
         make_float2(hi(a.x), hi(a.y)), make_float2(hi(bb.x), hi(bb.y)));
    } else if constexpr (NV == 2) {
      *reinterpret_cast<float2*>(d) = make_float2(lo(a.x), lo(a.y));
      if (row0 + 1 < H) *reinterpret_cast<float2*>(d + cb) = make_float2(lo(bb.x), lo(bb.y));
      if (row0 + 2 < H) *reinterpret_cast<float2*>(d + 2 * cb) = make_float2(hi(a.x), hi(a.y));
      if (row0 + 3 < H) *reinterpret_cast<float2*>(d + 3 * cb) = make_float2(hi(bb.x), hi(bb.y));
    } else {
      *reinterpret_cast<double2*>(d) = make_double2(a.x, a.y);
      if (row0 + 1 < H) *reinterpret_cast<double2*>(d + cb) = make_double2(bb.x, bb.y);
    }
  };
#pragma unroll
  for (int q = 0; q < (L::R3 + 1) / 2; ++q)
    put(i + q * L::TF, x[q], csel(t0, x[(L::R3 - q) % L::R3], y[L::R3 - 1 - q]));
#pragma unroll
  for (int q = 0; q < L::R3 / 2; ++q)
    put(iy + q * L::TF, y[q], csel(t0, y[L::R3 - 1 - q], x[L::R3 - 1 - q]));
  if (t0) {  // column N / 2, its own partner
    const C h = L::R3 % 2 == 0 ? x[L::R3 / 2] : y[L::R3 / 2];
    put(N / 2, h, h);
  }
}

template <typename S, int N, bool RAG, int RQ>
__global__ void __launch_bounds__(RowCfg<N>::threads, RowCfg<N>::min_ctas) row_inverse(const RowInvArgs<typename Sc<S>::real> p) {
  using L = RowPasses<N>;
  using C = Cp<S>;
  using T = typename Sc<S>::real;
  constexpr int TP = RowCfg<N>::TP, NV = Sc<S>::NV;
  const int Q = blockDim.x / TP;  // at most RowCfg<N>::Q
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_launch();
  const auto* __restrict__ tw = static_cast<const typename Sc<S>::Tw*>(p.tw);
  int Sy, Sx, Wr, group, lgcb;
  const Cx<T>* __restrict__ src;
  T* out;
  T scale_hi, scale_lo;
  if constexpr (RAG) {
    const int2 e = p.ctas[blockIdx.x];
    const RagInv<T>& it = p.items[e.x];
    Sy = it.Sy;
    Sx = it.Sx;
    Wr = it.Wr;
    lgcb = it.lgcb;
    src = it.src;
    out = it.out;
    scale_hi = it.scale_hi;
    scale_lo = it.scale_lo;
    group = e.y;
  } else {
    const unsigned t = blockIdx.x / (unsigned)p.groups;
    const int l = p.l0 + (int)t / p.nk, k = p.k0 + (int)t % p.nk;
    Sy = p.Sy;
    Sx = p.Sx;
    Wr = p.Wr;
    lgcb = p.lgcb;
    src = p.src + (((long long)t * p.nblk * spectrum_rows(Sy, RQ)) << lgcb);
    out = p.out + (l * p.o_l + k * p.o_k) * Sy * (long long)Sx;
    scale_hi = p.scale_hi;
    scale_lo = p.scale_lo;
    group = (int)(blockIdx.x - t * (unsigned)p.groups);
  }
  const int f = threadIdx.x / TP, i = threadIdx.x - f * TP;
  const int row0 = (group * Q + f) * (2 * NV);
  C* z = reinterpret_cast<C*>(smem_raw) + f * RowCfg<N>::FS;
  const int cb = 1 << lgcb;
  const int SP = spectrum_rows(Sy, RQ);
  src += (long long)row0 * cb;
  const bool v0 = row0 < Sy, v1 = row0 + 1 < Sy, v2 = row0 + 2 < Sy, v3 = row0 + 3 < Sy;
  // rows A and B of each row pair at column c
  const auto get = [&](int c, C* a, C* b) {
    const Cx<T>* d = src + (long long)(c >> lgcb) * SP * cb + (c & (cb - 1)) * RQ;
    if constexpr (RQ == 4) {  // rows beyond the last are the circular result's next ones
      const Col4 e = v0 ? ld(reinterpret_cast<const Col4*>(d)) : Col4{};
      *a = {pack(e.r[0].x, e.r[2].x), pack(e.r[0].y, e.r[2].y)};
      *b = {pack(e.r[1].x, e.r[3].x), pack(e.r[1].y, e.r[3].y)};
    } else if constexpr (NV == 2) {
      const float2 o = make_float2(0.f, 0.f);
      const float2 e0 = v0 ? ld(reinterpret_cast<const float2*>(d)) : o;
      const float2 e1 = v1 ? ld(reinterpret_cast<const float2*>(d + cb)) : o;
      const float2 e2 = v2 ? ld(reinterpret_cast<const float2*>(d + 2 * cb)) : o;
      const float2 e3 = v3 ? ld(reinterpret_cast<const float2*>(d + 3 * cb)) : o;
      *a = {pack(e0.x, e2.x), pack(e0.y, e2.y)};
      *b = {pack(e1.x, e3.x), pack(e1.y, e3.y)};
    } else {
      const double2 o = make_double2(0.0, 0.0);
      const double2 e0 = v0 ? ld(reinterpret_cast<const double2*>(d)) : o;
      const double2 e1 = v1 ? ld(reinterpret_cast<const double2*>(d + cb)) : o;
      *a = {e0.x, e0.y};
      *b = {e1.x, e1.y};
    }
  };
  pdl_wait();
  // Z = A + i B, Z[N - c] = conj A + i conj B: the inverse transform of Z is
  // row a + i row b.  First pass of items o and S1 - o (o = 0: items 0 and
  // S1 / 2), which use the same columns.
  for (int o = i; o < L::S1 / 2; o += TP) {
    const bool o0 = o == 0;
    const int oy = o0 ? L::S1 / 2 : L::S1 - o;
    constexpr int M = L::R1 / 2;
    C x[L::R1], y[L::R1];
    C cx[M], cy[M];  // the conjugate columns' values
#pragma unroll
    for (int m = 0; m < M; ++m) {
      C a, b;
      get(o + m * L::S1, &a, &b);
      x[m] = cadd_i<1>(a, b);
      cx[m] = {add(a.x, b.y), sub(b.x, a.y)};
      if (m == 0 && o0) x[0] = {a.x, b.x};  // column 0 is real
      get(oy + m * L::S1, &a, &b);
      y[m] = cadd_i<1>(a, b);
      cy[m] = {add(a.x, b.y), sub(b.x, a.y)};
    }
#pragma unroll
    for (int m = M; m < L::R1; ++m) {
      x[m] = m == M ? cy[M - 1] : csel(o0, cx[m == M ? 0 : L::R1 - m], cy[L::R1 - 1 - m]);
      y[m] = csel(o0, cy[L::R1 - 1 - m], cx[L::R1 - 1 - m]);
    }
    if (o0) {  // column N / 2 is real
      C a, b;
      get(N / 2, &a, &b);
      x[M] = {a.x, b.x};
    }
    Dft<S, 1, L::R1>::run(x);
    Dft<S, 1, L::R1>::run(y);
    C* bx = z + L::in_block(o);
    C* by = z + L::in_block(oy);
    bx[0] = x[0];
    by[0] = y[0];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) {
      bx[q * L::P1] = cmul<true>(x[q], tw[(q - 1) * L::S1 + o]);
      by[q * L::P1] = cmul<true>(y[q], tw[(q - 1) * L::S1 + oy]);
    }
  }
  __syncthreads();
  mid_passes<S, 1, false, L, 1>(z, i, TP, tw);
  if (!v0) return;
  T* o0 = out + (long long)row0 * Sx;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int it = i + u * TP;
    C x[L::R3];
    const C* base = z + L::last_item(it);
#pragma unroll
    for (int m = 0; m < L::R3; ++m) x[m] = base[m];
    Dft<S, 1, L::R3>::run(x);
#pragma unroll
    for (int q = 0; q < L::R3; ++q) {
      int sx = it + q * L::TF + Wr - 1;
      if (sx >= N) sx -= N;
      if (sx >= Sx) continue;
      T* d = o0 + sx;
      if constexpr (NV == 2) {
        // the scale as a sum of two terms: rounds like a scaling in higher precision
        const f2 sh = pack(scale_hi, scale_hi), sl = pack(scale_lo, scale_lo);
        const f2 a = fma(x[q].x, sh, mul(x[q].x, sl)), b = fma(x[q].y, sh, mul(x[q].y, sl));
        d[0] = lo(a);
        if (v1) d[Sx] = lo(b);
        if (v2) d[2 * (long long)Sx] = hi(a);
        if (v3) d[3 * (long long)Sx] = hi(b);
      } else {
        d[0] = x[q].x;
        if (v1) d[Sx] = x[q].y;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Column kernels: a unit is one block of CB columns of one matrix (or pair),
// on TU threads, lanes over the block's columns (NV at a time) first; PU
// units per CTA (fewer in short launches).
// ---------------------------------------------------------------------------
template <typename S, int N>
struct ColCfg {
  using L = ColPasses<N>;
  static constexpr int CB = Sc<S>::NV == 2 ? (N <= 2048 ? 4 : 2) : 2;
  static constexpr int lgcb = CB == 4 ? 2 : 1;
  static constexpr int RQ = Sc<S>::NV == 2 && CB == 2 ? 4 : 1;  // rows side by side (but ragged batches: 1)
  static constexpr int LC = CB / Sc<S>::NV;  // lanes across a block's columns
  // Items a pass runs side by side: the count that issues the fewest lane
  // slots over the passes (a pass of n items takes ceil(n / JT) rounds of JT
  // lanes; FP64 pays for idle lanes as for busy ones: at 128 points, 16
  // against 8 of 16 lanes busy in the radix-16 pass).
  static constexpr int slots(int jt) {
    int c = 0;
    for (int r : {L::R1, L::Ra, L::R3})
      if (r > 1) c += (N / r + jt - 1) / jt * jt * r;
    return c;
  }
  static constexpr int best(int a, int b) {
    return a * LC > 256 ? b : b * LC > 256 ? a : slots(a) <= slots(b) ? a : b;
  }
  static constexpr int JT = best(L::TF, best(L::Ra > 1 ? N / L::Ra : L::S1, L::S1));
  static constexpr int TU = JT * LC;
  static constexpr int PU = TU >= 128 ? 1 : (127 + TU) / TU;
  static constexpr int threads = TU * PU;
  static constexpr int unit = L::rows * LC;        // shared-memory elements of a unit
  // CTAs per SM the registers are cut for: 64 registers a thread while no
  // radix exceeds 8, else 128.  FP32 transforms of three passes up to 2048
  // points have a dense form too, with `bufs` units in shared memory: 96
  // registers, 80 with radix 12 and one buffer, where shared memory has room
  // for the warps (column kernel, us, with 128 / 96 / 80 registers: 640 points
  // x 163 outputs 145 / 124 / 124; 768 x 113 183 / 139 / 117; 1024 x 64 125 /
  // 113 / 118 and col_forward slower at 80; 1536 x 28 162 / 128 / 137; 2560 x
  // 10 166 / 164 / 164; FP64 is bound by its pipe in all).  Launches of one
  // wave keep the 128 registers: one pair of 340x340 17.4 us, 18.2 dense.
  static constexpr bool has_dense = Sc<S>::NV == 2 && L::R1 > 8 && L::Ra > 1 && N <= 2048;
  static constexpr int ctas(int bufs, bool dense) {
    const int most = 227 * 1024 / (bufs * PU * unit * 16 + 1024), roomy = 512 / threads;
    const int want = (L::R1 <= 12 && bufs == 1 ? 768 : 640) / threads, fit = want < most ? want : most;
    if (L::R1 <= 8) return 1024 / threads;
    return !dense || fit < roomy ? roomy : fit;
  }
};

// A thread's columns of one row of a block, RQ elements apart.
template <int RQ>
__device__ __forceinline__ Cp<f2> load_row(const Cx<float>* g) {
  if constexpr (RQ == 1) {
    const float4 v = ld(reinterpret_cast<const float4*>(g));
    return {pack(v.x, v.z), pack(v.y, v.w)};
  }
  const float2 u = ld(reinterpret_cast<const float2*>(g)), v = ld(reinterpret_cast<const float2*>(g + RQ));
  return {pack(u.x, v.x), pack(u.y, v.y)};
}
template <int RQ>
__device__ __forceinline__ Cp<double> load_row(const Cx<double>* g) {
  const double2 v = ld(reinterpret_cast<const double2*>(g));
  return {v.x, v.y};
}
template <int RQ>
__device__ __forceinline__ void store_row(Cx<float>* g, Cp<f2> v) {
  if constexpr (RQ == 1) {
    *reinterpret_cast<float4*>(g) = make_float4(lo(v.x), lo(v.y), hi(v.x), hi(v.y));
    return;
  }
  *reinterpret_cast<float2*>(g) = make_float2(lo(v.x), lo(v.y));
  *reinterpret_cast<float2*>(g + RQ) = make_float2(hi(v.x), hi(v.y));
}
template <int RQ>
__device__ __forceinline__ void store_row(Cx<double>* g, Cp<double> v) {
  *reinterpret_cast<double2*>(g) = make_double2(v.x, v.y);
}

// Forward passes of one column block from global memory (H rows; g points at
// the thread's columns) up to, not including, the last; ends with a barrier.
template <typename S, int N, int RQ>
__device__ __forceinline__ void col_load_passes(Cp<S>* z, const Cx<typename Sc<S>::real>* __restrict__ g, int H,
                                                int j0, const typename Sc<S>::Tw* __restrict__ tw) {
  using L = ColPasses<N>;
  using K = ColCfg<S, N>;
  for (int o = j0; o < L::S1; o += K::JT) {
    Cp<S> x[L::R1];
#pragma unroll
    for (int m = 0; m < L::R1; ++m) {
      const int y = o + m * L::S1;
      x[m] = y < H ? load_row<RQ>(g + (L::S1 % RQ == 0 ? row_at<K::CB, RQ>(o) + m * L::S1 * K::CB
                                                             : row_at<K::CB, RQ>(y)))
                   : czero<S>();
    }
    Dft<S, -1, L::R1>::run(x);
    Cp<S>* base = z + L::in_block(o) * K::LC;
    base[0] = x[0];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) base[q * L::P1 * K::LC] = cmul<false>(x[q], tw[(q - 1) * L::S1 + o]);
  }
  __syncthreads();
  mid_passes<S, -1, false, L, K::LC>(z, j0, K::JT, tw);
}

// Place of the last pass's item j in shared memory: the item order of the
// column kernels (lanes over the middle digit) keeps neighbouring lanes an odd
// number of elements apart.
template <typename S, int N>
__device__ __forceinline__ int col_item(int j) {
  using L = ColPasses<N>;
  const int q1 = j / L::Ra, qa = j - q1 * L::Ra;
  return (q1 * L::P1 + qa * L::Pa) * ColCfg<S, N>::LC;
}

// Full spectra of the columns, in pass order: element (q TF + j) LC + lane
// holds output q of the last pass's item j.
template <typename S, int N, bool DENSE>
__global__ void __launch_bounds__(ColCfg<S, N>::threads, ColCfg<S, N>::ctas(1, DENSE)) col_forward(const ColFwdArgs<typename Sc<S>::real> p) {
  using L = ColPasses<N>;
  using C = Cp<S>;
  using K = ColCfg<S, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_launch();
  const auto* __restrict__ tw = static_cast<const typename Sc<S>::Tw*>(p.tw);
  const int pu = threadIdx.x / K::TU, t = threadIdx.x - pu * K::TU;
  const int c = t % K::LC, j0 = t / K::LC;
  C* z = reinterpret_cast<C*>(smem_raw) + pu * K::unit + c;
  const long long u = (long long)blockIdx.x * (blockDim.x / K::TU) + pu;
  const bool live = u < p.units, first = u < p.a_units;
  const long long v = !live ? 0 : first ? u : u - p.a_units;
  const ColFwdSide<typename Sc<S>::real> side = first ? p.a : p.b;
  pdl_wait();
  col_load_passes<S, N, K::RQ>(z, side.src + v * spectrum_rows(side.H, K::RQ) * K::CB + c * (Sc<S>::NV * K::RQ),
                                live ? side.H : 0, j0, tw);
  if (!live) return;
  C* dst = static_cast<C*>(side.dst) + v * N * K::LC + c;
  for (int j = j0; j < L::TF; j += K::JT) {
    C x[L::R3];
    const C* base = z + col_item<S, N>(j);
#pragma unroll
    for (int m = 0; m < L::R3; ++m) x[m] = base[m * K::LC];
    Dft<S, -1, L::R3>::run(x);
#pragma unroll
    for (int q = 0; q < L::R3; ++q) dst[(q * L::TF + j) * K::LC] = x[q];
  }
}

// Products of column blocks: for a left matrix and each of a group of its
// partners, the right columns' transform (unless RPRE: already transformed),
// the product with the left spectrum (LPRE: read from global memory;
// otherwise transformed once per group and kept in shared memory), and the
// inverse transform, whose rows go out in the output's row order.
template <typename S, int N, bool LPRE, bool RPRE, bool RAG, bool DENSE>
__global__ void __launch_bounds__(ColCfg<S, N>::threads, ColCfg<S, N>::ctas(LPRE ? 1 : 2, DENSE)) col_pairs(const ColArgs<typename Sc<S>::real> p) {
  using L = ColPasses<N>;
  using C = Cp<S>;
  using K = ColCfg<S, N>;
  using G = Cx<typename Sc<S>::real>;
  constexpr int NV = Sc<S>::NV, RQ = RAG ? 1 : K::RQ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_launch();
  const auto* __restrict__ tw = static_cast<const typename Sc<S>::Tw*>(p.tw);
  const int pu = threadIdx.x / K::TU, t = threadIdx.x - pu * K::TU;
  const int c = t % K::LC, j0 = t / K::LC;
  C* z = reinterpret_cast<C*>(smem_raw) + pu * K::unit + c;
  const int PU = blockDim.x / K::TU;  // units of this launch's CTAs, at most K::PU
  C* zl = z + (LPRE ? 0 : PU * K::unit);  // left spectrum
  const unsigned gu = blockIdx.x * PU + pu;
  unsigned blk;
  int ll = 0, ka = 0, nk, kc = 1, Hl, Hr, Sy, nblk;
  long long l = 0;
  bool live;
  const G* gl;  // row spectra of the left's and the (first) right's block
  const G* gr;
  G* out;
  if constexpr (RAG) {
    live = gu < (unsigned)p.n_units;
    const int2 e = p.units[live ? gu : 0];
    const RagCol<typename Sc<S>::real>& it = p.items[e.x];
    blk = (unsigned)e.y;
    Hl = it.Hl;
    Hr = it.Hr;
    Sy = it.Sy;
    nblk = it.nblk;
    nk = live ? 1 : 0;
    gl = it.left;
    gr = it.right;
    out = it.out;
  } else {
    nblk = p.nblk;
    // partners first, then lefts: the CTAs that read one block's spectra run
    // side by side and find them in the L2 cache
    const int kg = (int)(gu % (unsigned)p.n_kg);
    const unsigned rest = gu / (unsigned)p.n_kg;
    ll = (int)(rest % (unsigned)p.n_left);  // left of this launch
    blk = rest / (unsigned)p.n_left;
    live = blk < (unsigned)nblk;
    if (!live) blk = 0;
    l = p.l0 + (live ? ll : 0);
    kc = p.kc;
    ka = p.k0 + kg * kc;
    nk = live ? min(kc, p.k1 - ka) : 0;
    Hl = p.Hl;
    Hr = p.Hr;
    Sy = p.Sy;
    gl = static_cast<const G*>(p.left);
    gr = static_cast<const G*>(p.right);
    out = p.out;
  }
  const C* lspec = nullptr;
  pdl_wait();
  if constexpr (LPRE) {
    lspec = static_cast<const C*>(p.left) + (l * nblk + blk) * (long long)N * K::LC + c;
  } else {
    col_load_passes<S, N, RQ>(zl, gl + (l * nblk + blk) * (long long)spectrum_rows(Hl, RQ) * K::CB + c * (NV * RQ),
                          live ? Hl : 0, j0, tw);
    // each thread reads back the items it writes here: no barrier needed
    for (int j = j0; j < L::TF; j += K::JT) {
      C x[L::R3];
      C* base = zl + col_item<S, N>(j);
#pragma unroll
      for (int m = 0; m < L::R3; ++m) x[m] = base[m * K::LC];
      Dft<S, -1, L::R3>::run(x);
#pragma unroll
      for (int m = 0; m < L::R3; ++m) base[m * K::LC] = x[m];
    }
  }
  const long long n_k = RAG ? 1 : p.k1 - p.k0;
  for (int kk = 0; kk < kc; ++kk) {
    const int k = ka + kk;
    const bool act = kk < nk;
    const long long r = !RAG && act ? l * p.r_l + k * p.r_k - p.r_off : 0;
    if constexpr (!RPRE)
      col_load_passes<S, N, RQ>(z, gr + (r * nblk + blk) * (long long)spectrum_rows(Hr, RQ) * K::CB + c * (NV * RQ),
                            act ? Hr : 0, j0, tw);
    for (int j = j0; j < L::TF; j += K::JT) {
      // half of the left spectrum's values are on their way while the right's
      // last pass runs (all of them do not fit the registers): 4096 points,
      // 8 partners, 350 us against 387
      constexpr int PF = LPRE ? L::R3 / 2 : 0;
      C x[L::R3], ahead[PF > 0 ? PF : 1];
#pragma unroll
      for (int q = 0; q < PF; ++q) ahead[q] = ld(lspec + (q * L::TF + j) * K::LC);
      C* base = z + col_item<S, N>(j);
      if constexpr (RPRE) {
        const C* rspec = static_cast<const C*>(p.right) + (r * nblk + blk) * (long long)N * K::LC + c;
#pragma unroll
        for (int q = 0; q < L::R3; ++q) x[q] = ld(rspec + (q * L::TF + j) * K::LC);
      } else {
#pragma unroll
        for (int m = 0; m < L::R3; ++m) x[m] = base[m * K::LC];
        Dft<S, -1, L::R3>::run(x);
      }
      const C* lb = zl + col_item<S, N>(j);
#pragma unroll
      for (int q = 0; q < L::R3; ++q) x[q] = cmul<true>(q < PF ? ahead[q < PF ? q : 0] : LPRE ? ld(lspec + (q * L::TF + j) * K::LC) : lb[q * K::LC], x[q]);
      Dft<S, 1, L::R3>::run(x);
#pragma unroll
      for (int m = 0; m < L::R3; ++m) base[m * K::LC] = x[m];
    }
    __syncthreads();
    mid_passes<S, 1, true, L, K::LC>(z, j0, K::JT, tw);
    if (act) {
      const int SP = spectrum_rows(Sy, RQ);  // at most N: a multiple of 16
      G* o = out + ((ll * n_k + (RAG ? 0 : k - p.k0)) * nblk + blk) * (long long)SP * K::CB + c * (NV * RQ);
      for (int i = j0; i < L::S1; i += K::JT) {
        C x[L::R1];
        const C* base = z + L::in_block(i) * K::LC;
        x[0] = base[0];
#pragma unroll
        for (int q = 1; q < L::R1; ++q) x[q] = cmul<true>(base[q * L::P1 * K::LC], tw[(q - 1) * L::S1 + i]);
        Dft<S, 1, L::R1>::run(x);
#pragma unroll
        for (int m = 0; m < L::R1; ++m) {
          int sy = i + m * L::S1 + Hr - 1;
          if (sy >= N) sy -= N;
          if (sy < SP) store_row<RQ>(o + row_at<K::CB, RQ>(sy), x[m]);
        }
      }
    }
    if (kk + 1 < kc) __syncthreads();  // the next partner's passes overwrite z
  }
}

// What the host needs to launch the kernels of one length.
struct RowKernels {
  const void* forward;
  const void* inverse;
  const void* forward_rq4;  // for column kernels with rq = 4 (FP32 only)
  const void* inverse_rq4;
  const void* rag_forward;  // over a ragged batch's records (FP32 only)
  const void* rag_inverse;
  int threads, q, nv, smem;
};
struct ColFns {
  const void* forward;
  const void* pairs;       // left transformed in the kernel
  const void* pairs_lpre;  // left spectra from col_forward
  const void* pairs_pre;   // both
  const void* rag_pairs;   // `pairs` over a ragged batch's records (FP32 only)
};
struct ColKernels {
  ColFns roomy, dense;  // (the same where a length has one form)
  int threads, pu, lgcb, rq, unit_smem;  // of pu units; shared memory of one buffer
  // the form for a launch of `blocks` CTAs on `sms` SMs: dense beyond one wave
  const ColFns& form(long long blocks, int sms) const { return blocks > (long long)sms * (512 / threads) ? dense : roomy; }
};
// false: no kernels for this length
bool row_kernels_f32(int n, RowKernels* k);
bool row_kernels_f64(int n, RowKernels* k);
bool col_kernels_f32(int n, ColKernels* k);
bool col_kernels_f64(int n, ColKernels* k);
bool col_kernels_f32_long(int n, ColKernels* k);  // the longer half of the lengths
bool col_kernels_f64_long(int n, ColKernels* k);

template <typename S, int N>
RowKernels row_kernels_of() {
  RowKernels k{};
  k.forward = (const void*)&row_forward<S, N, false, 1>;
  k.inverse = (const void*)&row_inverse<S, N, false, 1>;
  if constexpr (Sc<S>::NV == 2) {
    k.forward_rq4 = (const void*)&row_forward<S, N, false, 4>;
    k.inverse_rq4 = (const void*)&row_inverse<S, N, false, 4>;
    k.rag_forward = (const void*)&row_forward<S, N, true, 1>;
    k.rag_inverse = (const void*)&row_inverse<S, N, true, 1>;
  }
  k.threads = RowCfg<N>::threads;
  k.q = RowCfg<N>::Q;
  k.nv = Sc<S>::NV;
  k.smem = RowCfg<N>::smem;
  return k;
}
template <typename S, int N, bool DENSE>
ColFns col_fns_of() {
  ColFns k{};
  k.forward = (const void*)&col_forward<S, N, DENSE>;
  k.pairs = (const void*)&col_pairs<S, N, false, false, false, DENSE>;
  k.pairs_lpre = (const void*)&col_pairs<S, N, true, false, false, DENSE>;
  k.pairs_pre = (const void*)&col_pairs<S, N, true, true, false, DENSE>;
  if constexpr (Sc<S>::NV == 2) k.rag_pairs = (const void*)&col_pairs<S, N, false, false, true, DENSE>;
  return k;
}
template <typename S, int N>
ColKernels col_kernels_of() {
  using K = ColCfg<S, N>;
  ColKernels k{};
  k.roomy = col_fns_of<S, N, false>();
  k.dense = col_fns_of<S, N, K::has_dense>();
  k.threads = K::threads;
  k.pu = K::PU;
  k.lgcb = K::lgcb;
  k.rq = K::RQ;
  k.unit_smem = K::PU * K::unit * 16;
  return k;
}
#define XC_ROW_CASE(N_, ...)              \
  case N_:                                \
    *k = row_kernels_of<XC_FFT_S, N_>();  \
    return true;
#define XC_COL_CASE(N_, ...)              \
  case N_:                                \
    *k = col_kernels_of<XC_FFT_S, N_>();  \
    return true;

}  // namespace fe
}  // namespace xc
