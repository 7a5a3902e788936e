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
// Transforms are decimation-in-frequency over two or three radix passes
// N = R1 [R2] R3.  A pass reads and writes the same places, so a pass costs
// one shared-memory round trip and one barrier.  The column kernel never
// leaves digit-reversed order: left and right spectra are in the same order,
// and the inverse (decimation in time) starts from it, so its innermost
// forward pass, the product and the first inverse pass happen in registers.
// The row kernels transform two real rows as one complex row.
#pragma once

#include <cstdint>

#include "xc_common.cuh"

namespace xc {
namespace fe {

template <typename T>
struct CxOf;
template <>
struct CxOf<float> {
  using type = float2;
};
template <>
struct CxOf<double> {
  using type = double2;
};
template <typename T>
using Cx = typename CxOf<T>::type;

template <typename T>
__device__ __forceinline__ Cx<T> mk(T x, T y) {
  Cx<T> r;
  r.x = x;
  r.y = y;
  return r;
}
template <typename C>
__device__ __forceinline__ C cadd(C a, C b) {
  a.x += b.x;
  a.y += b.y;
  return a;
}
template <typename C>
__device__ __forceinline__ C csub(C a, C b) {
  a.x -= b.x;
  a.y -= b.y;
  return a;
}
// a * b, or a * conj(b)
template <bool CONJ, typename C>
__device__ __forceinline__ C cmul(C a, C b) {
  C r;
  if (CONJ) {
    r.x = a.x * b.x + a.y * b.y;
    r.y = a.y * b.x - a.x * b.y;
  } else {
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.y * b.x + a.x * b.y;
  }
  return r;
}
// a * (S i): S = -1 for forward transforms, +1 for inverse ones
template <int S, typename C>
__device__ __forceinline__ C mul_i(C a) {
  C r;
  r.x = S > 0 ? -a.y : a.y;
  r.y = S > 0 ? a.x : -a.x;
  return r;
}

// ---------------------------------------------------------------------------
// In-register transforms of R values, natural order in and out,
// X[k] = sum_n x[n] exp(S 2 pi i n k / R).
// ---------------------------------------------------------------------------
template <typename T, int S, int R>
struct Dft;

template <typename T, int S>
struct Dft<T, S, 2> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    const C a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
  }
};

template <typename T, int S>
struct Dft<T, S, 4> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    const C a = cadd(x[0], x[2]), b = csub(x[0], x[2]);
    const C c = cadd(x[1], x[3]), d = mul_i<S>(csub(x[1], x[3]));
    x[0] = cadd(a, c);
    x[1] = cadd(b, d);
    x[2] = csub(a, c);
    x[3] = csub(b, d);
  }
};

template <typename T, int S>
struct Dft<T, S, 3> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    constexpr T h = T(0.8660254037844386467637231707529362);  // sin(2 pi / 3)
    const C s = cadd(x[1], x[2]), d = csub(x[1], x[2]);
    const C m = mk<T>(x[0].x - T(0.5) * s.x, x[0].y - T(0.5) * s.y);
    const C r = mul_i<S>(mk<T>(h * d.x, h * d.y));
    x[0] = cadd(x[0], s);
    x[1] = cadd(m, r);
    x[2] = csub(m, r);
  }
};

// Odd prime R by symmetry: sums and differences of x[n], x[R-n].
template <typename T, int S>
struct Dft<T, S, 5> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    constexpr T c1 = T(0.3090169943749474241022934171828191), c2 = T(-0.8090169943749474241022934171828191);
    constexpr T s1 = T(0.9510565162951535721164393333793821), s2 = T(0.5877852522924731291687059546390728);
    const C a1 = cadd(x[1], x[4]), b1 = csub(x[1], x[4]);
    const C a2 = cadd(x[2], x[3]), b2 = csub(x[2], x[3]);
    const C m1 = mk<T>(x[0].x + c1 * a1.x + c2 * a2.x, x[0].y + c1 * a1.y + c2 * a2.y);
    const C m2 = mk<T>(x[0].x + c2 * a1.x + c1 * a2.x, x[0].y + c2 * a1.y + c1 * a2.y);
    const C r1 = mul_i<S>(mk<T>(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y));
    const C r2 = mul_i<S>(mk<T>(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y));
    x[0] = cadd(x[0], cadd(a1, a2));
    x[1] = cadd(m1, r1);
    x[4] = csub(m1, r1);
    x[2] = cadd(m2, r2);
    x[3] = csub(m2, r2);
  }
};

template <typename T, int S>
struct Dft<T, S, 7> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    constexpr T c1 = T(0.6234898018587335305250048840042398), c2 = T(-0.2225209339563144042889025644967948),
                c3 = T(-0.9009688679024191262361023195074451);
    constexpr T s1 = T(0.7818314824680298087084445266740578), s2 = T(0.9749279121818236070181316829939312),
                s3 = T(0.4338837391175581204757683328483587);
    const C a1 = cadd(x[1], x[6]), b1 = csub(x[1], x[6]);
    const C a2 = cadd(x[2], x[5]), b2 = csub(x[2], x[5]);
    const C a3 = cadd(x[3], x[4]), b3 = csub(x[3], x[4]);
    const C m1 = mk<T>(x[0].x + c1 * a1.x + c2 * a2.x + c3 * a3.x, x[0].y + c1 * a1.y + c2 * a2.y + c3 * a3.y);
    const C m2 = mk<T>(x[0].x + c2 * a1.x + c3 * a2.x + c1 * a3.x, x[0].y + c2 * a1.y + c3 * a2.y + c1 * a3.y);
    const C m3 = mk<T>(x[0].x + c3 * a1.x + c1 * a2.x + c2 * a3.x, x[0].y + c3 * a1.y + c1 * a2.y + c2 * a3.y);
    const C r1 = mul_i<S>(mk<T>(s1 * b1.x + s2 * b2.x + s3 * b3.x, s1 * b1.y + s2 * b2.y + s3 * b3.y));
    const C r2 = mul_i<S>(mk<T>(s2 * b1.x - s3 * b2.x - s1 * b3.x, s2 * b1.y - s3 * b2.y - s1 * b3.y));
    const C r3 = mul_i<S>(mk<T>(s3 * b1.x - s1 * b2.x + s2 * b3.x, s3 * b1.y - s1 * b2.y + s2 * b3.y));
    x[0] = cadd(x[0], cadd(a1, cadd(a2, a3)));
    x[1] = cadd(m1, r1);
    x[6] = csub(m1, r1);
    x[2] = cadd(m2, r2);
    x[5] = csub(m2, r2);
    x[3] = cadd(m3, r3);
    x[4] = csub(m3, r3);
  }
};

template <typename T, int S>
struct Dft<T, S, 8> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    constexpr T h = T(0.7071067811865475244008443621048490);
    C e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    Dft<T, S, 4>::run(e);
    Dft<T, S, 4>::run(o);
    // o[k] *= exp(S 2 pi i k / 8)
    const C i1 = mul_i<S>(o[1]), i3 = mul_i<S>(o[3]);
    o[1] = mk<T>(h * (o[1].x + i1.x), h * (o[1].y + i1.y));
    o[2] = mul_i<S>(o[2]);
    o[3] = mk<T>(h * (i3.x - o[3].x), h * (i3.y - o[3].y));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = cadd(e[k], o[k]);
      x[k + 4] = csub(e[k], o[k]);
    }
  }
};

template <typename T, int S>
struct Dft<T, S, 16> {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    constexpr T h = T(0.7071067811865475244008443621048490);
    constexpr T c = T(0.9238795325112867561281831893967882), s = T(0.3826834323650897717284599840303988);
    const T sg = S > 0 ? T(1) : T(-1);
    C y[4][4];  // [n2][k1]
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) y[n2][n1] = x[4 * n1 + n2];
      Dft<T, S, 4>::run(y[n2]);
    }
    // y[n2][k1] *= exp(S 2 pi i n2 k1 / 16)
    const C w1 = mk<T>(c, sg * s), w3 = mk<T>(s, sg * c), w9 = mk<T>(-c, -sg * s);
    auto eighth = [](C v) {  // exp(S pi i / 4)
      const C i = mul_i<S>(v);
      return mk<T>(h * (v.x + i.x), h * (v.y + i.y));
    };
    y[1][1] = cmul<false>(y[1][1], w1);
    y[1][2] = eighth(y[1][2]);
    y[1][3] = cmul<false>(y[1][3], w3);
    y[2][1] = eighth(y[2][1]);
    y[2][2] = mul_i<S>(y[2][2]);
    y[2][3] = eighth(mul_i<S>(y[2][3]));
    y[3][1] = cmul<false>(y[3][1], w3);
    y[3][2] = eighth(mul_i<S>(y[3][2]));
    y[3][3] = cmul<false>(y[3][3], w9);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      C z[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
      Dft<T, S, 4>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) x[k1 + 4 * k2] = z[k2];
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
template <typename T, int S, int A, int B>
struct DftPfa {
  using C = Cx<T>;
  static __device__ __forceinline__ void run(C* x) {
    constexpr int R = A * B;
    C y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = x[(B * n1 + A * n2) % R];
      // n k / R = n1 k1 / A + n2 k2 / B (mod 1): B n1 k / R = n1 k / A
      Dft<T, S, A>::run(y[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      C z[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
      Dft<T, S, B>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) x[crt(A, B, k1, k2)] = z[k2];
    }
  }
};
template <typename T, int S>
struct Dft<T, S, 6> : DftPfa<T, S, 2, 3> {};
template <typename T, int S>
struct Dft<T, S, 10> : DftPfa<T, S, 2, 5> {};
template <typename T, int S>
struct Dft<T, S, 12> : DftPfa<T, S, 4, 3> {};
template <typename T, int S>
struct Dft<T, S, 14> : DftPfa<T, S, 2, 7> {};

// ---------------------------------------------------------------------------
// Lengths and their passes.  R1 >= R2 >= R3 where possible; R2 = 1: two
// passes.  All lengths are multiples of 16, at most 25% apart (33% below 64).
// ---------------------------------------------------------------------------
#define XC_FFT_LENGTHS(X)                                                                                   \
  X(16, 4, 1, 4) X(32, 8, 1, 4) X(48, 8, 1, 6) X(64, 8, 1, 8) X(80, 10, 1, 8) X(96, 12, 1, 8)              \
  X(112, 14, 1, 8) X(128, 16, 1, 8) X(160, 16, 1, 10) X(192, 16, 1, 12) X(224, 16, 1, 14) X(256, 16, 1, 16) \
  X(320, 8, 8, 5) X(384, 8, 8, 6) X(448, 8, 8, 7) X(512, 8, 8, 8) X(640, 10, 8, 8) X(768, 12, 8, 8)         \
  X(896, 14, 8, 8) X(1024, 16, 8, 8) X(1280, 16, 10, 8) X(1536, 16, 12, 8) X(1792, 16, 14, 8)              \
  X(2048, 16, 16, 8) X(2560, 16, 16, 10) X(3072, 16, 16, 12) X(3584, 16, 16, 14) X(4096, 16, 16, 16)

template <int N>
struct Fac;
#define XC_FAC(N_, A_, B_, C_)                             \
  template <>                                              \
  struct Fac<N_> {                                         \
    static constexpr int R1 = A_, R2 = B_, R3 = C_;        \
    static_assert(A_ * B_ * C_ == N_, "factors of length"); \
  };
XC_FFT_LENGTHS(XC_FAC)
#undef XC_FAC

// Derived geometry of a length.  Element (q1, q2, m) of the pass structure --
// index q1 S1 + q2 R3 + m -- lies at q1 P1 + q2 PR + m in shared memory: odd
// strides, so that the passes that walk q1 or q2 across lanes hit different
// banks.
template <int N>
struct Len {
  static constexpr int R1 = Fac<N>::R1, R2 = Fac<N>::R2, R3 = Fac<N>::R3;
  static constexpr bool three = R2 > 1;
  static constexpr int S1 = N / R1;         // stride of the first pass
  static constexpr int PR = R3 | 1;
  static constexpr int P1 = (R2 * PR) | 1;
  static constexpr int rows = R1 * P1;      // padded length
  static constexpr int rmax = R1 > R3 ? R1 : R3;
  static constexpr int tw1 = 0;             // twiddles of pass 1: (R1 - 1) x S1, [q - 1][o]
  static constexpr int tw2 = (R1 - 1) * S1;  // of pass 2: (R2 - 1) x R3, [q - 1][o]
  static constexpr int ntw = tw2 + (three ? (R2 - 1) * R3 : 0);
  static __device__ __forceinline__ int pos(int i) {  // padded place of index i
    const int q1 = i / S1, o = i - q1 * S1;
    if (!three) return q1 * P1 + o;
    const int q2 = o / R3;
    return q1 * P1 + q2 * PR + (o - q2 * R3);
  }
};

// ---------------------------------------------------------------------------
// Layout of the half spectra between the kernels: matrix by matrix, blocks of
// CB = 2^lgcb columns, [block][row][column in block], columns 0..N/2 rounded
// up to whole blocks.  A row pair's share of a block is contiguous (row
// kernels), and so is a whole block (column kernels).
// ---------------------------------------------------------------------------
template <typename T>
struct RowSide {
  const T* src;  // matrices, H x W each
  Cx<T>* dst;    // half spectra of their rows
  int H, W;
  int groups;    // CTAs per matrix
};
template <typename T>
struct RowFwdArgs {
  RowSide<T> a, b;    // blocks [0, a_blocks) on side a, the rest on side b
  unsigned a_blocks;
  int nblk, lgcb;
  const Cx<T>* tw;
};

template <typename T>
struct ColArgs {
  const Cx<T>* left;   // row spectra of the lefts, or (LPRE) their full spectra
  const Cx<T>* right;  // the same of the rights (RPRE)
  Cx<T>* out;          // column-inverted products, Sy rows in output order
  int Hl, Hr, Sy;
  int nblk;
  int n_left;          // lefts l0 .. l0 + n_left - 1 of this launch
  int l0, k0, k1;      // partners k0 .. k1 - 1 of each
  int n_kg, kc;        // partner groups of kc partners
  long long r_l, r_k, r_off;  // right(l, k) = l r_l + k r_k - r_off within `right`
  const Cx<T>* tw;
};
template <typename T>
struct ColFwdArgs {
  const Cx<T>* src;    // row spectra, H rows
  Cx<T>* dst;          // full spectra, N rows in pass order
  int H, nblk;
  long long units;     // matrices x nblk
  const Cx<T>* tw;
};
template <typename T>
struct RowInvArgs {
  const Cx<T>* src;    // [output of this launch][block][Sy][CB]
  T* out;
  int Sy, Sx, Wr;
  int groups;          // CTAs per output
  int nblk, lgcb;
  int l0, k0, nk;      // output index t of the launch: l = l0 + t / nk, k = k0 + t % nk
  long long o_l, o_k;
  T scale_hi, scale_lo;
  const Cx<T>* tw;
};

// Row kernels: one transform (a row pair) on N / R3 threads, Q of them per CTA.
template <int N>
struct RowCfg {
  static constexpr int TF = N / Len<N>::R3;
  static constexpr int fit(int q) { return 2 * q * TF <= 320 ? fit(2 * q) : q; }
  static constexpr int Q = fit(1);
  static constexpr int threads = Q * TF;
  static constexpr int FS = Len<N>::rows + (21 - Len<N>::rows % 16) % 16;  // = 5 mod 16: transforms on different banks
  template <typename T>
  static constexpr int smem() {
    return Q * FS * (int)sizeof(Cx<T>);
  }
};

template <typename C>
struct alignas(16) Vec16 {  // 16 bytes of complex values
  static constexpr int V = 16 / (int)sizeof(C);
  C v[V];
};

// The middle pass of a three-pass transform, in place.
template <typename T, int S, int N, int STEP>
__device__ __forceinline__ void mid_pass(Cx<T>* z, int it0, int step, const Cx<T>* __restrict__ tw) {
  using L = Len<N>;
  using C = Cx<T>;
  for (int it = it0; it < N / L::R2; it += step) {
    const int b = it / L::R3, o = it - b * L::R3;
    C* base = z + (b * L::P1 + o) * STEP;
    C x[L::R2];
    if (S < 0) {
#pragma unroll
      for (int m = 0; m < L::R2; ++m) x[m] = base[m * L::PR * STEP];
      Dft<T, S, L::R2>::run(x);
      base[0] = x[0];
#pragma unroll
      for (int q = 1; q < L::R2; ++q)
        base[q * L::PR * STEP] = cmul<false>(x[q], __ldg(tw + L::tw2 + (q - 1) * L::R3 + o));
    } else {
      x[0] = base[0];
#pragma unroll
      for (int q = 1; q < L::R2; ++q)
        x[q] = cmul<true>(base[q * L::PR * STEP], __ldg(tw + L::tw2 + (q - 1) * L::R3 + o));
      Dft<T, S, L::R2>::run(x);
#pragma unroll
      for (int m = 0; m < L::R2; ++m) base[m * L::PR * STEP] = x[m];
    }
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(RowCfg<N>::threads) row_forward(const RowFwdArgs<T> p) {
  using L = Len<N>;
  using C = Cx<T>;
  using V16 = Vec16<C>;
  constexpr int TF = RowCfg<N>::TF, Q = RowCfg<N>::Q, V = V16::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* s = reinterpret_cast<C*>(smem_raw);
  const bool first = blockIdx.x < p.a_blocks;
  const unsigned b = first ? blockIdx.x : blockIdx.x - p.a_blocks;
  const int H = first ? p.a.H : p.b.H, W = first ? p.a.W : p.b.W;
  const unsigned groups = (unsigned)(first ? p.a.groups : p.b.groups);
  const T* __restrict__ src = first ? p.a.src : p.b.src;
  C* __restrict__ dst = first ? p.a.dst : p.b.dst;
  const long long mat = b / groups;
  const int rp0 = (int)(b - (unsigned)mat * groups) * Q;
  const int f = threadIdx.x / TF, i = threadIdx.x - f * TF;
  C* z = s + f * RowCfg<N>::FS;
  {
    const int row = 2 * (rp0 + f);
    const int w0 = row < H ? W : 0, w1 = row + 1 < H ? W : 0;
    const T* r0 = src + (mat * H + (row < H ? row : 0)) * (long long)W;
    const T* r1 = r0 + (row + 1 < H ? W : 0);
    if (i < L::S1) {
      C x[L::R1];
#pragma unroll
      for (int m = 0; m < L::R1; ++m) {
        const int k = i + m * L::S1;
        x[m] = mk<T>(k < w0 ? __ldg(r0 + k) : T(0), k < w1 ? __ldg(r1 + k) : T(0));
      }
      Dft<T, -1, L::R1>::run(x);
      C* base = z + (L::three ? (i / L::R3) * L::PR + i % L::R3 : i);
      base[0] = x[0];
#pragma unroll
      for (int q = 1; q < L::R1; ++q) base[q * L::P1] = cmul<false>(x[q], __ldg(p.tw + (q - 1) * L::S1 + i));
    }
  }
  __syncthreads();
  if constexpr (L::three) {
    mid_pass<T, -1, N, 1>(z, i, TF, p.tw);
    __syncthreads();
  }
  {
    const int q1 = i % L::R1, q2 = i / L::R1;
    C x[L::R3];
    const C* base = z + q1 * L::P1 + q2 * L::PR;
#pragma unroll
    for (int m = 0; m < L::R3; ++m) x[m] = base[m];
    Dft<T, -1, L::R3>::run(x);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < L::R3; ++q) z[i + q * TF] = x[q];  // natural order
  }
  __syncthreads();
  // The two rows' spectra: A = (Z[c] + conj Z[-c]) / 2, B = (Z[c] - conj Z[-c]) / 2i.
  const int cb = 1 << p.lgcb, lgh = p.lgcb - (V == 2 ? 1 : 0);
  const int total = p.nblk * (Q << lgh);
  dst += mat * p.nblk * (long long)H * cb;
  for (int u = threadIdx.x; u < total; u += Q * TF) {
    const int h = u & ((1 << lgh) - 1), ff = (u >> lgh) % Q, blk = (u >> lgh) / Q;
    const int row = 2 * (rp0 + ff);
    if (row >= H) continue;
    const C* zz = s + ff * RowCfg<N>::FS;
    V16 a, bb;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int c = blk * cb + h * V + v;
      const C zc = zz[c], zn = zz[c == 0 ? 0 : N - c];
      a.v[v] = mk<T>(T(0.5) * (zc.x + zn.x), T(0.5) * (zc.y - zn.y));
      bb.v[v] = mk<T>(T(0.5) * (zc.y + zn.y), T(0.5) * (zn.x - zc.x));
    }
    C* d = dst + ((long long)blk * H + row) * cb + h * V;
    *reinterpret_cast<V16*>(d) = a;
    if (row + 1 < H) *reinterpret_cast<V16*>(d + cb) = bb;
  }
}

template <typename T, int N>
__global__ void __launch_bounds__(RowCfg<N>::threads) row_inverse(const RowInvArgs<T> p) {
  using L = Len<N>;
  using C = Cx<T>;
  using V16 = Vec16<C>;
  constexpr int TF = RowCfg<N>::TF, Q = RowCfg<N>::Q, V = V16::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* s = reinterpret_cast<C*>(smem_raw);
  const int t = (int)(blockIdx.x / (unsigned)p.groups);
  const int rp0 = (int)(blockIdx.x - (unsigned)t * (unsigned)p.groups) * Q;
  // Z = A + i B of every row pair, whose inverse transform is row a + i row b
  const int cb = 1 << p.lgcb, lgh = p.lgcb - (V == 2 ? 1 : 0);
  const int total = p.nblk * (Q << lgh);
  const C* src = p.src + (long long)t * p.nblk * p.Sy * cb;
#pragma unroll 4
  for (int u = threadIdx.x; u < total; u += Q * TF) {
    const int h = u & ((1 << lgh) - 1), ff = (u >> lgh) % Q, blk = (u >> lgh) / Q;
    const int row = 2 * (rp0 + ff);
    V16 a, bb;
#pragma unroll
    for (int v = 0; v < V; ++v) a.v[v] = bb.v[v] = mk<T>(T(0), T(0));
    const C* d = src + ((long long)blk * p.Sy + row) * cb + h * V;
    if (row < p.Sy) a = *reinterpret_cast<const V16*>(d);
    if (row + 1 < p.Sy) bb = *reinterpret_cast<const V16*>(d + cb);
    C* zz = s + ff * RowCfg<N>::FS;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int c = blk * cb + h * V + v;
      if (c > N / 2) continue;
      if (c == 0 || c == N / 2) {
        zz[L::pos(c)] = mk<T>(a.v[v].x, bb.v[v].x);
      } else {
        zz[L::pos(c)] = mk<T>(a.v[v].x - bb.v[v].y, a.v[v].y + bb.v[v].x);
        zz[L::pos(N - c)] = mk<T>(a.v[v].x + bb.v[v].y, bb.v[v].x - a.v[v].y);
      }
    }
  }
  __syncthreads();
  const int f = threadIdx.x / TF, i = threadIdx.x - f * TF;
  C* z = s + f * RowCfg<N>::FS;
  if (i < L::S1) {
    C x[L::R1];
    C* base = z + (L::three ? (i / L::R3) * L::PR + i % L::R3 : i);
#pragma unroll
    for (int m = 0; m < L::R1; ++m) x[m] = base[m * L::P1];
    Dft<T, 1, L::R1>::run(x);
    base[0] = x[0];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) base[q * L::P1] = cmul<true>(x[q], __ldg(p.tw + (q - 1) * L::S1 + i));
  }
  __syncthreads();
  if constexpr (L::three) {
    // decimation in frequency with the conjugate twiddles
    for (int it = i; it < N / L::R2; it += TF) {
      const int b = it / L::R3, o = it - b * L::R3;
      C* base = z + b * L::P1 + o;
      C x[L::R2];
#pragma unroll
      for (int m = 0; m < L::R2; ++m) x[m] = base[m * L::PR];
      Dft<T, 1, L::R2>::run(x);
      base[0] = x[0];
#pragma unroll
      for (int q = 1; q < L::R2; ++q)
        base[q * L::PR] = cmul<true>(x[q], __ldg(p.tw + L::tw2 + (q - 1) * L::R3 + o));
    }
    __syncthreads();
  }
  {
    const int q1 = i % L::R1, q2 = i / L::R1;
    C x[L::R3];
    const C* base = z + q1 * L::P1 + q2 * L::PR;
#pragma unroll
    for (int m = 0; m < L::R3; ++m) x[m] = base[m];
    Dft<T, 1, L::R3>::run(x);
    const int row = 2 * (rp0 + f);
    if (row >= p.Sy) return;
    const int l = p.l0 + t / p.nk, k = p.k0 + t % p.nk;
    T* o0 = p.out + ((l * p.o_l + k * p.o_k) * p.Sy + row) * (long long)p.Sx;
    const bool two = row + 1 < p.Sy;
#pragma unroll
    for (int q = 0; q < L::R3; ++q) {
      int sx = i + q * TF + p.Wr - 1;
      if (sx >= N) sx -= N;
      if (sx >= p.Sx) continue;
      // the scale as a sum of two terms: rounds like a scaling in higher precision
      T va, vb;
      if constexpr (sizeof(T) == 4) {
        va = fmaf(x[q].x, p.scale_hi, x[q].x * p.scale_lo);
        vb = fmaf(x[q].y, p.scale_hi, x[q].y * p.scale_lo);
      } else {
        va = x[q].x * p.scale_hi;
        vb = x[q].y * p.scale_hi;
      }
      o0[sx] = va;
      if (two) o0[p.Sx + sx] = vb;
    }
  }
}

// ---------------------------------------------------------------------------
// Column kernels: a unit is one block of CB columns of one matrix (or pair),
// on TU threads, lanes over the block's columns first; PU units per CTA.
// ---------------------------------------------------------------------------
template <typename T, int N>
struct ColCfg {
  static constexpr int CB = sizeof(T) == 4 ? (N <= 2048 ? 4 : 2) : 2;
  static constexpr int lgcb = CB == 4 ? 2 : 1;
  static constexpr int TU = (N / Len<N>::R3) * CB <= 512 ? (N / Len<N>::R3) * CB : (N / Len<N>::R1) * CB;
  static constexpr int PU = TU >= 128 ? 1 : 128 / TU;
  static constexpr int threads = TU * PU;
  static constexpr int JT = TU / CB;             // items side by side in a pass
  static constexpr int unit = Len<N>::rows * CB;  // shared-memory elements of a unit
  static constexpr int nblk = (N / 2 + 1 + CB - 1) / CB;  // blocks when N is the row length (callers pass theirs)
};

// Forward passes of one column block from global memory (H rows of CB
// columns) up to, not including, the last; ends with a barrier.
template <typename T, int N>
__device__ __forceinline__ void col_load_passes(Cx<T>* z, const Cx<T>* __restrict__ g, int H, int j0, int c,
                                                const Cx<T>* __restrict__ tw) {
  using L = Len<N>;
  using C = Cx<T>;
  using K = ColCfg<T, N>;
  for (int o = j0; o < L::S1; o += K::JT) {
    C x[L::R1];
#pragma unroll
    for (int m = 0; m < L::R1; ++m) {
      const int y = o + m * L::S1;
      x[m] = y < H ? __ldg(g + (long long)y * K::CB + c) : mk<T>(T(0), T(0));
    }
    Dft<T, -1, L::R1>::run(x);
    C* base = z + (L::three ? (o / L::R3) * L::PR + o % L::R3 : o) * K::CB + c;
    base[0] = x[0];
#pragma unroll
    for (int q = 1; q < L::R1; ++q) base[q * L::P1 * K::CB] = cmul<false>(x[q], __ldg(tw + (q - 1) * L::S1 + o));
  }
  __syncthreads();
  if constexpr (L::three) {
    mid_pass<T, -1, N, K::CB>(z + c, j0, K::JT, tw);
    __syncthreads();
  }
}

// Place of the last pass's item j (its R3 values follow each other by CB).
template <typename T, int N>
__device__ __forceinline__ int col_item(int j) {
  using L = Len<N>;
  const int q1 = j / L::R2, q2 = j - q1 * L::R2;
  return (q1 * L::P1 + q2 * L::PR) * ColCfg<T, N>::CB;
}

// Full spectra of the columns, in pass order: row q N/R3 + j holds output q
// of the last pass's item j.
template <typename T, int N>
__global__ void __launch_bounds__(ColCfg<T, N>::threads) col_forward(const ColFwdArgs<T> p) {
  using L = Len<N>;
  using C = Cx<T>;
  using K = ColCfg<T, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pu = threadIdx.x / K::TU, t = threadIdx.x - pu * K::TU;
  const int c = t % K::CB, j0 = t / K::CB;
  C* z = reinterpret_cast<C*>(smem_raw) + pu * K::unit;
  const long long u = (long long)blockIdx.x * K::PU + pu;
  const bool live = u < p.units;
  col_load_passes<T, N>(z, p.src + (live ? u : 0) * p.H * K::CB, live ? p.H : 0, j0, c, p.tw);
  if (!live) return;
  C* dst = p.dst + u * N * K::CB + c;
  for (int j = j0; j < N / L::R3; j += K::JT) {
    C x[L::R3];
    const C* base = z + col_item<T, N>(j) + c;
#pragma unroll
    for (int m = 0; m < L::R3; ++m) x[m] = base[m * K::CB];
    Dft<T, -1, L::R3>::run(x);
#pragma unroll
    for (int q = 0; q < L::R3; ++q) dst[(q * (N / L::R3) + j) * K::CB] = x[q];
  }
}

// Products of column blocks: for a left matrix and each of a group of its
// partners, the right columns' transform (unless RPRE: already transformed),
// the product with the left spectrum (LPRE: read from global memory;
// otherwise transformed once per group and kept in shared memory), and the
// inverse transform, whose rows go out in the output's row order.
template <typename T, int N, bool LPRE, bool RPRE>
__global__ void __launch_bounds__(ColCfg<T, N>::threads) col_pairs(const ColArgs<T> p) {
  using L = Len<N>;
  using C = Cx<T>;
  using K = ColCfg<T, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int pu = threadIdx.x / K::TU, t = threadIdx.x - pu * K::TU;
  const int c = t % K::CB, j0 = t / K::CB;
  C* z = reinterpret_cast<C*>(smem_raw) + pu * K::unit;
  C* zl = z + (LPRE ? 0 : K::PU * K::unit);  // left spectrum
  const long long gu = (long long)blockIdx.x * K::PU + pu;
  const int blk = (int)(gu % p.nblk);
  const long long rest = gu / p.nblk;
  const int kg = (int)(rest % p.n_kg);
  const long long ll = rest / p.n_kg;  // left of this launch
  const bool live = ll < p.n_left;
  const long long l = p.l0 + (live ? ll : 0);
  const int ka = p.k0 + kg * p.kc, nk = live ? min(p.kc, p.k1 - ka) : 0;
  constexpr int NJ = N / L::R3;
  const C* lspec = nullptr;
  if constexpr (LPRE) {
    lspec = p.left + (l * p.nblk + blk) * (long long)N * K::CB + c;
  } else {
    col_load_passes<T, N>(zl, p.left + (l * p.nblk + blk) * (long long)p.Hl * K::CB, live ? p.Hl : 0, j0, c, p.tw);
    // each thread reads back the items it writes here: no barrier needed
    for (int j = j0; j < NJ; j += K::JT) {
      C x[L::R3];
      C* base = zl + col_item<T, N>(j) + c;
#pragma unroll
      for (int m = 0; m < L::R3; ++m) x[m] = base[m * K::CB];
      Dft<T, -1, L::R3>::run(x);
#pragma unroll
      for (int m = 0; m < L::R3; ++m) base[m * K::CB] = x[m];
    }
  }
  const long long n_k = p.k1 - p.k0;
  for (int kk = 0; kk < p.kc; ++kk) {
    const int k = ka + kk;
    const bool act = kk < nk;
    const long long r = act ? l * p.r_l + k * p.r_k - p.r_off : 0;
    if constexpr (!RPRE)
      col_load_passes<T, N>(z, p.right + (r * p.nblk + blk) * (long long)p.Hr * K::CB, act ? p.Hr : 0, j0, c, p.tw);
    for (int j = j0; j < NJ; j += K::JT) {
      C x[L::R3];
      C* base = z + col_item<T, N>(j) + c;
      C lv[L::R3];
      if constexpr (LPRE) {
#pragma unroll
        for (int q = 0; q < L::R3; ++q) lv[q] = __ldg(lspec + (q * NJ + j) * K::CB);
      }
      if constexpr (RPRE) {
        const C* rspec = p.right + (r * p.nblk + blk) * (long long)N * K::CB + c;
#pragma unroll
        for (int q = 0; q < L::R3; ++q) x[q] = __ldg(rspec + (q * NJ + j) * K::CB);
      } else {
#pragma unroll
        for (int m = 0; m < L::R3; ++m) x[m] = base[m * K::CB];
        Dft<T, -1, L::R3>::run(x);
      }
      const C* lb = zl + col_item<T, N>(j) + c;
#pragma unroll
      for (int q = 0; q < L::R3; ++q) x[q] = cmul<true>(LPRE ? lv[q] : lb[q * K::CB], x[q]);
      Dft<T, 1, L::R3>::run(x);
#pragma unroll
      for (int m = 0; m < L::R3; ++m) base[m * K::CB] = x[m];
    }
    __syncthreads();
    if constexpr (L::three) {
      mid_pass<T, 1, N, K::CB>(z + c, j0, K::JT, p.tw);
      __syncthreads();
    }
    if (act) {
      C* out = p.out + ((ll * n_k + (k - p.k0)) * p.nblk + blk) * (long long)p.Sy * K::CB + c;
      for (int o = j0; o < L::S1; o += K::JT) {
        C x[L::R1];
        const C* base = z + (L::three ? (o / L::R3) * L::PR + o % L::R3 : o) * K::CB + c;
        x[0] = base[0];
#pragma unroll
        for (int q = 1; q < L::R1; ++q) x[q] = cmul<true>(base[q * L::P1 * K::CB], __ldg(p.tw + (q - 1) * L::S1 + o));
        Dft<T, 1, L::R1>::run(x);
#pragma unroll
        for (int m = 0; m < L::R1; ++m) {
          int sy = o + m * L::S1 + p.Hr - 1;
          if (sy >= N) sy -= N;
          if (sy < p.Sy) out[(long long)sy * K::CB] = x[m];
        }
      }
    }
    if (kk + 1 < p.kc) __syncthreads();  // the next partner's passes overwrite z
  }
}

// What the host needs to launch the kernels of one length.
struct RowKernels {
  const void* forward;
  const void* inverse;
  int threads, q, smem;
};
struct ColKernels {
  const void* forward;
  const void* pairs;       // left transformed in the kernel
  const void* pairs_lpre;  // left spectra from col_forward
  const void* pairs_pre;   // both
  int threads, pu, lgcb, unit_smem;  // shared memory of one unit buffer
};
// false: no kernels for this length
bool row_kernels_f32(int n, RowKernels* k);
bool row_kernels_f64(int n, RowKernels* k);
bool col_kernels_f32(int n, ColKernels* k);
bool col_kernels_f64(int n, ColKernels* k);

#define XC_ROW_CASE(N_, A_, B_, C_)                                                       \
  case N_:                                                                                \
    *k = RowKernels{(const void*)&row_forward<XC_FFT_T, N_>, (const void*)&row_inverse<XC_FFT_T, N_>, \
                    RowCfg<N_>::threads, RowCfg<N_>::Q, RowCfg<N_>::smem<XC_FFT_T>()};    \
    return true;
#define XC_COL_CASE(N_, A_, B_, C_)                                                                             \
  case N_:                                                                                                      \
    *k = ColKernels{(const void*)&col_forward<XC_FFT_T, N_>, (const void*)&col_pairs<XC_FFT_T, N_, false, false>, \
                    (const void*)&col_pairs<XC_FFT_T, N_, true, false>,                                         \
                    (const void*)&col_pairs<XC_FFT_T, N_, true, true>, ColCfg<XC_FFT_T, N_>::threads,           \
                    ColCfg<XC_FFT_T, N_>::PU, ColCfg<XC_FFT_T, N_>::lgcb,                                       \
                    ColCfg<XC_FFT_T, N_>::PU * ColCfg<XC_FFT_T, N_>::unit * (int)sizeof(Cx<XC_FFT_T>)};         \
    return true;

}  // namespace fe
}  // namespace xc
