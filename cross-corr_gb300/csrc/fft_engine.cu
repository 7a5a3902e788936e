// fft_engine.cu -- planning and launches of the fused FFT correlation
// (kernels in fft_engine.cuh).
//
// A problem runs as three kernels per chunk of outputs: row transforms of the
// inputs, column transforms + product + inverse columns, inverse rows.  The
// zero padding, the conjugate product, the quadrant swap, the scale and the
// crop of the separate-kernel path (fft_pipeline.cu's stages) happen inside
// them, rows of zeros are never transformed or stored, and the intermediate
// spectra cross memory twice instead of eight times.
#include "fft_engine.h"

#include <algorithm>
#include <cmath>
#include <vector>

namespace xc {
namespace fe {

namespace {

struct Factors {
  int n, r1, ra, rb, r3;
};
#define XC_FACTORS(N_, A_, B_, C_, D_) {N_, A_, B_, C_, D_},
constexpr Factors kRows[] = {XC_FFT_ROWS(XC_FACTORS)};
#undef XC_FACTORS
#define XC_FACTORS(N_, A_, B_, D_) {N_, A_, B_, 1, D_},
constexpr Factors kCols[] = {XC_FFT_COLS(XC_FACTORS)};
#undef XC_FACTORS
constexpr int kLengths = (int)(sizeof(kRows) / sizeof(kRows[0]));
static_assert(sizeof(kRows) == sizeof(kCols), "the same lengths on both axes");

const Factors* factors(int n, bool rows) {
  for (int i = 0; i < kLengths; ++i)
    if (kRows[i].n == n) return rows ? &kRows[i] : &kCols[i];
  return nullptr;
}

// exp(-2 pi i k / n): the angle is reduced to the first octant, where sine
// and cosine are accurate to the last place.
void root(long long k, long long n, double* re, double* im) {
  k %= n;
  const double pi = 3.14159265358979323846264338327950288;
  const long long e = 8 * k;  // in octants of n
  const int oct = (int)(e / n);
  double c, s;
  const auto angle = [&](long long num) { return 2.0 * pi * ((double)num / (double)n); };  // num / n of a turn
  switch (oct) {
    case 0: c = std::cos(angle(k)); s = std::sin(angle(k)); break;
    case 1: c = std::sin(angle(n - 4 * k) / 4); s = std::cos(angle(n - 4 * k) / 4); break;
    case 2: c = -std::sin(angle(4 * k - n) / 4); s = std::cos(angle(4 * k - n) / 4); break;
    case 3: c = -std::cos(angle(n - 2 * k) / 2); s = std::sin(angle(n - 2 * k) / 2); break;
    case 4: c = -std::cos(angle(2 * k - n) / 2); s = -std::sin(angle(2 * k - n) / 2); break;
    case 5: c = -std::sin(angle(3 * n - 4 * k) / 4); s = -std::cos(angle(3 * n - 4 * k) / 4); break;
    case 6: c = std::sin(angle(4 * k - 3 * n) / 4); s = -std::cos(angle(4 * k - 3 * n) / 4); break;
    default: c = std::cos(angle(n - k)); s = -std::sin(angle(n - k)); break;
  }
  *re = c;
  *im = -s;
}

// The table of a pass structure: [q - 1][o] of every pass but the last.
template <typename Put>
void each_twiddle(const Factors& f, Put put) {
  const int s1 = f.n / f.r1, sa = s1 / f.ra;
  for (int q = 1; q < f.r1; ++q)
    for (int o = 0; o < s1; ++o) put((long long)o * q, f.n);
  for (int q = 1; q < f.ra; ++q)
    for (int o = 0; o < sa; ++o) put((long long)o * q, s1);
  for (int q = 1; q < f.rb; ++q)
    for (int o = 0; o < f.r3; ++o) put((long long)o * q, sa);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

xc_status raise_limit(const void* fn, int bytes) {
  if (bytes > 48 * 1024) XC_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return XC_OK;
}

template <typename Args>
xc_status launch(const void* fn, long long blocks, int threads, int smem, Args& args, cudaStream_t stream) {
  if (blocks > 0x7fffffffLL) return fail(XC_ERR_INVALID_ARGUMENT, "problem too large for one launch");
  void* a[] = {&args};
  // Programmatic dependent launch: the next kernel's CTAs may become resident
  // while this one's last ones run; each waits for the whole previous grid
  // (griddepcontrol.wait) before it touches memory.
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  XC_CUDA_TRY(cudaLaunchKernelExC(&cfg, fn, a));
  return XC_OK;
}

// Transforms (or units) of `threads` threads per CTA for a launch of `count`:
// as few as give every SM one CTA, whole warps, at most `most` (128-thread CTAs
// put a small problem on a few SMs; n_to_mn 4 + 8, 56x56: 18.0 us with those,
// 14.6 with this rule and the one for short launches below).
int per_cta(long long count, int most, int threads, int sms) {
  const long long even = (count + sms - 1) / sms, warp = div_up(32, threads);
  return (int)std::min<long long>(most, std::max(even, warp));
}

template <typename T>
xc_status run(const Engine& e, const void* left, const void* right, void* out, char* ws, cudaStream_t stream) {
  const Geometry& g = e.g;
  const char* tw = static_cast<const char*>(e.tw);
  Cx<T>* al = reinterpret_cast<Cx<T>*>(ws + e.off_al);
  Cx<T>* ar = reinterpret_cast<Cx<T>*>(ws + e.off_ar);
  char* fl = ws + e.off_fl;
  char* fr = ws + e.off_fr;
  Cx<T>* b = reinterpret_cast<Cx<T>*>(ws + e.off_b);
  const int lgcb = e.ck.lgcb, nblk = e.nblk;
  const int row_threads = e.rk.threads / e.rk.q, row_smem = e.rk.smem / e.rk.q;
  const int unit_threads = e.ck.threads / e.ck.pu, unit_smem = e.ck.unit_smem / e.ck.pu;
  const auto transforms = [&](long long mats, int H) { return mats * div_up(H, 2 * e.rk.nv); };
  const Scales sc = spectrum_scales(e.nx, e.ny, sizeof(T) == 8);

  // rows of `nr` rights from the r0-th on, and (first) of all lefts.  FP64
  // applies all of the result's scale here, in a product that is there anyway:
  // its range ends 900 binades further down than FP32's.
  const auto rows = [&](bool lefts, long long r0, long long nr) {
    const int q = per_cta((lefts ? transforms(e.pm.n_left, g.Hl) : 0) + transforms(nr, g.Hr), e.rk.q, row_threads, e.sms);
    const int rows_per_cta = 2 * e.rk.nv * q;
    RowFwdArgs<T> a{};
    a.a = RowSide<T>{static_cast<const T*>(left), al, g.Hl, g.Wl, div_up(g.Hl, rows_per_cta),
                     (T)sc.left};
    a.b = RowSide<T>{static_cast<const T*>(right) + r0 * g.Hr * g.Wr, ar, g.Hr, g.Wr, div_up(g.Hr, rows_per_cta),
                     (T)(sizeof(T) == 8 ? sc.right * sc.rest : sc.right)};
    const long long ab = lefts ? (long long)e.pm.n_left * a.a.groups : 0;
    if (ab + nr * a.b.groups > 0x7fffffffLL) return fail(XC_ERR_INVALID_ARGUMENT, "problem too large for one launch");
    a.a_blocks = (unsigned)ab;
    a.nblk = nblk;
    a.lgcb = lgcb;
    a.tw = tw;
    a.zeros = reinterpret_cast<const T*>(tw + e.zeros);
    return launch(e.rk.forward, ab + nr * a.b.groups, q * row_threads, q * row_smem, a, stream);
  };
  // full spectra of the lefts and of `nr` rights
  const auto columns = [&](long long nr) {
    ColFwdArgs<T> a{{al, fl, g.Hl}, {ar, fr, g.Hr}, (long long)e.pm.n_left * nblk, (e.pm.n_left + nr) * nblk, tw + e.tw_col};
    const int pu = per_cta(a.units, e.ck.pu, unit_threads, e.sms);
    return launch(e.ck.form(div_up(a.units, e.ck.pu), e.sms).forward, div_up(a.units, pu), pu * unit_threads,
                  pu * unit_smem, a, stream);
  };

  if (e.shared) XC_TRY(rows(true, 0, e.n_right));
  if (e.shared) XC_TRY(columns(e.n_right));
  for (int k0 = 0; k0 < e.pm.K; k0 += e.k_chunk) {
    const int k1 = std::min(e.pm.K, k0 + e.k_chunk), nk = k1 - k0;
    if (!e.shared) {
      XC_TRY(rows(k0 == 0, k0 * e.pm.r_k, nk * e.pm.r_k));
      if (e.lpre && k0 == 0) XC_TRY(columns(0));
    }
    for (int l0 = 0; l0 < e.pm.n_left; l0 += e.l_chunk) {
      const int nl = std::min(e.pm.n_left - l0, e.l_chunk);
      {
        ColArgs<T> a{};
        a.left = e.shared || e.lpre ? static_cast<void*>(fl) : al;
        a.right = e.shared ? static_cast<void*>(fr) : ar;
        a.out = b;
        a.Hl = g.Hl;
        a.Hr = g.Hr;
        a.Sy = g.Sy;
        a.nblk = nblk;
        a.n_left = nl;
        a.l0 = l0;
        a.k0 = k0;
        a.k1 = k1;
        a.kc = std::min(e.kc, nk);
        a.n_kg = div_up(nk, a.kc);
        a.r_l = e.pm.r_l;
        a.r_k = e.pm.r_k;
        a.r_off = e.shared ? 0 : k0 * e.pm.r_k;
        a.tw = tw + e.tw_col;
        const long long units = (long long)nl * a.n_kg * nblk;
        const int pu = per_cta(units, e.ck.pu, unit_threads, e.sms);
        const ColFns& fns = e.ck.form((units + e.ck.pu - 1) / e.ck.pu, e.sms);
        const void* fn = e.shared ? fns.pairs_pre : e.lpre ? fns.pairs_lpre : fns.pairs;
        XC_TRY(launch(fn, (units + pu - 1) / pu, pu * unit_threads, pu * unit_smem * (e.shared || e.lpre ? 1 : 2), a,
                      stream));
      }
      {
        const int q = per_cta(transforms((long long)nl * nk, g.Sy), e.rk.q, row_threads, e.sms);
        RowInvArgs<T> a{};
        a.src = b;
        a.out = static_cast<T*>(out);
        a.Sy = g.Sy;
        a.Sx = g.Sx;
        a.Wr = g.Wr;
        a.groups = div_up(g.Sy, 2 * e.rk.nv * q);
        a.nblk = nblk;
        a.lgcb = lgcb;
        a.l0 = l0;
        a.k0 = k0;
        a.nk = nk;
        a.o_l = e.pm.o_l;
        a.o_k = e.pm.o_k;
        a.scale_hi = (T)sc.rest;
        a.scale_lo = (T)(sc.rest - (double)a.scale_hi);
        a.tw = tw;
        XC_TRY(launch(e.rk.inverse, (long long)nl * nk * a.groups, q * row_threads, q * row_smem, a, stream));
      }
    }
  }
  return XC_OK;
}

}  // namespace

Scales spectrum_scales(int nx, int ny, bool early) {
  Scales s;
  int e = 0;
  const double m = std::frexp((double)nx * (double)ny, &e);  // nx ny = m 2^e, 1/2 <= m < 1
  const int end = early ? 0 : e / 2;
  e -= end;
  s.left = std::ldexp(1.0, -(e / 2));
  s.right = std::ldexp(1.0, -(e - e / 2));
  s.rest = std::ldexp(1.0 / m, -end);
  return s;
}

int length_for(int n) {
  for (const Factors& f : kRows)
    if (f.n >= n) return f.n;
  return 0;
}

size_t twiddle_bytes(int n, bool rows, xc_dtype dtype) {
  size_t count = 0;
  each_twiddle(*factors(n, rows), [&](long long, long long) { ++count; });
  return align256((dtype == XC_F32 ? sizeof(float2) : sizeof(double2)) * count);
}

void fill_twiddles(int n, bool rows, xc_dtype dtype, void* out) {
  float* of = static_cast<float*>(out);
  double* od = static_cast<double*>(out);
  each_twiddle(*factors(n, rows), [&](long long k, long long m) {
    double re, im;
    root(k, m, &re, &im);
    if (dtype == XC_F32) {
      of[0] = (float)re;
      of[1] = (float)im;
      of += 2;
    } else {
      od[0] = re;
      od[1] = im;
      od += 2;
    }
  });
}

xc_status engine_plan(Engine* e, xc_dtype dtype, const Geometry& g, const PairMap& pm, long long n_right,
                      size_t ws_bytes) {
  e->ready = false;
  e->dtype = dtype;
  e->g = g;
  e->pm = pm;
  e->n_right = n_right;
  e->nx = length_for(g.Sx);
  e->ny = length_for(g.Sy);
  if (e->nx == 0 || e->ny == 0) return XC_OK;
  const bool f32 = dtype == XC_F32;
  if (!(f32 ? row_kernels_f32(e->nx, &e->rk) : row_kernels_f64(e->nx, &e->rk)) ||
      !(f32 ? col_kernels_f32(e->ny, &e->ck) : col_kernels_f64(e->ny, &e->ck)))
    return XC_OK;
  if (e->ck.rq == 4) {
    e->rk.forward = e->rk.forward_rq4;
    e->rk.inverse = e->rk.inverse_rq4;
  }
  const size_t ce = f32 ? sizeof(float2) : sizeof(double2);
  const int cb = 1 << e->ck.lgcb;
  e->nblk = div_up(e->nx / 2 + 1, cb);
  const size_t row = (size_t)e->nblk * cb * ce;  // bytes of one spectrum row
  const auto rows = [&](int H) { return row * spectrum_rows(H, e->ck.rq); };
  e->sms = sm_count_cached();
  // FP64 keeps the library transforms unless the launches fill the GPU: a
  // transform's chain of FP64 instructions is long, and their shorter ones
  // spread a small problem better.  Over 303 problems of up to 256x256 the
  // kernels take 0.5 to 2.3 times as long below 1.1 million points of output
  // (2 million where spectra are shared), beyond it 0.42 to 0.91 times.
  const bool n_to_m = pm.r_l == 0 && pm.n_left > 1;
  const long long points = (long long)pm.n_left * pm.K * e->nx * e->ny;
  if (!f32 && points < (n_to_m ? 2 << 20 : 1100 << 10)) return XC_OK;
  // Short FP32 launches (one wave of the column kernel) take every pair by
  // itself, both column transforms included: three kernels instead of four or
  // five, the SMs have nothing else to do (n_to_m 2 + 2, 56x56: 14.4 us,
  // 27.3 in five kernels of full CTAs).
  const long long pair_units = (long long)pm.n_left * pm.K * e->nblk;
  const bool brief = f32 && 2 * e->ck.unit_smem <= 227 * 1024 &&
                     pair_units <= (long long)e->sms * (512 / e->ck.threads) * e->ck.pu;
  e->shared = n_to_m && !brief;
  e->lpre = false;
  // The left spectra are made first (col_forward) when several partners use
  // them: transforming the left's columns in the column kernel doubles the
  // serial work before its first product (one_to_many 256x256 x 64: column
  // kernel 47 us against 32).  Short launches with few partners save that
  // kernel instead.  The whole chain, us, left in the column kernel / first:
  // 640 points 1 partner 17.7 / 25.5, 2: 24.2 / 26.7, 3: 32.0 / 27.4; 1024: 1:
  // 23.2 / 29.8, 2: 33.2 / 29.3; 2048: 1: 37.8 / 36.9; 4096: 1: 155 / 148.
  // The other way runs where the workspace has no room for the full spectra
  // (one pair whose length is rounded up by much, 700x700: 32 us; it fell back
  // to the library transforms and took 119).
  const bool lpre = !brief && (pm.K >= 4 || (pm.K > 1 && (!f32 || pm.K * e->ny >= 1920)) || e->ny > 2048);

  // Workspace: row spectra of the lefts and of a chunk of rights, full
  // spectra of shared matrices, column-inverted products of a chunk: all
  // partners in one chunk unless the workspace is smaller (shorter chunks,
  // whose spectra stay in the L2 cache, measured slower: the launches' ramps
  // cost more than the traffic; 2048x2048 x 16: 1.78 ms in one chunk, 2.06 in
  // sixteen; 256x256 x 64: 86 us in one, 112 in two).
  const size_t ar1 = rows(g.Hr), b1 = rows(g.Sy);
  size_t off = 0;
  const auto take = [&](size_t bytes) {
    const size_t at = off;
    off += align256(bytes);
    return at;
  };
  if (e->shared) {
    e->off_fl = take(row * e->ny * pm.n_left);
    e->off_fr = take(row * e->ny * n_right);
    const size_t at = off;
    e->off_al = take(rows(g.Hl) * pm.n_left);
    e->off_ar = take(ar1 * n_right);
    const size_t a_end = off;
    e->off_b = at;  // products replace the row spectra, which are done with by then
    off = at;
    if (at + b1 > ws_bytes) return XC_OK;
    const long long fit = std::max<long long>(1, (long long)((ws_bytes - at) / b1));
    // whole lefts while one's products fit, else partners of one left; even chunks
    const int lfit = (int)std::min<long long>(pm.n_left, std::max<long long>(1, fit / pm.K));
    e->l_chunk = div_up(pm.n_left, div_up(pm.n_left, lfit));
    const int kfit = (int)std::min<long long>(pm.K, fit);
    e->k_chunk = e->l_chunk > 1 ? pm.K : div_up(pm.K, div_up(pm.K, kfit));
    off = std::max(a_end, at + align256(b1 * e->l_chunk * e->k_chunk));
    e->kc = 1;
  } else {
    e->l_chunk = pm.n_left;
    const size_t al1 = rows(g.Hl) * pm.n_left, fl1 = row * e->ny * pm.n_left;
    const auto place = [&](bool first, int most) {
      for (int c = 1; c <= most; ++c) {  // as few chunks of partners as fit, even ones
        const int k = div_up(pm.K, c);
        off = 0;
        if (first) e->off_fl = take(fl1);
        else e->off_al = take(al1);
        e->off_ar = take(ar1 * pm.r_k * k);
        // the first products replace the lefts' row spectra once those are transformed
        e->off_b = take(std::max(b1 * pm.n_left * k, first ? al1 : 0));
        if (first) e->off_al = e->off_b;
        if (off > ws_bytes) continue;
        e->lpre = first;
        e->k_chunk = k;
        // Without left spectra made first a unit transforms its left block once
        // for a group of partners: all of them where the units nearly fill a
        // wave of CTAs (0.8 of it), else as many as leave two waves.  One group
        // of all partners left the SMs idle: one_to_many 232x26 x 98, 9 units,
        // 509 us, 25 one by one (library transforms 71); FP64 75x319 by 263x9 x
        // 68, 97 units, 5978 us, 1123 in groups of five (2182).
        const long long units = (long long)pm.n_left * e->nblk, wave = (long long)e->sms * (512 / e->ck.threads) * e->ck.pu;
        const bool filled = 10 * units >= 8 * wave;
        e->kc = first || brief ? 1 : filled ? k : (int)std::max<long long>(1, std::min<long long>(k, k * units / (2 * wave)));
        return true;
      }
      return false;
    };
    // The preferred way in one chunk, the other in one, either in several.
    // Short launches that need several chunks (lengths rounded up by much)
    // stay with the library transforms while they are small: n_to_m 4 + 16,
    // 72x72 (1.6 million points) 23.9 us there, 32 in two chunks; 1 + 24, 16x16
    // by 128x128 21.7 and 29.4; but 4 + 16, 100x100 (3.2 million) 42.8 and 34.8.
    const bool room = 2 * e->ck.unit_smem <= 227 * 1024;  // both blocks' in the column kernel
    bool placed = false;
    for (int most : {1, brief && points < (2 << 20) ? 1 : pm.K})
      for (bool first : {lpre, !lpre}) placed = placed || ((first || room) && place(first, most));
    if (!placed) return XC_OK;
  }
  e->bytes = off;
  if (e->bytes > ws_bytes) return XC_OK;

  XC_TRY(raise_limit(e->rk.forward, e->rk.smem));
  XC_TRY(raise_limit(e->rk.inverse, e->rk.smem));
  for (const ColFns& f : {e->ck.roomy, e->ck.dense}) {
    XC_TRY(raise_limit(f.forward, e->ck.unit_smem));
    XC_TRY(raise_limit(f.pairs_lpre, e->ck.unit_smem));
    XC_TRY(raise_limit(f.pairs_pre, e->ck.unit_smem));
    if (2 * e->ck.unit_smem <= 227 * 1024) XC_TRY(raise_limit(f.pairs, 2 * e->ck.unit_smem));
  }
  e->tw_col = twiddle_bytes(e->nx, true, dtype);
  e->zeros = e->tw_col + twiddle_bytes(e->ny, false, dtype);
  std::vector<char> host(e->zeros + (size_t)e->nx * (f32 ? 4 : 8), 0);
  fill_twiddles(e->nx, true, dtype, host.data());
  fill_twiddles(e->ny, false, dtype, host.data() + e->tw_col);
  XC_CUDA_TRY(cudaMalloc(&e->tw, host.size()));
  const xc_status st = upload(e->tw, host.data(), host.size());
  if (st != XC_OK) {
    engine_release(e);
    return st;
  }
  e->ready = true;
  return XC_OK;
}

xc_status engine_run(const Engine& e, const void* left, const void* right, void* out, char* ws, cudaStream_t stream) {
  return e.dtype == XC_F32 ? run<float>(e, left, right, out, ws, stream)
                           : run<double>(e, left, right, out, ws, stream);
}

void engine_release(Engine* e) {
  cudaFree(e->tw);
  e->tw = nullptr;
  e->ready = false;
}

}  // namespace fe
}  // namespace xc
