// direct_cyclic.cu -- definition-based correlation of uniform batches by
// cyclic column classes (FP32 in packed pairs, FP64), sm_103a.
//
// For a left row r and a right row y the shifts dx take part with
// L[r][x + dx] R[y][x].  Lanes that own neighbouring shifts have overlaps of
// different lengths, and a warp runs as long as its longest lane: over a warp
// of 64 neighbouring shifts the plain tiled kernel multiplies 1.28 times the
// algorithmic count at 256 columns and 2.2 times at 64.  Here a lane owns a
// class of shifts instead, v, v - P, v - 2P, ... for the left width P (rounded
// up to TSX): it walks the right row once, x = 0 .. Wr - 1, reading the left
// row cyclically from v, and changes to the next shift of the class whenever
// it passes the left row's end.  Every lane has the same number of products,
// whatever its class: the only surplus is one block of TSX columns per wrap
// (the block that holds the end is multiplied for both shifts, the left row
// zero-padded by a block on both sides) and the rounding to blocks.
//
//  * A lane owns TSX = 32 bytes of neighbouring classes x TSY row shifts.
//    Lanes run over (row-shift tile, class): a warp takes 32 consecutive ones,
//    so narrow matrices fill it with several row-shift tiles.
//  * Two forms of the lane order.  Flat: lanes run on over (tile, class), and a
//    CTA holds whole left rows.  Windowed, for left rows much wider than the
//    right ones: a warp takes 32 classes of one tile, the CTA's warps the same
//    classes of neighbouring tiles, and shared memory holds the columns those
//    classes walk over, unrolled: the row's chunks with one chunk of zeros
//    after the last, repeated, so that a lane moves one chunk per step, wrap
//    or not.
//  * Loops: blocks of TSX right columns outermost, then left rows; each left
//    row's window (2 TSX values per lane) serves TSY right rows, which the
//    whole warp reads at one or two addresses.  The column blocks are the
//    outer loop because a lane wraps between blocks: it hands over its sums
//    once per wrap, not once per row.
//  * TSY right rows stay in registers while the 2 TSY - 1 left rows they meet
//    pass: every product of the body is wanted, 16 of 17 instructions are FMAs.
//    Scalar FP32 FMAs: packed ones (fma.rn.f32x2) over neighbouring shifts need
//    the odd pairs built by moves, 1.75 per odd FMA, and took 17.3 ms where
//    this takes 9.8 (one_to_many 256x256 x 64; the tiled kernel 14.0).
//  * A CTA holds a block of `hb` right rows of one pair and the left rows that
//    its row-shift tiles meet, loaded whole before the products (a CTA's loads
//    overlap another's products).  Results go through a small transpose
//    buffer, so that each instruction covers 32 consecutive outputs.
//  * The wider matrix of a pair takes the left's part: correlating the right
//    with the left gives the same outputs, mirrored.  (But for rights of a few
//    rows, see cyc_launch; a lane then wraps more than once.)
//  * With one block of right rows the output is written; with several, it
//    starts zeroed and each block adds (red.global.add).  The zeros are a
//    kernel whose dependent launch this one is, so that its CTAs load their
//    rows meanwhile (one pair of 128x128: 24.6 us, 28.5 after a memset).  hb
//    bounds an FP32 chain to 4096 products, as the tiled kernel's flushes do.
//    The order in which blocks add is not fixed, so results of more than two
//    blocks differ between runs in their last places.  CTAs that walk over all
//    blocks of their tiles instead, in order, repeat bit for bit, but their
//    loads differ by what their tiles meet: one_to_many 256x256 x 64 10.3 ms
//    against 9.9, x 16 3.0 against 2.6, 300x300 by 40x40 x 64 588 us against 499.
//
// What bounds it: instruction issue (83% of the slots, FMA pipe 76%; a bare
// loop of such bodies reaches 62 of the 75 TFLOP/s of independent FMAs) in
// FP32, the FP64 pipe in FP64.
#include <algorithm>
#include <type_traits>

#include "xc_common.cuh"
#include "xc_internal.h"

namespace xc {

namespace {


template <typename T>
struct CycArgs {
  const T* left;
  const T* right;
  T* out;
  int Hl, Wl, Hr, Wr, Sy, Sx;
  PairMap pm;
  int C;        // classes of TSX columns: ceil(Wl / TSX)
  int NB;       // blocks of TSX right columns
  int hb, n_rb;  // right rows per block, blocks
  int ST;       // row-shift tiles of a block: ceil((Hl + hb - 1) / TSY)
  int groups;   // CTAs per (pair, block)
  int win;      // class groups of 32 per row-shift tile (windowed form), 0: flat
  int chunks;   // windowed: chunks per left row in shared memory
  int l_rows, l_pitch, r_pitch;  // shared memory: left rows, bytes per row
  int accumulate;
};

// The sums of a lane (TSY x TSX) and a left row's window.
template <typename T, int TSY>
struct Tile {
  static constexpr int TSX = 32 / (int)sizeof(T);
  static constexpr int V = 16 / (int)sizeof(T);  // values per 16-byte load
  T acc[TSY][TSX];
  T w[2 * TSX];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int t = 0; t < TSY; ++t)
#pragma unroll
      for (int q = 0; q < TSX; ++q) acc[t][q] = T(0);
  }
  static __device__ __forceinline__ void load(T* d, const char* s) {
    if constexpr (sizeof(T) == 4) {
      const float4 v = *reinterpret_cast<const float4*>(s);
      d[0] = v.x;
      d[1] = v.y;
      d[2] = v.z;
      d[3] = v.w;
    } else {
      const double2 v = *reinterpret_cast<const double2*>(s);
      d[0] = v.x;
      d[1] = v.y;
    }
  }
  __device__ __forceinline__ void window(const char* w0, const char* w1) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      load(w + h * V, w0 + 16 * h);
      load(w + TSX + h * V, w1 + 16 * h);
    }
  }
  static __device__ __forceinline__ void right(T* v, const char* r) {
#pragma unroll
    for (int h = 0; h < 2; ++h) load(v + h * V, r + 16 * h);
  }
  __device__ __forceinline__ void row(const T* v, int t) {
#pragma unroll
    for (int x = 0; x < TSX; ++x)
#pragma unroll
      for (int q = 0; q < TSX; ++q) acc[t][q] = fma(w[x + q], v[x], acc[t][q]);
  }
  // TSY right rows against the 2 TSY - 1 left rows they meet at the tile's row
  // shifts: left row i meets right row i - t at shift t, and no other
  // combination is multiplied.  The right rows stay in registers.  One body of
  // TSY^2 TSX^2 products; a longer one (groups of rows rotating through the
  // registers, twice the code) missed the instruction cache.
  __device__ __forceinline__ void block(const char* w0, const char* w1, int w_step, const char* r, int r_step) {
    T v[TSY][TSX];
#pragma unroll
    for (int y = 0; y < TSY; ++y) right(v[y], r + y * r_step);
#pragma unroll
    for (int i = 0; i < 2 * TSY - 1; ++i) {
      window(w0, w1);
#pragma unroll
      for (int t = 0; t < TSY; ++t)
        if (t <= i && i - t < TSY) row(v[i - t], t);
      w0 += w_step;
      w1 += w_step;
    }
  }
  __device__ __forceinline__ void put(T* buf, int t) const {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if constexpr (sizeof(T) == 4)
        *reinterpret_cast<float4*>(buf + h * V) =
            make_float4(acc[t][h * V], acc[t][h * V + 1], acc[t][h * V + 2], acc[t][h * V + 3]);
      else
        *reinterpret_cast<double2*>(buf + h * V) = make_double2(acc[t][h * V], acc[t][h * V + 1]);
    }
  }
  __device__ __forceinline__ T get(int t, int q) const { return acc[t][q]; }
};

// Byte offset of a left row's 32-byte chunk: 16 bytes of padding per 128, so
// that lanes 32 bytes apart read from different banks.
__host__ __device__ __forceinline__ int chunk_at(int e) { return e * 32 + (e >> 2) * 16; }

// Rows of a matrix into shared memory in chunks of 16 bytes: row i at dst +
// i pitch, chunk j, from column col(j) on, at `at(j)`; rows outside [0, H) and
// columns outside [0, W) are zeros.  The chunks of all rows are dealt over the
// CTA's threads.
template <typename T, typename Col, typename At>
__device__ __forceinline__ void stage_rows(char* dst, int pitch, const T* __restrict__ src, int row0, int n_rows,
                                           int H, int W, int chunks, Col col, At at) {
  constexpr int V = 16 / (int)sizeof(T);
  const bool vec = W % V == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  const int total = n_rows * chunks;
#pragma unroll 4
  for (int k = threadIdx.x; k < total; k += blockDim.x) {
    const int i = k / chunks, j = k - i * chunks;
    const int r = row0 + i, c = col(j);
    const bool in = r >= 0 && r < H;
    const T* s = src + (long long)(in ? r : 0) * W + c;
    T v[V];
    if (vec && in && c >= 0 && c < W) {
      if constexpr (sizeof(T) == 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(s));
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
        v[3] = q.w;
      } else {
        const double2 q = __ldg(reinterpret_cast<const double2*>(s));
        v[0] = q.x;
        v[1] = q.y;
      }
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q) v[q] = in && !vec && c + q >= 0 && c + q < W ? __ldg(s + q) : T(0);
    }
    char* d = dst + i * pitch + at(j);
    if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<double2*>(d) = make_double2(v[0], v[1]);
  }
}

// One output's sum over a block's right rows by the definition: left row y +
// dy, column x + dx.  For outputs whose sum came out as NaN: the zero columns
// and rows around the matrices make NaN of an infinity, and of a NaN, that the
// shift does not meet.  A sum that is NaN stays one, so the loop ends there.
// One lane walks one output's overlap, at many times a product's cost in the
// kernel's body: one NaN in the left of one_to_many 256x256 x 64 makes 9.8 ms
// 18.5, one value of a hundred 25.1 (the tiled kernel, which spreads it, 14.0);
// one infinity costs nothing (9.7: only sums that are NaN are made again).
template <typename T>
__device__ __forceinline__ T overlap_sum(const T* __restrict__ L, const T* __restrict__ R, int Hl, int Wl, int rows,
                                         int Wr, int dy, int dx) {
  T s = T(0);
  const int y1 = min(rows, Hl - dy), xa = max(0, -dx), x1 = min(Wr, Wl - dx);
  for (int y = max(0, -dy); y < y1; ++y) {
    const T* l = L + (long long)(y + dy) * Wl + dx;
    const T* r = R + (long long)y * Wr;
    for (int x = xa; x < x1; ++x) s = fma(__ldg(l + x), __ldg(r + x), s);
    if (s != s) break;
  }
  return s;
}

// Zeros for the blocks to add to.  Launched in stream order: everything before
// it is done when it starts, so the correlation kernel, which may start right
// after it did, can read its inputs without waiting.
template <typename T>
__global__ void __launch_bounds__(256) zero_kernel(T* out, long long n) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int V = 16 / (int)sizeof(T);
  const long long head = min(n, (long long)((16 - (reinterpret_cast<uintptr_t>(out) & 15)) & 15) / (int)sizeof(T));
  const long long nv = (n - head) / V, tail = head + nv * V;
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i0 < head) out[i0] = T(0);
  if (i0 < n - tail) out[tail + i0] = T(0);
  for (long long i = i0; i < nv; i += (long long)gridDim.x * blockDim.x)
    reinterpret_cast<float4*>(out + head)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// FLIP: `left` holds the pairs' right matrices and `right` the left ones, and
// the outputs are mirrored.  (A form of its own: the choice of address at run
// time cost 1 to 4% of the other launches.)
template <typename T, int TSY, bool WIN, bool FLIP>
__global__ void __launch_bounds__(256, 2) cyclic_kernel(const CycArgs<T> p) {
  using Tl = Tile<T, TSY>;
  constexpr int TSX = Tl::TSX;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  char* sl = reinterpret_cast<char*>(smem_raw);        // left rows
  char* sr = sl + (size_t)p.l_rows * p.l_pitch;        // right rows
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* buf = reinterpret_cast<T*>(sr + (size_t)p.hb * p.r_pitch) + warp * (TSY * 32 * TSX);

  unsigned bid = blockIdx.x;
  const int g = (int)(bid % (unsigned)p.groups);
  bid /= (unsigned)p.groups;
  const int rb = (int)(bid % (unsigned)p.n_rb);
  bid /= (unsigned)p.n_rb;
  const int k = (int)(bid % (unsigned)p.pm.K), l = (int)(bid / (unsigned)p.pm.K);
  const long long lefts = l, rights = l * p.pm.r_l + k * p.pm.r_k;
  const T* __restrict__ L = p.left + (FLIP ? rights : lefts) * p.Hl * p.Wl;
  const int b0 = rb * p.hb, hbj = min(p.hb, p.Hr - b0);
  const T* __restrict__ R = p.right + ((FLIP ? lefts : rights) * p.Hr + b0) * (long long)p.Wr;
  T* out = p.out + (l * p.pm.o_l + k * p.pm.o_k) * p.Sy * (long long)p.Sx + (FLIP ? p.Sy * (long long)p.Sx - 1 : 0);

  // This CTA's tiles u0 .. u1; left row (u - u0) TSY + i of shared memory is
  // row u TSY - (hb - 1) + i of the matrix, which right row i - t of the block
  // meets at row shift t of tile u.
  constexpr int V = 16 / (int)sizeof(T);
  int u0, u1, c0 = 0;
  if constexpr (WIN) {
    c0 = g % p.win * 32;
    u0 = g / p.win * nw;
    u1 = min(p.ST, u0 + nw) - 1;
  } else {
    u0 = g * nw * 32 / p.C;
    u1 = min(p.ST - 1, ((g + 1) * nw * 32 - 1) / p.C);
  }
  const int n_rows = (u1 - u0 + 1) * TSY + p.hb - 1;
  const int row0 = u0 * TSY - (p.hb - 1);
  const auto at = [](int j) { return chunk_at(j >> 1) + (j & 1) * 16; };
  if constexpr (WIN) {
    const int period = p.C + 1;
    stage_rows(sl, p.l_pitch, L, row0, n_rows, p.Hl, p.Wl, 2 * p.chunks,
               [&](int j) {
                 const int q = (c0 + (j >> 1)) % period;
                 return q < p.C ? q * TSX + (j & 1) * V : p.Wl;
               },
               at);
  } else {
    stage_rows(sl, p.l_pitch, L, row0, n_rows, p.Hl, p.Wl, 2 * (p.C + 2), [](int j) { return j * V - TSX; }, at);
  }
  stage_rows(sr, p.r_pitch, R, 0, p.hb, hbj, p.Wr, 2 * p.NB, [](int j) { return j * V; },
             [](int j) { return j * 16; });
  asm volatile("griddepcontrol.wait;" ::: "memory");  // for the zeros
  __syncthreads();

  int u, c, uw0, uw1;
  bool live;
  if constexpr (WIN) {
    uw0 = uw1 = u = u0 + warp;
    if (u > u1) return;
    live = c0 + lane < p.C;
    c = live ? c0 + lane : c0;
  } else {
    const int w0 = (g * nw + warp) * 32, n_ids = p.C * p.ST;
    if (w0 >= n_ids) return;
    const int id = w0 + lane;
    live = id < n_ids;
    u = live ? id / p.C : u1;
    c = live ? id - u * p.C : 0;
    uw0 = w0 / p.C;
    uw1 = min(p.ST - 1, (w0 + 31) / p.C);
  }
  // Groups of TSY right rows some lane of the warp has left rows for: group j
  // meets left rows u TSY - (hb - 1) + j TSY + (0 .. 2 TSY - 2).
  const int j0 = max(0, (p.hb - 1 - uw1 * TSY - (2 * TSY - 2) + TSY - 1) / TSY);
  const int j1 = min((hbj + TSY - 1) / TSY, (p.Hl + p.hb - 1 - uw0 * TSY + TSY - 1) / TSY);
  const char* lrow = sl + (size_t)((u - u0) * TSY) * p.l_pitch;

  Tl a;
  a.zero();
  int e = c, b = 0, m = 0;  // left block, right block, wraps so far
  const int my_steps = p.NB + (p.NB + c) / p.C;
  const int steps = (int)__reduce_max_sync(0xffffffffu, (unsigned)my_steps);
  // output of class element q, row shift t, after m wraps
  const int sy = u * TSY - (b0 + p.hb - 1) + p.Hr - 1;  // of t = 0
  const int sx = c * TSX + p.Wr - 1;                    // of q = 0, m = 0
  const int P = p.C * TSX;
  // a sum that is NaN is made again from what its shift meets (`redo`)
  const auto emit = [&](int oy, int ox, T v) {
    const long long at = (long long)oy * p.Sx + ox;
    T* dst = FLIP ? out - at : out + at;
    if (p.accumulate) atomicAdd(dst, v);  // result unused: red.global.add
    else *dst = v;
  };
  const auto redo = [&](int oy, int ox) {
    emit(oy, ox,
         overlap_sum(L, R, p.Hl, p.Wl, hbj, p.Wr, oy - (p.Hr - 1) + b0, ox - (p.Wr - 1)));
  };
  // the warp's buffer, as the sums of segment mm of every lane in `mask`
  const auto flush = [&](int mm, unsigned mask) {
    __syncwarp();
    unsigned bad = 0;  // NaN sums, by j TSY + t
#pragma unroll
    for (int j = 0; j < TSX; ++j) {
      const int from = j * (32 / TSX) + lane / TSX;
      const int fy = __shfl_sync(0xffffffffu, sy, from);
      const int fx = __shfl_sync(0xffffffffu, sx, from) - mm * P + lane % TSX;
      if (!((mask >> from) & 1u) || fx < 0 || fx >= p.Sx) continue;
#pragma unroll
      for (int t = 0; t < TSY; ++t)
        if (fy + t >= 0 && fy + t < p.Sy) {
          const T v = buf[t * (32 * TSX) + j * 32 + lane];
          if (v == v) emit(fy + t, fx, v);
          else bad |= 1u << (j * TSY + t);
        }
    }
    while (__any_sync(0xffffffffu, bad != 0)) {
      const int i = bad ? __ffs((int)bad) - 1 : 0, j = i / TSY;
      const int from = j * (32 / TSX) + lane / TSX;
      const int fy = __shfl_sync(0xffffffffu, sy, from) + i % TSY;
      const int fx = __shfl_sync(0xffffffffu, sx, from) - mm * P + lane % TSX;
      if (bad) redo(fy, fx);
      bad &= bad - 1;
    }
    __syncwarp();
  };

  for (int s = 0; s < steps; ++s) {
    const int at0 = WIN ? c - c0 + s : e + 1;
    const char* w_lo = lrow + chunk_at(at0);
    const char* w_hi = lrow + chunk_at(at0 + 1);
    const char* rq = sr + b * 32 + j0 * TSY * p.r_pitch;
    w_lo += j0 * TSY * p.l_pitch;
    w_hi += j0 * TSY * p.l_pitch;
#pragma unroll 1
    for (int j = j0; j < j1; ++j) {
      a.block(w_lo, w_hi, p.l_pitch, rq, p.r_pitch);
      w_lo += TSY * p.l_pitch;
      w_hi += TSY * p.l_pitch;
      rq += TSY * p.r_pitch;
    }
    // next block; a lane at the left row's end hands over and wraps, a lane
    // that is done before the warp's last step hands over too
    const bool wrap = e == p.C - 1;
    const bool done = !wrap && b == p.NB - 1;
    if ((wrap || done) && s + 1 < steps && s < my_steps) {
      if (m == 0) {
#pragma unroll
        for (int t = 0; t < TSY; ++t) a.put(buf + t * (32 * TSX) + lane * TSX, t);
      } else if (live) {
        unsigned bad = 0;
#pragma unroll
        for (int t = 0; t < TSY; ++t)
#pragma unroll
          for (int q = 0; q < TSX; ++q) {
            const int x = sx - m * P + q;
            if (sy + t >= 0 && sy + t < p.Sy && x >= 0 && x < p.Sx) {
              const T v = a.get(t, q);
              if (v == v) emit(sy + t, x, v);
              else bad |= 1u << (t * TSX + q);
            }
          }
        for (; bad; bad &= bad - 1) {
          const int i = __ffs((int)bad) - 1;
          redo(sy + i / TSX, sx - m * P + i % TSX);
        }
      }
      a.zero();
    }
    if (wrap) {
      e = -1;
      ++m;
    } else if (!done) {
      ++e;
      ++b;
    }
  }
  // Lanes that took every step hold their last segment (the same one, m, in
  // all of them); the buffer holds segment 0 of the others and of wrapped ones.
  const bool last = my_steps == steps;
  // a wrap at the very last step would move on to a segment without products
  const int mm = steps - p.NB;
  const unsigned live_mask = __ballot_sync(0xffffffffu, live);
  const unsigned last_mask = __ballot_sync(0xffffffffu, live && last);
  if (mm > 0) flush(0, live_mask);
  if (last) {
#pragma unroll
    for (int t = 0; t < TSY; ++t) a.put(buf + t * (32 * TSX) + lane * TSX, t);
  }
  flush(mm, mm > 0 ? last_mask : live_mask);
}

struct CycPlan {
  int tsy, hb, nw, win, chunks, n_rb, ST, groups, l_rows, l_pitch, r_pitch, smem;
  long long warps;  // over all pairs and blocks
};

// The plan for `hb` right rows per block and nw warps per CTA, in the flat or
// the windowed form.
template <typename T>
bool cyc_layout(const Geometry& g, long long pairs, int TSY, int hb, int nw, bool windowed, CycPlan* c) {
  constexpr int TSX = 32 / (int)sizeof(T);
  const int C = div_up(g.Wl, TSX), NB = div_up(g.Wr, TSX);
  hb = div_up(hb, TSY) * TSY;
  c->tsy = TSY;
  c->hb = hb;
  c->n_rb = div_up(g.Hr, hb);
  c->ST = div_up((long)g.Hl + hb - 1, TSY);
  const long long ids = (long long)C * c->ST;
  if (ids > (1LL << 30)) return false;
  c->win = windowed ? div_up(C, 32) : 0;
  long long w, chunks;
  if (windowed) {
    c->nw = std::min(nw, c->ST);
    c->groups = c->win * div_up(c->ST, c->nw);
    w = (long long)c->win * c->ST;
    c->l_rows = c->nw * TSY + hb - 1;
    chunks = 32LL + NB + (NB + C - 1) / C + 1;  // first chunks of 32 lanes, every step, the window's second chunk
  } else {
    w = (ids + 31) / 32;
    c->nw = (int)std::min<long long>(nw, w);
    c->groups = (int)((w + c->nw - 1) / c->nw);
    const long long span = (32LL * c->nw + C - 2) / C + 1;  // tiles a CTA's lanes can touch
    c->l_rows = (int)std::min<long long>(span, c->ST) * TSY + hb - 1;
    chunks = C + 2;
  }
  if (chunks > 8192) return false;
  c->chunks = (int)chunks;
  c->warps = pairs * c->n_rb * w;
  c->l_pitch = chunk_at(c->chunks - 1) + 32;
  c->r_pitch = NB * 32;
  const long long smem = (long long)c->l_rows * c->l_pitch + (long long)hb * c->r_pitch +
                         (long long)c->nw * TSY * 32 * TSX * (long long)sizeof(T);
  c->smem = (int)std::min<long long>(smem, 1 << 30);
  return smem <= 227 * 1024 && pairs * c->n_rb * c->groups <= 0x7fffffffLL;
}

// Share of the SMs' warp slots (16 per SM) the shape's busy lanes fill.
double cyc_fill(const CycPlan& c, int C) {
  const int res = std::min(16, (227 * 1024) / (c.smem + 1024) * c.nw);
  return res / 16.0 * (c.win ? (double)C / (32.0 * c.win) : 1.0);
}

// Row shifts per lane, right rows per block and warps per CTA: the first shape
// of the list that gives the launch enough warps, the last one otherwise.
// Longer blocks load and add less per product (a block adds each of its
// outputs once), more warps fill the GPU.  Measured (us; FP32 unless said):
//   one_to_many 256x256 x 64   4 shifts, 16 rows 9767; 4, 8: 10276; 4, 4: 11170; 2, 16: 10956
//   n_to_m 3x6, 201x183 by 75x59   4, 16: 167 (4 warps per CTA) and 196 (8); 4, 8: 173; 2, 8: 199
//   one pair of 128x128        4, 8: 41; 2, 8: 29; 2, 4: 27; 2, 2: 29
//   n_to_mn 8 + 32, 64x64 FP64   2, 16: 1281; 2, 8: 1199; 2, 4: 1027; 2, 2: 1021
//   one pair of 1x300, FP32    1, 1: 10.8; 2, 2: 17.2 (the tiled kernel 10.7)
//   n_to_m 4x8, 16x300 by 1x300 FP64   1, 1: 121; 2, 2: 312 (309)
//   n_to_m 8x9, 314x403 by 1x1, FP32   1, 1: 60.6; 2, 2: 52.6
// FP64 wants more warps (its pipe is the bound, and an uneven share of the SMs
// shows), FP32 chains stay within 4096 products as in the tiled kernel.  Rights
// of one row take 1 shift and 1 row, which multiplies nothing else; in FP32 with
// a single column block of a wider left, where outputs and not products cost,
// only launches that 2 shifts do not fill.
template <typename T>
bool cyc_plan(const Geometry& g, long long pairs, CycPlan* best) {
  constexpr bool f32 = sizeof(T) == 4;
  constexpr int TSX = 32 / (int)sizeof(T);
  struct Shape {
    int tsy, hb;
  };
  constexpr Shape shapes[] = {{4, 16}, {4, 8}, {2, 8}, {2, 4}, {2, 2}, {1, 1}};
  const int chain = f32 ? 4096 / g.Wr : 1 << 30;
  if (chain < 2) return false;  // rows too wide for a chain of two
  const long long enough = (f32 ? 6LL : 32LL) * sm_count_cached();
  bool found = false;
  for (const Shape& sh : shapes) {
    if (sh.hb > chain || (!f32 && sh.tsy == 4) || (sh.hb > 2 && sh.hb / 2 >= g.Hr)) continue;
    if (g.Hr > 1 ? sh.hb == 1 : sh.hb == 2 && (!f32 || g.Wr > TSX || g.Wl <= TSX)) continue;
    CycPlan c;
    // CTAs of eight warps share more of their left rows; four-warp ones spread
    // a short launch more evenly.  The form that fills more warp slots.
    bool fits = false;
    const int C = div_up(g.Wl, 32 / (int)sizeof(T));
    for (int nw : {8, 4, 2, 1})
      for (bool windowed : {false, true}) {
        CycPlan t;
        if (!cyc_layout<T>(g, pairs, sh.tsy, sh.hb, nw, windowed, &t)) continue;
        if (nw == 8 && t.warps < 64LL * sm_count_cached()) continue;
        if (fits && cyc_fill(t, C) <= cyc_fill(c, C)) continue;
        c = t;
        fits = true;
      }
    if (!fits) continue;
    *best = c;
    found = true;
    if (c.warps >= enough) break;
  }
  return found;
}

template <typename T>
xc_status cyc_launch(const T* left, const T* right, T* out, Geometry g, const PairMap& pm, cudaStream_t stream,
                     bool add, bool* taken) {
  constexpr int TSX = 32 / (int)sizeof(T);
  // A left narrower than the right changes places with it: few classes wrap
  // often, and every wrap costs a surplus block and a hand-over (16x16 by
  // 128x128 27.6 us, 8.1 with places changed; x 24 43.0 and 16.4).  Not where
  // the right has one to three rows and the left many: in the left's part those
  // few rows meet a few right rows each, most of a block's products are of
  // zeros.  There the wraps cost less once the lanes (a left row's classes, over
  // all pairs) fill the GPU: 1000x1 by 1x8 x 64 50.4 us, 6.6 in its place; 300x4 by
  // 2x40 x 64 21.3 and 16.9; 238x160 by 1x227, 105 pairs, 352 and 152; but one
  // pair of 300x1 by 1x40 5.2 and 8.2, of 300x2 by 1x8 4.8 and 5.2, 20x60 by 1x300
  // x 64 17.8 and 24.9.
  const int C = div_up(g.Wl, TSX);
  const long long lanes = (long long)pm.n_left * pm.K * g.Hl * C;
  const bool columns = g.Hl > g.Hr && ((g.Hr == 1 && C == 1 && g.Wr <= 8 && (g.Hl < 64 || lanes >= 2000)) ||
                                       (g.Hr <= 3 && g.Hl >= 64 && lanes >= (g.Hr == 1 && C == 1 ? 9000 : 16000)));
  const bool flip = g.Wl < g.Wr && !columns;
  if (flip) {
    std::swap(g.Hl, g.Hr);
    std::swap(g.Wl, g.Wr);
    std::swap(left, right);
  }
  CycPlan c;
  *taken = cyc_plan<T>(g, (long long)pm.n_left * pm.K, &c);
  if (!*taken) return XC_OK;
  CycArgs<T> a;
  a.left = left;
  a.right = right;
  a.out = out;
  a.Hl = g.Hl;
  a.Wl = g.Wl;
  a.Hr = g.Hr;
  a.Wr = g.Wr;
  a.Sy = g.Sy;
  a.Sx = g.Sx;
  a.pm = pm;
  a.C = flip ? div_up(g.Wl, TSX) : C;
  a.NB = div_up(g.Wr, TSX);
  a.hb = c.hb;
  a.n_rb = c.n_rb;
  a.ST = c.ST;
  a.groups = c.groups;
  a.win = c.win;
  a.chunks = c.chunks;
  a.l_rows = c.l_rows;
  a.l_pitch = c.l_pitch;
  a.r_pitch = c.r_pitch;
  a.accumulate = add || c.n_rb > 1 ? 1 : 0;
  const long long blocks = (long long)pm.n_left * pm.K * c.n_rb * c.groups;
  if (c.n_rb > 1 && !add) {
    const long long n_out = (long long)(pm.n_left - 1) * pm.o_l + (long long)(pm.K - 1) * pm.o_k + 1;
    const long long n = n_out * g.Sy * g.Sx;
    const long long want = (n * (long long)sizeof(T) + 4095) / 4096;  // 16 bytes a thread
    zero_kernel<T><<<(unsigned)std::min<long long>(8LL * sm_count_cached(), want), 256, 0, stream>>>(out, n);
    XC_CUDA_TRY(cudaGetLastError());
  }
  const auto pick = [&](auto tsy) -> void (*)(const CycArgs<T>) {
    constexpr int Y = decltype(tsy)::value;
    if (c.win) return flip ? cyclic_kernel<T, Y, true, true> : cyclic_kernel<T, Y, true, false>;
    return flip ? cyclic_kernel<T, Y, false, true> : cyclic_kernel<T, Y, false, false>;
  };
  void (*kern)(const CycArgs<T>) = nullptr;
  if constexpr (sizeof(T) == 4) {
    if (c.tsy == 4) kern = pick(std::integral_constant<int, 4>());
  }
  if (c.tsy == 2) kern = pick(std::integral_constant<int, 2>());
  if (c.tsy == 1) kern = pick(std::integral_constant<int, 1>());
  XC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  const int slot = kernel_timer_begin(stream);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(32u * c.nw);
  cfg.dynamicSmemBytes = (size_t)c.smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = c.n_rb > 1 && !add ? 1 : 0;  // without the zero kernel before it, in stream order
  XC_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a));
  kernel_timer_end(slot, stream);
  return XC_OK;
}

}  // namespace

xc_status direct_cyclic(xc_dtype dtype, const void* left, const void* right, void* out, const Geometry& g,
                        const PairMap& pm, cudaStream_t stream, bool add, bool* taken) {
  if (dtype == XC_F32)
    return cyc_launch<float>((const float*)left, (const float*)right, (float*)out, g, pm, stream, add, taken);
  return cyc_launch<double>((const double*)left, (const double*)right, (double*)out, g, pm, stream, add, taken);
}

}  // namespace xc
