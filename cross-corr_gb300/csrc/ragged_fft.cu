// ragged_fft.cu -- pairs of a ragged batch through the fused FFT kernels.
//
// Pairs of any sizes share the launches of their transform lengths: the
// kernels take their geometry from records in device memory and their place
// from a list entry per CTA, so a batch is a few dozen launches (one per
// length and phase) however many pairs it has.
#include "ragged_fft.h"

#include <algorithm>
#include <cstring>
#include <map>

#include "fft_engine.h"
#include "xc_common.cuh"

namespace xc {
namespace fe {

namespace {

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Lengths, kernels and workspace of one pair.
struct PairPlan {
  int nx, ny, nblk;
  ColKernels ck;
  RowKernels rk;
  size_t al, ar, b, bytes;  // offsets within the pair's workspace
};
bool plan_pair(const Geometry& g, PairPlan* p) {
  p->nx = length_for(g.Sx);
  p->ny = length_for(g.Sy);
  if (p->nx == 0 || p->ny == 0 || !row_kernels_f32(p->nx, &p->rk) || !col_kernels_f32(p->ny, &p->ck)) return false;
  const int cb = 1 << p->ck.lgcb;
  p->nblk = div_up(p->nx / 2 + 1, cb);
  const size_t row = (size_t)p->nblk * cb * sizeof(Cx<float>);
  p->al = 0;
  p->ar = align256(row * g.Hl);
  p->b = p->ar + align256(row * g.Hr);
  p->bytes = p->b + align256(row * g.Sy);
  return true;
}

// Chunks of consecutive pairs whose workspaces fit `cap` together.
std::vector<size_t> chunk_starts(const std::vector<PairPlan>& plans, size_t cap, size_t* most) {
  std::vector<size_t> starts;
  size_t used = 0;
  *most = 0;
  for (size_t i = 0; i < plans.size(); ++i) {
    if (i == 0 || used + plans[i].bytes > cap) {
      starts.push_back(i);
      used = 0;
    }
    used += plans[i].bytes;
    *most = std::max(*most, used);
  }
  starts.push_back(plans.size());
  return starts;
}

// Host image of the device tables.
struct Image {
  std::vector<char> bytes;
  template <typename T>
  size_t put(const std::vector<T>& v) {
    const size_t at = align256(bytes.size());
    bytes.resize(at + v.size() * sizeof(T));
    std::memcpy(bytes.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
};

template <typename Rec>
struct Group {  // the records and CTA (or unit) list of one length
  std::vector<Rec> items;
  std::vector<int2> list;
  size_t items_at = 0, list_at = 0;
};

template <typename Args>
std::vector<char> blob(const Args& a) {
  std::vector<char> v(sizeof(a));
  std::memcpy(v.data(), &a, sizeof(a));
  return v;
}

xc_status raise_limit(const void* fn, int bytes) {
  if (bytes > 48 * 1024) XC_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return XC_OK;
}

}  // namespace

bool ragged_fft_takes(const Geometry& g) {
  PairPlan p;
  // the ragged column kernel keeps both blocks in shared memory
  return plan_pair(g, &p) && 2 * p.ck.unit_smem <= 227 * 1024;
}

size_t ragged_fft_workspace(const std::vector<FftPair>& pairs, size_t cap) {
  std::vector<PairPlan> plans(pairs.size());
  for (size_t i = 0; i < pairs.size(); ++i) plan_pair(pairs[i].g, &plans[i]);
  size_t most = 0;
  chunk_starts(plans, cap, &most);
  return most;
}

xc_status ragged_fft_build(RaggedFft* f, const std::vector<FftPair>& pairs, void* workspace, size_t cap) {
  using T = float;
  ragged_fft_release(f);
  std::vector<PairPlan> plans(pairs.size());
  for (size_t i = 0; i < pairs.size(); ++i)
    if (!plan_pair(pairs[i].g, &plans[i])) return fail(XC_ERR_UNSUPPORTED, "pair beyond the FFT kernels' lengths");
  size_t most = 0;
  const std::vector<size_t> starts = chunk_starts(plans, cap, &most);
  Image image;
  // twiddles of every length in use, and a row of zeros
  std::map<int, size_t> twx, twy;
  int longest = 0;
  for (const PairPlan& p : plans) {
    longest = std::max(longest, p.nx);
    for (int rows = 0; rows < 2; ++rows) {
      const int n = rows ? p.nx : p.ny;
      auto& m = rows ? twx : twy;
      if (m.count(n)) continue;
      std::vector<char> t(twiddle_bytes(n, rows != 0, XC_F32));
      fill_twiddles(n, rows != 0, XC_F32, t.data());
      m[n] = image.put(t);
    }
  }
  const size_t zeros = image.put(std::vector<float>(longest, 0.0f));

  struct Chunk {
    std::map<int, Group<RagRow<T>>> fwd;
    std::map<int, Group<RagCol<T>>> col;
    std::map<int, Group<RagInv<T>>> inv;
  };
  std::vector<Chunk> chunks(starts.size() - 1);
  for (size_t c = 0; c + 1 < starts.size(); ++c) {
    Chunk& ch = chunks[c];
    char* ws = static_cast<char*>(workspace);
    for (size_t i = starts[c]; i < starts[c + 1]; ++i) {
      const PairPlan& p = plans[i];
      const Geometry& g = pairs[i].g;
      Cx<T>* al = reinterpret_cast<Cx<T>*>(ws + p.al);
      Cx<T>* ar = reinterpret_cast<Cx<T>*>(ws + p.ar);
      Cx<T>* b = reinterpret_cast<Cx<T>*>(ws + p.b);
      ws += p.bytes;
      const Scales sc = spectrum_scales(p.nx, p.ny, true);
      const int rows = 2 * p.rk.nv * p.rk.q;
      Group<RagRow<T>>& gf = ch.fwd[p.nx];
      for (int side = 0; side < 2; ++side) {
        const int H = side ? g.Hr : g.Hl;
        for (int q = 0; q < div_up(H, rows); ++q) gf.list.push_back(make_int2((int)gf.items.size(), q));
        gf.items.push_back(RagRow<T>{side ? pairs[i].right : pairs[i].left, side ? ar : al, H, side ? g.Wr : g.Wl,
                                     p.ck.lgcb, (T)(side ? sc.right : sc.left)});
      }
      Group<RagCol<T>>& gc = ch.col[p.ny];
      for (int k = 0; k < p.nblk; ++k) gc.list.push_back(make_int2((int)gc.items.size(), k));
      gc.items.push_back(RagCol<T>{al, ar, b, g.Hl, g.Hr, g.Sy, p.nblk});
      Group<RagInv<T>>& gi = ch.inv[p.nx];
      for (int q = 0; q < div_up(g.Sy, rows); ++q) gi.list.push_back(make_int2((int)gi.items.size(), q));
      const T hi = (T)sc.rest;
      gi.items.push_back(RagInv<T>{b, pairs[i].out, g.Sy, g.Sx, g.Wr, p.ck.lgcb, hi, (T)(sc.rest - (double)hi)});
    }
    const auto put = [&](auto& groups) {
      for (auto& kv : groups) {
        kv.second.items_at = image.put(kv.second.items);
        kv.second.list_at = image.put(kv.second.list);
      }
    };
    put(ch.fwd);
    put(ch.col);
    put(ch.inv);
  }
  XC_CUDA_TRY(cudaMalloc(&f->tables, image.bytes.size()));
  const xc_status up = upload(f->tables, image.bytes.data(), image.bytes.size());
  if (up != XC_OK) {
    ragged_fft_release(f);
    return up;
  }
  const char* base = static_cast<const char*>(f->tables);
  for (Chunk& ch : chunks) {
    std::vector<RaggedFft::Launch> fwd, col, inv;
    for (auto& kv : ch.fwd) {
      RowKernels rk{};
      row_kernels_f32(kv.first, &rk);
      RowFwdArgs<T> a{};
      a.tw = base + twx[kv.first];
      a.zeros = reinterpret_cast<const T*>(base + zeros);
      a.items = reinterpret_cast<const RagRow<T>*>(base + kv.second.items_at);
      a.ctas = reinterpret_cast<const int2*>(base + kv.second.list_at);
      fwd.push_back({rk.rag_forward, (unsigned)kv.second.list.size(), rk.threads, rk.smem, blob(a)});
    }
    for (auto& kv : ch.col) {
      ColKernels ck{};
      col_kernels_f32(kv.first, &ck);
      ColArgs<T> a{};
      a.tw = base + twy[kv.first];
      a.items = reinterpret_cast<const RagCol<T>*>(base + kv.second.items_at);
      a.units = reinterpret_cast<const int2*>(base + kv.second.list_at);
      a.n_units = (int)kv.second.list.size();
      const int blocks = div_up(a.n_units, ck.pu);
      col.push_back({ck.form(blocks, sm_count_cached()).rag_pairs, (unsigned)blocks, ck.threads, 2 * ck.unit_smem, blob(a)});
    }
    for (auto& kv : ch.inv) {
      RowKernels rk{};
      row_kernels_f32(kv.first, &rk);
      RowInvArgs<T> a{};
      a.tw = base + twx[kv.first];
      a.items = reinterpret_cast<const RagInv<T>*>(base + kv.second.items_at);
      a.ctas = reinterpret_cast<const int2*>(base + kv.second.list_at);
      inv.push_back({rk.rag_inverse, (unsigned)kv.second.list.size(), rk.threads, rk.smem, blob(a)});
    }
    for (auto* ph : {&fwd, &col, &inv}) {
      for (const RaggedFft::Launch& l : *ph) XC_TRY(raise_limit(l.fn, l.smem));
      // most work first, so that the streams end together
      std::stable_sort(ph->begin(), ph->end(), [](const RaggedFft::Launch& x, const RaggedFft::Launch& y) {
        return (double)x.blocks * x.threads > (double)y.blocks * y.threads;
      });
      f->phases.push_back(std::move(*ph));
    }
  }
  return XC_OK;
}

xc_status ragged_fft_enqueue(const RaggedFft& f, const cudaStream_t* streams, int n_streams, cudaEvent_t fork,
                             const cudaEvent_t* joins) {
  for (const auto& phase : f.phases) {
    const int used = std::max(1, std::min(n_streams, (int)phase.size()));
    if (used > 1) {
      XC_CUDA_TRY(cudaEventRecord(fork, streams[0]));
      for (int k = 1; k < used; ++k) XC_CUDA_TRY(cudaStreamWaitEvent(streams[k], fork, 0));
    }
    xc_status st = XC_OK;
    std::vector<double> load(used, 0.0);
    for (const RaggedFft::Launch& l : phase) {
      const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      load[k] += (double)l.blocks * l.threads;
      void* args[] = {const_cast<char*>(l.args.data())};
      const cudaError_t e =
          cudaLaunchKernel(l.fn, dim3(l.blocks), dim3((unsigned)l.threads), args, (size_t)l.smem, streams[k]);
      if (e != cudaSuccess) {
        st = from_cuda(e, "ragged FFT launch");
        break;
      }
    }
    // every forked stream joins, also after an error, so that a capture can end
    for (int k = 1; k < used; ++k) {
      cudaEventRecord(joins[k], streams[k]);
      cudaStreamWaitEvent(streams[0], joins[k], 0);
    }
    XC_TRY(st);
  }
  return XC_OK;
}

void ragged_fft_release(RaggedFft* f) {
  cudaFree(f->tables);
  f->tables = nullptr;
  f->phases.clear();
}

}  // namespace fe
}  // namespace xc
