// Engine of libtbpm_b200: buffers, launch plans, CUDA-graph replay and the
// drivers behind the C ABI.  The numerics live in tbpm_kernels.cuh.
//
// Data layout in HBM (one context):
//   Hamiltonian  indptr int32[N+1], indices int32[nnz], hop complex[nnz] in the
//                context precision (+ dx, dy real[nnz] for the current operator)
//   A            the state block being propagated, row-interleaved [N][ld]
//   X, Y         the two Chebyshev work vectors p_{k-1}, p_{k-2}  [N][ld]
//   wf0          the initial states (correlation reference)       [N][B]
//   partials     block partial sums of the fused reductions
//   out          per-step reduced values [rows][ld][nv] (FP64)
//   ctr          device step counter + finalize completion counter
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <optional>
#include <type_traits>

#include "tbpm_engine.cuh"
#include "tbpm_dc_kernels.cuh"
#include "tbpm_seg_kernels.cuh"
#include "tbpm_kernels.cuh"
#include "tbpm_ring_kernels.cuh"
#include "tbpm_pq_gemm.cuh"
#include "tbpm_pair_kernels.cuh"
#include "tbpm_more_kernels.cuh"
#include "tbpm_scan.cuh"
#include "tbpm_poly_kernels.cuh"


namespace tbpm {

void throw_cuda(cudaError_t e, const char* what) {
  (void)cudaGetLastError();  // clear sticky-free errors
  const int code = e == cudaErrorMemoryAllocation ? TBPM_ERR_OOM : TBPM_ERR_CUDA;
  throw Error{code, std::string(what) + ": " + cudaGetErrorString(e)};
}

void DevMem::ensure(size_t n) {
  if (n <= bytes && p) return;
  release();
  if (n == 0) n = 16;
  n = (n + 255) & ~(size_t)255;
  TBPM_CK(cudaMalloc(&p, n));
  bytes = n;
}

void DevMem::release() {
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
}

void GraphCache::reset() {
  if (exec) cudaGraphExecDestroy(exec);
  exec = nullptr;
  key.clear();
  steps = 0;
}

Expansion time_step_expansion(const double* bes, int n_bes) {
  // propagation.f90:33-48 with img_dt = +i (forward); backward columns are
  // selected through neg_mask (alpha -> -alpha).
  Expansion e;
  e.n_terms = n_bes;
  e.alpha1_re = 0.0;
  e.alpha1_im = -1.0;
  e.alpha_re = 0.0;
  e.alpha_im = -2.0;
  e.beta = 1.0;
  for (int s = 0; s < 2; ++s) {
    e.w[s].resize(n_bes);
    e.w[s][0] = bes[0];
    for (int k = 1; k < n_bes; ++k) e.w[s][k] = 2 * bes[k];
  }
  return e;
}

Expansion fermi_expansion(const double* coef_a, int n_a, const double* coef_b, int n_b,
                          unsigned long long set_b_mask) {
  // propagation.f90:66-81: T0 = H psi, T1 = 2 H T0 - psi, p2 = 2 H p1 - p0.
  Expansion e;
  e.n_terms = std::max(n_a, n_b);
  e.alpha1_re = 1.0;
  e.alpha1_im = 0.0;
  e.alpha_re = 2.0;
  e.alpha_im = 0.0;
  e.beta = -1.0;
  e.w[0].assign(e.n_terms, 0.0);
  e.w[1].assign(e.n_terms, 0.0);
  for (int k = 0; k < n_a; ++k) e.w[0][k] = coef_a[k];
  for (int k = 0; k < n_b; ++k) e.w[1][k] = coef_b[k];
  e.set_mask = set_b_mask;
  return e;
}

namespace {

constexpr int kSMs = 148;

template <typename R, int V_>
struct Prec {
  using Real = R;
  static constexpr int V = V_;
};

template <class F>
void dispatch(int prec, int V, F&& f) {
  if (prec == TBPM_PREC_FP64 && V == 2)
    f(Prec<double, 2>{});
  else if (prec == TBPM_PREC_FP64)
    f(Prec<double, 1>{});
  else if (V == 4)
    f(Prec<float, 4>{});
  else if (V == 2)
    f(Prec<float, 2>{});
  else
    f(Prec<float, 1>{});
}

inline size_t real_size(int prec) { return prec == TBPM_PREC_FP64 ? 8 : 4; }

int num_sms(int device) {
  static std::atomic<int> cached[64];
  if (device < 0 || device >= 64) return kSMs;
  if (!cached[device]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        v <= 0) {
      (void)cudaGetLastError();
      v = kSMs;
    }
    cached[device] = v;
  }
  return cached[device];
}

// Resident blocks per SM of `kernel` at the given block shape (cached for all contexts
// of the process, which may be driven from several threads).
template <class K>
int resident_per_sm(K kernel, int threads, size_t smem) {
  static std::mutex mutex;
  static std::vector<std::pair<std::pair<const void*, long long>, int>> cache;
  std::lock_guard<std::mutex> lock(mutex);
  const void* key = reinterpret_cast<const void*>(kernel);
  const long long shape = (long long)threads * (1ll << 32) + (long long)smem;
  for (const auto& e : cache)
    if (e.first.first == key && e.first.second == shape) return e.second;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem) != cudaSuccess) {
    (void)cudaGetLastError();
    nb = 1;
  }
  nb = std::max(nb, 1);
  cache.push_back({{key, shape}, nb});
  return nb;
}

// Block shape (threads = rpp rows x tpr threads per row) and a persistent
// grid: at most the number of blocks that are resident at once, so that the
// grid-stride kernels sweep the rows as one narrow band.  A positive
// opts.rows_per_tile instead sizes the grid as ceil(n_rows / rows_per_tile)
// (for tuning experiments).
template <class K>
Tile pick_tile(const tbpm_ctx* c, int64_t n_rows, int tpr, K kernel, size_t smem_per_thread,
               int default_threads = 256) {
  Tile t;
  int want = c->opts.threads_per_block > 0 ? c->opts.threads_per_block : default_threads;
  want = std::min(std::max(want, 32), 256);  // the kernels are bounded to 256 threads
  t.rpp = std::max(1, want / tpr);
  while (t.rpp * tpr > 256 && t.rpp > 1) --t.rpp;
  t.threads = t.rpp * tpr;
  const int64_t n_tiles = (n_rows + t.rpp - 1) / t.rpp;
  int64_t grid;
  if (c->opts.rows_per_tile > 0) {
    grid = (n_rows + c->opts.rows_per_tile - 1) / c->opts.rows_per_tile;
  } else {
    const int per_sm = resident_per_sm(kernel, t.threads, smem_per_thread * t.threads);
    grid = (int64_t)per_sm * num_sms(c->device);
  }
  grid = std::min<int64_t>(std::max<int64_t>(grid, 1), std::max<int64_t>(n_tiles, 1));
  t.grid = (int)grid;
  t.rows_per_tile = t.rpp;
  return t;
}

// ---- small utility kernels -------------------------------------------------

// dst[r*ld + col0 + s] = src[s*n + r]   (host C-order states -> interleaved)
template <typename R>
__global__ void interleave_kernel(const double2* src, int ns, int64_t n, int ld, int col0,
                                  typename Cx<R>::t* dst) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= n * ns) return;
  const int64_t r = gid / ns;
  const int s = (int)(gid - r * ns);
  const double2 v = src[(int64_t)s * n + r];
  typename Cx<R>::t o;
  o.x = (R)v.x;
  o.y = (R)v.y;
  dst[r * ld + col0 + s] = o;
}

// dst[s*n + r] = src[r*ld + col0 + s]   (interleaved -> host C-order states)
template <typename R>
__global__ void deinterleave_kernel(const typename Cx<R>::t* src, int ns, int64_t n, int ld,
                                    int col0, double2* dst) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= n * ns) return;
  const int s = (int)(gid / n);
  const int64_t r = gid - (int64_t)s * n;
  const typename Cx<R>::t v = src[r * ld + col0 + s];
  dst[gid] = make_double2((double)v.x, (double)v.y);
}


inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

// ---- launch helpers ----------------------------------------------------------

struct Counters {
  int* step;
  unsigned int* done;
};

Counters counters(tbpm_ctx* c, int which) {
  int* base = c->ctr.as<int>();
  return Counters{base + 2 * which, reinterpret_cast<unsigned int*>(base + 2 * which + 1)};
}

void reset_counters(tbpm_ctx* c, int which) {
  TBPM_CK(cudaMemsetAsync(c->ctr.as<int>() + 2 * which, 0, 2 * sizeof(int), c->stream));
}

void launch_finalize(tbpm_ctx* c, int grid_parts, int n_values, Counters k, double* out) {
  finalize_kernel<<<n_values, 256, 0, c->stream>>>(c->partials.as<double>(), grid_parts, n_values,
                                                    k.step, k.done, out);
  TBPM_CK(cudaGetLastError());
  c->launches++;
}

// Block partials of the fused reductions.  A persistent grid needs at most
// 192 values x (32 blocks per SM x SMs); reserving that much up front keeps
// every later request inside the buffer, so no allocation happens while a
// CUDA graph is being captured.
void ensure_partials(tbpm_ctx* c, size_t n_doubles) {
  const size_t floor_doubles = (size_t)192 * 32 * num_sms(c->device);
  c->partials.ensure(std::max(n_doubles, floor_doubles) * sizeof(double));
}

// Launch shapes of the four compiled modes of the Chebyshev-term kernel, and
// for each mode whether the shared-memory ring kernel runs it.
struct TermTiles {
  Tile t[4];
  bool ring[4] = {false, false, false, false};
  RingShape rs[4] = {};
  const int* win = nullptr;  // window records (ring_window_kernel); null: no windows
};

// Consumer threads of the ring kernel of a mode.
template <typename R, int V>
int ring_items(int mode, bool win) {
  if (mode == 0) return win ? kRingItems<R, V, 0, true> : kRingItems<R, V, 0, false>;
  if (mode == 1) return win ? kRingItems<R, V, 1, true> : kRingItems<R, V, 1, false>;
  if (mode == 2) return win ? kRingItems<R, V, 2, true> : kRingItems<R, V, 2, false>;
  if (mode == 4) return kRingItems<R, V, 4, false>;
  return kRingItems<R, V, 3, false>;
}

// Ring layout for rows of tpr packs in kernel mode `mode` (ref_tpr: packs per
// row of the MODE 2 correlation reference, 0 for none); stages == 0 when the
// ring does not apply (rows that are not a multiple of 16 bytes, or fewer than
// two stages fit into the shared memory of one of kRingMinBlocks blocks per SM).
template <typename R, int V>
RingShape ring_shape(const tbpm_ctx* c, int tpr, int mode, int ref_tpr, bool win = false,
                     int items = 0) {
  RingShape s{};
  if (items == 0) items = ring_items<R, V>(mode, win);
  const size_t row_bytes = (size_t)tpr * sizeof(Pack<R, V>);
  if (row_bytes % 16 != 0 || tpr < 1 || tpr > items) return s;
  const int TR = items / tpr;
  const Ham& h = c->ham;
  const size_t cs = sizeof(typename Cx<R>::t);
  // CSR entries one stage holds: the mean row length of O over a tile with 25%
  // slack, plus the widening to 16-byte boundaries; denser tiles read their
  // entries from global memory instead
  const double per_row = h.n > 0 ? (double)h.nnz / (double)h.n : 0.0;
  int cap = (int)std::ceil(per_row * TR * 1.25) + 8;
  cap = (cap + 3) & ~3;
  auto al = [](size_t b) { return (int)((b + 127) & ~(size_t)127); };
  const int tile = al((size_t)TR * row_bytes);
  int off = 0;
  s.hdr_off = -1;
  s.win_off = -1;
  s.win_rows = 0;
  if (win) {
    // window layout: the table, then rows of p_{k-1} for three tiles and a
    // margin (graphene: its own rows and the two neighbouring rows of cells)
    s.hdr_off = off;
    off += kRingWinHdr;
    s.win_rows = 3 * TR + 16;
    s.win_off = off;
    off += al((size_t)s.win_rows * row_bytes);
  }
  s.pin_off = off;
  off += tile;
  s.own_off = -1;
  if (!win) {
    s.own_off = off;
    off += tile;
  }
  s.acc_off = -1;
  if (mode == 1 || mode == 2) {
    s.acc_off = off;
    off += tile;
  }
  s.diag_off = off;
  off += al((size_t)(TR + 2) * cs);
  s.ip_off = off;
  off += al((size_t)(TR + 8) * 4);
  s.ix_off = off;
  off += al((size_t)cap * 4);
  s.hop_off = off;
  off += al((size_t)cap * cs);
  // MODE 2: the correlation reference's rows too, when they are whole 16-byte units
  s.ref_off = -1;
  const size_t ref_row = (size_t)ref_tpr * sizeof(Pack<R, V>);
  if (mode == 2 && ref_tpr > 0 && ref_row % 16 == 0) {
    s.ref_off = off;
    off += al((size_t)TR * ref_row);
  }
  s.stage_bytes = off;
  // kRingMinBlocks resident blocks per SM (228 KB of shared memory, 1 KB
  // reserved per block)
  const int budget = (228 * 1024) / kRingMinBlocks - 1024 - 256;
  const int S = std::min(kRingMaxStages, budget / off);
  if (S < 2) return RingShape{};
  s.rows = TR;
  s.stages = S;
  s.cap = cap;
  s.bar_off = S * off;
  s.smem_bytes = s.bar_off + 2 * S * 8;
  // MODE 2 and 3 reduce their partials in the stage buffers
  if ((size_t)s.bar_off < (size_t)items * V * 3 * sizeof(double)) return RingShape{};
  return s;
}

template <typename R, int V, int MODE, bool WIN>
int ring_blocks_per_sm(const tbpm_ctx* c, const RingShape& rs) {
  static std::atomic<bool> attr_set[64];
  const int dev = c->device;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    TBPM_CK(cudaFuncSetAttribute(cheb_ring_kernel<R, V, MODE, WIN>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    attr_set[dev] = true;
  }
  return resident_per_sm(cheb_ring_kernel<R, V, MODE, WIN>, kRingItems<R, V, MODE, WIN> + 32, (size_t)rs.smem_bytes);
}

// The window records for tiles of `rows` rows on the current Hamiltonian,
// built (asynchronously, on the context stream) when missing or stale; null
// during a graph capture that finds none (recorded in c->pair_requests).
const int* window_plan(tbpm_ctx* c, int rows) {
  WindowPlan* p = nullptr;
  for (auto& e : c->windows)
    if (e->rows == rows) p = e.get();
  if (p && p->ham_gen == c->ham.gen) return p->win.as<int>();
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  TBPM_CK(cudaStreamIsCapturing(c->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    PairRequest q{};
    q.rows = rows;
    q.kind = 1;
    c->pair_requests.push_back(q);
    return nullptr;
  }
  if (!p) {
    c->windows.push_back(std::make_unique<WindowPlan>());
    p = c->windows.back().get();
  }
  const Ham& h = c->ham;
  const int64_t nt = (h.n + rows - 1) / rows;
  p->rows = rows;
  p->ham_gen = h.gen;
  p->n_tiles = (int)nt;
  p->win.ensure((size_t)nt * kRingWinInts * 4);
  p->n_gather.ensure(16);
  TBPM_CK(cudaMemsetAsync(p->n_gather.p, 0, 4, c->stream));
  const int grid = (int)std::min<int64_t>(blocks_for(nt, 128), (int64_t)kSMs * 16);
  ring_window_kernel<<<grid, 128, 0, c->stream>>>(h.indptr.as<int32_t>(),
                                                   h.indices.as<int32_t>(), h.n, rows, (int)nt,
                                                   3 * rows + 16, p->win.as<int>(),
                                                   p->n_gather.as<unsigned>());
  TBPM_CK(cudaGetLastError());
  return p->win.as<int>();
}

#ifndef TBPM_F32V4_THREADS
#define TBPM_F32V4_THREADS 128
#endif
template <typename R, int V>
TermTiles term_tiles(tbpm_ctx* c, int64_t n_rows, int tpr, int ref_tpr = 0) {
  TermTiles tt;
  // measured on B200 (2048^2 graphene, 16 states): 128-thread blocks for FP64,
  // 256 for FP32
  const int th = sizeof(R) == 8 ? 128 : (V == 4 ? TBPM_F32V4_THREADS : 256);
  tt.t[0] = pick_tile(c, n_rows, tpr, cheb_term_kernel<R, V, 0>, 0, th);
  tt.t[1] = pick_tile(c, n_rows, tpr, cheb_term_kernel<R, V, 1>, 0, th);
  tt.t[2] = pick_tile(c, n_rows, tpr, cheb_term_kernel<R, V, 2>, V * 3 * sizeof(double), th);
  tt.t[3] = pick_tile(c, n_rows, tpr, cheb_term_kernel<R, V, 3>, V * 2 * sizeof(double), th);
  // row windows (term_kernel 4) where every mode's window layout fits and the
  // plan exists.  (Measured on B200, 2048^2 graphene, 16 states: 31.3 ms per
  // step against 28.2 ms with gathers; each row of p_{k-1} is staged by three
  // tiles, while the gathers of in-tile neighbours hit L1.)
  const bool want_win = c->opts.term_kernel == 4;
  bool win = false;
  if (want_win && c->opts.term_kernel != 1) {
    win = true;
    for (int m = 0; m < 3; ++m) win = win && ring_shape<R, V>(c, tpr, m, ref_tpr, true).stages >= 2;
    if (win) {
      tt.win = window_plan(c, ring_items<R, V>(0, true) / tpr);
      win = tt.win != nullptr;
    }
  }
  // the automatic choice keeps small problems (fewer than two ring tiles per
  // SM) on the grid-stride kernel, whose smaller tiles spread them over more
  // SMs (measured on B200: 100^2 graphene, one state, 256 steps, 16 ms against
  // 21 ms with the ring)
  const bool small = c->opts.term_kernel == 0 && tpr <= kRingConsumers &&
                     (n_rows + kRingConsumers / tpr - 1) / (kRingConsumers / tpr) <
                         2 * (int64_t)num_sms(c->device);
  if (c->opts.term_kernel != 1 && !small) {
    for (int m = 0; m < 4; ++m) {
      // mode 3 always gathers
      const RingShape rs = ring_shape<R, V>(c, tpr, m, ref_tpr, win && m < 3);
      if (rs.stages == 0) continue;
      const int per_sm = m == 3 ? ring_blocks_per_sm<R, V, 3, false>(c, rs)
                         : win ? (m == 0   ? ring_blocks_per_sm<R, V, 0, true>(c, rs)
                                : m == 1 ? ring_blocks_per_sm<R, V, 1, true>(c, rs)
                                         : ring_blocks_per_sm<R, V, 2, true>(c, rs))
                             : (m == 0   ? ring_blocks_per_sm<R, V, 0, false>(c, rs)
                                : m == 1 ? ring_blocks_per_sm<R, V, 1, false>(c, rs)
                                         : ring_blocks_per_sm<R, V, 2, false>(c, rs));
      const int64_t tiles = (n_rows + rs.rows - 1) / rs.rows;
      Tile t;
      t.threads = ring_items<R, V>(m, win && m < 3) + 32;
      t.rpp = rs.rows;
      t.rows_per_tile = rs.rows;
      t.grid = (int)std::max<int64_t>(
          1, std::min<int64_t>((int64_t)per_sm * num_sms(c->device), tiles));
      tt.t[m] = t;
      tt.ring[m] = true;
      tt.rs[m] = rs;
    }
  }
  return tt;
}

// Returns the grid of the launch (needed by the finalize of mode 2).
template <typename R, int V>
int launch_term(tbpm_ctx* c, const TermTiles& tt, const TermArgs<R, V>& a) {
  const int mode = a.partials ? (a.acc ? 2 : 3) : (a.c.nflush > 0 ? 1 : 0);
  const Tile& t = tt.t[mode];
  if (tt.ring[mode]) {
    RingArgs<R, V> ra;
    ra.t = a;
    ra.s = tt.rs[mode];
    ra.status = c->status.as<unsigned int>();
    ra.win = tt.win;
    ra.tiles = nullptr;
    ra.n_tiles = 0;
    const size_t smem = (size_t)ra.s.smem_bytes;
    if (mode == 3) {
      cheb_ring_kernel<R, V, 3, false><<<t.grid, t.threads, smem, c->stream>>>(ra);
    } else if (tt.win) {
      if (mode == 2)
        cheb_ring_kernel<R, V, 2, true><<<t.grid, t.threads, smem, c->stream>>>(ra);
      else if (mode == 1)
        cheb_ring_kernel<R, V, 1, true><<<t.grid, t.threads, smem, c->stream>>>(ra);
      else
        cheb_ring_kernel<R, V, 0, true><<<t.grid, t.threads, smem, c->stream>>>(ra);
    } else if (mode == 2) {
      cheb_ring_kernel<R, V, 2, false><<<t.grid, t.threads, smem, c->stream>>>(ra);
    } else if (mode == 1) {
      cheb_ring_kernel<R, V, 1, false><<<t.grid, t.threads, smem, c->stream>>>(ra);
    } else {
      cheb_ring_kernel<R, V, 0, false><<<t.grid, t.threads, smem, c->stream>>>(ra);
    }
  } else if (mode == 3) {
    const size_t smem = (size_t)t.threads * V * 2 * sizeof(double);
    cheb_term_kernel<R, V, 3><<<t.grid, t.threads, smem, c->stream>>>(a);
  } else if (mode == 2) {
    const size_t smem = (size_t)t.threads * V * 3 * sizeof(double);
    cheb_term_kernel<R, V, 2><<<t.grid, t.threads, smem, c->stream>>>(a);
  } else if (mode == 1) {
    cheb_term_kernel<R, V, 1><<<t.grid, t.threads, 0, c->stream>>>(a);
  } else {
    cheb_term_kernel<R, V, 0><<<t.grid, t.threads, 0, c->stream>>>(a);
  }
  TBPM_CK(cudaGetLastError());
  c->launches++;
  return t.grid;
}

// Tiles of packed realisations for the ring kernel's mode 4: none crosses a
// realisation.  rows == 0: the mode does not apply (no ring, or a row's packs
// are no power of two, so that a warp does not hold whole rows).
struct SegTiles {
  RingShape rs{};
  int grid = 0;
  int n_tiles = 0;
  int warps = 0;
  std::vector<int2> tiles;
  std::vector<int> first;  // first tile of every realisation, and the end
};

template <typename R, int V>
SegTiles seg_tiles(const tbpm_ctx* c, const std::vector<int64_t>& off, int tpr) {
  SegTiles t;
  if (c->opts.term_kernel == 1 || c->opts.rows_per_tile > 0 || tpr > 32 || (tpr & (tpr - 1)))
    return t;
  t.rs = ring_shape<R, V>(c, tpr, 4, 0);
  if (t.rs.stages == 0) return t;
  t.warps = ring_items<R, V>(4, false) / 32;
  for (size_t k = 0; k + 1 < off.size(); ++k) {
    t.first.push_back((int)t.tiles.size());
    for (int64_t r = off[k]; r < off[k + 1]; r += t.rs.rows)
      t.tiles.push_back(make_int2((int)r, (int)std::min<int64_t>(t.rs.rows, off[k + 1] - r)));
  }
  t.first.push_back((int)t.tiles.size());
  t.n_tiles = (int)t.tiles.size();
  const int per_sm = ring_blocks_per_sm<R, V, 4, false>(c, t.rs);
  t.grid = std::max(1, std::min(per_sm * num_sms(c->device), t.n_tiles));
  return t;
}

template <typename R, int V>
void launch_seg_term(tbpm_ctx* c, const SegTiles& t, const int2* tiles,
                     const TermArgs<R, V>& a) {
  RingArgs<R, V> ra;
  ra.t = a;
  ra.s = t.rs;
  ra.status = c->status.as<unsigned int>();
  ra.win = nullptr;
  ra.tiles = tiles;
  ra.n_tiles = t.n_tiles;
  cheb_ring_kernel<R, V, 4, false>
      <<<t.grid, t.warps * 32 + 32, (size_t)t.rs.smem_bytes, c->stream>>>(ra);
  TBPM_CK(cudaGetLastError());
  c->launches++;
}

// ---- paired terms (tbpm_pair_kernels.cuh) --------------------------------

template <typename R, int V>
int pair_blocks_per_sm(const tbpm_ctx* c, size_t smem) {
  static std::atomic<bool> attr_set[64];
  const int dev = c->device;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    TBPM_CK(cudaFuncSetAttribute(cheb_pair_kernel<R, V>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    attr_set[dev] = true;
  }
  return resident_per_sm(cheb_pair_kernel<R, V>, kRingThreads, smem);
}

#ifndef TBPM_PAIR_LAG
#define TBPM_PAIR_LAG 2
#endif
// L2 the rows between a tile's two terms may occupy: the second term finds
// p_k, p_{k-1} and the CSR slice of its tile in L2 while the tiles started
// in between (the margin plus the dependency lag) fit in this budget.
constexpr size_t kPairL2Window = 48ull << 20;

// Build the plan for tiles of `rows` rows on the device: dependency lists
// (pair_fwd/rev/merge_kernel), the item sequence (pair_seq_kernel), zeroed
// flags and counters.  usable: every list fits kPairDeps and, unless forced,
// at least 90% of the tiles have their last dependency within the L2 window.
void build_pair_plan(tbpm_ctx* c, PairPlan& p, const PairRequest& q) {
  const Ham& h = c->ham;
  cudaStream_t st = c->stream;
  const int TR = q.rows;
  const int64_t nt64 = (h.n + TR - 1) / TR;
  if (nt64 < 1 || nt64 > (1 << 29)) throw Error{TBPM_ERR_ARG, "too many row tiles to pair"};
  const int nt = (int)nt64;
  p.rows = TR;
  p.grid = q.grid;
  p.ham_gen = h.gen;
  p.forced = q.force;
  p.usable = false;
  p.n_tiles = nt;
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t b_list = al((size_t)nt * kPairDeps * 4), b_t = al((size_t)nt * 4),
               b_t1 = al((size_t)(nt + 1) * 4), b_off = al((size_t)(nt + 2) * 8);
  const size_t b_scan = al(scan_bytes(nt + 1));
  c->pair_tmp.ensure(2 * b_list + 3 * b_t + 2 * b_t1 + b_off + 256 + b_scan);
  char* w = c->pair_tmp.as<char>();
  int* fwd = reinterpret_cast<int*>(w);
  int* rev = reinterpret_cast<int*>(w += b_list);
  int* fcnt = reinterpret_cast<int*>(w += b_list);
  int* rcnt = reinterpret_cast<int*>(w += b_t);
  int* ready = reinterpret_cast<int*>(w += b_t);
  int* cnt_b = reinterpret_cast<int*>(w += b_t);
  int* g_cnt = reinterpret_cast<int*>(w += b_t1);
  int64_t* off_b = reinterpret_cast<int64_t*>(w += b_t1);
  unsigned* flags2 = reinterpret_cast<unsigned*>(w += b_off);  // [0] bad, [1] near
  p.seq.ensure((size_t)2 * nt * sizeof(int4));
  p.deps.ensure((size_t)nt * kPairDeps * 4);
  p.flags.ensure((size_t)nt * 4);
  p.sync.ensure(sizeof(PairSync));
  TBPM_CK(cudaMemsetAsync(rcnt, 0, (size_t)nt * 4, st));
  TBPM_CK(cudaMemsetAsync(cnt_b, 0, (size_t)(nt + 1) * 4, st));
  TBPM_CK(cudaMemsetAsync(g_cnt, 0, (size_t)(nt + 1) * 4, st));
  TBPM_CK(cudaMemsetAsync(flags2, 0, 8, st));
  TBPM_CK(cudaMemsetAsync(p.flags.p, 0, (size_t)nt * 4, st));
  TBPM_CK(cudaMemsetAsync(p.sync.p, 0, sizeof(PairSync), st));
  // a second term goes TBPM_PAIR_LAG items per block (plus the stages in
  // flight) after its last dependency, counted in first terms
  const int margin = q.grid * (q.stages + TBPM_PAIR_LAG) / 2;
  const long long window = (long long)(kPairL2Window / std::max<size_t>(3 * q.tile_bytes, 1));
  const int near = (int)std::max<long long>(0, std::min<long long>(window - margin, nt));
  const int gw = (int)std::min<int64_t>((nt + 7) / 8, (int64_t)kSMs * 16);
  const int gt = (int)std::min<int64_t>(blocks_for(nt, 256), (int64_t)kSMs * 16);
  pair_fwd_kernel<<<gw, 256, 0, st>>>(h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.n, TR,
                                      nt, fwd, fcnt, flags2);
  pair_rev_kernel<<<gt, 256, 0, st>>>(fwd, fcnt, nt, rev, rcnt, flags2);
  pair_merge_kernel<<<gt, 256, 0, st>>>(fwd, fcnt, rev, rcnt, nt, margin, near,
                                        p.deps.as<int>(), ready, cnt_b, flags2, flags2 + 1);
  TBPM_CK(cudaGetLastError());
  scan_counts(cnt_b, nt + 1, off_b, reinterpret_cast<int64_t*>(w + 256), st);
  pair_seq_kernel<<<gt, 256, 0, st>>>(h.indptr.as<int32_t>(), h.n, TR, nt, ready, off_b, g_cnt,
                                      p.seq.as<int4>());
  TBPM_CK(cudaGetLastError());
  unsigned host[2] = {0, 0};
  TBPM_CK(cudaMemcpyAsync(host, flags2, 8, cudaMemcpyDeviceToHost, st));
  TBPM_CK(cudaStreamSynchronize(st));
  p.usable = host[0] == 0 && (q.force || (double)host[1] >= 0.9 * (double)nt);
}

// The plan for tiles of q.rows rows on the current Hamiltonian, built when
// missing or stale; null when pairs do not apply.  During a graph capture a
// missing plan is recorded in c->pair_requests instead (ensure_graph builds it
// and captures again) and this call returns null.
PairPlan* pair_plan(tbpm_ctx* c, const PairRequest& q) {
  PairPlan* p = nullptr;
  for (auto& e : c->pairs)
    if (e->rows == q.rows) p = e.get();
  if (p && p->ham_gen == c->ham.gen && p->grid == q.grid && p->forced == q.force)
    return p->usable ? p : nullptr;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  TBPM_CK(cudaStreamIsCapturing(c->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) {
    c->pair_requests.push_back(q);
    return nullptr;
  }
  if (!p) {
    c->pairs.push_back(std::make_unique<PairPlan>());
    p = c->pairs.back().get();
  }
  build_pair_plan(c, *p, q);
  return p->usable ? p : nullptr;
}

template <typename R, int V>
void launch_pair(tbpm_ctx* c, const PairPlan& pp, const RingShape& rs, const TermArgs<R, V>& a0,
                 const TermArgs<R, V>& a1) {
  PairArgs<R, V> pa;
  pa.t[0] = a0;
  pa.t[1] = a1;
  pa.s = rs;
  pa.seq = pp.seq.as<int4>();
  pa.n_items = 2 * pp.n_tiles;
  pa.deps = pp.deps.as<int>();
  pa.flags = pp.flags.as<unsigned>();
  pa.sync = pp.sync.as<PairSync>();
  pa.status = c->status.as<unsigned int>();
  // cooperative: every block of the grid is resident at once (the items of a
  // block wait on items of other blocks)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)pp.grid);
  cfg.blockDim = dim3(kRingThreads);
  cfg.dynamicSmemBytes = (size_t)rs.smem_bytes + pair_extra_smem<R, V>();
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TBPM_CK(cudaLaunchKernelEx(&cfg, cheb_pair_kernel<R, V>, pa));
  c->launches++;
}

double matrix_bytes(const Ham& h) {
  const double s = h.prec == TBPM_PREC_FP64 ? 16 : 8;
  return (double)(h.n + 1) * 4 + (double)h.nnz * (4 + s) + (h.has_diag ? (double)h.n * s : 0.0);
}

// Allows `kernel` the shared memory of its next launch.  The limit belongs to the
// function, not to the launch, and other threads launch it for other contexts: it is
// set once per device, to the most the kernel can have.
template <class K>
void qe_smem_attr(K kernel, size_t bytes) {
  // (a kernel's static shared memory counts towards the default 48 KB too)
  if (bytes <= 40 * 1024) return;
  static std::mutex mutex;
  static std::vector<std::pair<const void*, int>> set;
  int dev = 0;
  TBPM_CK(cudaGetDevice(&dev));
  const std::pair<const void*, int> key(reinterpret_cast<const void*>(kernel), dev);
  std::lock_guard<std::mutex> lock(mutex);
  if (std::find(set.begin(), set.end(), key) != set.end()) return;
  cudaFuncAttributes fa;
  TBPM_CK(cudaFuncGetAttributes(&fa, kernel));
  TBPM_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               227 * 1024 - (int)fa.sharedSizeBytes));
  set.push_back(key);
}

// Longest wait on a grid barrier.
constexpr unsigned long long kGridWaitNs = 2000000000ull;

// Launch of a kernel with a grid barrier: every block is resident at once, so the
// barrier cannot wait on a block that has not started.
template <class K, class Args>
void launch_cooperative(tbpm_ctx* c, K kernel, int grid, int threads, size_t smem,
                        const Args& args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TBPM_CK(cudaLaunchKernelEx(&cfg, kernel, args));
}

// Matrix and two vectors up to which one launch beats a launch per term: the crossover,
// above what L2 holds (126 MB), since the lines that stay still save a launch (measured
// on B200, us per term of the DOS moments, one launch / ring):
//   FP64  131,072 orbitals x  8 states,  44 MB:  9.2 / 16.5
//         720,000           x  1,        83 MB:  9.5 / 17.3
//         320,000           x  5,        78 MB: 17.3 / 26.0
//        1,280,000          x  1,       148 MB: 27.2 / 35.5
//         720,000           x  4,       152 MB: 36.7 / 40.3
//         320,000           x 16,       191 MB: 57.6 / 55.7
//   FP32  720,000           x  4,        84 MB: 13.7 / 26.0
//         320,000           x 16,        99 MB: 25.6 / 33.1
// Moments reuse two vectors; windows of vectors and accumulators leave less of L2 to
// each, so their line lies lower.
constexpr double kPersistMoments = 160e6, kPersistOther = 90e6;
// Launch shape of cheb_persist_kernel, for problems of at most `most` bytes; grid == 0
// when it does not apply.
struct PersistShape {
  int grid = 0, threads = 0;
};

template <typename R, int V>
PersistShape persist_shape(const tbpm_ctx* c, int ld, double most = kPersistOther) {
  PersistShape s;
  const tbpm_options& o = c->opts;
  if (o.term_kernel != 0 || o.threads_per_block > 0 || o.rows_per_tile > 0) return s;
  const Ham& h = c->ham;
  const int tpr = ld / V;
  constexpr int TMAX = kPersistThreads<R, V>;
  if (tpr > TMAX) return s;
  const double bytes = matrix_bytes(h) + 2.0 * (double)h.n * ld * 2 * sizeof(R);
  const int sms = num_sms(c->device);
  if (bytes > most) return s;
  const int64_t per_sm = (h.n + sms - 1) / sms;
  const int rpp = (int)std::min<int64_t>(std::max<int64_t>(per_sm, (128 + tpr - 1) / tpr),
                                         TMAX / tpr);
  s.threads = rpp * tpr;
  s.grid = (int)std::min<int64_t>(sms, (h.n + rpp - 1) / rpp);
  return s;
}

// The arguments that every use of cheb_persist_kernel shares: terms k0..k1 with
// p_k = alpha H p_{k-1} - p_{k-2} (turn: times (-i)^k) on a ring of vectors.
template <typename R, int V>
PersistArgs<R, V> persist_args(const tbpm_ctx* c, double alpha, int k0, int k1, int ld,
                               const Pack<R, V>* p0, Pack<R, V>* const* ring, int slots,
                               bool turn) {
  const Ham& h = c->ham;
  PersistArgs<R, V> a{};
  a.indptr = h.indptr.as<int32_t>();
  a.indices = h.indices.as<int32_t>();
  a.hop = h.hop.as<typename Cx<R>::t>();
  a.diag = h.has_diag ? h.diag.as<typename Cx<R>::t>() : nullptr;
  a.n_rows = h.n;
  a.tpr = ld / V;
  a.p0 = p0;
  for (int q = 0; q < slots; ++q) a.ring[q] = ring[q];
  a.slots = slots;
  a.alpha = alpha;
  a.turn = turn ? 1 : 0;
  a.k0 = k0;
  a.k1 = k1;
  a.bar = c->ctr.as<unsigned int>() + 12;
  a.status = c->status.as<unsigned int>();
  a.absent = 0;
  a.wait_ns = kGridWaitNs;
  return a;
}

template <bool ACC, typename R, int V>
void launch_persist(tbpm_ctx* c, const PersistShape& s, const PersistArgs<R, V>& a) {
  const size_t smem = !ACC && a.k_dots >= a.k0
                          ? (size_t)kPersistBatch * s.threads * V * 2 * sizeof(double)
                          : 0;
  qe_smem_attr(cheb_persist_kernel<R, V, ACC>, smem);
  TBPM_CK(cudaMemsetAsync(a.bar, 0, sizeof(unsigned int), c->stream));
  launch_cooperative(c, cheb_persist_kernel<R, V, ACC>, s.grid, s.threads, smem, a);
  c->launches++;
}

// The moments' terms k0..k1 of a tiny problem by cheb_cluster_kernel: block partials
// to c->partials, the number of blocks returned (0: it does not apply).  The even
// vectors are in A, the odd ones in X; both are written back when `keep`.
template <typename R, int V>
int launch_cluster(tbpm_ctx* c, double alpha, int k0, int k1, bool keep, int ld, Pack<R, V>* A,
                   Pack<R, V>* X) {
  const tbpm_options& o = c->opts;
  if (o.term_kernel != 0 || o.threads_per_block > 0 || o.rows_per_tile > 0) return 0;
  const Ham& h = c->ham;
  const int tpr = ld / V;
  constexpr int TMAX = kClusterThreads<R, V>;
  if (h.n > (1 << 20) || tpr > TMAX) return 0;
  // at least two rows: the quotient's multiplier 2^32 / rows has 32 bits
  const int rows = std::max(2, (int)((h.n + kClusterBlocks - 1) / kClusterBlocks));
  const int rpp = std::max(std::min(rows, TMAX / tpr), (128 + tpr - 1) / tpr);
  const int threads = rpp * tpr;
  if (rows > kClusterItems * rpp) return 0;
  const size_t smem = 2 * (size_t)rows * tpr * sizeof(Pack<R, V>) +
                      (size_t)kPersistBatch * threads * V * 2 * sizeof(double);
  // (the products' slots start at a multiple of 8 bytes: packs are that or more)
  if (smem > 200 * 1024 || threads > TMAX) return 0;
  auto kernel = cheb_cluster_kernel<R, V>;
  TBPM_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  qe_smem_attr(kernel, smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterBlocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kClusterBlocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n_clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&n_clusters, kernel, &cfg) != cudaSuccess ||
      n_clusters < 1) {
    (void)cudaGetLastError();
    return 0;
  }
  ensure_partials(c, (size_t)(k1 - k0 + 1) * ld * 2 * kClusterBlocks);
  ClusterArgs<R, V> a;
  a.indptr = h.indptr.as<int32_t>();
  a.indices = h.indices.as<int32_t>();
  a.hop = h.hop.as<typename Cx<R>::t>();
  a.diag = h.has_diag ? h.diag.as<typename Cx<R>::t>() : nullptr;
  a.n_rows = (int)h.n;
  a.tpr = tpr;
  a.even = A;
  a.odd = X;
  a.alpha = alpha;
  a.k0 = k0;
  a.k1 = k1;
  a.keep = keep ? 1 : 0;
  a.rows = rows;
  a.magic = (unsigned)(((1ull << 32) + rows - 1) / rows);
  a.partials = c->partials.as<double>();
  TBPM_CK(cudaLaunchKernelEx(&cfg, kernel, a));
  c->launches++;
  return kClusterBlocks;
}

// Expansions of this many terms or more run in one launch on small problems (a
// time step's 16 to 20 stay single launches, which CUDA graphs replay).
constexpr int kPersistMinTerms = 64;

// Enqueue one expansion (one time step, or one Fermi operator) on the block A.
// When `partials_out` is set the last term also produces <ref|psi>, <psi|psi>
// block partials and a finalize launch stores them in out[*step].
template <typename R, int V>
void enqueue_expansion(tbpm_ctx* c, const Expansion& ex, int ld, Pack<R, V>* A, Pack<R, V>* X,
                       Pack<R, V>* Y, const Pack<R, V>* ref, int ref_ld, double* partials_out,
                       Counters k_ctr, Pack<R, V>* A_out = nullptr) {
  // A holds psi (p_0) on entry; the expansion result goes to A_out (default A).
  if (!A_out) A_out = A;
  const Ham& h = c->ham;
  const int tpr = ld / V;
  const TermTiles tt = term_tiles<R, V>(c, h.n, tpr, ref ? ref_ld / V : 0);
  const bool want = partials_out != nullptr;
  if (want) ensure_partials(c, (size_t)ld * 3 * tt.t[2].grid);
  int last_grid = 0;
  auto buf = [&](int k) { return (k & 1) ? X : Y; };
  const int n = ex.n_terms;
  int last_flush = -1;
  const size_t sv = 2 * sizeof(R);
  const double vec = (double)h.n * ld * sv;
  const double mat = (double)(h.n + 1) * 4 + (double)h.nnz * (4 + 2 * sizeof(R)) +
                     (h.has_diag ? (double)h.n * 2 * sizeof(R) : 0.0);
  std::vector<TermArgs<R, V>> terms(std::max(n, 1));
  std::vector<double> term_bytes(std::max(n, 1), 0.0);
  for (int k = 1; k < n; ++k) {
    TermArgs<R, V>& a = terms[k];
    a = TermArgs<R, V>{};
    a.indptr = h.indptr.as<int32_t>();
    a.indices = h.indices.as<int32_t>();
    a.hop = h.hop.as<typename Cx<R>::t>();
    a.diag = h.has_diag ? h.diag.as<typename Cx<R>::t>() : nullptr;
    a.n_rows = h.n;
    a.rows_per_tile = tt.t[0].rows_per_tile;
    a.tpr = tpr;
    a.c.neg_mask = ex.neg_mask;
    a.c.set_mask = ex.set_mask;
    double bytes = mat + vec;  // gather of p_{k-1}
    if (k == 1) {
      a.c.alpha_re = ex.alpha1_re;
      a.c.alpha_im = ex.alpha1_im;
      a.c.beta = 0.0;
      a.gather = A;
      a.pin = nullptr;
      a.pout = X;
      a.c.nflush = 0;
      bytes += vec;
    } else {
      a.c.alpha_re = ex.alpha_re;
      a.c.alpha_im = ex.alpha_im;
      a.c.beta = ex.beta;
      a.gather = buf(k - 1);
      a.pin = (k == 2) ? A : buf(k);
      a.pout = (k < n - 1) ? buf(k) : nullptr;
      bytes += vec * (a.pout ? 2 : 1);
      const int pending = k - last_flush;
      const bool flush = (k == 2) || pending == 3 || k == n - 1;
      if (flush) {
        a.c.nflush = pending;
        a.c.acc_init = (k == 2) ? 1 : 0;
        for (int s = 0; s < 2; ++s) {
          a.c.w[s][0] = pending >= 3 ? ex.w[s][k - 2] : 0.0;
          a.c.w[s][1] = pending >= 2 ? ex.w[s][k - 1] : 0.0;
          a.c.w[s][2] = ex.w[s][k];
        }
        a.acc = A_out;
        last_flush = k;
        bytes += vec * (a.c.acc_init ? 1 : 2);
      }
    }
    if (k == n - 1 && want) {
      a.ref = ref;
      a.ref_tpr = ref ? ref_ld / V : 0;
      a.partials = c->partials.as<double>();
      if (ref) bytes += (double)h.n * ref_ld * sv;
    }
    term_bytes[k] = bytes;
  }
  // With term_kernel 3, terms k, k+1 run as one paired launch where the plan
  // applies, except a last term with correlation partials and two flush terms
  // in a row (the second would stage accumulator rows the first wrote in the
  // same launch).  (Measured on B200, 2048^2 graphene: the paired launches
  // move the bytes of the model but take longer than two ring launches; the
  // automatic choice is the ring.)
  PairPlan* pp = nullptr;
  RingShape prs{};
  const int tk = c->opts.term_kernel;
  if (n >= 3 && tk == 3 && tt.ring[1])
    prs = ring_shape<R, V>(c, tpr, 1, 0, false, kRingConsumers);
  if (prs.stages >= 2) {
    const size_t smem = (size_t)prs.smem_bytes + pair_extra_smem<R, V>();
    if (smem <= 227 * 1024) {
      const int per_sm = pair_blocks_per_sm<R, V>(c, smem);
      const int64_t tiles = (h.n + prs.rows - 1) / prs.rows;
      PairRequest q;
      q.rows = prs.rows;
      q.grid = (int)std::max<int64_t>(
          1, std::min<int64_t>((int64_t)per_sm * num_sms(c->device), tiles));
      q.stages = prs.stages;
      q.tile_bytes = (size_t)prs.rows * tpr * sizeof(Pack<R, V>);
      q.force = true;
      pp = pair_plan(c, q);
    }
  }
  int k_first = 1;
  const PersistShape ps = n >= kPersistMinTerms && ex.neg_mask == 0
                              ? persist_shape<R, V>(c, ld)
                              : PersistShape{};
  const double alpha = ex.alpha_re != 0.0 ? ex.alpha_re : -ex.alpha_im;
  const bool turn = ex.alpha_re == 0.0;
  // the recurrences of the one-launch kernel: real alpha with beta = -1, or -i
  // times it with beta = 1, and half of alpha in the first term
  const bool fits = (turn ? ex.beta == 1.0 : ex.alpha_im == 0.0 && ex.beta == -1.0) &&
                    2 * ex.alpha1_re == ex.alpha_re && 2 * ex.alpha1_im == ex.alpha_im;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (ps.grid > 0) TBPM_CK(cudaStreamIsCapturing(c->stream, &capturing));
  if (ps.grid > 0 && fits && capturing == cudaStreamCaptureStatusNone) {
    // all but the last term, which also carries the products with `ref`
    std::vector<double> w(ex.w[0]);
    w.insert(w.end(), ex.w[1].begin(), ex.w[1].end());
    c->wts.ensure(w.size() * sizeof(double));
    TBPM_CK(cudaMemcpyAsync(c->wts.p, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice,
                            c->stream));
    Pack<R, V>* ring[2] = {Y, X};
    PersistArgs<R, V> a = persist_args<R, V>(c, alpha, 1, n - 2, ld, A, ring, 2, turn);
    a.acc = A_out;
    a.w = c->wts.as<double>();
    a.n_w = n;
    a.set_mask = ex.set_mask;
    launch_persist<true>(c, ps, a);
    for (int k = 1; k < n - 1; ++k) c->model_bytes += term_bytes[k];
    k_first = n - 1;
  }
  for (int k = k_first; k < n;) {
    const bool pair = pp && k + 1 < n && !(want && k + 1 == n - 1) &&
                      !(terms[k].c.nflush > 0 && terms[k + 1].c.nflush > 0);
    if (pair) {
      launch_pair<R, V>(c, *pp, prs, terms[k], terms[k + 1]);
      // the second term reads p_k, its own p_{k-1} rows and the matrix from L2
      c->model_bytes += term_bytes[k] + term_bytes[k + 1] - mat - 2 * vec;
      k += 2;
    } else {
      last_grid = launch_term<R, V>(c, tt, terms[k]);
      c->model_bytes += term_bytes[k];
      k += 1;
    }
  }
  if (want) launch_finalize(c, last_grid, ld * 3, k_ctr, partials_out);
}

template <typename R, int V>
void enqueue_corr(tbpm_ctx* c, const Pack<R, V>* x, const Pack<R, V>* ref, int ld, int ref_ld,
                  double* out, Counters k_ctr) {
  const int tpr = ld / V;
  const Tile t = pick_tile(c, c->ham.n, tpr, corr_kernel<R, V>, V * 3 * sizeof(double));
  ensure_partials(c, (size_t)ld * 3 * t.grid);
  const size_t smem = (size_t)t.threads * V * 3 * sizeof(double);
  corr_kernel<R, V><<<t.grid, t.threads, smem, c->stream>>>(
      x, ref, c->ham.n, t.rows_per_tile, tpr, ref ? ref_ld / V : 0, c->partials.as<double>());
  TBPM_CK(cudaGetLastError());
  c->launches++;
  launch_finalize(c, t.grid, ld * 3, k_ctr, out);
}

// Random states of the reference distribution into dst (row-interleaved, ld
// columns starting at column 0).  keys[col] = iseed * 49741.
template <typename R, int V>
void gen_states(tbpm_ctx* c, const StateKeys& keys, int ld, int kind, Pack<R, V>* dst) {
  if constexpr (sizeof(R) == 8 && V == 2) {
    // Same memory layout; generating with one value per thread keeps the
    // normalisation sums grouped as for every other FP64 caller (e.g.
    // tbpm_random_states), so the states do not depend on the vector width.
    gen_states<R, 1>(c, keys, ld, kind, reinterpret_cast<Pack<R, 1>*>(dst));
    return;
  }
  const int tpr = ld / V;
  const Tile t = pick_tile(c, c->ham.n, tpr, gen_state_kernel<R, V>, V * sizeof(double));
  ensure_partials(c, (size_t)ld * t.grid);
  c->small.ensure(sizeof(double) * kMaxCols * 2);
  reset_counters(c, 1);
  const size_t smem = (size_t)t.threads * V * sizeof(double);
  gen_state_kernel<R, V><<<t.grid, t.threads, smem, c->stream>>>(
      keys, kind, c->ham.n, t.rows_per_tile, tpr, 0, nullptr, 1, dst, c->partials.as<double>());
  TBPM_CK(cudaGetLastError());
  c->launches++;
  launch_finalize(c, t.grid, ld, counters(c, 1), c->small.as<double>());
  gen_state_kernel<R, V><<<t.grid, t.threads, 0, c->stream>>>(
      keys, kind, c->ham.n, t.rows_per_tile, tpr, 1, c->small.as<double>(), 1, dst, nullptr);
  TBPM_CK(cudaGetLastError());
  c->launches++;
}

// Host states (complex128 [ns][n]) -> columns [col0, col0+ns) of dst.
template <typename R>
void upload_states(tbpm_ctx* c, const double* host, int ns, int ld, int col0, void* dst) {
  const int64_t n = c->ham.n;
  const size_t bytes = (size_t)n * ns * 16;
  c->stage.ensure(bytes);
  TBPM_CK(cudaMemcpyAsync(c->stage.p, host, bytes, cudaMemcpyHostToDevice, c->stream));
  interleave_kernel<R><<<blocks_for(n * ns, 256), 256, 0, c->stream>>>(
      c->stage.as<double2>(), ns, n, ld, col0, reinterpret_cast<typename Cx<R>::t*>(dst));
  TBPM_CK(cudaGetLastError());
  c->launches++;
}

void check_status(tbpm_ctx* c);

// Columns [col0, col0+ns) of src -> host complex128 [ns][n] (synchronous).
template <typename R>
void download_states(tbpm_ctx* c, const void* src, int ns, int ld, int col0, double* host) {
  const int64_t n = c->ham.n;
  const size_t bytes = (size_t)n * ns * 16;
  c->stage.ensure(bytes);
  deinterleave_kernel<R><<<blocks_for(n * ns, 256), 256, 0, c->stream>>>(
      reinterpret_cast<const typename Cx<R>::t*>(src), ns, n, ld, col0, c->stage.as<double2>());
  TBPM_CK(cudaGetLastError());
  c->launches++;
  TBPM_CK(cudaMemcpyAsync(host, c->stage.p, bytes, cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
  check_status(c);
}

void ensure_vectors(tbpm_ctx* c, int ld, int ref_ld) {
  const size_t vb = (size_t)c->ham.n * ld * 2 * real_size(c->ham.prec);
  c->A.ensure(vb);
  c->X.ensure(vb);
  c->Y.ensure(vb);
  c->wf0.ensure((size_t)c->ham.n * std::max(ref_ld, 1) * 2 * real_size(c->ham.prec));
  c->ctr.ensure(16 * sizeof(int));
}

StateKeys make_keys(int seed, int first_sample, int n_states, int rank, int n_ran_samples) {
  // tbpm.f90:57 iseed = seed*(i_sample + rank*n_ran_samples); random.f90:52
  // iseed0 = iseed*49741 seeds the stream.
  StateKeys k{};
  for (int i = 0; i < n_states && i < kMaxCols; ++i) {
    const long long iseed = (long long)seed * ((long long)first_sample + i +
                                               (long long)rank * n_ran_samples);
    k.key[i] = iseed * 49741LL;
  }
  return k;
}

#ifndef TBPM_FP32_V4
#define TBPM_FP32_V4 1
#endif
int pick_V(int prec, int ld, int group, int requested = 0) {
  const bool can2 = ld % 2 == 0 && group % 2 == 0;
  // FP64: two complex128 per thread (256-bit accesses) unless one is requested
  // (measured on B200, 2048^2 graphene, 16 states: 33.7 vs 37.6 ms per step)
  if (prec == TBPM_PREC_FP64) return requested != 1 && can2 ? 2 : 1;
  if (requested == 1) return 1;
  // FP32: four complex64 per thread (256-bit accesses) when the widths allow
  const bool can4 = ld % 4 == 0 && group % 4 == 0;
  if (requested == 2 || TBPM_FP32_V4 == 0) return can2 ? 2 : 1;
  return can4 ? 4 : (can2 ? 2 : 1);
}

void require_ham(const tbpm_ctx* c, bool need_dxy) {
  if (c->ham.n <= 0) throw Error{TBPM_ERR_STATE, "no Hamiltonian uploaded"};
  if (c->ham.prec != c->opts.precision)
    throw Error{TBPM_ERR_STATE,
                "the uploaded Hamiltonian has a different precision than the context options; "
                "upload it again"};
  if (need_dxy && !c->ham.has_dxy)
    throw Error{TBPM_ERR_ARG, "dx/dy are required (current operator) but were not uploaded"};
}

int batch_size(const tbpm_ctx* c) {
  int b = c->opts.batch > 0 ? c->opts.batch : 16;
  return std::min(b, kMaxCols);
}

// ---- CUDA graph replay of a per-step program ---------------------------------

// Capture G steps of `step` as the context's CUDA graph unless the cached one
// has the same key and length.  The launches and modelled bytes of one step
// are recorded with the graph (every captured step enqueues the same work),
// so replays account for them without another capture.  The graph is also
// uploaded to the device here, so its first launch carries no set-up work.
template <class Fn>
void ensure_graph(tbpm_ctx* c, const std::vector<unsigned char>& key, Fn&& step, int G) {
  if (c->graph.exec && c->graph.key == key && c->graph.steps == G) return;
  c->graph.reset();
  const int64_t l0 = c->launches;
  const double b0 = c->model_bytes;
  cudaGraph_t g = nullptr;
  // a capture that asked for paired-term plans is discarded; the plans are
  // built (outside the capture) and the steps captured again
  for (int attempt = 0;; ++attempt) {
    c->pair_requests.clear();
    TBPM_CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeRelaxed));
    try {
      for (int i = 0; i < G; ++i) step();
    } catch (...) {
      cudaGraph_t gx = nullptr;
      cudaStreamEndCapture(c->stream, &gx);
      if (gx) cudaGraphDestroy(gx);
      c->launches = l0;
      c->model_bytes = b0;
      c->pair_requests.clear();
      throw;
    }
    TBPM_CK(cudaStreamEndCapture(c->stream, &g));
    if (c->pair_requests.empty() || attempt > 0) break;
    cudaGraphDestroy(g);
    g = nullptr;
    c->launches = l0;
    c->model_bytes = b0;
    const std::vector<PairRequest> reqs = c->pair_requests;
    c->pair_requests.clear();
    for (const PairRequest& q : reqs) {
      if (q.kind == 1)
        window_plan(c, q.rows);
      else
        pair_plan(c, q);
    }
  }
  c->pair_requests.clear();
  cudaError_t e = cudaGraphInstantiate(&c->graph.exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    c->graph.exec = nullptr;
    c->launches = l0;
    c->model_bytes = b0;
    throw_cuda(e, "cudaGraphInstantiate");
  }
  // capture does not execute: keep the per-step counts, undo the totals
  c->graph.l_step = (c->launches - l0) / G;
  c->graph.b_step = (c->model_bytes - b0) / G;
  c->launches = l0;
  c->model_bytes = b0;
  c->graph.key = key;
  c->graph.steps = G;
  TBPM_CK(cudaGraphUpload(c->graph.exec, c->stream));
}

int graph_length(const tbpm_ctx* c, int graph_steps) {
  return graph_steps > 0 ? graph_steps
                         : (c->opts.steps_per_graph > 0 ? c->opts.steps_per_graph : 16);
}

// Enqueue n_steps of `step`: replay a CUDA graph of G captured steps as often
// as it fits (G = graph_steps if positive, else opts.steps_per_graph), the
// remainder directly.
template <class Fn>
void run_steps(tbpm_ctx* c, int n_steps, const std::vector<unsigned char>& key, Fn&& step,
               int graph_steps = 0) {
  if (n_steps <= 0) return;
  const int G = graph_length(c, graph_steps);
  int done = 0;
  if (c->opts.use_graphs && n_steps >= G) {
    ensure_graph(c, key, step, G);
    while (n_steps - done >= G) {
      TBPM_CK(cudaGraphLaunch(c->graph.exec, c->stream));
      c->launches += c->graph.l_step * G;
      c->model_bytes += c->graph.b_step * G;
      done += G;
    }
  }
  for (; done < n_steps; ++done) step();
}

template <typename T>
void key_push(std::vector<unsigned char>& k, const T& v) {
  const unsigned char* p = reinterpret_cast<const unsigned char*>(&v);
  k.insert(k.end(), p, p + sizeof(T));
}

std::vector<unsigned char> plan_key(const tbpm_ctx* c, int kind, int ld, int V,
                                    const Expansion& ex) {
  std::vector<unsigned char> k;
  key_push(k, kind);
  key_push(k, ld);
  key_push(k, V);
  key_push(k, c->ham.prec);
  key_push(k, c->ham.n);
  key_push(k, c->ham.nnz);
  key_push(k, c->ham.has_diag);
  key_push(k, c->ham.has_dxy);
  key_push(k, c->ham.rescale);
  key_push(k, c->ham.gen);
  key_push(k, c->opts.term_kernel);
  const void* ptrs[] = {c->ham.indptr.p, c->ham.indices.p, c->ham.hop.p,  c->ham.dx.p,
                        c->ham.dy.p,     c->ham.diag.p,    c->A.p,        c->X.p,
                        c->Y.p,          c->wf0.p,         c->partials.p, c->out.p,
                        c->ctr.p};
  for (const void* p : ptrs) key_push(k, p);
  key_push(k, c->opts.threads_per_block);
  key_push(k, c->opts.rows_per_tile);
  key_push(k, ex.n_terms);
  key_push(k, ex.neg_mask);
  key_push(k, ex.set_mask);
  for (int s = 0; s < 2; ++s)
    for (double w : ex.w[s]) key_push(k, w);
  return k;
}

// ---- norm check (funcs.f90:175-192) -----------------------------------------

double effective_thr(const tbpm_ctx* c, double thr) {
  if (c->ham.prec == TBPM_PREC_FP32) return std::max(thr, c->opts.fp32_chk_thr);
  return thr;
}

// 0 when the norm passes check_norm (funcs.f90:175-192); TBPM_ERR_NAN when it
// is NaN or infinite; TBPM_ERR_NORM when it is off the reference by more than thr.
int norm_broken(double norm, double ref, double thr) {
  const double d = std::fabs(norm - ref);
  if (!std::isfinite(norm) || !std::isfinite(d)) return TBPM_ERR_NAN;
  return d > thr ? TBPM_ERR_NORM : 0;
}

void raise_norm(const char* where, int t, int code) {
  char buf[320];
  if (code == TBPM_ERR_NAN)
    std::snprintf(buf, sizeof buf,
                  "%s: the wave function norm is NaN or infinite at time step %d. Check the "
                  "initial states and the Hamiltonian for non-finite values.",
                  where, t);
  else
    std::snprintf(buf, sizeof buf,
                  "%s: wave function norm gets broken during propagation (time step %d). "
                  "Check the Hermitianity of the Hamiltonian, then try increasing 'rescale'.",
                  where, t);
  throw Error{code, buf};
}

// After a synchronisation: TBPM_ERR_TIMEOUT if a bounded wait of a kernel ran
// out since the last check (the word is cleared).
void check_status(tbpm_ctx* c) {
  unsigned int st = 0;
  TBPM_CK(cudaMemcpy(&st, c->status.p, sizeof st, cudaMemcpyDeviceToHost));
  if (st) {
    TBPM_CK(cudaMemset(c->status.p, 0, sizeof st));
    throw Error{TBPM_ERR_TIMEOUT,
                "a bounded device-side wait of a kernel ran out; the results of this call are "
                "invalid"};
  }
}

void read_out(tbpm_ctx* c, std::vector<double>& host, size_t n_doubles) {
  host.resize(n_doubles);
  TBPM_CK(cudaStreamSynchronize(c->stream));
  check_status(c);
  if (n_doubles)
    TBPM_CK(cudaMemcpy(host.data(), c->out.p, n_doubles * sizeof(double), cudaMemcpyDeviceToHost));
}

// ---- polynomial routes (tbpm_poly_kernels.cuh) --------------------------------

// Shortest run that takes a polynomial route.  The line is one of equality, not of speed:
// below it a call returns the bits of sessions (checkpointed runs) and of every term
// kernel, which tests and users rely on for short runs.  Moments are the faster side from
// 4 steps on (measured on B200, DOS, FP64, ms time-stepped / moments: 20,000 orbitals x 1
// state, 20 steps 2.2 / 0.34, 63 steps 4.7 / 0.47; 2M x 16, 20 steps 131 / 17, 63 steps
// 411 / 41).
constexpr int kPolyMinSteps = 64;
// Longest run (moments_pay and filters_pay judge the runs below it).
constexpr int kPolyMaxSteps = 65536;
// Largest deviation |P(x) - exp(-i tau x)| over the spectrum for which powers
// of P count as unitary (the default Bessel precision leaves 1e-14).
constexpr double kPolyUnitary = 1e-12;
// The recurrence runs on y = H/a with a this much above the Gershgorin bound: at
// the edge of [-1, 1] a rounding error grows by 1/sin(theta) per term, 7 here,
// against k at the very edge; the margin costs 1% more terms.
constexpr double kPolyMargin = 1.01;
// With a norm-check threshold below this the check would see the rounding of
// the time steps themselves; such a run is time-stepped.
constexpr double kPolyMinThr = 1e-11;
// Largest |tau| T |(H - H^+)/2| of a run.  Time stepping lets the states grow or decay
// with the anti-Hermitian part of H, moments take H as Hermitian: the product bounds what
// that changes in a curve (FP32: the states' own rounding is above it), and twice the
// product is the largest drift of the squared norm, of which the norm check has to see
// anything near its threshold.
constexpr double kPolySkew64 = 1e-11, kPolySkew32 = 1e-5;

struct PolyPlan {
  float alpha = 0;         // 2/a, a float, so that both precisions run the same y = H/a
  long double a = 0;       // 2/alpha
  double tau = 0;          // P(x) ~ exp(-i tau x)
  const double* bes = nullptr;
  int n_bes = 0;
};

const Spectrum& ham_spectrum(tbpm_ctx* c) {
  Spectrum& sp = c->spec;
  const Ham& h = c->ham;
  if (sp.gen == h.gen && h.gen != 0) return sp;
  c->poly.ensure(256);
  TBPM_CK(cudaMemsetAsync(c->poly.p, 0, 3 * sizeof(unsigned long long), c->stream));
  const int grid = (int)std::min<int64_t>(blocks_for(h.n, 256), (int64_t)num_sms(c->device) * 16);
  auto launch = [&](auto tag) {
    using R = decltype(tag);
    using C = typename Cx<R>::t;
    // values that are conjugates in FP64 stay so when rounded to FP32
    const double tol = sizeof(R) == 8 ? 1e-14 : 1.2e-7;
    const double rounding = sizeof(R) == 8 ? 4.5e-16 : 1.2e-7;  // two ulps, one
    ham_spectrum_kernel<R><<<grid, 256, 0, c->stream>>>(
        h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<C>(),
        h.has_diag ? h.diag.as<C>() : nullptr, h.n, tol, rounding,
        c->poly.as<unsigned long long>());
  };
  if (h.prec == TBPM_PREC_FP64)
    launch(double{});
  else
    launch(float{});
  TBPM_CK(cudaGetLastError());
  c->launches++;
  unsigned long long info[3];
  TBPM_CK(cudaMemcpyAsync(info, c->poly.p, sizeof info, cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
  std::memcpy(&sp.bound, &info[0], sizeof(double));
  std::memcpy(&sp.skew, &info[1], sizeof(double));
  sp.hermitian = info[2] == 0;
  sp.gen = h.gen;
  return sp;
}

// P(x) = sum_k w_k T_k(x), w_k = (2 - delta_k0) (-i)^k bes_k (propagation.f90:33-48)
void step_polynomial(const PolyPlan& pp, long double x, long double* re, long double* im) {
  long double t0 = 1.0L, t1 = x;
  *re = pp.bes[0];
  *im = 0.0L;
  for (int k = 1; k < pp.n_bes; ++k) {
    const long double w = 2.0L * pp.bes[k] * t1;
    switch (k & 3) {
      case 0: *re += w; break;
      case 1: *im -= w; break;
      case 2: *re -= w; break;
      default: *im += w; break;
    }
    const long double t2 = 2.0L * x * t1 - t0;
    t0 = t1;
    t1 = t2;
  }
}

// Whether powers of the step polynomial of `bes` on the resident Hamiltonian may
// be expanded over the whole run: H Hermitian, its spectrum bounded, and P
// unitary on it.  Everything else (a series for another operator, a rescale
// factor below the spectral radius, a non-Hermitian H) is time-stepped as before.
bool poly_route(tbpm_ctx* c, const double* bes, int n_bes, int n_timestep, int chk_step,
                double chk_thr, PolyPlan* pp) {
  if (n_timestep < kPolyMinSteps || n_timestep > kPolyMaxSteps) return false;
  const bool check = chk_step >= 2 && chk_step <= n_timestep;
  if (check && !(effective_thr(c, chk_thr) >= kPolyMinThr)) return false;
  const Spectrum& sp = ham_spectrum(c);
  if (!sp.hermitian || !(sp.bound < 4.0)) return false;
  const double want = 2.0 / std::max(sp.bound * kPolyMargin, 1.0 / 1024);
  float alpha = (float)want;
  if ((double)alpha > want) alpha = std::nextafter(alpha, 0.0f);
  pp->alpha = alpha;
  pp->a = 2.0L / (long double)alpha;
  pp->bes = bes;
  pp->n_bes = n_bes;
  double tau = 0.0;  // -i P'(0) / P(0), T_k'(0) = k sin(k pi / 2)
  for (int k = 1; k < n_bes; k += 2) tau += 2.0 * k * bes[k];
  pp->tau = tau;
  if (!(std::fabs(tau) < 1e3)) return false;
  double drift = c->ham.prec == TBPM_PREC_FP64 ? kPolySkew64 : kPolySkew32;
  if (check) drift = std::min(drift, 0.25 * effective_thr(c, chk_thr));
  if (!(std::fabs(tau) * n_timestep * sp.skew <= drift)) return false;
  for (int j = 0; j <= 64; ++j) {
    const long double x = pp->a * (long double)(j - 32) / 32.0L;
    long double re, im;
    step_polynomial(*pp, x, &re, &im);
    const long double dr = re - cosl(tau * x), di = im + sinl(tau * x);
    if (!(std::fabs((double)dr) <= kPolyUnitary && std::fabs((double)di) <= kPolyUnitary))
      return false;
  }
  return true;
}

// Seconds of one term on a block of ld columns: a launch and the bytes (measured on
// B200, about 6 TB/s; small problems 2.2 us in a CUDA graph or the one-launch kernel,
// 4.5 us as single launches, 8 us a time-stepped term of packed samples with its sums).
double term_seconds(const tbpm_ctx* c, int ld, double launch) {
  const double vec = (double)c->ham.n * ld * 2 * real_size(c->ham.prec);
  return launch + (matrix_bytes(c->ham) + 3.0 * vec) / 6e12;
}

// Whether moments are the faster side.  The terms grow with the run, the transforms
// from moments to curves with its square: M (M + T) cosines and powers per 8 columns
// take 7.5 ps each (measured: 2.2e6 nodes x 60,000 steps 38 s, where 200 orbitals are
// time-stepped in 9.7 s; 1.5e5 x 4096 0.26 s against 0.67 s).
bool moments_pay(const tbpm_ctx* c, const PolyPlan& pp, int T, int ld, int n_cols,
                 double step_launch) {
  const double M = std::fabs(pp.tau) * (double)pp.a * T;
  return 7.5e-12 * M * (M + T) * ((n_cols + 7) / 8) + 0.5 * M * term_seconds(c, ld, 2.2e-6) <
         (double)T * (pp.n_bes - 1) * term_seconds(c, ld, step_launch);
}

// Number of Chebyshev coefficients of exp(-i z y) on [-1, 1] above 1e-17, i.e.
// one more than the last k with |J_k(z)| > 1e-17 (Miller's downward recurrence
// normalised by J_0 + 2 sum J_2k = 1).
int bessel_degree(double z) {
  z = std::max(std::fabs(z), 1e-2);
  const int top = (int)(z + 30 * std::cbrt(z) + 40);
  std::vector<double> J(top + 2, 0.0);
  J[top] = 1e-300;
  for (int k = top; k > 0; --k) {
    J[k - 1] = 2.0 * k / z * J[k] - J[k + 1];
    if (std::fabs(J[k - 1]) > 1e200)
      for (int q = k - 1; q <= top; ++q) J[q] *= 1e-200;
  }
  double norm = J[0];
  for (int k = 2; k <= top; k += 2) norm += 2.0 * J[k];
  int last = 2;
  for (int k = 0; k <= top; ++k)
    if (std::fabs(J[k] / norm) > 1e-17) last = k;
  return last + 1;
}

// The powers' bases at the M Gauss-Chebyshev nodes of [-a, a], in extended
// precision: an error of a node's phase grows with the power.
std::vector<PolyNode> poly_nodes(const PolyPlan& pp, int M) {
  const long double pi = 3.14159265358979323846264338327950288L;
  std::vector<PolyNode> nodes(M);
  for (int j = 0; j < M; ++j) {
    long double re, im;
    step_polynomial(pp, pp.a * cosl(pi * (j + 0.5L) / M), &re, &im);
    const long double turns = atan2l(im, re) / (2.0L * pi);
    nodes[j].hi = (double)turns;
    nodes[j].lo = (double)(turns - (long double)nodes[j].hi);
    nodes[j].lnabs = (double)(0.5L * log1pl(re * re + im * im - 1.0L));
  }
  return nodes;
}

// w[k] with P(x)^m = sum_k w[k] (-i)^k T_k(x/a), k < bessel_degree: the even
// coefficients of a power of P are real, the odd ones imaginary, and the
// nodes j and M-1-j differ only in the sign of x, so half of them suffice.
std::vector<double> power_weights(const PolyPlan& pp, int m) {
  const int M = std::max(4, bessel_degree(pp.tau * (double)pp.a * m));
  const std::vector<PolyNode> nodes = poly_nodes(pp, M);
  const double pi = 3.14159265358979323846;
  std::vector<double> re(M), im(M), tab(4 * (size_t)M);
  for (int j = 0; j < M; ++j) {
    const long double t = (long double)m * ((long double)nodes[j].hi + nodes[j].lo);
    const long double f = 2 * 3.14159265358979323846264338327950288L * (t - roundl(t));
    const double g = std::exp(m * nodes[j].lnabs);
    re[j] = g * (double)cosl(f);
    im[j] = g * (double)sinl(f);
  }
  for (int q = 0; q < 4 * M; ++q) tab[q] = std::cos(pi * q / (2.0 * M));
  std::vector<double> w(M);
  for (int k = 0; k < M; ++k) {
    const std::vector<double>& f = (k & 1) ? im : re;
    double s = 0.0;
    for (int j = 0, q = k; j < M / 2; ++j) {  // q = k (2j + 1) mod 4M
      s += f[j] * tab[q];
      q += 2 * k;
      if (q >= 4 * M) q -= 4 * M;
    }
    s *= 2.0;
    if (M & 1) s += f[M / 2] * tab[(size_t)((int64_t)k * M % (4 * M))];
    s *= (k ? 2.0 : 1.0) / M;
    // (-i)^k: 1, -i, -1, i
    const int q = k & 3;
    w[k] = (q == 0 || q == 3) ? s : -s;
  }
  return w;
}

// m time steps as one expansion on y = H/a: p_k = (-i)^k T_k(y) psi.
Expansion power_expansion(const PolyPlan& pp, int m) {
  Expansion e;
  e.w[0] = power_weights(pp, m);
  e.w[1] = e.w[0];
  e.n_terms = (int)e.w[0].size();
  e.alpha1_im = -0.5 * (double)pp.alpha;
  e.alpha_im = -(double)pp.alpha;
  e.beta = 1.0;
  return e;
}

// Arguments of the term p_k = (2/a) H p_{k-1} - p_{k-2} (k >= 1), or, with
// `turn`, of the same vectors times (-i)^k.
template <typename R, int V>
TermArgs<R, V> poly_term(const tbpm_ctx* c, const PolyPlan& pp, int k, int tpr,
                         const Pack<R, V>* pm1, const Pack<R, V>* pm2, Pack<R, V>* pk,
                         bool turn = false) {
  const Ham& h = c->ham;
  TermArgs<R, V> a{};
  a.indptr = h.indptr.as<int32_t>();
  a.indices = h.indices.as<int32_t>();
  a.hop = h.hop.as<typename Cx<R>::t>();
  a.diag = h.has_diag ? h.diag.as<typename Cx<R>::t>() : nullptr;
  a.n_rows = h.n;
  a.tpr = tpr;
  a.gather = pm1;
  a.pin = k >= 2 ? pm2 : nullptr;
  a.pout = pk;
  const double alpha = (k == 1 ? 0.5 : 1.0) * (double)pp.alpha;
  if (turn)
    a.c.alpha_im = -alpha;
  else
    a.c.alpha_re = alpha;
  a.c.beta = k >= 2 ? (turn ? 1.0 : -1.0) : 0.0;
  return a;
}

// The same on two buffers, p_0 in A: p_k overwrites p_{k-2}.
template <typename R, int V>
TermArgs<R, V> poly_term2(const tbpm_ctx* c, const PolyPlan& pp, int k, int tpr, Pack<R, V>* A,
                          Pack<R, V>* X) {
  Pack<R, V>* dst = (k & 1) ? X : A;
  return poly_term<R, V>(c, pp, k, tpr, (k & 1) ? A : X, dst, dst);
}

// Terms whose block partials are reduced together: as many as fit 64 MB.
int moment_chunk(int terms, int64_t doubles_per_term) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(terms, (64ll << 20) / (doubles_per_term * 8)));
}

// Terms 1..K with the products of every term: sums[((k-1)*ld + col)*2 + q],
// q = 0: <p_k|p_k>, 1: Re <p_k|p_{k-1}>.  p_0 is in A, X is scratch.
template <typename R, int V>
void enqueue_moment_terms(tbpm_ctx* c, const PolyPlan& pp, int K, int ld, Pack<R, V>* A,
                          Pack<R, V>* X, double* sums) {
  const double bytes = matrix_bytes(c->ham) + 3.0 * (double)c->ham.n * ld * 2 * sizeof(R);
  int k0 = 1;
  // every route leaves p_k in A (k even) or X (k odd), where the next chunk takes it
  auto reduce = [&](int terms, int blocks) {
    const int64_t n_vals = (int64_t)terms * ld * 2;
    reduce_rows_kernel<<<(int)std::min<int64_t>(n_vals, 65535), 256, 0, c->stream>>>(
        c->partials.as<double>(), blocks, n_vals, sums + (int64_t)(k0 - 1) * ld * 2);
    TBPM_CK(cudaGetLastError());
    c->launches++;
    c->model_bytes += terms * bytes;
    k0 += terms;
  };
  while (k0 <= K) {
    const int m = moment_chunk(K - k0 + 1, (int64_t)ld * 2 * kClusterBlocks);
    const int blocks = launch_cluster<R, V>(c, pp.alpha, k0, k0 + m - 1, k0 + m <= K, ld, A, X);
    if (blocks == 0) break;
    reduce(m, blocks);
  }
  if (k0 > K) return;
  const PersistShape ps = persist_shape<R, V>(c, ld, kPersistMoments);
  while (ps.grid > 0 && k0 <= K) {
    const int m = moment_chunk(K - k0 + 1, (int64_t)ld * 2 * ps.grid);
    ensure_partials(c, (size_t)m * ld * 2 * ps.grid);
    Pack<R, V>* ring[2] = {A, X};
    PersistArgs<R, V> a =
        persist_args<R, V>(c, pp.alpha, k0, k0 + m - 1, ld, A, ring, 2, false);
    a.k_dots = K;
    a.partials = c->partials.as<double>();
    launch_persist<false>(c, ps, a);
    reduce(m, ps.grid);
  }
  if (k0 > K) return;
  const int tpr = ld / V;
  const TermTiles tt = term_tiles<R, V>(c, c->ham.n, tpr);
  const int grid = tt.t[3].grid;
  const int64_t per_term = (int64_t)ld * 2 * grid;
  ensure_partials(c, (size_t)moment_chunk(K, per_term) * per_term);
  while (k0 <= K) {
    const int m = moment_chunk(K - k0 + 1, per_term);
    for (int i = 0; i < m; ++i) {
      TermArgs<R, V> a = poly_term2<R, V>(c, pp, k0 + i, tpr, A, X);
      a.partials = c->partials.as<double>() + (int64_t)i * per_term;
      launch_term<R, V>(c, tt, a);
    }
    reduce(m, grid);
  }
}

// Moments of n_cols columns -> correlation functions and norms in c->out (the
// rows of moment_curve_kernel); mu, rho: n_cols*M doubles each.
void enqueue_moment_curves(tbpm_ctx* c, const PolyPlan& pp, int M, int T, int n_cols,
                           const double* sums, int64_t stride, const double* mu0,
                           int mu0_stride, double* mu, double* rho, PolyNode* nodes,
                           int chk_step, int t_ref = 1, bool have_nodes = false) {
  const int64_t total = (int64_t)n_cols * M;
  moment_gather_kernel<<<(int)std::min<int64_t>(blocks_for(total, 256), 4096), 256, 0,
                         c->stream>>>(sums, stride, mu0, mu0_stride, n_cols, M, mu);
  const unsigned cg = (unsigned)((n_cols + kMomentCols - 1) / kMomentCols);
  moment_density_kernel<<<dim3((unsigned)M, cg), 128, 0, c->stream>>>(mu, n_cols, M, rho);
  TBPM_CK(cudaGetLastError());
  if (!have_nodes) {  // the host evaluates them while the terms run
    const std::vector<PolyNode> host = poly_nodes(pp, M);
    TBPM_CK(cudaMemcpyAsync(nodes, host.data(), sizeof(PolyNode) * M, cudaMemcpyHostToDevice,
                            c->stream));
  }
  moment_curve_kernel<<<dim3((unsigned)(T + 3), cg), 128, 0, c->stream>>>(
      nodes, mu, rho, n_cols, M, T, t_ref, std::max(chk_step - 1, 1), c->out.as<double>());
  TBPM_CK(cudaGetLastError());
  c->launches += 3;
}

// check_norm on the curves of enqueue_moment_curves (host: c->out): the norms after t_chk
// and t_ref steps, and no moment above mu_0.  A recurrence of M/2 terms whose rounding
// errors grow by at most 7 each leaves a moment within 7 M rounding errors of mu_0.
void check_moments(const tbpm_ctx* c, const std::vector<double>& host, int T, int M, int n_cols,
                   int chk_step, double chk_thr, const char* who) {
  if (chk_step < 2 || chk_step > T) return;
  const double thr = effective_thr(c, chk_thr);
  const double eps = c->ham.prec == TBPM_PREC_FP64 ? 1.1e-16 : 6e-8;
  for (int v = 0; v < n_cols; ++v) {
    const double* ref = &host[((size_t)(T + 1) * n_cols + v) * 2];
    const double* chk = &host[((size_t)(T + 2) * n_cols + v) * 2];
    if (const int bad = norm_broken(chk[0], ref[0], thr)) raise_norm(who, chk_step, bad);
    if (!(chk[1] <= ref[0] * (1 + 1e-12 + 64.0 * M * eps)))
      raise_norm(who, chk_step, TBPM_ERR_NORM);
  }
}

// dos_batch by moments of the whole run: C(t) = <wf0|P(H)^t|wf0>.
template <typename R, int V>
void dos_moments(tbpm_ctx* c, const PolyPlan& pp, int ns, const StateKeys* keys,
                 const double* host_wf0, int n_timestep, int chk_step, double chk_thr, int n_avg,
                 double* corr, double* corr_per_state, int state_offset) {
  const int T = n_timestep;
  const int M = std::max(4, bessel_degree(pp.tau * (double)pp.a * T));
  const int K = M / 2;
  c->graph.reset();
  c->sess.active = false;
  const size_t vb = (size_t)c->ham.n * ns * 2 * sizeof(R);
  c->A.ensure(vb);
  c->X.ensure(vb);
  c->ctr.ensure(16 * sizeof(int));
  c->small.ensure(sizeof(double) * kMaxCols * 3);
  c->out.ensure((size_t)(T + 3) * ns * 2 * sizeof(double));
  const size_t n_sums = (size_t)K * ns * 2, n_mu = (size_t)ns * M;
  c->poly.ensure((n_sums + 2 * n_mu) * sizeof(double) + sizeof(PolyNode) * M);
  double* sums = c->poly.as<double>();
  double* mu = sums + n_sums;
  double* rho = mu + n_mu;
  PolyNode* nodes = reinterpret_cast<PolyNode*>(rho + n_mu);
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  if (keys)
    gen_states<R, V>(c, *keys, ns, c->opts.state_kind, A);
  else
    upload_states<R>(c, host_wf0, ns, ns, 0, A);
  reset_counters(c, 2);
  enqueue_corr<R, V>(c, A, nullptr, ns, 0, c->small.as<double>(), counters(c, 2));
  enqueue_moment_terms<R, V>(c, pp, K, ns, A, X, sums);
  enqueue_moment_curves(c, pp, M, T, ns, sums, (int64_t)ns * 2, c->small.as<double>() + 2, 3, mu,
                        rho, nodes, chk_step);
  std::vector<double> host;
  read_out(c, host, (size_t)(T + 3) * ns * 2);
  // as in dos_batch: after chk_step - 1 steps against after the first
  check_moments(c, host, T, M, ns, chk_step, chk_thr, "tbpm_dos");
  for (int b = 0; b < ns; ++b)
    for (int t = 0; t <= T; ++t) {
      const double* v = &host[((size_t)t * ns + b) * 2];
      corr[2 * t] += v[0] / n_avg;
      corr[2 * t + 1] += v[1] / n_avg;
      if (corr_per_state) {
        double* o = corr_per_state + 2 * ((size_t)(state_offset + b) * (T + 1) + t);
        o[0] = v[0];
        o[1] = v[1];
      }
    }
}

// ---- DOS ----------------------------------------------------------------------

template <typename R, int V>
void dos_session_begin(tbpm_ctx* c, const Expansion& ex, int ns, const StateKeys* keys,
                       const double* host_wf0, int rows_cap) {
  c->graph.reset();
  ensure_vectors(c, ns, ns);
  c->out.ensure((size_t)rows_cap * ns * 3 * sizeof(double));
  auto* A = c->A.as<Pack<R, V>>();
  auto* W = c->wf0.as<Pack<R, V>>();
  if (keys)
    gen_states<R, V>(c, *keys, ns, c->opts.state_kind, W);
  else
    upload_states<R>(c, host_wf0, ns, ns, 0, W);
  TBPM_CK(cudaMemcpyAsync(A, W, (size_t)c->ham.n * ns * 2 * sizeof(R), cudaMemcpyDeviceToDevice,
                          c->stream));
  reset_counters(c, 0);
  enqueue_corr<R, V>(c, A, W, ns, ns, c->out.as<double>(), counters(c, 0));
  c->sess.active = true;
  c->sess.kind = 1;
  c->sess.ld = ns;
  c->sess.V = V;
  c->sess.rows_cap = rows_cap;
  c->sess.rows_enqueued = 1;
  c->sess.ex = ex;
}

// Resume a DOS session from exported state: initial states wf0, current states
// psi (complex128 [ns][n]) and the n_done recorded rows (corr complex, norms).
// n_done == 0 starts a fresh session from the given states (row 0 recorded).
template <typename R, int V>
void dos_session_resume(tbpm_ctx* c, const Expansion& ex, int ns, const double* wf0,
                        const double* psi, const double* corr, const double* norms, int n_done,
                        int rows_cap) {
  if (n_done == 0) {
    dos_session_begin<R, V>(c, ex, ns, nullptr, wf0, rows_cap);
    return;
  }
  c->graph.reset();
  ensure_vectors(c, ns, ns);
  c->out.ensure((size_t)rows_cap * ns * 3 * sizeof(double));
  upload_states<R>(c, wf0, ns, ns, 0, c->wf0.p);
  upload_states<R>(c, psi, ns, ns, 0, c->A.p);
  std::vector<double> rows((size_t)n_done * ns * 3);
  for (int r = 0; r < n_done; ++r)
    for (int b = 0; b < ns; ++b) {
      double* v = &rows[((size_t)r * ns + b) * 3];
      v[0] = corr[2 * ((size_t)r * ns + b)];
      v[1] = corr[2 * ((size_t)r * ns + b) + 1];
      v[2] = norms[(size_t)r * ns + b];
    }
  TBPM_CK(cudaMemcpyAsync(c->out.p, rows.data(), rows.size() * sizeof(double),
                          cudaMemcpyHostToDevice, c->stream));
  // device step counter = next row to record; completion counter = 0
  const int ctr[2] = {n_done, 0};
  TBPM_CK(cudaMemcpyAsync(counters(c, 0).step, ctr, sizeof(ctr), cudaMemcpyHostToDevice,
                          c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));  // host staging buffers go out of scope
  c->sess.active = true;
  c->sess.kind = 1;
  c->sess.ld = ns;
  c->sess.V = V;
  c->sess.rows_cap = rows_cap;
  c->sess.rows_enqueued = n_done;
  c->sess.ex = ex;
}

// Enqueue n_steps DOS time steps of the active session; with n_steps == 0 and
// graphs enabled, only capture (and upload) the session's step graph when
// the session has room for at least one graph's worth of steps.
template <typename R, int V>
void dos_session_advance(tbpm_ctx* c, int n_steps) {
  Session& s = c->sess;
  if (!s.active || s.kind != 1) throw Error{TBPM_ERR_STATE, "no DOS session active"};
  if (s.rows_enqueued + n_steps > s.rows_cap)
    throw Error{TBPM_ERR_ARG, "session capacity (n_timestep) exceeded"};
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  auto* Y = c->Y.as<Pack<R, V>>();
  auto* W = c->wf0.as<Pack<R, V>>();
  const int ld = s.ld;
  const Expansion& ex = s.ex;
  auto step = [&]() {
    enqueue_expansion<R, V>(c, ex, ld, A, X, Y, W, ld, c->out.as<double>(), counters(c, 0));
  };
  if (n_steps == 0) {
    const int G = graph_length(c, 0);
    if (c->opts.use_graphs && s.rows_cap - s.rows_enqueued >= G)
      ensure_graph(c, plan_key(c, 1, ld, V, ex), step, G);
    return;
  }
  run_steps(c, n_steps, plan_key(c, 1, ld, V, ex), step);
  s.rows_enqueued += n_steps;
}

// Run one batch of DOS states and accumulate into corr (complex, n_t+1),
// optionally storing per-state correlations.
template <typename R, int V>
void dos_batch(tbpm_ctx* c, const Expansion& ex, int ns, const StateKeys* keys,
               const double* host_wf0, int n_timestep, int chk_step, double chk_thr,
               int n_avg, double* corr, double* corr_per_state, int state_offset,
               int total_states) {
  dos_session_begin<R, V>(c, ex, ns, keys, host_wf0, n_timestep + 1);
  const double thr = effective_thr(c, chk_thr);
  std::vector<double> host;
  // tbpm.f90:71-79: the norm of wf_t(t-1) is checked at t == chk_step against
  // norm_ref = <wf_1|wf_1>; rows hold the state after `row` steps.
  const bool check = chk_step >= 2 && chk_step <= n_timestep;
  int done = 0;
  if (check) {
    dos_session_advance<R, V>(c, chk_step - 1);
    done = chk_step - 1;
    read_out(c, host, (size_t)(done + 1) * ns * 3);
    for (int b = 0; b < ns; ++b) {
      const double ref = host[((size_t)1 * ns + b) * 3 + 2];
      const double nv = host[((size_t)(chk_step - 1) * ns + b) * 3 + 2];
      if (const int bad_ = norm_broken(nv, ref, thr))
        raise_norm("tbpm_dos", chk_step, bad_);
    }
  }
  dos_session_advance<R, V>(c, n_timestep - done);
  read_out(c, host, (size_t)(n_timestep + 1) * ns * 3);
  c->sess.active = false;
  // tbpm.f90:58-86: corr(t) += corrval / n_ran_samples, sample by sample
  for (int b = 0; b < ns; ++b) {
    for (int t = 0; t <= n_timestep; ++t) {
      const double re = host[((size_t)t * ns + b) * 3 + 0];
      const double im = host[((size_t)t * ns + b) * 3 + 1];
      corr[2 * t] += re / n_avg;
      corr[2 * t + 1] += im / n_avg;
      if (corr_per_state) {
        double* o = corr_per_state + 2 * ((size_t)(state_offset + b) * (n_timestep + 1) + t);
        o[0] = re;
        o[1] = im;
      }
    }
  }
  (void)total_states;
}


// ---- batches of uneven realisations (block-diagonal packing) -----------------

// One DOS propagation of n_seg packed realisations x ns states each.  corr:
// complex [n_seg][n_timestep+1], averaged over the ns states of a realisation;
// corr_per_state (optional): complex [n_seg][ns][n_timestep+1].  The whole
// propagation is captured as a single CUDA graph and launched once.  V only
// changes how term-kernel threads map onto the columns of a row; the
// row-interleaved layout read by the segment kernels is the same for every V.
template <typename R, int V>
void dos_segmented_run(tbpm_ctx* c, const Expansion& ex, const std::vector<int64_t>& off,
                       int ns, int seed, int n_timestep, int chk_step, double chk_thr,
                       double* corr, double* corr_per_state) {
  using C = typename Cx<R>::t;
  const int n_seg = (int)off.size() - 1;
  const int64_t n = c->ham.n;
  int64_t max_len = 0;
  for (int k = 0; k < n_seg; ++k) max_len = std::max<int64_t>(max_len, off[k + 1] - off[k]);
  const int64_t rows_per_chunk = 4096;
  const int n_chunks = (int)std::max<int64_t>(1, (max_len + rows_per_chunk - 1) / rows_per_chunk);
  const int rpp = std::max(1, 256 / ns);
  const int threads = rpp * ns;
  const int n_values = n_seg * ns * 3;
  c->graph.reset();
  c->sess.active = false;
  ensure_vectors(c, ns, ns);
  c->seg.ensure(sizeof(int64_t) * off.size());
  TBPM_CK(cudaMemcpyAsync(c->seg.p, off.data(), sizeof(int64_t) * off.size(),
                          cudaMemcpyHostToDevice, c->stream));
  ensure_partials(c, (size_t)n_values * n_chunks);
  c->small.ensure(sizeof(double) * std::max<size_t>((size_t)n_seg * ns, kMaxCols * 2));
  c->out.ensure((size_t)(n_timestep + 1) * n_values * sizeof(double));
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  auto* Y = c->Y.as<Pack<R, V>>();
  auto* W = c->wf0.as<Pack<R, V>>();
  const dim3 grid(n_chunks, n_seg);
  // random states, normalised per realisation
  reset_counters(c, 1);
  seg_state_kernel<R><<<grid, threads, 0, c->stream>>>(
      c->seg.as<int64_t>(), ns, (long long)seed, c->opts.state_kind, rows_per_chunk, 0, nullptr,
      nullptr, c->partials.as<double>());
  TBPM_CK(cudaGetLastError());
  launch_finalize(c, n_chunks, n_seg * ns, counters(c, 1), c->small.as<double>());
  seg_state_kernel<R><<<grid, threads, 0, c->stream>>>(
      c->seg.as<int64_t>(), ns, (long long)seed, c->opts.state_kind, rows_per_chunk, 1,
      c->small.as<double>(), reinterpret_cast<C*>(W), nullptr);
  TBPM_CK(cudaGetLastError());
  c->launches += 2;
  TBPM_CK(cudaMemcpyAsync(A, W, (size_t)n * ns * sizeof(C), cudaMemcpyDeviceToDevice, c->stream));
  reset_counters(c, 0);
  auto seg_corr = [&]() {
    seg_corr_kernel<R><<<grid, threads, 0, c->stream>>>(
        c->seg.as<int64_t>(), ns, rows_per_chunk, reinterpret_cast<const C*>(A),
        reinterpret_cast<const C*>(W), c->partials.as<double>());
    TBPM_CK(cudaGetLastError());
    c->launches++;
    c->model_bytes += 2.0 * (double)n * ns * sizeof(C);
    launch_finalize(c, n_chunks, n_values, counters(c, 0), c->out.as<double>());
  };
  seg_corr();  // row 0: <wf0|wf0>
  auto step = [&]() {
    enqueue_expansion<R, V>(c, ex, ns, A, X, Y, nullptr, 0, nullptr, Counters{});
    seg_corr();
  };
  std::vector<unsigned char> key = plan_key(c, 4, ns, V, ex);
  key_push(key, n_seg);
  const double thr = effective_thr(c, chk_thr);
  std::vector<double> host;
  int done = 0;
  const bool check = chk_step >= 2 && chk_step <= n_timestep;
  if (check) {
    run_steps(c, chk_step - 1, key, step, chk_step - 1);
    done = chk_step - 1;
    read_out(c, host, (size_t)(done + 1) * n_values);
    for (int v = 0; v < n_seg * ns; ++v) {
      const double ref = host[((size_t)1 * n_seg * ns + v) * 3 + 2];
      const double nv = host[((size_t)done * n_seg * ns + v) * 3 + 2];
      if (const int bad_ = norm_broken(nv, ref, thr))
        raise_norm("tbpm_dos_segmented", chk_step, bad_);
    }
    c->graph.reset();
  }
  run_steps(c, n_timestep - done, key, step, n_timestep - done);
  read_out(c, host, (size_t)(n_timestep + 1) * n_values);
  c->graph.reset();
  for (int k = 0; k < n_seg; ++k)
    for (int t = 0; t <= n_timestep; ++t) {
      double re = 0, im = 0;
      for (int b = 0; b < ns; ++b) {
        const double* v = &host[(((size_t)t * n_seg + k) * ns + b) * 3];
        re += v[0] / ns;
        im += v[1] / ns;
        if (corr_per_state) {
          double* o = corr_per_state + 2 * (((size_t)k * ns + b) * (n_timestep + 1) + t);
          o[0] = v[0];
          o[1] = v[1];
        }
      }
      corr[2 * ((size_t)k * (n_timestep + 1) + t)] = re;
      corr[2 * ((size_t)k * (n_timestep + 1) + t) + 1] = im;
    }
}

// Whether no entry of the resident Hamiltonian couples two realisations.  Moments
// need that: <p_k|p_k> over a part of the rows is a moment of that part's states only
// when H maps the part onto itself.
bool segments_closed(tbpm_ctx* c, const std::vector<int64_t>& off) {
  const int n_seg = (int)off.size() - 1;
  int64_t max_len = 0;
  for (int k = 0; k < n_seg; ++k) max_len = std::max<int64_t>(max_len, off[k + 1] - off[k]);
  c->seg.ensure(sizeof(int64_t) * off.size());
  c->poly.ensure(256);
  TBPM_CK(cudaMemcpyAsync(c->seg.p, off.data(), sizeof(int64_t) * off.size(),
                          cudaMemcpyHostToDevice, c->stream));
  TBPM_CK(cudaMemsetAsync(c->poly.p, 0, sizeof(unsigned int), c->stream));
  const unsigned chunks =
      (unsigned)std::min<int64_t>(blocks_for(std::max<int64_t>(max_len, 1), 256), 64);
  seg_closed_kernel<<<dim3(chunks, (unsigned)n_seg), 256, 0, c->stream>>>(
      c->seg.as<int64_t>(), c->ham.indptr.as<int32_t>(), c->ham.indices.as<int32_t>(),
      c->poly.as<unsigned int>());
  TBPM_CK(cudaGetLastError());
  c->launches++;
  unsigned int coupled = 0;
  TBPM_CK(cudaMemcpyAsync(&coupled, c->poly.p, sizeof coupled, cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
  return coupled == 0;
}

// dos_segmented_run by moments: the terms of all realisations run as one block
// row-interleaved state block, seg_dots_kernel forms the two products of every
// term per (segment, state).
template <typename R, int V>
bool dos_segmented_moments(tbpm_ctx* c, const PolyPlan& pp, const std::vector<int64_t>& off,
                           int ns, int seed, int n_timestep, int chk_step, double chk_thr,
                           double* corr, double* corr_per_state) {
  using C = typename Cx<R>::t;
  const int n_seg = (int)off.size() - 1;
  const int n_cols = n_seg * ns;
  const int T = n_timestep;
  const int64_t n = c->ham.n;
  const int M = std::max(4, bessel_degree(pp.tau * (double)pp.a * T));
  const int K = M / 2;
  // a batch of very many tiny realisations would need more moments than states
  if ((n_cols + kMomentCols - 1) / kMomentCols > 65535 || (double)n_cols * M * 32 > 4e9)
    return false;
  int64_t max_len = 0;
  for (int k = 0; k < n_seg; ++k) max_len = std::max<int64_t>(max_len, off[k + 1] - off[k]);
  // the states' chunks set the order of their normalisation sums, as in
  // dos_segmented_run; the products take about 16 blocks per SM
  const int64_t rows_per_chunk = 4096;
  const int n_chunks = (int)std::max<int64_t>(1, (max_len + rows_per_chunk - 1) / rows_per_chunk);
  const int rpp = std::max(1, 256 / ns);
  const int threads = rpp * ns;
  const int64_t dot_rows = std::max<int64_t>(4 * rpp, n / (16 * (int64_t)num_sms(c->device)) + 1);
  const int dot_chunks = (int)std::max<int64_t>(1, (max_len + dot_rows - 1) / dot_rows);
  c->graph.reset();
  c->sess.active = false;
  const size_t vb = (size_t)n * ns * sizeof(C);
  c->A.ensure(vb);
  c->X.ensure(vb);
  c->ctr.ensure(16 * sizeof(int));
  c->seg.ensure(sizeof(int64_t) * off.size());
  TBPM_CK(cudaMemcpyAsync(c->seg.p, off.data(), sizeof(int64_t) * off.size(),
                          cudaMemcpyHostToDevice, c->stream));
  const int tpr = ns / V;
  const SegTiles st = seg_tiles<R, V>(c, off, tpr);
  const int64_t seg_stride = (int64_t)st.n_tiles * st.warps * ns * 2;
  const int64_t per_term = std::max<int64_t>((int64_t)n_cols * 2 * dot_chunks, seg_stride);
  // (a chunk's terms are the y axis of seg_tile_reduce_kernel's grid: 65,535 at most)
  const int chunk = (int)std::max<int64_t>(
      1, std::min<int64_t>({(int64_t)K + 1, (64ll << 20) / (per_term * 8), (int64_t)65535}));
  ensure_partials(c, std::max<size_t>((size_t)chunk * per_term, (size_t)n_cols * n_chunks));
  c->small.ensure(sizeof(double) * std::max<size_t>((size_t)n_cols, kMaxCols * 2));
  c->out.ensure((size_t)(T + 3) * n_cols * 2 * sizeof(double));
  const size_t n_sums = (size_t)(K + 1) * n_cols * 2, n_mu = (size_t)n_cols * M;
  c->poly.ensure((n_sums + 2 * n_mu) * sizeof(double) + sizeof(PolyNode) * M);
  double* sums = c->poly.as<double>();
  double* mu = sums + n_sums;
  double* rho = mu + n_mu;
  PolyNode* nodes = reinterpret_cast<PolyNode*>(rho + n_mu);
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  const dim3 grid(n_chunks, n_seg);
  reset_counters(c, 1);
  seg_state_kernel<R><<<grid, threads, 0, c->stream>>>(
      c->seg.as<int64_t>(), ns, (long long)seed, c->opts.state_kind, rows_per_chunk, 0, nullptr,
      nullptr, c->partials.as<double>());
  TBPM_CK(cudaGetLastError());
  launch_finalize(c, n_chunks, n_cols, counters(c, 1), c->small.as<double>());
  seg_state_kernel<R><<<grid, threads, 0, c->stream>>>(
      c->seg.as<int64_t>(), ns, (long long)seed, c->opts.state_kind, rows_per_chunk, 1,
      c->small.as<double>(), reinterpret_cast<C*>(A), nullptr);
  TBPM_CK(cudaGetLastError());
  c->launches += 2;
  const TermTiles tt = term_tiles<R, V>(c, n, tpr);
  const double bytes = matrix_bytes(c->ham) + (st.grid > 0 ? 3.0 : 5.0) * (double)vb;
  auto dots = [&](const Pack<R, V>* x, const Pack<R, V>* y, double* out) {
    seg_dots_kernel<R><<<dim3(dot_chunks, n_seg), threads, 0, c->stream>>>(
        c->seg.as<int64_t>(), ns, dot_rows, reinterpret_cast<const C*>(x),
        reinterpret_cast<const C*>(y), out);
    TBPM_CK(cudaGetLastError());
    c->launches++;
  };
  auto reduce_dots = [&](int k, int count) {  // rows k .. k + count - 1 of the sums
    const int64_t n_vals = (int64_t)count * n_cols * 2;
    reduce_rows_kernel<<<(int)std::min<int64_t>(n_vals, 65535), 256, 0, c->stream>>>(
        c->partials.as<double>(), dot_chunks, n_vals, sums + (int64_t)k * n_cols * 2);
    TBPM_CK(cudaGetLastError());
    c->launches++;
  };
  int k0 = 0;
  if (st.grid > 0) {
    // the products come out of the terms (20 samples, 1.4M rows, 4 FP64 states, 128
    // steps: 32.8 ms with a separate pass over both vectors per term, 50 us and 39 us;
    // 27.6 ms with them here)
    ScratchScope scope(c->scratch);
    TempMem tiles(c->scratch), first(c->scratch);
    tiles.ensure(st.tiles.size() * sizeof(int2));
    first.ensure(st.first.size() * sizeof(int));
    TBPM_CK(cudaMemcpyAsync(tiles.p, st.tiles.data(), st.tiles.size() * sizeof(int2),
                            cudaMemcpyHostToDevice, c->stream));
    TBPM_CK(cudaMemcpyAsync(first.p, st.first.data(), st.first.size() * sizeof(int),
                            cudaMemcpyHostToDevice, c->stream));
    dots(A, A, c->partials.as<double>());
    reduce_dots(0, 1);
    for (k0 = 1; k0 <= K; k0 += chunk) {
      const int m = std::min(chunk, K + 1 - k0);
      for (int i = 0; i < m; ++i) {
        TermArgs<R, V> a = poly_term2<R, V>(c, pp, k0 + i, tpr, A, X);
        a.partials = c->partials.as<double>() + (int64_t)i * seg_stride;
        launch_seg_term<R, V>(c, st, tiles.as<int2>(), a);
        c->model_bytes += bytes;
      }
      seg_tile_reduce_kernel<<<dim3((unsigned)n_seg, (unsigned)m), 256, 0, c->stream>>>(
          c->partials.as<double>(), seg_stride, first.as<int>(), st.warps, ns * 2,
          sums + (int64_t)k0 * n_cols * 2);
      TBPM_CK(cudaGetLastError());
      c->launches++;
    }
    TBPM_CK(cudaStreamSynchronize(c->stream));  // the tables go out of scope
  }
  for (; k0 <= K; k0 += chunk) {  // row 0 of the sums: <p_0|p_0>
    const int m = std::min(chunk, K + 1 - k0);
    for (int i = 0; i < m; ++i) {
      const int k = k0 + i;
      Pack<R, V>* x = (k & 1) ? X : A;
      Pack<R, V>* y = (k & 1) || k == 0 ? A : X;
      if (k >= 1) launch_term<R, V>(c, tt, poly_term2<R, V>(c, pp, k, tpr, A, X));
      dots(x, y, c->partials.as<double>() + (int64_t)i * n_cols * 2 * dot_chunks);
      c->model_bytes += bytes;
    }
    reduce_dots(k0, m);
  }
  enqueue_moment_curves(c, pp, M, T, n_cols, sums + (int64_t)n_cols * 2, (int64_t)n_cols * 2,
                        sums, 2, mu, rho, nodes, chk_step);
  std::vector<double> host;
  read_out(c, host, (size_t)(T + 3) * n_cols * 2);
  check_moments(c, host, T, M, n_cols, chk_step, chk_thr, "tbpm_dos_segmented");
  for (int k = 0; k < n_seg; ++k)
    for (int t = 0; t <= T; ++t) {
      double re = 0, im = 0;
      for (int b = 0; b < ns; ++b) {
        const double* v = &host[((size_t)t * n_cols + k * ns + b) * 2];
        re += v[0] / ns;
        im += v[1] / ns;
        if (corr_per_state) {
          double* o = corr_per_state + 2 * (((size_t)k * ns + b) * (T + 1) + t);
          o[0] = v[0];
          o[1] = v[1];
        }
      }
      corr[2 * ((size_t)k * (T + 1) + t)] = re;
      corr[2 * ((size_t)k * (T + 1) + t) + 1] = im;
    }
  return true;
}

// ---- several time steps per expansion (combine_kernel) ---------------------------

// Weights of P^1 .. P^m; the last one's length is the number of vectors.
struct StepsPlan {
  int m = 0;
  std::vector<std::vector<double>> w;
};

StepsPlan steps_plan(const PolyPlan& pp, int m) {
  StepsPlan sp;
  sp.m = m;
  for (int j = 1; j <= m; ++j) sp.w.push_back(power_weights(pp, j));
  return sp;
}

// states[j] = P(H)^(j+1) psi, j < m <= sp.m, for blocks of ld columns.  psi may be
// states[sp.m-1].  ring: window + 2 blocks for the vectors of the recurrence; the
// outputs are updated once per `window` vectors (at most kCombineWindow).
template <typename R, int V>
void enqueue_steps(tbpm_ctx* c, const PolyPlan& pp, const StepsPlan& sp, int m, int ld,
                   Pack<R, V>* psi, const std::vector<Pack<R, V>*>& ring,
                   const std::vector<Pack<R, V>*>& states) {
  using C = typename Cx<R>::t;
  const int64_t n = c->ham.n;
  const double vb = (double)n * ld * sizeof(C);
  const int tpr = ld / V;
  const int window = (int)ring.size() - 2;
  const TermTiles tt = term_tiles<R, V>(c, n, tpr);
  const double term_bytes = matrix_bytes(c->ham) + 3.0 * vb;
  auto vec = [&](int k) { return k == 0 ? psi : ring[k % ring.size()]; };
  const int n_vec = (int)sp.w[m - 1].size();
  CombineArgs<R> a{};
  a.total = n * ld;
  a.m = m;
  for (int j = 0; j < m; ++j) a.out[j] = reinterpret_cast<C*>(states[j]);
  const int grid = sizeof(R) == 8 ? blocks_for(a.total, 256)
                                  : (int)std::min<int64_t>(blocks_for((a.total + 15) / 16, 8),
                                                           (int64_t)num_sms(c->device) * 4);
  const PersistShape ps = persist_shape<R, V>(c, ld);
  for (int k0 = 0; k0 < n_vec; k0 += window) {
    const int len = std::min(window, n_vec - k0);
    if (ps.grid > 0 && k0 + len > 1) {
      launch_persist<false>(c, ps,
                            persist_args<R, V>(c, pp.alpha, std::max(k0, 1), k0 + len - 1, ld, psi,
                                               ring.data(), (int)ring.size(), true));
      c->model_bytes += (k0 + len - std::max(k0, 1)) * term_bytes;
    }
    for (int q = 0; q < len; ++q) {
      const int k = k0 + q;
      if (k >= 1 && ps.grid == 0) {
        launch_term<R, V>(c, tt,
                          poly_term<R, V>(c, pp, k, tpr, vec(k - 1), k >= 2 ? vec(k - 2) : nullptr,
                                          vec(k), true));
        c->model_bytes += term_bytes;
      }
      a.p[q] = reinterpret_cast<const C*>(vec(k));
    }
    a.np = len;
    // outputs are ordered by degree: those that end before this window are done
    a.j0 = 0;
    while (a.j0 < m - 1 && (int)sp.w[a.j0].size() <= k0) ++a.j0;
    a.init = k0 == 0 ? 1 : 0;
    for (int j = 0; j < m; ++j)
      for (int q = 0; q < kCombineWindow; ++q)
        a.w[j][q] = q < len && k0 + q < (int)sp.w[j].size() ? sp.w[j][k0 + q] : 0.0;
    if constexpr (sizeof(R) == 8) {
      if (m <= 4)
        combine_kernel<R, 4><<<grid, 256, 0, c->stream>>>(a);
      else if (m <= 8)
        combine_kernel<R, 8><<<grid, 256, 0, c->stream>>>(a);
      else
        combine_kernel<R, 16><<<grid, 256, 0, c->stream>>>(a);
    } else {
      // blocks of a multiple of four values keep their 16-byte boundaries
      bool wide = a.total % 4 == 0;
      for (int q = 0; q < len; ++q) wide = wide && reinterpret_cast<uintptr_t>(a.p[q]) % 16 == 0;
      for (int j = 0; j < m; ++j) wide = wide && reinterpret_cast<uintptr_t>(a.out[j]) % 16 == 0;
      if (wide) combine_mma_kernel<true><<<grid, 256, 0, c->stream>>>(a);
      else combine_mma_kernel<false><<<grid, 256, 0, c->stream>>>(a);
    }
    TBPM_CK(cudaGetLastError());
    c->launches++;
    c->model_bytes += vb * (len + (m - a.j0) * (k0 == 0 ? 1 : 2));
  }
}

template <typename R>
constexpr int most_steps = sizeof(R) == 8 ? 16 : 8;  // (combine_mma_kernel: 8 outputs)

// Time steps per expansion and vectors per update for blocks of vb bytes.
struct StepsShape {
  int m = 0;  // 0: none fits
  int window = 0;
};

// Reserves `mem` for the states and the window of the largest shape that fits, with
// `extra` further blocks: m + window + extra blocks of vb bytes, beside `other` bytes of
// buffers to come, in the memory that is free or held by `mem` itself.  (What another
// buffer holds from an earlier, larger call is not free.)  Someone else may take memory
// after the query; a shape whose allocation fails is passed over for the next one.
// Model of a step of phase pi/2 in passes over the block (time stepping: 57): 18 at
// (16, 32), 20 at (16, 16), 24 at (8, 16), 27 at (8, 8), 36 at (4, 8).  Windows of 32
// instead of 16 vectors: AC 561 -> 541 ms (256,000 cells x 8 states), FP32 DC 201 -> 183
// ms.  FP32 states take 8 steps at most: the 16 outputs' FP64 products cost more than the
// terms they save (DC 183 ms at 8, 212 ms at 16).
StepsShape reserve_steps(DevMem& mem, size_t vb, int extra, size_t other, int m_max,
                         size_t cap = SIZE_MAX) {
  const size_t reserve = (size_t)2 << 30;
  for (const StepsShape s : {StepsShape{16, kCombineWindow}, StepsShape{16, 16},
                             StepsShape{8, kCombineWindow}, StepsShape{8, 16}, StepsShape{8, 8},
                             StepsShape{4, 8}}) {
    const size_t need = vb * (size_t)(s.m + s.window + extra);
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
      (void)cudaGetLastError();
      return StepsShape{};
    }
    if (s.m > m_max || need > cap || need + other + reserve > free_b + mem.bytes) continue;
    try {
      mem.ensure(need);
      return s;
    } catch (const Error& e) {
      if (e.code != TBPM_ERR_OOM) throw;
    }
  }
  return StepsShape{};
}

// Blocks of several steps can fill the device; they are given back after the
// call when they hold more than this.
constexpr size_t kKeepBytes = (size_t)12 << 30;
void trim(DevMem& m) {
  if (m.bytes > kKeepBytes) m.release();
}

// Room for the blocks of enqueue_steps behind the block in c->A (ld columns; X
// and Y serve as two blocks of the ring), reserved before c->A is filled.
template <typename R>
StepsShape steps_room(tbpm_ctx* c, const PolyPlan* pp, int ld, int ref_ld) {
  StepsShape s;
  if (pp) {
    const size_t vb = (size_t)c->ham.n * ld * 2 * sizeof(R);
    c->X.ensure(vb);
    c->Y.ensure(vb);
    c->wf0.ensure((size_t)c->ham.n * ref_ld * 2 * sizeof(R));
    // still to come: the staging of states that come from the host
    s = reserve_steps(c->A, vb, 1, (size_t)c->ham.n * ref_ld * 16, most_steps<R>);
  }
  ensure_vectors(c, ld, ref_ld);
  return s;
}

// Propagates the block in c->A by enqueue_steps and hands every state to `each`.
template <typename R, int V>
struct StepsRun {
  const PolyPlan* pp;
  StepsPlan sp;
  int ld;
  Pack<R, V>* psi = nullptr;
  std::vector<Pack<R, V>*> ring, states;

  StepsRun(tbpm_ctx* c, const PolyPlan* plan, const StepsShape& s, int ld_) : pp(plan), ld(ld_) {
    if (s.m == 0) return;
    const size_t vb = (size_t)c->ham.n * ld * 2 * sizeof(R);
    auto block = [&](int i) { return reinterpret_cast<Pack<R, V>*>(c->A.as<char>() + vb * i); };
    sp = steps_plan(*plan, s.m);
    psi = block(0);
    ring = {c->X.as<Pack<R, V>>(), c->Y.as<Pack<R, V>>()};
    for (int q = 0; q < s.window; ++q) ring.push_back(block(1 + q));
    for (int j = 0; j < s.m; ++j) states.push_back(block(1 + s.window + j));
  }

  template <class F>
  void run(tbpm_ctx* c, int n_steps, F&& each) {
    while (n_steps > 0) {
      const int m = std::min(n_steps, sp.m);
      enqueue_steps<R, V>(c, *pp, sp, m, ld, psi, ring, states);
      for (int j = 0; j < m; ++j) each(states[j]);
      if (m < sp.m) std::swap(states[m - 1], states[sp.m - 1]);
      psi = states[sp.m - 1];
      n_steps -= m;
    }
  }
};

// ---- AC ---------------------------------------------------------------------

template <typename R, int V>
void ac_batch(tbpm_ctx* c, const Expansion& ex_time, const Expansion& ex_fermi, int nb,
              const StateKeys* keys, const double* host_wf0, int n_timestep, int chk_step,
              double chk_thr, int n_avg, double* corr, const PolyPlan* pp) {
  const int ld = 3 * nb;
  c->graph.reset();
  c->sess.active = false;
  const StepsShape shape = steps_room<R>(c, pp, ld, nb);
  c->out.ensure((size_t)std::max(n_timestep, 1) * nb * 9 * sizeof(double));
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  auto* Y = c->Y.as<Pack<R, V>>();
  auto* W = c->wf0.as<Pack<R, V>>();
  const Ham& h = c->ham;
  if (keys)
    gen_states<R, V>(c, *keys, nb, c->opts.state_kind, W);
  else
    upload_states<R>(c, host_wf0, nb, nb, 0, W);
  // [J_x wf0 | J_y wf0 | wf0] (tbpm.f90:277-278)
  current_apply_kernel<R><<<blocks_for(h.n * nb, 256), 256, 0, c->stream>>>(
      h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<typename Cx<R>::t>(),
      h.dx.as<R>(), h.dy.as<R>(), h.rescale, h.n, nb,
      reinterpret_cast<const typename Cx<R>::t*>(W), reinterpret_cast<typename Cx<R>::t*>(A));
  TBPM_CK(cudaGetLastError());
  c->launches++;
  // Fermi operators (tbpm.f90:279-281): 1-F on the current columns, F on wf0
  enqueue_expansion<R, V>(c, ex_fermi, ld, A, X, Y, nullptr, 0, nullptr, Counters{});
  const Tile tj = pick_tile(c, h.n, nb, jcorr_kernel<R>, 9 * sizeof(double));
  const size_t smem_j = (size_t)tj.threads * 9 * sizeof(double);
  reset_counters(c, 0);
  auto jcorr = [&](const Pack<R, V>* x) {
    ensure_partials(c, (size_t)nb * 9 * tj.grid);
    jcorr_kernel<R><<<tj.grid, tj.threads, smem_j, c->stream>>>(
        h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<typename Cx<R>::t>(),
        h.dx.as<R>(), h.dy.as<R>(), h.rescale, h.n, tj.rows_per_tile, nb,
        reinterpret_cast<const typename Cx<R>::t*>(x), c->partials.as<double>());
    TBPM_CK(cudaGetLastError());
    c->launches++;
    c->model_bytes += (double)(h.n + 1) * 4 + (double)h.nnz * (4 + 4 * sizeof(R)) +
                      (double)h.n * nb * 3 * 2 * sizeof(R);
    launch_finalize(c, tj.grid, nb * 9, counters(c, 0), c->out.as<double>());
  };
  // row 0: after the Fermi operators (t = 1, not accumulated; its psi2 norm is
  // the norm reference of tbpm.f90:307)
  jcorr(A);
  auto step = [&]() {
    enqueue_expansion<R, V>(c, ex_time, ld, A, X, Y, nullptr, 0, nullptr, Counters{});
    jcorr(A);
  };
  const double thr = effective_thr(c, chk_thr);
  std::vector<double> host;
  int done = 0;  // propagation steps enqueued; row r = after r steps
  const bool check = chk_step >= 2 && chk_step <= n_timestep;
  const auto key = plan_key(c, 2, ld, V, ex_time);
  StepsRun<R, V> many(c, pp, shape, ld);
  auto advance = [&](int n_steps) {
    if (shape.m > 0)
      many.run(c, n_steps, jcorr);
    else
      run_steps(c, n_steps, key, step);
  };
  if (check) {
    // at t == chk_step psi2 has been propagated chk_step-2 times
    advance(chk_step - 2);
    done = chk_step - 2;
    read_out(c, host, (size_t)(done + 1) * nb * 9);
    for (int b = 0; b < nb; ++b) {
      const double ref = host[(size_t)b * 9 + 8];
      const double nv = host[((size_t)done * nb + b) * 9 + 8];
      if (const int bad_ = norm_broken(nv, ref, thr))
        raise_norm("tbpm_accond", chk_step, bad_);
    }
  }
  advance((n_timestep - 1) - done);
  const int rows = std::max(n_timestep, 1);
  read_out(c, host, (size_t)rows * nb * 9);
  // corr(k, t) for t = 2..n_timestep is row t-1 (tbpm.f90:346-349)
  for (int b = 0; b < nb; ++b)
    for (int t = 2; t <= n_timestep; ++t)
      for (int k = 0; k < 4; ++k) {
        const double re = host[((size_t)(t - 1) * nb + b) * 9 + 2 * k];
        const double im = host[((size_t)(t - 1) * nb + b) * 9 + 2 * k + 1];
        corr[2 * (k + 4 * (size_t)(t - 1))] += re / n_avg;
        corr[2 * (k + 4 * (size_t)(t - 1)) + 1] += im / n_avg;
      }
}


// ---- DC -----------------------------------------------------------------------

// One batch of nb states of tbpm_dccond (tbpm.f90:586-698), or, with qe_acc
// set, of tbpm_eigenstates (tbpm.f90:753-813): phase 1 only, then every
// quasi-eigenstate is normalised and acc[r][i] += |QE_i(r)|^2 / n_avg.
// The QE kernels may need more than the default 48 KB of dynamic shared
// memory (row tiles).  The attribute belongs to the current device, so it is
// set before every launch that needs it (a host-side call, once per window).
#ifndef TBPM_QE_MMA
#define TBPM_QE_MMA 1  // quasi-eigenstate accumulation on mma.sync f64 (0: FMA kernel)
#endif
template <typename R>
void qe_accum_attr(size_t bytes) {
  qe_smem_attr(qe_accum_kernel<R>, bytes);
}

// Whether nb states' quasi-eigenstates at n_en energies come from filters.  Their
// tables (values on the nodes, coefficients, window factors) have to stay small beside
// QE, and the transforms of the filters, M^2 n_en products of 1.9 ps, are to cost less
// than the steps they save: 8192 steps, 911 energies, 200 orbitals 1017 ms with filters,
// 739 ms time-stepped; 183 energies 263 and 709 ms; 4096 steps, 455 energies 162 and 354.
bool filters_pay(const tbpm_ctx* c, const PolyPlan& pp, int T, int nb, int n_en) {
  const double M = std::fabs(pp.tau) * (double)pp.a * T;
  const double transform =
      1.9e-12 * M * M * n_en + 7.5e-12 * M * (M + T) * ((nb + 7) / 8);
  return 16.0 * n_en * (M + T) < 1e9 &&
         transform + M * term_seconds(c, nb, 2.2e-6) <
             (double)T * (pp.n_bes - 1) * term_seconds(c, 2 * nb, 4.5e-6);
}

// Phase 1 on the polynomial route: QE_i = f_i(H) wf0 by the energies' filters
// (filter_values_kernel), and the DOS correlation from the moments of the same
// vectors' first half.  dos (complex [T] per state, interleaved [t][nb]) may be null.
template <typename R, int V>
void dc_filter(tbpm_ctx* c, const PolyPlan& pp, int nb, const Pack<R, V>* W, int T, double t_step,
               const std::vector<double>& en_sel, int chk_step, double chk_thr, const char* who,
               std::vector<double>* dos) {
  using C = typename Cx<R>::t;
  const int64_t n = c->ham.n;
  const int n_en = (int)en_sel.size();
  const int M = std::max(4, bessel_degree(pp.tau * (double)pp.a * T));
  const int K = M / 2;
  const int last = n_en > 0 ? M - 1 : K;  // last Chebyshev vector needed
  const size_t vb = (size_t)n * nb * sizeof(C);
  constexpr int slots = kFilterWindow + 2;
  c->A.ensure(vb * slots);
  c->out.ensure((size_t)(T + 3) * nb * 2 * sizeof(double));
  c->small.ensure(sizeof(double) * kMaxCols * 3);
  const size_t n_sums = (size_t)K * nb * 2, n_mu = (size_t)nb * M, n_f = (size_t)M * n_en;
  const size_t n_c = (size_t)T * n_en;  // window and phase factors (complex)
  c->poly.ensure((n_sums + 2 * n_mu + 2 * n_f + 2 * n_c) * sizeof(double) + sizeof(PolyNode) * M);
  double2* factors = c->poly.as<double2>();
  double* sums = c->poly.as<double>() + 2 * n_c;
  double* mu = sums + n_sums;
  double* rho = mu + n_mu;
  double* f = rho + n_mu;
  double* coef = f + n_f;
  PolyNode* nodes = reinterpret_cast<PolyNode*>(coef + n_f);
  const std::vector<PolyNode> host_nodes = poly_nodes(pp, M);
  TBPM_CK(cudaMemcpyAsync(nodes, host_nodes.data(), sizeof(PolyNode) * M, cudaMemcpyHostToDevice,
                          c->stream));
  if (n_en > 0) {
    // Hanning window and phases as the time-stepped phase 1 forms them
    std::vector<double2> hf(n_c);
    const double pi = 3.14159265358979323846;
    for (int tt = 1; tt <= T; ++tt) {
      const double Wh = 0.5 * (1 + std::cos(pi * tt / T));
      for (int i = 0; i < n_en; ++i) {
        const double x = en_sel[i] * (double)tt * t_step;
        hf[(size_t)(tt - 1) * n_en + i] = make_double2(Wh * std::cos(x), Wh * std::sin(x));
      }
    }
    TBPM_CK(cudaMemcpyAsync(factors, hf.data(), sizeof(double2) * n_c, cudaMemcpyHostToDevice,
                            c->stream));
    filter_values_kernel<<<dim3((unsigned)((M + 31) / 32), (unsigned)((n_en + 7) / 8)), 256, 0,
                           c->stream>>>(nodes, M, factors, n_en, T, f);
    filter_coef_kernel<<<dim3((unsigned)M, (unsigned)((n_en + 255) / 256)), 256, 0, c->stream>>>(
        f, M, n_en, coef);
    TBPM_CK(cudaGetLastError());
    c->launches += 2;
    TBPM_CK(cudaStreamSynchronize(c->stream));  // the host vectors go out of scope
  }
  reset_counters(c, 2);
  enqueue_corr<R, V>(c, W, nullptr, nb, 0, c->small.as<double>(), counters(c, 2));
  const int tpr = nb / V;
  const TermTiles tt = term_tiles<R, V>(c, n, tpr);
  const int grid3 = tt.t[3].grid;
  const int64_t per_term = (int64_t)nb * 2 * grid3;
  const int chunk = moment_chunk(K, per_term);
  ensure_partials(c, (size_t)chunk * per_term);
  auto vec = [&](int k) -> Pack<R, V>* {
    return k == 0 ? const_cast<Pack<R, V>*>(W)
                  : reinterpret_cast<Pack<R, V>*>(c->A.as<char>() + vb * (k % slots));
  };
  const double term_bytes = matrix_bytes(c->ham) + 3.0 * (double)vb;
  C* qe = c->qe.as<C>();
  const int rt = qe_filter_rows<R>(nb);
  const int64_t tiles = (n + rt - 1) / rt;
  const int groups = ((n_en + 7) / 8 + kQeMmaWarps * kQeMmaMT - 1) / (kQeMmaWarps * kQeMmaMT);
  const dim3 qgrid((unsigned)std::min<int64_t>(tiles, (int64_t)num_sms(c->device) * 2),
                   (unsigned)std::max(groups, 1));
  const size_t qsmem = qe_filter_smem<R>(nb);
  qe_smem_attr(qe_filter_mma_kernel<R>, qsmem);
  const PersistShape ps = persist_shape<R, V>(c, nb);
  std::vector<Pack<R, V>*> ring(slots);
  for (int q = 0; q < slots; ++q)
    ring[q] = reinterpret_cast<Pack<R, V>*>(c->A.as<char>() + vb * q);
  auto reduce_terms = [&](int k, int count, int grid) {  // terms k .. k + count - 1
    const int64_t n_vals = (int64_t)count * nb * 2;
    reduce_rows_kernel<<<(int)std::min<int64_t>(n_vals, 65535), 256, 0, c->stream>>>(
        c->partials.as<double>(), grid, n_vals, sums + (int64_t)(k - 1) * nb * 2);
    TBPM_CK(cudaGetLastError());
    c->launches++;
  };
  int pend = 0;  // terms whose block partials wait for their reduction
  for (int w0 = 0; w0 <= last; w0 += kFilterWindow) {
    const int w1 = std::min(w0 + kFilterWindow - 1, last);
    const int k_lo = std::max(w0, 1);
    if (ps.grid > 0 && k_lo <= w1) {
      ensure_partials(c, (size_t)kFilterWindow * nb * 2 * ps.grid);
      PersistArgs<R, V> a =
          persist_args<R, V>(c, pp.alpha, k_lo, w1, nb, W, ring.data(), slots, false);
      a.k_dots = K;
      a.partials = c->partials.as<double>();
      launch_persist<false>(c, ps, a);
      c->model_bytes += (w1 - k_lo + 1) * term_bytes;
      if (k_lo <= K) reduce_terms(k_lo, std::min(w1, K) - k_lo + 1, ps.grid);
    }
    for (int k = k_lo; ps.grid == 0 && k <= w1; ++k) {
      TermArgs<R, V> a = poly_term<R, V>(c, pp, k, tpr, vec(k - 1), k >= 2 ? vec(k - 2) : nullptr,
                                         vec(k));
      if (k <= K) a.partials = c->partials.as<double>() + (int64_t)pend * per_term;
      launch_term<R, V>(c, tt, a);
      c->model_bytes += term_bytes;
      if (k <= K && (++pend == chunk || k == K)) {
        reduce_terms(k - pend + 1, pend, grid3);
        pend = 0;
      }
    }
    if (n_en == 0) continue;
    FilterPtrs<R> win{};
    for (int k = w0; k <= w1; ++k) win.p[k - w0] = reinterpret_cast<const C*>(vec(k));
    qe_filter_mma_kernel<R><<<qgrid, kQeMmaWarps * 32, qsmem, c->stream>>>(
        qe, n, n_en, nb, win, w1 - w0 + 1, coef + (int64_t)w0 * n_en, w0 == 0 ? 1 : 0);
    TBPM_CK(cudaGetLastError());
    c->launches++;
    c->model_bytes += (double)n * n_en * nb * sizeof(C) * (w0 == 0 ? 1 : 2) +
                      (double)(w1 - w0 + 1) * (double)vb;
  }
  const bool check = chk_step >= 2 && chk_step <= T;
  if (!dos && !check) return;
  enqueue_moment_curves(c, pp, M, T, nb, sums, (int64_t)nb * 2, c->small.as<double>() + 2, 3, mu,
                        rho, nodes, chk_step, 0, true);
  std::vector<double> host;
  read_out(c, host, (size_t)(T + 3) * nb * 2);
  // tbpm.f90:611-614: after chk_step - 1 steps against <wf0|wf0>; P and its
  // conjugate have the same norms
  check_moments(c, host, T, M, nb, chk_step, chk_thr, who);
  if (dos) dos->assign(host.begin() + (size_t)nb * 2, host.begin() + (size_t)(T + 1) * nb * 2);
}

template <typename R, int V>
void dc_batch(tbpm_ctx* c, const Expansion& ex_pm, const Expansion& ex_fwd, int nb,
              const StateKeys* keys, const double* host_wf0, int n_timestep, double t_step,
              const std::vector<double>& en_sel, int chk_step, double chk_thr, int n_avg,
              int n_energies, double* dos_corr, double* dc_corr, double* qe_acc = nullptr,
              const char* who = "tbpm_dccond", int en_out0 = 0, bool add_dos = true,
              const PolyPlan* pp = nullptr) {
  const bool filters = pp && filters_pay(c, *pp, n_timestep, nb, (int)en_sel.size());
  using C = typename Cx<R>::t;
  const Ham& h = c->ham;
  const int64_t n = h.n;
  const int ld = 2 * nb;
  const int n_en = (int)en_sel.size();
  const int T1 = std::min(kMaxWindow, std::max(n_timestep, 1));  // phase-1 window
  const int T2 = std::min(8, std::max(n_timestep, 1));           // phase-2 window
  const size_t vb = (size_t)n * ld * 2 * sizeof(R);
  c->graph.reset();
  c->sess.active = false;
  if (!filters) {
    c->X.ensure(vb);
    c->Y.ensure(vb);
    c->A.ensure(vb * (size_t)(std::max(T1, T2) + 1));
  }
  c->wf0.ensure((size_t)n * nb * 2 * sizeof(R));
  c->ctr.ensure(16 * sizeof(int));
  c->out.ensure((size_t)std::max(n_timestep, 1) * ld * 3 * sizeof(double));
  c->small.ensure(sizeof(double) * 3 * kMaxCols * 2);
  const size_t qe_bytes = (size_t)n * std::max(n_en, 1) * nb * 2 * sizeof(R);
  c->qe.ensure(qe_bytes);
  c->coef.ensure(sizeof(double2) * (size_t)kMaxWindow * std::max(n_en, 1));
  auto slot = [&](int s) { return reinterpret_cast<Pack<R, V>*>(c->A.as<char>() + vb * s); };
  auto* W = c->wf0.as<Pack<R, V>>();
  C* qe = c->qe.as<C>();
  if (keys)
    gen_states<R, V>(c, *keys, nb, c->opts.state_kind, W);
  else
    upload_states<R>(c, host_wf0, nb, nb, 0, W);
  std::vector<double> host;
  std::optional<Phase> phase;
  phase.emplace("tbpm_dccond: quasi-eigenstates");
  int t = 1;
  if (filters) {
    std::vector<double> dos;
    dc_filter<R, V>(c, *pp, nb, W, n_timestep, t_step, en_sel, chk_step, chk_thr, who,
                    dos_corr && add_dos ? &dos : nullptr);
    if (dos_corr && add_dos)
      for (int b = 0; b < nb; ++b)
        for (int tt = 1; tt <= n_timestep; ++tt) {
          dos_corr[2 * (tt - 1)] += dos[((size_t)(tt - 1) * nb + b) * 2] / n_avg;
          dos_corr[2 * (tt - 1) + 1] += dos[((size_t)(tt - 1) * nb + b) * 2 + 1] / n_avg;
        }
  } else {
    auto* X = c->X.as<Pack<R, V>>();
    auto* Y = c->Y.as<Pack<R, V>>();
    // wf_t_pos = wf_t_neg = wf0 in the slot read by the first step
    dup_columns_kernel<R><<<blocks_for(n * nb, 256), 256, 0, c->stream>>>(
        reinterpret_cast<const C*>(W), n, nb, reinterpret_cast<C*>(slot(T1 - 1)));
    TBPM_CK(cudaGetLastError());
    c->launches++;
    // norm_ref = <wf0|wf0> (tbpm.f90:606) for every column
    reset_counters(c, 2);
    enqueue_corr<R, V>(c, slot(T1 - 1), nullptr, ld, 0, c->small.as<double>(), counters(c, 2));
    std::vector<double> norm_ref(3 * ld);
    TBPM_CK(cudaMemcpyAsync(norm_ref.data(), c->small.p, norm_ref.size() * sizeof(double),
                            cudaMemcpyDeviceToHost, c->stream));
    TBPM_CK(cudaStreamSynchronize(c->stream));
    const double thr = effective_thr(c, chk_thr);
    reset_counters(c, 0);
    const bool check = chk_step >= 2 && chk_step <= n_timestep;
    std::vector<double2> coef_host((size_t)kMaxWindow * std::max(n_en, 1));
    const double pi = 3.14159265358979323846;
    // ---- phase 1: +/- dt propagation, DOS correlation, QE accumulation ----
    bool first_window = true;
    while (t <= n_timestep) {
      int len = std::min(T1, n_timestep - t + 1);
      if (check && t <= chk_step - 1 && t + len - 1 > chk_step - 1) len = chk_step - t;
      for (int tau = 0; tau < len; ++tau) {
        Pack<R, V>* in = slot(tau == 0 ? T1 - 1 : tau - 1);
        enqueue_expansion<R, V>(c, ex_pm, ld, in, X, Y, W, nb, c->out.as<double>(),
                                counters(c, 0), slot(tau));
      }
      if (n_en > 0) {
        for (int tau = 0; tau < len; ++tau) {
          const int tt = t + tau;
          const double Wh = 0.5 * (1 + std::cos(pi * tt / n_timestep));  // Hanning
          for (int i = 0; i < n_en; ++i) {
            const double x = en_sel[i] * (double)tt * t_step;
            coef_host[(size_t)tau * n_en + i] = make_double2(Wh * std::cos(x), Wh * std::sin(x));
          }
        }
        TBPM_CK(cudaMemcpyAsync(c->coef.p, coef_host.data(), sizeof(double2) * len * n_en,
                                cudaMemcpyHostToDevice, c->stream));
        StatePtrs<R> win{};
        for (int tau = 0; tau < len; ++tau) win.p[tau] = reinterpret_cast<const C*>(slot(tau));
        const int64_t total = n * n_en * nb;
        if (TBPM_QE_MMA) {
          // FP64 tensor-path products (qe_accum_mma_kernel)
          const int rt = qe_mma_rows(nb);
          const int64_t tiles = (n + rt - 1) / rt;
          const int groups = ((n_en + 7) / 8 + kQeMmaWarps * kQeMmaMT - 1) / (kQeMmaWarps * kQeMmaMT);
          const dim3 grid((unsigned)std::min<int64_t>(tiles, (int64_t)num_sms(c->device) * 4),
                          (unsigned)groups);
          const size_t qsmem = qe_mma_smem(nb);
          qe_smem_attr(qe_accum_mma_kernel<R>, qsmem);
          qe_accum_mma_kernel<R><<<grid, kQeMmaWarps * 32, qsmem, c->stream>>>(
              qe, n, n_en, nb, win, len, c->coef.as<double2>(), first_window ? 1 : 0,
              reinterpret_cast<const C*>(W));
        } else {
          const int qthreads = qe_accum_threads(n_en, nb);
          const int n_chunks = (n_en * nb + kQeG * qthreads - 1) / (kQeG * qthreads);
          const int64_t tiles = (n + qe_accum_rows<R>(nb) - 1) / qe_accum_rows<R>(nb);
          const dim3 grid((unsigned)std::min<int64_t>(tiles, (int64_t)kSMs * 16),
                          (unsigned)n_chunks);
          const size_t qsmem = qe_accum_smem<R>(n_en, nb);
          qe_accum_attr<R>(qsmem);
          qe_accum_kernel<R><<<grid, qthreads, qsmem, c->stream>>>(
              qe, n, n_en, nb, win, len, c->coef.as<double2>(), first_window ? 1 : 0,
              reinterpret_cast<const C*>(W));
        }
        TBPM_CK(cudaGetLastError());
        c->launches++;
        c->model_bytes += (double)total * 2 * sizeof(R) * (first_window ? 1 : 2) +
                          (double)len * n * ld * 2 * sizeof(R);
      }
      // the window ring: the next window reads the last state from slot T1-1
      if (len != T1 && t + len - 1 < n_timestep)
        TBPM_CK(cudaMemcpyAsync(slot(T1 - 1), slot(len - 1), vb, cudaMemcpyDeviceToDevice,
                                c->stream));
      TBPM_CK(cudaStreamSynchronize(c->stream));  // coef_host is reused
      first_window = false;
      t += len;
      if (check && t == chk_step) {
        // tbpm.f90:611-614: at t == chk_step the states after chk_step-1 steps
        read_out(c, host, (size_t)(chk_step - 1) * ld * 3);
        for (int b = 0; b < ld; ++b) {
          const double nv = host[((size_t)(chk_step - 2) * ld + b) * 3 + 2];
          if (const int bad_ = norm_broken(nv, norm_ref[(size_t)b * 3 + 2], thr))
            raise_norm(who, chk_step, bad_);
        }
      }
    }
  }
  if (qe_acc) {
    // tbpm.f90:803-813: QE_i / |QE_i|, then |.|^2 averaged over samples
    const int n_ib = n_en * nb;
    const int64_t rpt = std::max<int64_t>(64, n / ((int64_t)kSMs * 8));
    const int pgrid = (int)((n + rpt - 1) / rpt);
    ensure_partials(c, (size_t)n_ib * pgrid);
    c->small.ensure(sizeof(double) * std::max(n_ib, 64));
    qe_sqnorm_kernel<R><<<pgrid, std::min(256, ((n_ib + 31) / 32) * 32), 0, c->stream>>>(
        qe, n, rpt, n_ib, c->partials.as<double>());
    TBPM_CK(cudaGetLastError());
    reduce_rows_kernel<<<std::min(n_ib, 65535), 256, 0, c->stream>>>(
        c->partials.as<double>(), pgrid, n_ib, c->small.as<double>());
    TBPM_CK(cudaGetLastError());
    const int64_t total = n * n_en;
    const int grid = (int)std::min<int64_t>(blocks_for(total, 256), (int64_t)kSMs * 32);
    qe_density_kernel<R><<<grid, 256, 0, c->stream>>>(qe, n, n_en, nb, c->small.as<double>(),
                                                     1.0 / n_avg, qe_acc);
    TBPM_CK(cudaGetLastError());
    c->launches += 3;
    c->model_bytes += 2.0 * (double)n * n_ib * 2 * sizeof(R) + 2.0 * total * 8;
    TBPM_CK(cudaStreamSynchronize(c->stream));
    check_status(c);
    return;
  }
  if (!filters) read_out(c, host, (size_t)n_timestep * ld * 3);
  if (!filters && add_dos)
    for (int b = 0; b < nb; ++b)
      for (int tt = 1; tt <= n_timestep; ++tt) {
        dos_corr[2 * (tt - 1)] += host[((size_t)(tt - 1) * ld + b) * 3 + 0] / n_avg;
        dos_corr[2 * (tt - 1) + 1] += host[((size_t)(tt - 1) * ld + b) * 3 + 1] / n_avg;
      }
  if (n_en == 0) return;
  // ---- phase 2 ----
  phase.emplace("tbpm_dccond: current correlations");
  const int n_ib = n_en * nb;
  // about four blocks per SM over the row ranges and the chunks
  const ProjShape psh = proj_shape(n_en, nb);
  const int64_t chunks = (int64_t)psh.n_bc * psh.n_ec;
  const int64_t want = std::max<int64_t>(1, 4 * (int64_t)num_sms(c->device) / chunks);
  const int64_t rows_per_block = std::max<int64_t>(64, (n + want - 1) / want);
  const int pgrid = (int)((n + rows_per_block - 1) / rows_per_block);
  const int parts = pgrid * psh.ws;
  const size_t psmem = proj_smem<R>(psh);
  qe_smem_attr(qe_project_kernel<R>, psmem);
  auto project = [&](const StatePtrs<R>& u, int len, int K) {
    qe_project_kernel<R><<<dim3((unsigned)pgrid, (unsigned)chunks), kProjWarps * 32, psmem,
                           c->stream>>>(qe, n, rows_per_block, n_en, nb, u, len, K,
                                        c->partials.as<double>());
    TBPM_CK(cudaGetLastError());
    const int64_t n_vals = (int64_t)2 * len * K * n_ib;
    reduce_rows_kernel<<<(int)std::min<int64_t>(n_vals, 65535), 256, 0, c->stream>>>(
        c->partials.as<double>(), parts, n_vals, c->small.as<double>());
    TBPM_CK(cudaGetLastError());
    c->launches += 2;
  };
  ensure_partials(c, (size_t)2 * 2 * T2 * n_ib * parts);
  c->small.ensure(sizeof(double) * std::max<size_t>((size_t)2 * T2 * 2 * n_ib, 64));
  // |<wf0|QE_i>| per (energy, state)
  {
    StatePtrs<R> w{};
    w.p[0] = reinterpret_cast<const C*>(W);
    project(w, 1, 1);
  }
  std::vector<double> proj(2 * n_ib);
  TBPM_CK(cudaMemcpyAsync(proj.data(), c->small.p, proj.size() * sizeof(double),
                          cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
  std::vector<double> amp(n_ib);
  for (int ib = 0; ib < n_ib; ++ib) amp[ib] = std::hypot(proj[2 * ib], proj[2 * ib + 1]);
  // wf0_J = [J_x wf0 | J_y wf0] (tbpm.f90:654-655), propagated step by step, or
  // several steps per expansion where their blocks fit beside QE
  StepsShape shape;
  if (pp) {
    // a memory budget covers QE and these blocks together
    size_t cap = SIZE_MAX;
    if (c->opts.dc_budget_gb > 0) {
      const size_t budget = (size_t)(c->opts.dc_budget_gb * 1073741824.0);
      cap = budget > qe_bytes ? budget - qe_bytes : 0;
    }
    shape = reserve_steps(c->A, vb, 2 + T2, 0, most_steps<R>, cap);
    if (shape.m == 0) {
      c->X.ensure(vb);
      c->Y.ensure(vb);
      c->A.ensure(vb * (size_t)(T2 + 1));
    }
  }
  std::vector<Pack<R, V>*> ring, states, us;
  for (int q = 0; q < T2; ++q) us.push_back(slot(q));
  StepsPlan sp;
  if (shape.m > 0) {
    sp = steps_plan(*pp, std::min(shape.m, std::max(n_timestep - 1, 1)));
    for (int q = 0; q < shape.window + 2; ++q) ring.push_back(slot(T2 + q));
    for (int q = 0; q < sp.m; ++q) states.push_back(slot(T2 + shape.window + 2 + q));
  } else {
    states.push_back(slot(pp ? T2 : std::max(T1, T2)));
  }
  Pack<R, V>* wj = states.back();
  int made = 0, used = 0;  // states of the current expansion
  jj_apply_kernel<R><<<blocks_for(n * ld, 256), 256, 0, c->stream>>>(
      h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<C>(), h.dx.as<R>(), h.dy.as<R>(),
      h.rescale, n, nb, reinterpret_cast<const C*>(W), nb, 0, 0, reinterpret_cast<C*>(wj));
  TBPM_CK(cudaGetLastError());
  c->launches++;
  std::vector<double> vals;
  for (t = 1; t <= n_timestep; t += T2) {
    const int len = std::min(T2, n_timestep - t + 1);
    StatePtrs<R> u{};
    for (int tau = 0; tau < len; ++tau) {
      const int tt = t + tau;
      if (tt >= 2 && shape.m > 0) {
        if (used == made) {
          made = std::min(sp.m, n_timestep - tt + 1);
          used = 0;
          enqueue_steps<R, V>(c, *pp, sp, made, ld, wj, ring, states);
        }
        wj = states[used++];
      } else if (tt >= 2) {
        enqueue_expansion<R, V>(c, ex_fwd, ld, wj, c->X.as<Pack<R, V>>(), c->Y.as<Pack<R, V>>(),
                                nullptr, 0, nullptr, Counters{});
      }
      C* uq = reinterpret_cast<C*>(us[tau]);
      jj_apply_kernel<R><<<blocks_for(n * ld, 256), 256, 0, c->stream>>>(
          h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<C>(), h.dx.as<R>(),
          h.dy.as<R>(), h.rescale, n, nb, reinterpret_cast<const C*>(wj), ld, 0, nb, uq);
      TBPM_CK(cudaGetLastError());
      c->launches++;
      u.p[tau] = uq;
    }
    project(u, len, 2);
    const int64_t n_vals = (int64_t)2 * len * 2 * n_ib;
    c->model_bytes += (double)n * n_ib * 2 * sizeof(R) + (double)len * n * ld * 2 * sizeof(R);
    vals.resize(n_vals);
    TBPM_CK(cudaMemcpyAsync(vals.data(), c->small.p, n_vals * sizeof(double),
                            cudaMemcpyDeviceToHost, c->stream));
    TBPM_CK(cudaStreamSynchronize(c->stream));
    for (int tau = 0; tau < len; ++tau)
      for (int k = 0; k < 2; ++k)
        for (int i = 0; i < n_en; ++i)
          for (int b = 0; b < nb; ++b) {
            const int ib = i * nb + b;
            const int64_t o = ((int64_t)(tau * 2 + k) * n_ib + ib) * 2;
            const double a = amp[ib];
            const size_t d = 2 * ((size_t)k + 2 * ((size_t)(en_out0 + i) +
                                                   (size_t)n_energies * (t + tau - 1)));
            dc_corr[d] += vals[o] / a / n_avg;
            dc_corr[d + 1] += vals[o + 1] / a / n_avg;
          }
  }
  check_status(c);  // (once: a read of the word per window cost 1.3% of the run)
}

// ---- dynamical polarisation -------------------------------------------------------

// One batch of nb states and nq q-points of tbpm_dyn_pol (tbpm.f90:436-488).
// The block holds psi1 for every (q-point, state) and psi2 for every state:
// psi2 does not depend on q, so it is propagated once for all q-points of the
// batch instead of once per q-point.
template <typename R, int V>
void dynpol_batch(tbpm_ctx* c, const Expansion& ex_time, const Expansion& ex_fermi, int nb,
                  int nq, const QBlock& qb, const double* sx, const double* sy, const double* sz,
                  const StateKeys* keys, const double* host_wf0, int n_timestep, int chk_step,
                  double chk_thr, int n_avg, int q0, int n_q_total, double* corr,
                  const PolyPlan* pp) {
  using C = typename Cx<R>::t;
  const int ld = (nq + 1) * nb;
  const int tpr = nq * nb;
  c->graph.reset();
  c->sess.active = false;
  const StepsShape shape = steps_room<R>(c, pp, ld, nb);
  c->out.ensure((size_t)std::max(n_timestep, 1) * tpr * 3 * sizeof(double));
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  auto* Y = c->Y.as<Pack<R, V>>();
  auto* W = c->wf0.as<Pack<R, V>>();
  const Ham& h = c->ham;
  if (keys)
    gen_states<R, V>(c, *keys, nb, c->opts.state_kind, W);
  else
    upload_states<R>(c, host_wf0, nb, nb, 0, W);
  const int64_t total = h.n * ld;
  dens_init_kernel<R><<<(int)std::min<int64_t>(blocks_for(total, 256), (int64_t)kSMs * 32), 256,
                        0, c->stream>>>(reinterpret_cast<const C*>(W), sx, sy, sz, qb, nq, nb,
                                        h.n, reinterpret_cast<C*>(A));
  TBPM_CK(cudaGetLastError());
  c->launches++;
  // Fermi operators (tbpm.f90:458-461): 1-F on every psi1 column, F on psi2
  enqueue_expansion<R, V>(c, ex_fermi, ld, A, X, Y, nullptr, 0, nullptr, Counters{});
  const Tile td = pick_tile(c, h.n, tpr, dens_corr_kernel<R>, 3 * sizeof(double));
  const size_t smem = (size_t)td.threads * 3 * sizeof(double);
  reset_counters(c, 0);
  auto dcorr = [&](const Pack<R, V>* x) {
    ensure_partials(c, (size_t)tpr * 3 * td.grid);
    dens_corr_kernel<R><<<td.grid, td.threads, smem, c->stream>>>(
        reinterpret_cast<const C*>(x), sx, sy, sz, qb, nq, nb, h.n, c->partials.as<double>());
    TBPM_CK(cudaGetLastError());
    c->launches++;
    c->model_bytes += (double)h.n * ld * 2 * sizeof(R) + (double)h.n * 24;
    launch_finalize(c, td.grid, tpr * 3, counters(c, 0), c->out.as<double>());
  };
  dcorr(A);  // t = 1 (tbpm.f90:463-470); its psi2 norm is the norm reference
  auto step = [&]() {
    enqueue_expansion<R, V>(c, ex_time, ld, A, X, Y, nullptr, 0, nullptr, Counters{});
    dcorr(A);
  };
  auto key = plan_key(c, 5, ld, V, ex_time);
  key_push(key, nq);
  key_push(key, sx);
  for (int k = 0; k < nq; ++k)
    for (int d = 0; d < 3; ++d) key_push(key, qb.q[k][d]);
  StepsRun<R, V> many(c, pp, shape, ld);
  auto advance = [&](int n_steps) {
    if (shape.m > 0)
      many.run(c, n_steps, dcorr);
    else
      run_steps(c, n_steps, key, step);
  };
  const double thr = effective_thr(c, chk_thr);
  std::vector<double> host;
  int done = 0;
  const bool check = chk_step >= 2 && chk_step <= n_timestep;
  if (check) {
    // tbpm.f90:479: at t == chk_step psi2 has been propagated chk_step-2 times
    advance(chk_step - 2);
    done = chk_step - 2;
    read_out(c, host, (size_t)(done + 1) * tpr * 3);
    for (int b = 0; b < nb; ++b) {
      const double ref = host[(size_t)b * 3 + 2];
      const double nv = host[((size_t)done * tpr + b) * 3 + 2];
      if (const int bad_ = norm_broken(nv, ref, thr))
        raise_norm("tbpm_dyn_pol", chk_step, bad_);
    }
  }
  advance((n_timestep - 1) - done);
  read_out(c, host, (size_t)n_timestep * tpr * 3);
  for (int k = 0; k < nq; ++k)
    for (int b = 0; b < nb; ++b)
      for (int t = 1; t <= n_timestep; ++t)
        corr[(q0 + k) + (size_t)n_q_total * (t - 1)] +=
            host[((size_t)(t - 1) * tpr + k * nb + b) * 3 + 1] / n_avg;
}

// ---- Kubo-Bastin mu_mn ------------------------------------------------------------

// scatter site amplitudes into a zeroed vector (tbpm.f90:1005-1008)
template <typename R>
__global__ void scatter_sites_kernel(const int32_t* sites, const double2* vals, int n_sites,
                                     typename Cx<R>::t* v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_sites) return;
  typename Cx<R>::t o;
  o.x = (R)vals[i].x;
  o.y = (R)vals[i].y;
  v[sites[i]] = o;
}

// Slices of the N rows for the split-K contraction: at most four blocks per SM
// (two waves of the two that are resident; one block more would start a third:
// 25 slices of 24 tiles took 2.5 ms where 24 take 1.75 ms), slices a multiple of the
// 16-row step.
struct PqSplit {
  int slices;
  int64_t rows;
};

PqSplit pq_split(const tbpm_ctx* c, int64_t n, int m, int nk) {
  const int64_t tiles = (int64_t)((m + kPqTile - 1) / kPqTile) * ((nk + kPqTile - 1) / kPqTile);
  const int64_t want = std::max<int64_t>(1, 4 * (int64_t)num_sms(c->device) / tiles);
  const int64_t max_slices = std::max<int64_t>(1, n / (16 * kPqK));
  const int64_t sl = std::min(want, max_slices);
  int64_t rows = (n + sl - 1) / sl;
  rows = (rows + kPqK - 1) / kPqK * kPqK;
  PqSplit p;
  p.rows = rows;
  p.slices = (int)((n + rows - 1) / rows);
  return p;
}

// One state of tbpm_kbdc (tbpm.f90:898-957).  Q holds J_a T_j(H) psi for all
// j (N x nk, column-major); the bra vectors T_i(H) J_x psi are generated in
// chunks of kc columns and contracted with Q by one complex GEMM per chunk
// (pq_dmma_kernel in FP64, pq_gemm_kernel in FP32, split over N, and
// pq_reduce_kernel): the nk^2 inner products of the reference as a
// (kc x N) . (N x nk) product.
template <typename R>
void kbdc_state(tbpm_ctx* c, int nk, int direction, const double* g_dev, double scale,
                double2* mu_dev) {
  using C = typename Cx<R>::t;
  const Ham& h = c->ham;
  const int64_t n = h.n;
  const int kc = std::min(nk, 128);
  const size_t vb = (size_t)n * sizeof(C);
  C* Q = c->A.as<C>();
  C* P = c->X.as<C>();
  C* ring = c->Y.as<C>();  // 5 vectors: T ring (3) and the P carry (2)
  C* psi = c->wf0.as<C>();
  double2* ws = nullptr;  // split partials of the contraction (c->qe)
  const int grid = (int)std::min<int64_t>(blocks_for(n, 256), (int64_t)kSMs * 16);
  const C* diag = h.has_diag ? h.diag.as<C>() : nullptr;
  const R* dj = direction == 1 ? h.dx.as<R>() : h.dy.as<R>();
  auto hmv = [&](double alpha, double beta, const C* x, const C* z, C* y) {
    cheb_vec_kernel<R><<<grid, 256, 0, c->stream>>>(h.indptr.as<int32_t>(),
                                                   h.indices.as<int32_t>(), h.hop.as<C>(), diag,
                                                   n, alpha, beta, x, z, y);
    TBPM_CK(cudaGetLastError());
    c->launches++;
  };
  auto cur = [&](const R* d, const C* x, C* y) {
    current_vec_kernel<R><<<grid, 256, 0, c->stream>>>(h.indptr.as<int32_t>(),
                                                      h.indices.as<int32_t>(), h.hop.as<C>(),
                                                      d, h.rescale, n, x, y);
    TBPM_CK(cudaGetLastError());
    c->launches++;
  };
  // ket side: Q_j = J_a T_j(H) psi  (tbpm.f90:905-929), with T_{j+1} from the same
  // pass over the matrix
  C* t[3] = {ring, ring + n, ring + 2 * n};
  TBPM_CK(cudaMemcpyAsync(t[0], psi, vb, cudaMemcpyDeviceToDevice, c->stream));
  for (int j = 0; j < nk; ++j) {
    cheb_current_kernel<R><<<grid, 256, 0, c->stream>>>(
        h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<C>(), diag, dj, h.rescale, n,
        j == 0 ? 1.0 : 2.0, j == 0 ? 0.0 : -1.0, t[j % 3], j == 0 ? nullptr : t[(j + 2) % 3],
        j + 1 < nk ? t[(j + 1) % 3] : nullptr, Q + (size_t)j * n);
    TBPM_CK(cudaGetLastError());
    c->launches++;
  }
  // bra side in chunks: P_i = T_i(H) J_x psi, then mu[i0:i0+kc, :] += P^H Q
  C* carry[2] = {ring + 3 * n, ring + 4 * n};
  for (int i0 = 0; i0 < nk; i0 += kc) {
    const int m = std::min(kc, nk - i0);
    for (int ii = 0; ii < m; ++ii) {
      const int i = i0 + ii;
      C* pi = P + (size_t)ii * n;
      // the two previous bra vectors: in this chunk or carried from the last one
      const C* pm1 = ii >= 1 ? P + (size_t)(ii - 1) * n : carry[1];
      const C* pm2 = ii >= 2 ? P + (size_t)(ii - 2) * n : (ii == 1 ? carry[1] : carry[0]);
      if (i == 0)
        cur(h.dx.as<R>(), psi, pi);  // p_0 = J_x psi (tbpm.f90:932)
      else if (i == 1)
        hmv(1.0, 0.0, pm1, nullptr, pi);  // p_1 = H p_0 (:938)
      else
        hmv(2.0, -1.0, pm1, pm2, pi);  // p_i = 2 H p_i-1 - p_i-2 (:950)
    }
    const PqSplit sp = pq_split(c, n, m, nk);
    // a short last chunk may take more slices than the full chunks it was sized for
    c->qe.ensure((size_t)sp.slices * m * nk * sizeof(double2));
    ws = c->qe.as<double2>();
    const dim3 pgrid((nk + kPqTile - 1) / kPqTile, (m + kPqTile - 1) / kPqTile, sp.slices);
    if constexpr (sizeof(R) == 8) {
      qe_smem_attr(pq_dmma_kernel, kPqSmem);
      pq_dmma_kernel<<<pgrid, 128, kPqSmem, c->stream>>>(P, Q, n, m, nk, sp.rows, ws);
    } else {
      pq_gemm_kernel<R><<<pgrid, 256, 0, c->stream>>>(P, Q, n, m, nk, sp.rows, ws);
    }
    TBPM_CK(cudaGetLastError());
    pq_reduce_kernel<<<(int)std::min<int64_t>(blocks_for((int64_t)m * nk, 256), 4096), 256, 0,
                       c->stream>>>(ws, sp.slices, m, nk, i0, g_dev, scale, mu_dev);
    TBPM_CK(cudaGetLastError());
    c->launches += 2;
    // carry the last two bra vectors into the next chunk
    if (i0 + m < nk) {  // m == kc >= 2 here
      TBPM_CK(cudaMemcpyAsync(carry[0], P + (size_t)(m - 2) * n, vb, cudaMemcpyDeviceToDevice,
                              c->stream));
      TBPM_CK(cudaMemcpyAsync(carry[1], P + (size_t)(m - 1) * n, vb, cudaMemcpyDeviceToDevice,
                              c->stream));
    }
  }
  c->model_bytes += (double)nk * (2.0 * ((double)(h.n + 1) * 4 + (double)h.nnz * (4 + 2 * sizeof(R))) +
                                  7.0 * n * sizeof(C)) +
                    2.0 * (double)nk * n * sizeof(C);
}

// ---- Haydock recursion ---------------------------------------------------------------

// propagation.f90:85-155 for the start vector already in wf0 (single column);
// a (complex) and b of every depth are written to sc[0 .. 3*n_depth).
template <typename R>
void haydock_state(tbpm_ctx* c, int n_depth, double h_rescale, double* sc) {
  using C = typename Cx<R>::t;
  const Ham& h = c->ham;
  // Enough threads for one row each, spread over the SMs.  Blocks of 768 have the
  // registers to load a row ahead; past five rows a thread (their own rows no longer
  // fit the shared memory in FP64) the more loads in flight of 1024 win.  Measured on
  // B200, us per depth, 768 / 1024: FP64 320,000 orbitals 10.5 / 11.8, 524,288 12.6 /
  // 14.0, 980,000 28.3 / 25.8; FP32 320,000 11.0 / 12.0, 980,000 19.4 / 18.7.
  const int sms = num_sms(c->device);
  const int64_t per_sm = (h.n + sms - 1) / sms;
  const bool large = h.n > 5 * (int64_t)sms * 768;
  auto kernel = large ? haydock_kernel<R, 1024> : haydock_kernel<R, 768>;
  const int threads = (int)std::min<int64_t>(
      large ? 1024 : 768, std::max<int64_t>(128, (per_sm + 31) / 32 * 32));
  const int grid = (int)std::min<int64_t>(sms, (h.n + threads - 1) / threads);
  ensure_partials(c, (size_t)3 * grid);
  c->ctr.ensure(16 * sizeof(int));
  HaydockArgs<R> a;
  a.indptr = h.indptr.as<int32_t>();
  a.indices = h.indices.as<int32_t>();
  a.hop = h.hop.as<C>();
  a.diag = h.has_diag ? h.diag.as<C>() : nullptr;
  a.n_rows = h.n;
  a.rescale = h_rescale;
  a.w0 = c->wf0.as<C>();
  a.w1 = c->X.as<C>();
  a.y = c->Y.as<C>();
  a.n_depth = n_depth;
  a.a = sc;
  a.b = sc + 2 * n_depth;
  a.partials = c->partials.as<double>();
  const int64_t items = (h.n + (int64_t)grid * threads - 1) / ((int64_t)grid * threads);
  const size_t item_bytes = 3 * (size_t)threads * sizeof(C);
  a.cap = (int)std::min<int64_t>(items, (int64_t)(kHaydockSmem / item_bytes));
  a.bar = c->ctr.as<unsigned int>() + 12;
  a.status = c->status.as<unsigned int>();
  a.absent = 0;
  a.wait_ns = kGridWaitNs;
  TBPM_CK(cudaMemsetAsync(a.bar, 0, sizeof(unsigned int), c->stream));
  qe_smem_attr(kernel, a.cap * item_bytes);
  launch_cooperative(c, kernel, grid, threads, a.cap * item_bytes, a);
  c->launches++;
  c->model_bytes += (double)n_depth * (matrix_bytes(h) + 6.0 * h.n * sizeof(C));
}

// ---- psi(t) -------------------------------------------------------------------

// Two staging buffers of a call and the stream their copies run on.
struct FrameCopies {
  tbpm_ctx* c;
  size_t bytes;
  cudaStream_t stream = nullptr;
  cudaEvent_t ready = nullptr;
  int slot = 0;
  double* host = nullptr;  // destination of the staged frame, null: none

  FrameCopies(tbpm_ctx* ctx, size_t n) : c(ctx), bytes((n + 255) & ~(size_t)255) {
    c->stage.ensure(2 * bytes);
    TBPM_CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    const cudaError_t e = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      cudaStreamDestroy(stream);
      throw_cuda(e, "cudaEventCreateWithFlags");
    }
  }
  ~FrameCopies() {
    cudaStreamSynchronize(stream);
    cudaEventDestroy(ready);
    cudaStreamDestroy(stream);
  }
  FrameCopies(const FrameCopies&) = delete;
  FrameCopies& operator=(const FrameCopies&) = delete;

  double2* next() { return reinterpret_cast<double2*>(c->stage.as<char>() + slot * bytes); }
  // next() has been filled on the context stream; its copy goes to dst at flush()
  void stage(double* dst) {
    TBPM_CK(cudaEventRecord(ready, c->stream));
    host = dst;
  }
  // Copies the staged frame, complete when this returns (the other buffer is
  // then free for the next frame).
  void flush() {
    if (!host) return;
    double* dst = host;
    host = nullptr;
    TBPM_CK(cudaStreamWaitEvent(stream, ready, 0));
    TBPM_CK(cudaMemcpyAsync(dst, next(), (size_t)c->ham.n * 16, cudaMemcpyDeviceToHost, stream));
    TBPM_CK(cudaStreamSynchronize(stream));
    slot ^= 1;
  }
};

template <typename R>
void psi_t_run(tbpm_ctx* c, const Expansion& ex, const double* bes, int n_bes,
               const double* psi0, const int32_t* time_log, int n_log, int n_timestep,
               int chk_step, double chk_thr, double* psi_t) {
  constexpr int V = 1;
  c->graph.reset();
  c->sess.active = false;
  ensure_vectors(c, 1, 1);
  c->out.ensure((size_t)(n_timestep + 1) * 3 * sizeof(double));
  auto* A = c->A.as<Pack<R, V>>();
  auto* X = c->X.as<Pack<R, V>>();
  auto* Y = c->Y.as<Pack<R, V>>();
  upload_states<R>(c, psi0, 1, 1, 0, A);
  reset_counters(c, 0);
  enqueue_corr<R, V>(c, A, nullptr, 1, 0, c->out.as<double>(), counters(c, 0));
  const int64_t n = c->ham.n;
  auto step = [&]() {
    enqueue_expansion<R, V>(c, ex, 1, A, X, Y, nullptr, 0, c->out.as<double>(), counters(c, 0));
  };
  const auto key = plan_key(c, 3, 1, V, ex);
  const double thr = effective_thr(c, chk_thr);
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp);
  std::vector<double> host;
  int done = 0;  // steps enqueued
  int rows = 0;  // rows of c->out after the initial one
  int ptr = 0;
  int jump_m = 0;
  Expansion jump;
  // tbpm.f90:1071-1092: at iteration t the state after t-1 steps is logged if
  // requested, checked at t == chk_step, then propagated.  Between two such
  // times the state is not needed: on the polynomial route the m steps are one
  // expansion of about tau*a*m terms (512 x 480 graphene, one state, 64 steps
  // between frames: 260 terms instead of 1216).
  // Long intervals are taken in pieces: the weights of a piece cost the host the
  // square of its length (512 steps: about 2 ms, beside 1700 terms on the device).
  constexpr int kMaxJump = 512;
  auto advance_to = [&](int target) {
    while (poly && target > done) {
      const int m = std::min(target - done, kMaxJump);
      if (m != jump_m) {
        jump_m = m;
        jump = power_expansion(pp, m);
      }
      enqueue_expansion<R, V>(c, jump, 1, A, X, Y, nullptr, 0, c->out.as<double>(),
                              counters(c, 0));
      ++rows;
      done += m;
    }
    if (target > done) {
      run_steps(c, target - done, key, step);
      rows += target - done;
      done = target;
    }
  };
  // A logged state is converted into one of two staging buffers; its copy to the
  // host (which blocks the calling thread) is issued on a second stream after
  // the next propagation has been enqueued, so that both run at the same time.
  // (Five frames of 8 MB: 25 ms of which 15 were on the device.)
  FrameCopies frames(c, (size_t)n * 16);
  for (int t = 1; t <= n_timestep; ++t) {
    if (ptr < n_log && time_log[ptr] == t - 1) {
      advance_to(t - 1);
      frames.flush();
      deinterleave_kernel<R><<<blocks_for(n, 256), 256, 0, c->stream>>>(
          reinterpret_cast<const typename Cx<R>::t*>(A), 1, n, 1, 0, frames.next());
      TBPM_CK(cudaGetLastError());
      c->launches++;
      frames.stage(psi_t + 2 * (size_t)ptr * n);
      if (ptr < n_log - 1) ++ptr;
      else ptr = n_log;  // further matches impossible (sorted, unique)
    }
    if (t == chk_step) {
      advance_to(t - 1);
      read_out(c, host, (size_t)(rows + 1) * 3);
      if (const int bad_ = norm_broken(host[(size_t)rows * 3 + 2], host[2], thr))
        raise_norm("tbpm_psi_t", t, bad_);
    }
  }
  if (ptr < n_log && time_log[ptr] == n_timestep) {
    advance_to(n_timestep);
    frames.flush();
    deinterleave_kernel<R><<<blocks_for(n, 256), 256, 0, c->stream>>>(
        reinterpret_cast<const typename Cx<R>::t*>(A), 1, n, 1, 0, frames.next());
    TBPM_CK(cudaGetLastError());
    c->launches++;
    frames.stage(psi_t + 2 * (size_t)ptr * n);
  }
  frames.flush();
  TBPM_CK(cudaStreamSynchronize(c->stream));
  check_status(c);
}

// ---- Fermi coefficients (funcs.f90:60-123) --------------------------------------

// In-place iterative radix-2 FFT, X_k = sum_n x_n exp(sgn*2*pi*i*k*n/N).
void fft_radix2(std::vector<double>& re, std::vector<double>& im, int sgn) {
  const size_t n = re.size();
  for (size_t i = 1, j = 0; i < n; ++i) {
    size_t bit = n >> 1;
    for (; j & bit; bit >>= 1) j ^= bit;
    j ^= bit;
    if (i < j) {
      std::swap(re[i], re[j]);
      std::swap(im[i], im[j]);
    }
  }
  const double pi = 3.14159265358979323846;
  for (size_t len = 2; len <= n; len <<= 1) {
    const double ang = sgn * 2 * pi / (double)len;
    for (size_t i = 0; i < n; i += len) {
      for (size_t k = 0; k < len / 2; ++k) {
        const double wr = std::cos(ang * (double)k), wi = std::sin(ang * (double)k);
        const size_t a = i + k, b = i + k + len / 2;
        const double tr = re[b] * wr - im[b] * wi;
        const double ti = re[b] * wi + im[b] * wr;
        re[b] = re[a] - tr;
        im[b] = im[a] - ti;
        re[a] += tr;
        im[a] += ti;
      }
    }
  }
}

int fermi_coef(int nr_fermi, double beta, double mu, bool one_minus, double eps,
               std::vector<double>& coef) {
  if (nr_fermi < 4 || (nr_fermi & (nr_fermi - 1)))
    throw Error{TBPM_ERR_ARG, "nr_Fermi_fft_steps must be a power of two >= 4"};
  const double pi = 3.14159265358979323846;
  std::vector<double> re(nr_fermi), im(nr_fermi, 0.0);
  const double r0 = 2 * pi / nr_fermi;
  for (int i = 0; i < nr_fermi; ++i) {
    const double e = std::cos(i * r0);
    double f;  // funcs.f90:36-57
    if (e >= mu) {
      const double x = std::exp(beta * (mu - e));
      f = x / (1 + x);
    } else {
      const double x = std::exp(beta * (e - mu));
      f = 1 / (1 + x);
    }
    re[i] = one_minus ? 1.0 - f : f;
  }
  fft_radix2(re, im, -1);
  int n_cheb = nr_fermi / 2;
  coef.assign(nr_fermi + 1, 0.0);
  const double q = pi / n_cheb;
  const double cotq = std::cos(q) / std::sin(q);
  for (int k = 0; k < n_cheb; ++k) {
    // Jackson kernel with the first element halved (kpm.f90:8-29)
    const double g =
        k == 0 ? 0.5 : ((double)(n_cheb - k) * std::cos(q * k) + cotq * std::sin(q * k)) / n_cheb;
    coef[k] = g * re[k] / n_cheb;
  }
  for (int i = 0; i < n_cheb; ++i) {
    if (std::fabs(coef[i]) < eps && std::fabs(coef[i + 1]) < eps) {
      n_cheb = i + 1;
      break;
    }
  }
  coef.resize(n_cheb);
  return n_cheb;
}

// ---- Hamiltonian upload --------------------------------------------------------

// ---- upload of a host CSR: checked and split into H = D + O on the device ----

// Per row: status bit 1 when indptr decreases or leaves [0, nnz], bit 2 when a
// column index is out of range; off[r] = entries off the diagonal; *n_diag
// counts rows with a diagonal entry.
__global__ void csr_check_count_kernel(const int32_t* indptr, const int32_t* indices,
                                       int64_t n, int64_t nnz, int32_t* off,
                                       unsigned* status, unsigned long long* n_diag) {
  unsigned st = 0;
  unsigned long long nd = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = indptr[r], b = indptr[r + 1];
    if (a < 0 || b > nnz || b < a) {
      st |= 1u;
      off[r] = 0;
      continue;
    }
    int d = 0;
    for (int64_t j = a; j < b; ++j) {
      const int32_t cj = indices[j];
      if (cj < 0 || (int64_t)cj >= n) st |= 2u;
      d += (cj == r);
    }
    off[r] = (int32_t)(b - a - d);
    nd += d > 0;
  }
  if (st) atomicOr(status, st);
  for (int w = 16; w > 0; w >>= 1) nd += __shfl_xor_sync(0xffffffffu, nd, w);
  if ((threadIdx.x & 31) == 0 && nd) atomicAdd(n_diag, nd);
}

// Writes O (entries in CSR order, diagonal skipped) and D (diagonal entries
// summed from 0 in CSR order) in precision R, and dx/dy of O when given.
template <typename R>
__global__ void csr_split_kernel(const int32_t* indptr, const int32_t* indices,
                                 const double2* hop, const double* dx, const double* dy,
                                 int64_t n, const int64_t* off, int32_t* o_indptr,
                                 int32_t* o_indices, typename Cx<R>::t* o_hop, R* o_dx, R* o_dy,
                                 typename Cx<R>::t* diag) {
  using C = typename Cx<R>::t;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    int64_t p = off[r];
    o_indptr[r] = (int32_t)p;
    if (r == n - 1) o_indptr[n] = (int32_t)off[n];
    double gr = 0.0, gi = 0.0;
    for (int64_t j = indptr[r]; j < indptr[r + 1]; ++j) {
      const int32_t cj = indices[j];
      const double2 h = hop[j];
      if (cj == r) {
        gr += h.x;
        gi += h.y;
        continue;
      }
      o_indices[p] = cj;
      C v;
      v.x = (R)h.x;
      v.y = (R)h.y;
      o_hop[p] = v;
      if (o_dx) {
        o_dx[p] = (R)dx[j];
        o_dy[p] = (R)dy[j];
      }
      ++p;
    }
    if (diag) {
      C v;
      v.x = (R)gr;
      v.y = (R)gi;
      diag[r] = v;
    }
  }
}

void ham_upload(tbpm_ctx* c, const int32_t* indptr, const int32_t* indices, const double* hop,
                int64_t n, int64_t nnz, const double* dx, const double* dy, double rescale) {
  if (n < 1) throw Error{TBPM_ERR_ARG, "empty Hamiltonian (n_rows < 1)"};
  if (nnz < 0 || nnz > INT32_MAX) throw Error{TBPM_ERR_ARG, "nnz out of the int32 range"};
  if (n > INT32_MAX) throw Error{TBPM_ERR_ARG, "n_rows out of the int32 range"};
  if (indptr[0] != 0) throw Error{TBPM_ERR_ARG, "indptr[0] must be 0"};
  if ((int64_t)indptr[n] != nnz) throw Error{TBPM_ERR_ARG, "indptr[n_rows] != nnz"};
  // captured graphs stay valid: their key covers every buffer pointer and
  // Hamiltonian property they bake in, so a re-upload of the same shape reuses them
  c->sess.active = false;
  Ham& h = c->ham;
  h.n = 0;
  cudaStream_t st = c->stream;
  const bool with_dxy = dx && dy;
  // device copies of the caller's arrays (one grow-only buffer of the context,
  // 256-byte aligned parts), then the checks and the split run here
  const size_t nz = (size_t)std::max<int64_t>(nnz, 1);
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t b_ip = al((size_t)(n + 1) * 4), b_ix = al(nz * 4), b_hop = al(nz * 16);
  const size_t b_d = with_dxy ? al(nz * 8) : 0, b_cnt = al((size_t)n * 4);
  const size_t b_off = al((size_t)(n + 1) * 8), b_fl = 256, b_scan = al(scan_bytes(n));
  c->raw.ensure(b_ip + b_ix + b_hop + 2 * b_d + b_cnt + b_off + b_fl + b_scan);
  char* q = c->raw.as<char>();
  int32_t* rip = reinterpret_cast<int32_t*>(q);
  int32_t* rix = reinterpret_cast<int32_t*>(q += b_ip);
  double2* rhop = reinterpret_cast<double2*>(q += b_ix);
  double* rdx = reinterpret_cast<double*>(q += b_hop);
  double* rdy = reinterpret_cast<double*>(q += b_d);
  int32_t* cnt = reinterpret_cast<int32_t*>(q += b_d);
  int64_t* offs = reinterpret_cast<int64_t*>(q += b_cnt);
  unsigned* status = reinterpret_cast<unsigned*>(q += b_off);
  unsigned long long* n_diag = reinterpret_cast<unsigned long long*>(q + 8);
  TBPM_CK(cudaMemcpyAsync(rip, indptr, (size_t)(n + 1) * 4, cudaMemcpyHostToDevice, st));
  if (nnz) {
    TBPM_CK(cudaMemcpyAsync(rix, indices, (size_t)nnz * 4, cudaMemcpyHostToDevice, st));
    TBPM_CK(cudaMemcpyAsync(rhop, hop, (size_t)nnz * 16, cudaMemcpyHostToDevice, st));
    if (with_dxy) {
      TBPM_CK(cudaMemcpyAsync(rdx, dx, (size_t)nnz * 8, cudaMemcpyHostToDevice, st));
      TBPM_CK(cudaMemcpyAsync(rdy, dy, (size_t)nnz * 8, cudaMemcpyHostToDevice, st));
    }
  }
  TBPM_CK(cudaMemsetAsync(status, 0, 16, st));
  const int grid = (int)std::min<int64_t>(blocks_for(n, 256), (int64_t)kSMs * 16);
  csr_check_count_kernel<<<grid, 256, 0, st>>>(rip, rix, n, nnz, cnt, status, n_diag);
  TBPM_CK(cudaGetLastError());
  unsigned long long host_flags[2] = {0, 0};
  TBPM_CK(cudaMemcpyAsync(host_flags, status, 16, cudaMemcpyDeviceToHost, st));
  TBPM_CK(cudaStreamSynchronize(st));
  const unsigned bad = (unsigned)(host_flags[0] & 0xffffffffu);
  if (bad & 1u) throw Error{TBPM_ERR_ARG, "indptr must be non-decreasing"};
  if (bad & 2u) throw Error{TBPM_ERR_ARG, "column index out of range"};
  const int64_t n_off = scan_counts(cnt, n, offs, reinterpret_cast<int64_t*>(q + b_fl), st);
  const bool has_diag = host_flags[1] > 0;
  const size_t rs = c->opts.precision == TBPM_PREC_FP64 ? 8 : 4;
  h.indptr.ensure((size_t)(n + 1) * 4);
  h.indices.ensure((size_t)std::max<int64_t>(n_off, 1) * 4);
  h.hop.ensure((size_t)std::max<int64_t>(n_off, 1) * 2 * rs);
  if (has_diag) h.diag.ensure((size_t)n * 2 * rs);
  if (with_dxy) {
    h.dx.ensure((size_t)std::max<int64_t>(n_off, 1) * rs);
    h.dy.ensure((size_t)std::max<int64_t>(n_off, 1) * rs);
  }
  auto split = [&](auto tag) {
    using R = decltype(tag);
    using C = typename Cx<R>::t;
    csr_split_kernel<R><<<grid, 256, 0, st>>>(
        rip, rix, rhop, with_dxy ? rdx : nullptr, with_dxy ? rdy : nullptr, n, offs,
        h.indptr.as<int32_t>(), h.indices.as<int32_t>(), h.hop.as<C>(),
        with_dxy ? h.dx.as<R>() : nullptr, with_dxy ? h.dy.as<R>() : nullptr,
        has_diag ? h.diag.as<C>() : nullptr);
  };
  if (rs == 8)
    split(double{});
  else
    split(float{});
  TBPM_CK(cudaGetLastError());
  TBPM_CK(cudaStreamSynchronize(st));
  h.has_diag = has_diag;
  h.has_dxy = with_dxy;
  h.prec = c->opts.precision;
  h.n = n;
  h.nnz = n_off;
  h.rescale = rescale;
  ++h.gen;
}

}  // namespace

// ---------------------------------------------------------------------------
// drivers used by the C ABI
// ---------------------------------------------------------------------------

void drv_ham_upload(tbpm_ctx* c, const int32_t* indptr, const int32_t* indices,
                    const double* hop, int64_t n, int64_t nnz, const double* dx,
                    const double* dy, double rescale) {
  Phase phase("tbpm_ham_upload");
  if (!indptr || (nnz > 0 && (!indices || !hop))) throw Error{TBPM_ERR_ARG, "null CSR array"};
  ham_upload(c, indptr, indices, hop, n, nnz, dx, dy, rescale);
}

void drv_dos(tbpm_ctx* c, const double* bes, int n_bes, const double* wf0, int n_states,
             int seed, int rank, int n_ran_samples, int n_timestep, int chk_step,
             double chk_thr, double* corr, double* corr_per_state) {
  Phase phase("tbpm_dos");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_timestep < 1) throw Error{TBPM_ERR_ARG, "n_timestep must be >= 1"};
  if (n_states < 1) throw Error{TBPM_ERR_ARG, "n_ran_samples must be >= 1"};
  if (!corr) throw Error{TBPM_ERR_ARG, "null output"};
  c->launches = 0;
  c->model_bytes = 0;
  std::fill(corr, corr + 2 * (size_t)(n_timestep + 1), 0.0);
  const Expansion ex = time_step_expansion(bes, n_bes);
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp);
  const int B = batch_size(c);
  for (int s0 = 0; s0 < n_states; s0 += B) {
    const int ns = std::min(B, n_states - s0);
    StateKeys keys{};
    const StateKeys* kp = nullptr;
    if (!wf0) {
      keys = make_keys(seed, s0 + 1, ns, rank, n_ran_samples);
      kp = &keys;
    }
    const double* hw = wf0 ? wf0 + 2 * (size_t)s0 * c->ham.n : nullptr;
    dispatch(c->ham.prec, pick_V(c->ham.prec, ns, ns, c->opts.vector_width), [&](auto tag) {
      using P = decltype(tag);
      if (poly && moments_pay(c, pp, n_timestep, ns, ns, 2.2e-6))
        dos_moments<typename P::Real, P::V>(c, pp, ns, kp, hw, n_timestep, chk_step, chk_thr,
                                            n_states, corr, corr_per_state, s0);
      else
        dos_batch<typename P::Real, P::V>(c, ex, ns, kp, hw, n_timestep, chk_step, chk_thr,
                                          n_states, corr, corr_per_state, s0, n_states);
    });
  }
}

void drv_ac(tbpm_ctx* c, const double* bes, int n_bes, double beta, double mu,
            const double* wf0, int n_states, int seed, int rank, int n_ran_samples,
            int n_timestep, int nr_fermi, double fermi_precision, int chk_step, double chk_thr,
            double* corr) {
  Phase phase("tbpm_accond");
  require_ham(c, true);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_timestep < 1) throw Error{TBPM_ERR_ARG, "n_timestep must be >= 1"};
  if (n_states < 1) throw Error{TBPM_ERR_ARG, "n_ran_samples must be >= 1"};
  c->launches = 0;
  c->model_bytes = 0;
  std::fill(corr, corr + 2 * 4 * (size_t)n_timestep, 0.0);
  std::vector<double> cf, comf;
  const int nf = fermi_coef(nr_fermi, beta, mu, false, fermi_precision, cf);
  const int nomf = fermi_coef(nr_fermi, beta, mu, true, fermi_precision, comf);
  if (nf < 3 || nomf < 3) throw Error{TBPM_ERR_ARG, "Fermi expansion shorter than 3 terms"};
  const Expansion ex_time = time_step_expansion(bes, n_bes);
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp);
  const int B = std::min(batch_size(c), kMaxCols / 3);
  for (int s0 = 0; s0 < n_states; s0 += B) {
    const int nb = std::min(B, n_states - s0);
    unsigned long long set_b = 0;
    for (int b = 2 * nb; b < 3 * nb; ++b) set_b |= 1ull << b;
    const Expansion ex_fermi = fermi_expansion(comf.data(), nomf, cf.data(), nf, set_b);
    StateKeys keys{};
    const StateKeys* kp = nullptr;
    if (!wf0) {
      keys = make_keys(seed, s0 + 1, nb, rank, n_ran_samples);
      kp = &keys;
    }
    const double* hw = wf0 ? wf0 + 2 * (size_t)s0 * c->ham.n : nullptr;
    dispatch(c->ham.prec, pick_V(c->ham.prec, 3 * nb, nb, c->opts.vector_width), [&](auto tag) {
      using P = decltype(tag);
      ac_batch<typename P::Real, P::V>(c, ex_time, ex_fermi, nb, kp, hw, n_timestep, chk_step,
                                       chk_thr, n_states, corr, poly ? &pp : nullptr);
    });
  }
  trim(c->A);
}


// The states [first_state, first_state + n_states) of a DC run of n_avg states:
// their contributions, each divided by n_avg, are added to dos_corr / dc_corr
// in state order (zeroed first when `zero`).  Seeded states (wf0 == NULL)
// follow the seed rule with the run's n_ran_samples; wf0 holds this part's
// states.
void drv_dc_part(tbpm_ctx* c, const double* bes, int n_bes, const double* wf0, int first_state,
                 int n_states, int n_avg, int seed, int rank, int n_ran_samples, int n_timestep,
                 double t_step, const double* energies, int n_energies, const int32_t* en_inds,
                 int n_en_inds, int chk_step, double chk_thr, double* dos_corr, double* dc_corr,
                 bool zero) {
  Phase phase("tbpm_dccond");
  require_ham(c, true);
  if (first_state < 0 || n_avg < 1) throw Error{TBPM_ERR_ARG, "bad state range"};
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_timestep < 1) throw Error{TBPM_ERR_ARG, "n_timestep must be >= 1"};
  if (n_states < 1) throw Error{TBPM_ERR_ARG, "n_ran_samples must be >= 1"};
  if (n_en_inds < 0 || n_en_inds > n_energies || (n_en_inds > 0 && (!en_inds || !energies)))
    throw Error{TBPM_ERR_ARG, "bad energy selection"};
  if (!dos_corr || !dc_corr) throw Error{TBPM_ERR_ARG, "null output"};
  std::vector<double> en_sel(n_en_inds);
  for (int i = 0; i < n_en_inds; ++i) {
    if (en_inds[i] < 0 || en_inds[i] >= n_energies)
      throw Error{TBPM_ERR_ARG, "energy index out of range"};
    en_sel[i] = energies[en_inds[i]];
  }
  c->launches = 0;
  c->model_bytes = 0;
  if (zero) {
    std::fill(dos_corr, dos_corr + 2 * (size_t)n_timestep, 0.0);
    std::fill(dc_corr, dc_corr + 2 * 2 * (size_t)n_energies * n_timestep, 0.0);
  }
  const Expansion ex_fwd = time_step_expansion(bes, n_bes);
  // states per batch: the QE block (N x n_en x nb complex) must fit in memory.
  // When not even one state's block fits, the energies are taken in chunks:
  // every chunk repeats the propagation of the batch for its own energies
  // (the DOS correlation is taken from the first chunk only).
  int B = std::min(batch_size(c), kMaxCols / 2);
  int en_chunk = std::max(n_en_inds, 1);
  {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && n_en_inds > 0) {
      // per state: its QE block (N x n_en complex) plus its two columns in
      // the window ring (kMaxWindow + 1 slots) and in X, Y, wf0; buffers this
      // context already holds count as free
      const size_t held = c->qe.bytes + c->A.bytes + c->X.bytes + c->Y.bytes + c->wf0.bytes;
      const size_t avail = free_b + held;
      const size_t cx = 2 * real_size(c->ham.prec);
      const size_t ring = (size_t)c->ham.n * (size_t)(kMaxWindow + 4) * 2 * cx;
      const size_t qe_1 = (size_t)c->ham.n * cx;  // one energy of one state
      const size_t reserve = (size_t)6 << 30;
      size_t budget = avail > 2 * reserve ? avail - reserve : avail / 2;
      if (c->opts.dc_budget_gb > 0)
        budget = std::min(budget, (size_t)(c->opts.dc_budget_gb * 1073741824.0));
      const size_t per_state = (size_t)n_en_inds * qe_1 + ring;
      const int fit = (int)std::min<size_t>((size_t)B, budget / std::max<size_t>(per_state, 1));
      if (fit >= 1) {
        B = fit;
      } else {
        B = 1;
        en_chunk = budget > ring ? (int)std::min<size_t>((budget - ring) / qe_1, n_en_inds) : 0;
        if (en_chunk < 1)
          throw Error{TBPM_ERR_OOM,
                      "tbpm_dccond: one state's propagation ring does not fit in device memory"};
      }
    }
    (void)cudaGetLastError();
  }
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp);
  for (int s0 = 0; s0 < n_states; s0 += B) {
    const int nb = std::min(B, n_states - s0);
    Expansion ex_pm = ex_fwd;
    for (int b = nb; b < 2 * nb; ++b) ex_pm.neg_mask |= 1ull << b;
    StateKeys keys{};
    const StateKeys* kp = nullptr;
    if (!wf0) {
      keys = make_keys(seed, first_state + s0 + 1, nb, rank, n_ran_samples);
      kp = &keys;
    }
    const double* hw = wf0 ? wf0 + 2 * (size_t)s0 * c->ham.n : nullptr;
    for (int e0 = 0; e0 < std::max(n_en_inds, 1); e0 += en_chunk) {
      const std::vector<double> part(
          en_sel.begin() + std::min(e0, n_en_inds),
          en_sel.begin() + std::min(e0 + en_chunk, n_en_inds));
      dispatch(c->ham.prec, pick_V(c->ham.prec, 2 * nb, nb, c->opts.vector_width),
               [&](auto tag) {
                 using P = decltype(tag);
                 dc_batch<typename P::Real, P::V>(c, ex_pm, ex_fwd, nb, kp, hw, n_timestep,
                                                  t_step, part, chk_step, chk_thr, n_avg,
                                                  n_energies, dos_corr, dc_corr, nullptr,
                                                  "tbpm_dccond", e0, e0 == 0,
                                                  poly ? &pp : nullptr);
               });
    }
  }
  trim(c->A);
}

void drv_dc(tbpm_ctx* c, const double* bes, int n_bes, const double* wf0, int n_states,
            int seed, int rank, int n_ran_samples, int n_timestep, double t_step,
            const double* energies, int n_energies, const int32_t* en_inds, int n_en_inds,
            int chk_step, double chk_thr, double* dos_corr, double* dc_corr) {
  drv_dc_part(c, bes, n_bes, wf0, 0, n_states, n_states, seed, rank, n_ran_samples, n_timestep,
              t_step, energies, n_energies, en_inds, n_en_inds, chk_step, chk_thr, dos_corr,
              dc_corr, true);
}


void drv_dyn_pol(tbpm_ctx* c, const double* bes, int n_bes, double beta, double mu,
                 const double* sx, const double* sy, const double* sz, const double* q_points,
                 int n_q, const double* wf0, int n_states, int seed, int rank,
                 int n_ran_samples, int n_timestep, int nr_fermi, double fermi_precision,
                 int chk_step, double chk_thr, double* corr) {
  Phase phase("tbpm_dyn_pol");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_timestep < 1) throw Error{TBPM_ERR_ARG, "n_timestep must be >= 1"};
  if (n_states < 1) throw Error{TBPM_ERR_ARG, "n_ran_samples must be >= 1"};
  if (!sx || !sy || !sz) throw Error{TBPM_ERR_ARG, "site coordinates required"};
  if (!q_points || n_q < 1) throw Error{TBPM_ERR_ARG, "at least one q-point required"};
  if (!corr) throw Error{TBPM_ERR_ARG, "null output"};
  c->launches = 0;
  c->model_bytes = 0;
  std::fill(corr, corr + (size_t)n_q * n_timestep, 0.0);
  std::vector<double> cf, comf;
  const int nf = fermi_coef(nr_fermi, beta, mu, false, fermi_precision, cf);
  const int nomf = fermi_coef(nr_fermi, beta, mu, true, fermi_precision, comf);
  if (nf < 3 || nomf < 3) throw Error{TBPM_ERR_ARG, "Fermi expansion shorter than 3 terms"};
  const Expansion ex_time = time_step_expansion(bes, n_bes);
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp);
  const int64_t n = c->ham.n;
  ScratchScope scope(c->scratch);
  TempMem sites(c->scratch);
  sites.ensure((size_t)n * 3 * sizeof(double));
  double* dsx = sites.as<double>();
  TBPM_CK(cudaMemcpyAsync(dsx, sx, n * 8, cudaMemcpyHostToDevice, c->stream));
  TBPM_CK(cudaMemcpyAsync(dsx + n, sy, n * 8, cudaMemcpyHostToDevice, c->stream));
  TBPM_CK(cudaMemcpyAsync(dsx + 2 * n, sz, n * 8, cudaMemcpyHostToDevice, c->stream));
  const int B = std::min(std::min(batch_size(c), n_states), kMaxCols / 2);
  const int nq_max = std::max(1, kMaxCols / B - 1);
  for (int q0 = 0; q0 < n_q; q0 += nq_max) {
    const int nq = std::min(nq_max, n_q - q0);
    QBlock qb{};
    for (int k = 0; k < nq; ++k)
      for (int d = 0; d < 3; ++d) qb.q[k][d] = q_points[3 * (q0 + k) + d];
    for (int s0 = 0; s0 < n_states; s0 += B) {
      const int nb = std::min(B, n_states - s0);
      const int ld = (nq + 1) * nb;
      unsigned long long set_b = 0;
      for (int col = nq * nb; col < ld; ++col) set_b |= 1ull << col;
      const Expansion ex_fermi = fermi_expansion(comf.data(), nomf, cf.data(), nf, set_b);
      StateKeys keys{};
      const StateKeys* kp = nullptr;
      if (!wf0) {
        keys = make_keys(seed, s0 + 1, nb, rank, n_ran_samples);
        kp = &keys;
      }
      const double* hw = wf0 ? wf0 + 2 * (size_t)s0 * n : nullptr;
      dispatch(c->ham.prec, pick_V(c->ham.prec, ld, nb, c->opts.vector_width), [&](auto tag) {
        using P = decltype(tag);
        dynpol_batch<typename P::Real, P::V>(c, ex_time, ex_fermi, nb, nq, qb, dsx, dsx + n,
                                             dsx + 2 * n, kp, hw, n_timestep, chk_step, chk_thr,
                                             n_states, q0, n_q, corr, poly ? &pp : nullptr);
      });
    }
  }
  c->graph.reset();  // the graphs refer to the site buffer of this call
  trim(c->A);
}

void drv_eigenstates(tbpm_ctx* c, const double* bes, int n_bes, const double* wf0,
                     int n_states, int seed, int rank, int n_ran_samples, int n_timestep,
                     double t_step, const double* energies, int n_energies, int chk_step,
                     double chk_thr, double* wf_qe) {
  Phase phase("tbpm_eigenstates");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_timestep < 1) throw Error{TBPM_ERR_ARG, "n_timestep must be >= 1"};
  if (n_states < 1) throw Error{TBPM_ERR_ARG, "n_ran_samples must be >= 1"};
  if (!energies || n_energies < 1) throw Error{TBPM_ERR_ARG, "at least one energy required"};
  if (!wf_qe) throw Error{TBPM_ERR_ARG, "null output"};
  c->launches = 0;
  c->model_bytes = 0;
  const int64_t n = c->ham.n;
  const std::vector<double> en_sel(energies, energies + n_energies);
  const Expansion ex_fwd = time_step_expansion(bes, n_bes);
  ScratchScope scope(c->scratch);
  TempMem acc(c->scratch);
  acc.ensure((size_t)n * n_energies * sizeof(double));
  TBPM_CK(cudaMemsetAsync(acc.p, 0, (size_t)n * n_energies * sizeof(double), c->stream));
  int B = std::min(batch_size(c), kMaxCols / 2);
  {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) {
      const size_t cx = 2 * real_size(c->ham.prec);
      const size_t per_state =
          (size_t)n * ((size_t)n_energies * cx + (size_t)(kMaxWindow + 4) * 2 * cx);
      const size_t reserve = (size_t)6 << 30;
      const size_t budget = free_b > 2 * reserve ? free_b - reserve : free_b / 2;
      B = std::min(B, (int)std::max<size_t>(1, budget / std::max<size_t>(per_state, 1)));
    }
    (void)cudaGetLastError();
  }
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp);
  for (int s0 = 0; s0 < n_states; s0 += B) {
    const int nb = std::min(B, n_states - s0);
    Expansion ex_pm = ex_fwd;
    for (int b = nb; b < 2 * nb; ++b) ex_pm.neg_mask |= 1ull << b;
    StateKeys keys{};
    const StateKeys* kp = nullptr;
    if (!wf0) {
      keys = make_keys(seed, s0 + 1, nb, rank, n_ran_samples);
      kp = &keys;
    }
    const double* hw = wf0 ? wf0 + 2 * (size_t)s0 * n : nullptr;
    dispatch(c->ham.prec, pick_V(c->ham.prec, 2 * nb, nb, c->opts.vector_width), [&](auto tag) {
      using P = decltype(tag);
      dc_batch<typename P::Real, P::V>(c, ex_pm, ex_fwd, nb, kp, hw, n_timestep, t_step, en_sel,
                                       chk_step, chk_thr, n_states, n_energies, nullptr,
                                       nullptr, acc.as<double>(), "tbpm_eigenstates", 0, true,
                                       poly ? &pp : nullptr);
    });
  }
  // acc[r][i] is the Fortran (n_energies, n) layout of wf_QE
  TBPM_CK(cudaMemcpyAsync(wf_qe, acc.p, (size_t)n * n_energies * sizeof(double),
                          cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
}

void drv_kbdc(tbpm_ctx* c, const double* wf0, int n_states, int seed, int rank,
              int n_ran_samples, int n_kernel, int direction, double* mu) {
  Phase phase("tbpm_kbdc");
  require_ham(c, true);
  if (n_states < 1) throw Error{TBPM_ERR_ARG, "n_ran_samples must be >= 1"};
  if (n_kernel < 2) throw Error{TBPM_ERR_ARG, "n_kernel must be >= 2"};
  if (direction != 1 && direction != 2)
    throw Error{TBPM_ERR_ARG, "Error: wrong direction! (1: x, 2: y)"};
  if (!mu) throw Error{TBPM_ERR_ARG, "null output"};
  if (c->ham.n > (int64_t)INT32_MAX) throw Error{TBPM_ERR_ARG, "too many orbitals for the GEMM"};
  c->launches = 0;
  c->model_bytes = 0;
  c->graph.reset();
  c->sess.active = false;
  const int64_t n = c->ham.n;
  const size_t cs = 2 * real_size(c->ham.prec);
  const int kc = std::min(n_kernel, 128);
  ensure_vectors(c, 1, 1);
  c->A.ensure((size_t)n * n_kernel * cs);
  c->X.ensure((size_t)n * kc * cs);
  c->Y.ensure((size_t)n * 5 * cs);
  {
    const PqSplit sp = pq_split(c, n, kc, n_kernel);
    c->qe.ensure((size_t)sp.slices * kc * n_kernel * sizeof(double2));
  }
  // kpm.f90:8-29 Jackson kernel, first element halved
  std::vector<double> g(n_kernel);
  g[0] = 0.5;
  const double pi = 3.14159265358979323846;
  const double q = pi / n_kernel;
  const double cotq = std::cos(q) / std::sin(q);
  for (int k = 1; k < n_kernel; ++k)
    g[k] = ((double)(n_kernel - k) * std::cos(q * k) + cotq * std::sin(q * k)) / n_kernel;
  ScratchScope scope(c->scratch);
  TempMem gdev(c->scratch), mdev(c->scratch);
  gdev.ensure(sizeof(double) * n_kernel);
  mdev.ensure(sizeof(double2) * (size_t)n_kernel * n_kernel);
  TBPM_CK(cudaMemcpyAsync(gdev.p, g.data(), sizeof(double) * n_kernel, cudaMemcpyHostToDevice,
                          c->stream));
  TBPM_CK(cudaMemsetAsync(mdev.p, 0, sizeof(double2) * (size_t)n_kernel * n_kernel, c->stream));
  for (int s = 0; s < n_states; ++s) {
    if (wf0) {
      if (c->ham.prec == TBPM_PREC_FP64)
        upload_states<double>(c, wf0 + 2 * (size_t)s * n, 1, 1, 0, c->wf0.p);
      else
        upload_states<float>(c, wf0 + 2 * (size_t)s * n, 1, 1, 0, c->wf0.p);
    } else {
      const StateKeys keys = make_keys(seed, s + 1, 1, rank, n_ran_samples);
      if (c->ham.prec == TBPM_PREC_FP64)
        gen_states<double, 1>(c, keys, 1, c->opts.state_kind, c->wf0.as<Pack<double, 1>>());
      else
        gen_states<float, 1>(c, keys, 1, c->opts.state_kind, c->wf0.as<Pack<float, 1>>());
    }
    if (c->ham.prec == TBPM_PREC_FP64)
      kbdc_state<double>(c, n_kernel, direction, gdev.as<double>(), 1.0 / n_states,
                         mdev.as<double2>());
    else
      kbdc_state<float>(c, n_kernel, direction, gdev.as<double>(), 1.0 / n_states,
                        mdev.as<double2>());
  }
  TBPM_CK(cudaMemcpyAsync(mu, mdev.p, sizeof(double2) * (size_t)n_kernel * n_kernel,
                          cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
}

void drv_haydock(tbpm_ctx* c, const int32_t* sites, int n_sites, const double* wf_sites,
                 int n_samples, int n_depth, double h_rescale, double* coefa, double* coefb) {
  Phase phase("tbpm_haydock");
  require_ham(c, false);
  if (!sites || n_sites < 1 || !wf_sites || n_samples < 1)
    throw Error{TBPM_ERR_ARG, "site indices and site amplitudes required"};
  if (n_depth < 1) throw Error{TBPM_ERR_ARG, "recursion depth must be >= 1"};
  if (!coefa || !coefb) throw Error{TBPM_ERR_ARG, "null output"};
  const int64_t n = c->ham.n;
  for (int i = 0; i < n_sites; ++i)
    if (sites[i] < 0 || sites[i] >= n) throw Error{TBPM_ERR_ARG, "site index out of range"};
  c->launches = 0;
  c->model_bytes = 0;
  c->graph.reset();
  c->sess.active = false;
  const size_t cs = 2 * real_size(c->ham.prec);
  c->wf0.ensure((size_t)n * cs);
  c->X.ensure((size_t)n * cs);
  c->Y.ensure((size_t)n * cs);
  ScratchScope scope(c->scratch);
  TempMem dsites(c->scratch), dvals(c->scratch), sc(c->scratch);
  dsites.ensure(sizeof(int32_t) * n_sites);
  dvals.ensure(sizeof(double2) * n_sites);
  sc.ensure(sizeof(double) * 3 * (size_t)n_depth);
  TBPM_CK(cudaMemcpyAsync(dsites.p, sites, sizeof(int32_t) * n_sites, cudaMemcpyHostToDevice,
                          c->stream));
  std::fill(coefa, coefa + 2 * (size_t)n_depth, 0.0);
  std::fill(coefb, coefb + n_depth, 0.0);
  std::vector<double> host(3 * (size_t)n_depth);
  for (int s = 0; s < n_samples; ++s) {
    TBPM_CK(cudaMemsetAsync(c->wf0.p, 0, (size_t)n * cs, c->stream));
    TBPM_CK(cudaMemcpyAsync(dvals.p, wf_sites + 2 * (size_t)s * n_sites,
                            sizeof(double2) * n_sites, cudaMemcpyHostToDevice, c->stream));
    const int grid = (n_sites + 255) / 256;
    if (c->ham.prec == TBPM_PREC_FP64) {
      scatter_sites_kernel<double><<<grid, 256, 0, c->stream>>>(
          dsites.as<int32_t>(), dvals.as<double2>(), n_sites, c->wf0.as<double2>());
      haydock_state<double>(c, n_depth, h_rescale, sc.as<double>());
    } else {
      scatter_sites_kernel<float><<<grid, 256, 0, c->stream>>>(
          dsites.as<int32_t>(), dvals.as<double2>(), n_sites, c->wf0.as<float2>());
      haydock_state<float>(c, n_depth, h_rescale, sc.as<double>());
    }
    TBPM_CK(cudaGetLastError());
    TBPM_CK(cudaMemcpyAsync(host.data(), sc.p, host.size() * sizeof(double),
                            cudaMemcpyDeviceToHost, c->stream));
    TBPM_CK(cudaStreamSynchronize(c->stream));
    check_status(c);
    for (int d = 0; d < n_depth; ++d) {
      coefa[2 * d] += host[2 * d] / n_samples;
      coefa[2 * d + 1] += host[2 * d + 1] / n_samples;
      coefb[d] += host[2 * (size_t)n_depth + d] / n_samples;
    }
  }
}

// G00(E + i delta) on the energies from the recursion's coefficients.
void drv_haydock_green(tbpm_ctx* c, const double* coefa, const double* coefb, int n_depth,
                       const double* energies, int n_e, double delta, double* g) {
  Phase phase("tbpm_haydock_green");
  if (!coefa || !coefb || !energies || !g || n_depth < 1 || n_e < 1)
    throw Error{TBPM_ERR_ARG, "coefficients, energies and an output required"};
  const size_t n_in = 3 * (size_t)n_depth + n_e;
  c->small.ensure(sizeof(double) * (n_in + 2 * (size_t)n_e + 1));
  double* in = c->small.as<double>();
  double2* out = reinterpret_cast<double2*>(in + ((n_in + 1) & ~(size_t)1));
  std::vector<double> host(coefa, coefa + 2 * (size_t)n_depth);
  host.insert(host.end(), coefb, coefb + n_depth);
  host.insert(host.end(), energies, energies + n_e);
  TBPM_CK(cudaMemcpyAsync(in, host.data(), sizeof(double) * n_in, cudaMemcpyHostToDevice,
                          c->stream));
  haydock_green_kernel<<<blocks_for(n_e, 64), 64, 0, c->stream>>>(
      in, in + 2 * n_depth, n_depth, in + 3 * n_depth, n_e, delta, out);
  TBPM_CK(cudaGetLastError());
  TBPM_CK(cudaMemcpyAsync(g, out, sizeof(double2) * n_e, cudaMemcpyDeviceToHost, c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
}

void drv_cond_from_trace(tbpm_ctx* c, const double* mu_mn, int nk, const double* mu, int n_mu,
                         double h_rescale, double beta, int ne_integral, double* cond) {
  if (!mu_mn || nk < 1 || !cond || (n_mu > 0 && !mu)) throw Error{TBPM_ERR_ARG, "bad arguments"};
  if (ne_integral < 2) throw Error{TBPM_ERR_ARG, "ne_integral must be >= 2"};
  if ((size_t)nk * 2 * sizeof(double) > 200 * 1024)
    throw Error{TBPM_ERR_ARG, "n_kernel too large for the trace kernel (max 12800)"};
  const int ne = ne_integral - 1;
  ScratchScope scope(c->scratch);
  TempMem dmu(c->scratch), dsum(c->scratch);
  dmu.ensure(sizeof(double2) * (size_t)nk * nk);
  dsum.ensure(sizeof(double) * ne);
  TBPM_CK(cudaMemcpyAsync(dmu.p, mu_mn, sizeof(double2) * (size_t)nk * nk,
                          cudaMemcpyHostToDevice, c->stream));
  const size_t smem = (size_t)nk * 2 * sizeof(double);
  qe_smem_attr(gamma_trace_kernel, smem);
  gamma_trace_kernel<<<ne, 256, smem, c->stream>>>(dmu.as<double2>(), nk, ne_integral,
                                                   dsum.as<double>());
  TBPM_CK(cudaGetLastError());
  std::vector<double> sum(ne);
  TBPM_CK(cudaMemcpyAsync(sum.data(), dsum.p, sizeof(double) * ne, cudaMemcpyDeviceToHost,
                          c->stream));
  TBPM_CK(cudaStreamSynchronize(c->stream));
  // final integral over the Fermi distribution (analysis.f90:55-67)
  const double pi = 3.14159265358979323846;
  const double dE = pi / ne_integral;
  for (int i = 0; i < n_mu; ++i) {
    double dcx = 0.0;
    for (int k = 1; k <= ne; ++k) {
      const double e = k * dE;
      const double s = std::sin(e);
      const double div = s * s * s;
      const double en = std::cos(e) * h_rescale;
      double fd;
      if (en >= mu[i]) {
        const double x = std::exp(beta * (mu[i] - en));
        fd = x / (1 + x);
      } else {
        const double x = std::exp(beta * (en - mu[i]));
        fd = 1 / (1 + x);
      }
      dcx += sum[k - 1] * fd * dE / div;
    }
    cond[i] = dcx;
  }
}

void drv_dos_segmented(tbpm_ctx* c, const double* bes, int n_bes, const int64_t* seg_off,
                       int n_seg, int n_states, int seed, int n_timestep, int chk_step,
                       double chk_thr, double* corr, double* corr_per_state) {
  Phase phase("tbpm_dos_segmented");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_timestep < 1) throw Error{TBPM_ERR_ARG, "n_timestep must be >= 1"};
  if (n_states < 1 || n_states > kMaxCols) throw Error{TBPM_ERR_ARG, "1..64 states"};
  if (!seg_off || n_seg < 1 || n_seg > 65535) throw Error{TBPM_ERR_ARG, "1..65535 segments"};
  if (!corr) throw Error{TBPM_ERR_ARG, "null output"};
  std::vector<int64_t> off(seg_off, seg_off + n_seg + 1);
  if (off[0] != 0 || off[n_seg] != c->ham.n)
    throw Error{TBPM_ERR_ARG, "segment offsets must start at 0 and end at n_rows"};
  for (int k = 0; k < n_seg; ++k)
    if (off[k + 1] < off[k]) throw Error{TBPM_ERR_ARG, "segment offsets must not decrease"};
  c->launches = 0;
  c->model_bytes = 0;
  const Expansion ex = time_step_expansion(bes, n_bes);
  PolyPlan pp;
  const bool poly = poly_route(c, bes, n_bes, n_timestep, chk_step, chk_thr, &pp) &&
                    moments_pay(c, pp, n_timestep, n_states, n_seg * n_states, 8e-6) &&
                    segments_closed(c, off);
  dispatch(c->ham.prec, pick_V(c->ham.prec, n_states, n_states, c->opts.vector_width),
           [&](auto tag) {
             using P = decltype(tag);
             if (poly && dos_segmented_moments<typename P::Real, P::V>(
                             c, pp, off, n_states, seed, n_timestep, chk_step, chk_thr, corr,
                             corr_per_state))
               return;
             dos_segmented_run<typename P::Real, P::V>(c, ex, off, n_states, seed, n_timestep,
                                                       chk_step, chk_thr, corr, corr_per_state);
           });
}

void drv_psi_t(tbpm_ctx* c, const double* bes, int n_bes, const double* psi0,
               const int32_t* time_log, int n_log, int n_timestep, int chk_step,
               double chk_thr, double* psi_t) {
  Phase phase("tbpm_psi_t");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_log < 1 || !time_log) throw Error{TBPM_ERR_ARG, "time_log must not be empty"};
  for (int i = 0; i < n_log; ++i) {
    if (time_log[i] < 0 || time_log[i] > n_timestep)
      throw Error{TBPM_ERR_ARG, "time in time_log out of [0, n_timestep]"};
    if (i && time_log[i] <= time_log[i - 1])
      throw Error{TBPM_ERR_ARG, "time_log must be sorted and unique"};
  }
  c->launches = 0;
  c->model_bytes = 0;
  const Expansion ex = time_step_expansion(bes, n_bes);
  if (c->ham.prec == TBPM_PREC_FP64)
    psi_t_run<double>(c, ex, bes, n_bes, psi0, time_log, n_log, n_timestep, chk_step, chk_thr, psi_t);
  else
    psi_t_run<float>(c, ex, bes, n_bes, psi0, time_log, n_log, n_timestep, chk_step, chk_thr, psi_t);
}

void drv_random_states(tbpm_ctx* c, int64_t n, int seed, int first_sample, int n_states,
                       int rank, int n_ran_samples, int kind, double* wf) {
  Phase phase("tbpm_random_states");
  if (n < 1 || n_states < 1) throw Error{TBPM_ERR_ARG, "bad sizes"};
  c->sess.active = false;
  c->graph.reset();
  // the generator only needs the row count; use a temporary geometry
  const int64_t saved_n = c->ham.n;
  const int saved_prec = c->ham.prec;
  c->ham.n = n;
  c->ham.prec = TBPM_PREC_FP64;
  try {
    for (int s0 = 0; s0 < n_states; s0 += kMaxCols) {
      const int ns = std::min(kMaxCols, n_states - s0);
      const StateKeys keys = make_keys(seed, first_sample + s0, ns, rank, n_ran_samples);
      c->wf0.ensure((size_t)n * ns * 16);
      c->ctr.ensure(16 * sizeof(int));
      gen_states<double, 1>(c, keys, ns, kind, c->wf0.as<Pack<double, 1>>());
      download_states<double>(c, c->wf0.p, ns, ns, 0, wf + 2 * (size_t)s0 * n);
    }
  } catch (...) {
    c->ham.n = saved_n;
    c->ham.prec = saved_prec;
    throw;
  }
  c->ham.n = saved_n;
  c->ham.prec = saved_prec;
}

void drv_fermi_coef(int nr_fermi, double beta, double mu, int one_minus, double eps,
                    double* coef, int* n_cheb) {
  std::vector<double> cf;
  const int n = fermi_coef(nr_fermi, beta, mu, one_minus != 0, eps, cf);
  std::fill(coef, coef + nr_fermi, 0.0);
  std::copy(cf.begin(), cf.end(), coef);
  *n_cheb = n;
}

void drv_expansion_apply(tbpm_ctx* c, const Expansion& ex, double* wf, int n_states) {
  Phase phase("tbpm_expansion_apply");
  require_ham(c, false);
  if (n_states < 1 || n_states > kMaxCols) throw Error{TBPM_ERR_ARG, "1..64 states"};
  c->graph.reset();
  c->sess.active = false;
  const int ld = n_states;
  ensure_vectors(c, ld, 1);
  dispatch(c->ham.prec, pick_V(c->ham.prec, ld, ld, c->opts.vector_width), [&](auto tag) {
    using P = decltype(tag);
    using R = typename P::Real;
    constexpr int V = P::V;
    upload_states<R>(c, wf, n_states, ld, 0, c->A.p);
    enqueue_expansion<R, V>(c, ex, ld, c->A.as<Pack<R, V>>(), c->X.as<Pack<R, V>>(),
                            c->Y.as<Pack<R, V>>(), nullptr, 0, nullptr, Counters{});
    download_states<R>(c, c->A.p, n_states, ld, 0, wf);
  });
}

void drv_session_dos_begin(tbpm_ctx* c, const double* bes, int n_bes, int n_states, int seed,
                           int rank, int n_ran_samples, int n_timestep) {
  Phase phase("tbpm_session_dos_begin");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_states < 1 || n_states > kMaxCols) throw Error{TBPM_ERR_ARG, "1..64 states"};
  c->launches = 0;
  c->model_bytes = 0;
  const Expansion ex = time_step_expansion(bes, n_bes);
  const StateKeys keys = make_keys(seed, 1, n_states, rank, n_ran_samples);
  dispatch(c->ham.prec, pick_V(c->ham.prec, n_states, n_states, c->opts.vector_width), [&](auto tag) {
    using P = decltype(tag);
    dos_session_begin<typename P::Real, P::V>(c, ex, n_states, &keys, nullptr, n_timestep + 1);
    // capture the step graph now, so that the first advance only replays it
    dos_session_advance<typename P::Real, P::V>(c, 0);
  });
}

void drv_session_advance(tbpm_ctx* c, int n_steps) {
  Phase phase("tbpm_session_advance");
  if (!c->sess.active) throw Error{TBPM_ERR_STATE, "no session active"};
  if (n_steps < 0) throw Error{TBPM_ERR_ARG, "n_steps < 0"};
  dispatch(c->ham.prec, c->sess.V, [&](auto tag) {
    using P = decltype(tag);
    dos_session_advance<typename P::Real, P::V>(c, n_steps);
  });
}

void drv_session_dos_resume(tbpm_ctx* c, const double* bes, int n_bes, int n_states,
                            const double* wf0, const double* psi, const double* corr,
                            const double* norms, int n_done, int n_timestep) {
  Phase phase("tbpm_session_dos_resume");
  require_ham(c, false);
  if (!bes || n_bes < 3) throw Error{TBPM_ERR_ARG, "at least 3 Bessel coefficients required"};
  if (n_states < 1 || n_states > kMaxCols) throw Error{TBPM_ERR_ARG, "1..64 states"};
  if (!wf0) throw Error{TBPM_ERR_ARG, "null initial states"};
  if (n_done < 0 || n_done > n_timestep + 1) throw Error{TBPM_ERR_ARG, "bad number of rows"};
  if (n_done > 0 && (!psi || !corr || !norms)) throw Error{TBPM_ERR_ARG, "null session state"};
  c->launches = 0;
  c->model_bytes = 0;
  const Expansion ex = time_step_expansion(bes, n_bes);
  dispatch(c->ham.prec, pick_V(c->ham.prec, n_states, n_states, c->opts.vector_width),
           [&](auto tag) {
             using P = decltype(tag);
             dos_session_resume<typename P::Real, P::V>(c, ex, n_states, wf0, psi, corr, norms,
                                                        n_done, n_timestep + 1);
           });
}

void drv_session_export(tbpm_ctx* c, double* wf0, double* psi) {
  if (!c->sess.active) throw Error{TBPM_ERR_STATE, "no session active"};
  const int ns = c->sess.ld;
  TBPM_CK(cudaStreamSynchronize(c->stream));
  if (c->ham.prec == TBPM_PREC_FP64) {
    if (wf0) download_states<double>(c, c->wf0.p, ns, ns, 0, wf0);
    if (psi) download_states<double>(c, c->A.p, ns, ns, 0, psi);
  } else {
    if (wf0) download_states<float>(c, c->wf0.p, ns, ns, 0, wf0);
    if (psi) download_states<float>(c, c->A.p, ns, ns, 0, psi);
  }
}

// One block waits, with the ring kernels' bounded wait, on an mbarrier phase
// that nothing completes; the wait runs out after kRingWaitNs and records it
// in the status word like any ring kernel would.
__global__ void ring_wait_probe_kernel(unsigned int* status) {
  __shared__ __align__(8) unsigned long long bar;
  if (threadIdx.x != 0) return;
  const uint32_t b = ring_smem(&bar);
  ring_bar_init(b, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (!ring_wait(b, 0)) atomicOr(status, 1u);
}

void drv_selftest_wait_timeout(tbpm_ctx* c) {
  ring_wait_probe_kernel<<<1, 32, 0, c->stream>>>(c->status.as<unsigned int>());
  TBPM_CK(cudaGetLastError());
  TBPM_CK(cudaStreamSynchronize(c->stream));
  check_status(c);  // throws TBPM_ERR_TIMEOUT when the wait ran out
}

// A tiny launch of a kernel with a grid barrier (0: cheb_persist_kernel, 1:
// haydock_kernel) on two blocks and an empty matrix, whose first barrier expects one
// arrival more than there are blocks: every block gives up after 10 ms.
void drv_selftest_grid_wait(tbpm_ctx* c, int kernel, int report) {
  if (kernel < 0 || kernel > 1) throw Error{TBPM_ERR_ARG, "kernel must be 0 or 1"};
  constexpr int n = 64, threads = 128, grid = 2;
  constexpr unsigned long long wait_ns = 10000000ull;
  c->ctr.ensure(16 * sizeof(int));
  unsigned int* bar = c->ctr.as<unsigned int>() + 12;
  unsigned int* status = c->status.as<unsigned int>();
  ScratchScope scope(c->scratch);
  TempMem mem(c->scratch);
  const size_t vec = n * sizeof(double2), bytes = 3 * vec + 64 * sizeof(double) + (n + 1) * 4;
  mem.ensure(bytes);
  TBPM_CK(cudaMemsetAsync(mem.p, 0, bytes, c->stream));
  TBPM_CK(cudaMemsetAsync(bar, 0, sizeof(unsigned int), c->stream));
  auto* v = mem.as<double2>();
  double* sums = reinterpret_cast<double*>(v + 3 * n);
  const int32_t* indptr = reinterpret_cast<const int32_t*>(sums + 64);  // rows without entries
  if (kernel == 0) {
    PersistArgs<double, 1> a{};
    a.indptr = indptr;
    a.n_rows = n;
    a.tpr = 1;
    a.p0 = reinterpret_cast<Pack<double, 1>*>(v);
    a.ring[0] = reinterpret_cast<Pack<double, 1>*>(v + n);
    a.ring[1] = reinterpret_cast<Pack<double, 1>*>(v + 2 * n);
    a.slots = 2;
    a.alpha = 1.0;
    a.k0 = 1;
    a.k1 = 2;
    a.bar = bar;
    a.status = status;
    a.absent = 1;
    a.wait_ns = wait_ns;
    launch_cooperative(c, cheb_persist_kernel<double, 1, false>, grid, threads, 0, a);
  } else {
    HaydockArgs<double> a{};
    a.indptr = indptr;
    a.n_rows = n;
    a.rescale = 1.0;
    a.w0 = v;
    a.w1 = v + n;
    a.y = v + 2 * n;
    a.n_depth = 1;
    a.a = sums;
    a.b = sums + 2;
    a.partials = sums + 8;
    a.bar = bar;
    a.status = status;
    a.absent = 1;
    a.wait_ns = wait_ns;
    launch_cooperative(c, haydock_kernel<double, 768>, grid, threads, 0, a);
  }
  TBPM_CK(cudaStreamSynchronize(c->stream));
  if (report) check_status(c);
}

// Curves and norm check of a run of T steps, checked at its end, from given sums of its
// terms (one column, <p_0|p_0> = 1, y = H): what dos_moments does with its own.
void drv_selftest_moments(tbpm_ctx* c, const double* bes, int n_bes, const double* sums,
                          int n_terms, int T, double* corr) {
  if (!bes || n_bes < 3 || !sums || n_terms < 2 || T < 2 || !corr)
    throw Error{TBPM_ERR_ARG, "series, sums and an output required"};
  c->sess.active = false;
  PolyPlan pp;
  pp.alpha = 2.0f;
  pp.a = 1.0L;
  pp.bes = bes;
  pp.n_bes = n_bes;
  const int M = 2 * n_terms;
  c->out.ensure((size_t)(T + 3) * 2 * sizeof(double));
  const size_t n_sums = 2 * (size_t)n_terms;
  c->poly.ensure((n_sums + 1 + 2 * (size_t)M) * sizeof(double) + sizeof(PolyNode) * M);
  double* d = c->poly.as<double>();
  std::vector<double> in(sums, sums + n_sums);
  in.push_back(1.0);
  TBPM_CK(cudaMemcpyAsync(d, in.data(), in.size() * sizeof(double), cudaMemcpyHostToDevice,
                          c->stream));
  double* mu = d + in.size();
  enqueue_moment_curves(c, pp, M, T, 1, d, 2, d + n_sums, 1, mu, mu + M,
                        reinterpret_cast<PolyNode*>(mu + 2 * M), T);
  std::vector<double> host;
  read_out(c, host, (size_t)(T + 3) * 2);
  check_moments(c, host, T, M, 1, T, 1e-9, "tbpm_selftest_moments");
  std::copy(host.begin(), host.begin() + 2 * (T + 1), corr);
}

void drv_session_read(tbpm_ctx* c, double* corr, double* norms, int* n_done) {
  if (!c->sess.active) throw Error{TBPM_ERR_STATE, "no session active"};
  const int rows = c->sess.rows_enqueued, ld = c->sess.ld;
  std::vector<double> host;
  read_out(c, host, (size_t)rows * ld * 3);
  for (int r = 0; r < rows; ++r)
    for (int b = 0; b < ld; ++b) {
      const double* v = &host[((size_t)r * ld + b) * 3];
      if (corr) {
        corr[2 * ((size_t)r * ld + b)] = v[0];
        corr[2 * ((size_t)r * ld + b) + 1] = v[1];
      }
      if (norms) norms[(size_t)r * ld + b] = v[2];
    }
  if (n_done) *n_done = rows;
}

}  // namespace tbpm
