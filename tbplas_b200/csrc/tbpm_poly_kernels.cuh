// Kernels of the polynomial routes: functions of a Hermitian H that the TBPM
// drivers need are evaluated from Chebyshev vectors over the whole time range
// instead of one time step after the other.
//
// One time step of the reference applies the polynomial P(H) = sum_k w_k T_k(H)
// (propagation.f90:12-49), n_Bes - 1 products with H.  For Hermitian H with
// spectrum in [-a, a] every power P(H)^t is a polynomial in y = H/a whose
// Chebyshev coefficients vanish beyond k ~ tau*a*t (they are Bessel functions
// J_k(tau*a*t) up to the rounding of P), so T steps together need about
// tau*a*T products, not (n_Bes - 1)*T: for the DOS 3.0 per step instead of 19,
// and half of that again because <p_k|p_k> and <p_k|p_{k-1}> give the moments
// mu_2k and mu_2k-1.  Measured on B200, whole calls, before -> after: DOS of
// 1600 x 1500 graphene, 16 FP64 states, 64 steps: 1017 -> 103 ms; 1024 x 1000, 16
// FP32 states, 128 steps: 482 -> 45 ms; 100 x 100, one state, 256 steps: 14.3 ->
// 1.8 ms; 20 packed samples, 4 states, 128 steps: 178 -> 40 ms.  The error against
// exact propagation stays where it was (1e-15 to 1e-14).
//
//  ham_spectrum_kernel    Gershgorin bound of H and whether H is Hermitian.
//  moment_density_kernel  moments -> weights rho_j of Gauss-Chebyshev nodes.
//  moment_curve_kernel    C(t) = sum_j P(x_j)^t rho_j, and the norms.
//  cheb_persist_kernel    all terms of a small problem in one launch.
//  seg_dots_kernel        the two products per (segment, state) of packed samples.
//  filter_values_kernel,  the quasi-eigenstates' energy filters on the nodes and
//  filter_coef_kernel     their Chebyshev coefficients.
//  qe_filter_mma_kernel   QE += (filter coefficients) x (a window of Chebyshev
//                         vectors) on mma.sync f64.
//  combine_kernel         the states after 1..m time steps from the Chebyshev
//                         vectors of one expansion.
#pragma once

#include "tbpm_dc_kernels.cuh"
#include "tbpm_kernels.cuh"
#include "tbpm_seg_kernels.cuh"

namespace tbpm {

// Rows longer than this are not searched for their transposes.
constexpr int kSpectrumMaxRow = 64;

// info[0]: largest row sum |D_r| + sum_j |O_rj| (the bits of a non-negative
// double, ordered like it), info[1]: nonzero when H is not Hermitian to `tol`
// (relative) or a row is longer than kSpectrumMaxRow.  One thread per row; a
// row's transposed entries lie in its neighbours' rows, which are near in
// memory.  Runs once per Hamiltonian.
template <typename R>
__global__ void __launch_bounds__(256) ham_spectrum_kernel(const int32_t* indptr,
                                                           const int32_t* indices,
                                                           const typename Cx<R>::t* hop,
                                                           const typename Cx<R>::t* diag,
                                                           int64_t n, double tol,
                                                           unsigned long long* info) {
  double bound = 0.0;
  bool bad = false;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int j0 = indptr[r], j1 = indptr[r + 1];
    double s = 0.0;
    if (diag) {
      const typename Cx<R>::t d = diag[r];
      s = fabs((double)d.x);
      if (!(fabs((double)d.y) <= tol * fmax(1.0, s))) bad = true;
    }
    if (j1 - j0 > kSpectrumMaxRow) {
      bad = true;
      continue;
    }
    for (int j = j0; j < j1; ++j) {
      const int c = indices[j];
      const typename Cx<R>::t h = hop[j];
      s += hypot((double)h.x, (double)h.y);
      // the sums of all entries at (r, c) and at (c, r)
      double fr = 0.0, fi = 0.0, br = 0.0, bi = 0.0;
      for (int k = j0; k < j1; ++k)
        if (indices[k] == c) {
          fr += (double)hop[k].x;
          fi += (double)hop[k].y;
        }
      const int k1 = indptr[c + 1];
      if (k1 - indptr[c] > kSpectrumMaxRow) {
        bad = true;
        continue;
      }
      for (int k = indptr[c]; k < k1; ++k)
        if (indices[k] == (int)r) {
          br += (double)hop[k].x;
          bi += (double)hop[k].y;
        }
      const double lim = tol * (fabs(fr) + fabs(fi));
      if (!(fabs(fr - br) <= lim && fabs(fi + bi) <= lim)) bad = true;
    }
    if (!(s <= 1e300)) bad = true;
    bound = fmax(bound, s);
  }
  for (int w = 16; w > 0; w >>= 1) bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, w));
  const bool any = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(info, (unsigned long long)__double_as_longlong(bound));
    if (any) atomicOr(info + 1, 1ull);
  }
}

// ---- moments -> correlation function --------------------------------------

// A node x_j = a cos(pi (j + 1/2) / M): P(x_j) = exp(lnabs) exp(2 pi i (hi + lo)).
// The phase is kept in turns as an unevaluated sum of two doubles, so that
// its t-th multiple keeps full precision.
struct PolyNode {
  double hi, lo, lnabs;
};

// cos(pi k (j + 1/2) / M), the argument reduced in integers
__device__ __forceinline__ double node_cos(int64_t k, int64_t j, int64_t M) {
  const int64_t m = (k * (2 * j + 1)) % (4 * M);
  return cospi((double)m / (double)(2 * M));
}

// turns -> (cos, sin) of t times the node's phase
__device__ __forceinline__ void node_power(const PolyNode& p, double t, double* re, double* im) {
  const double q = t * p.hi;
  const double e = fma(t, p.hi, -q) + t * p.lo;  // q + e = t * (hi + lo)
  const double f = (q - rint(q)) + e;
  sincospi(2.0 * f, im, re);
}

// mu_m of column col from the sums of the terms: sums[(k-1)*stride + col*2 + q]
// with q = 0: <p_k|p_k>, 1: Re <p_k|p_{k-1}>, and mu0 = <p_0|p_0>:
// T_m T_n = (T_{m+n} + T_{|m-n|}) / 2.
__device__ __forceinline__ double moment_at(int m, const double* sums, int64_t stride, int col,
                                            double mu0) {
  if (m == 0) return mu0;
  const double mu1 = sums[(int64_t)col * 2 + 1];
  if (m == 1) return mu1;
  const double* s = sums + (int64_t)((m + 1) / 2 - 1) * stride + (int64_t)col * 2;
  return (m & 1) ? 2.0 * s[1] - mu1 : 2.0 * s[0] - mu0;
}

// mu[col*M + m] for every column (mu0[col*mu0_stride] = <p_0|p_0>)
static __global__ void __launch_bounds__(256) moment_gather_kernel(const double* sums,
                                                                   int64_t stride,
                                                                   const double* mu0,
                                                                   int mu0_stride, int n_cols,
                                                                   int M, double* mu) {
  const int64_t total = (int64_t)n_cols * M;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int m = (int)(g % M);
    const int col = (int)(g / M);
    mu[g] = moment_at(m, sums, stride, col, mu0[(int64_t)col * mu0_stride]);
  }
}

constexpr int kMomentCols = 8;  // columns that share one cosine / one power

// rho[col*M + j] = (1/M) sum_m (2 - delta_m0) mu[col*M + m] cos(m theta_j).
// Block (j, column chunk), threads over m; M^2 cosines in all (10^7 at 1024
// time steps), negligible beside the terms.
static __global__ void __launch_bounds__(128) moment_density_kernel(const double* mu, int n_cols,
                                                                    int M, double* rho) {
  __shared__ double red[128 / 32][kMomentCols];
  const int j = blockIdx.x;
  const int c0 = blockIdx.y * kMomentCols;
  const int nc = min(kMomentCols, n_cols - c0);
  double acc[kMomentCols];
#pragma unroll
  for (int c = 0; c < kMomentCols; ++c) acc[c] = 0.0;
  for (int m = threadIdx.x; m < M; m += 128) {
    const double w = (m ? 2.0 : 1.0) * node_cos(m, j, M);
#pragma unroll
    for (int c = 0; c < kMomentCols; ++c)
      if (c < nc) acc[c] += w * mu[(int64_t)(c0 + c) * M + m];
  }
#pragma unroll
  for (int c = 0; c < kMomentCols; ++c) {
    for (int s = 16; s > 0; s >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = acc[c];
  }
  __syncthreads();
  if (threadIdx.x < nc) {
    const double s = (red[0][threadIdx.x] + red[1][threadIdx.x]) +
                     (red[2][threadIdx.x] + red[3][threadIdx.x]);
    rho[(int64_t)(c0 + threadIdx.x) * M + j] = s / M;
  }
}

// Block (row, column chunk).  Rows 0..T: out = sum_j P(x_j)^t rho_j (re, im);
// rows T+1, T+2: the norm sum_j |P(x_j)|^(2t) rho_j after t = t_ref, t_chk
// steps.  out[(row*n_cols + col)*2 + {re, im}].
static __global__ void __launch_bounds__(128) moment_curve_kernel(const PolyNode* nodes,
                                                                  const double* rho, int n_cols,
                                                                  int M, int T, int t_ref,
                                                                  int t_chk, double* out) {
  __shared__ double red[128 / 32][2 * kMomentCols];
  const int row = blockIdx.x;
  const int c0 = blockIdx.y * kMomentCols;
  const int nc = min(kMomentCols, n_cols - c0);
  const bool norm = row > T;
  const double t = !norm ? (double)row : (row == T + 1 ? (double)t_ref : (double)t_chk);
  double ar[kMomentCols], ai[kMomentCols];
#pragma unroll
  for (int c = 0; c < kMomentCols; ++c) ar[c] = ai[c] = 0.0;
  for (int j = threadIdx.x; j < M; j += 128) {
    const PolyNode p = nodes[j];
    double re, im;
    if (norm) {
      re = exp(2.0 * t * p.lnabs);
      im = 0.0;
    } else {
      node_power(p, t, &re, &im);
      const double g = exp(t * p.lnabs);
      re *= g;
      im *= g;
    }
#pragma unroll
    for (int c = 0; c < kMomentCols; ++c)
      if (c < nc) {
        const double w = rho[(int64_t)(c0 + c) * M + j];
        ar[c] += re * w;
        ai[c] += im * w;
      }
  }
#pragma unroll
  for (int c = 0; c < kMomentCols; ++c) {
    for (int s = 16; s > 0; s >>= 1) {
      ar[c] += __shfl_xor_sync(0xffffffffu, ar[c], s);
      ai[c] += __shfl_xor_sync(0xffffffffu, ai[c], s);
    }
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5][2 * c] = ar[c];
      red[threadIdx.x >> 5][2 * c + 1] = ai[c];
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * nc)
    out[((int64_t)row * n_cols + c0) * 2 + threadIdx.x] =
        (red[0][threadIdx.x] + red[1][threadIdx.x]) + (red[2][threadIdx.x] + red[3][threadIdx.x]);
}

// ---- all terms of a small problem in one launch -----------------------------

template <typename R, int V>
struct PersistArgs {
  const int32_t* indptr;
  const int32_t* indices;
  const typename Cx<R>::t* hop;
  const typename Cx<R>::t* diag;
  int64_t n_rows;
  int tpr;
  Pack<R, V>* p0;    // p_0 on entry; overwritten by p_2, p_4, ...
  Pack<R, V>* p1;    // receives p_1, p_3, ...
  double alpha;      // 2 / a
  int n_terms;       // K
  double* partials;  // [((k-1)*ld*2 + col*2 + q) * gridDim.x + block]
  unsigned int* bar;     // grid barrier, zero on entry
  unsigned int* status;  // bit 0: a bounded wait ran out
};

// most threads of a block: 128 registers a thread for 32-byte packs, 102 for
// 16-byte ones, 64 for 8-byte ones
template <typename R, int V>
constexpr int kPersistThreads = sizeof(R) * V == 16 ? 512 : (sizeof(R) * V == 8 ? 640 : 1024);
constexpr int kPersistDeg = 4;  // row entries whose gathers are issued together
constexpr unsigned long long kPersistWaitNs = 2000000000ull;  // 2 s per wait

// The moments' terms p_k = (2/a) H p_{k-1} - p_{k-2}, k = 1..K, of a problem
// whose vectors stay in L2, under one cooperative launch: a grid barrier per
// term instead of a launch per term.  What bounds it is latency, not bytes: a
// barrier round trip and one gather.  The matrix entries of a thread's next
// item (a row's pack of V columns; up to kPersistDeg entries) are loaded as soon
// as those of the current item are used, so the first item's are in registers
// when the barrier opens.  p_k is read with L2-only loads, as other SMs wrote it
// in this launch.  The block's two products per column are reduced after its
// arrival on the barrier, while the other blocks arrive.
template <typename R, int V>
__global__ void __launch_bounds__((kPersistThreads<R, V>), 1)
    cheb_persist_kernel(const __grid_constant__ PersistArgs<R, V> a) {
  using C = typename Cx<R>::t;
  extern __shared__ double psm[];
  __shared__ int stop;
  const int tpr = a.tpr;
  const int slot = threadIdx.x / tpr;
  const int lane = threadIdx.x - slot * tpr;
  const int rpp = blockDim.x / tpr;
  const int64_t stride = (int64_t)gridDim.x * rpp;
  const int64_t n = a.n_rows;
  const bool in = slot < rpp;
  const int64_t r_first = (int64_t)blockIdx.x * rpp + slot;
  const int width = tpr * V * 2;
  const int ld2 = tpr * V * 2;
  if (threadIdx.x == 0) stop = 0;
  // matrix entries of the current item
  int j0 = 0, j1 = 0;
  int c[kPersistDeg];
  C h[kPersistDeg];
  C d;
  d.x = d.y = (R)0;
  auto load = [&](int64_t r) {
    j0 = __ldg(a.indptr + r);
    j1 = __ldg(a.indptr + r + 1);
#pragma unroll
    for (int u = 0; u < kPersistDeg; ++u) {
      c[u] = -1;
      if (j0 + u < j1) {
        c[u] = __ldg(a.indices + j0 + u);
        h[u] = ldg_c(a.hop + j0 + u);
      }
    }
    if (a.diag) d = ldg_c(a.diag + r);
  };
  const bool any = in && r_first < n;
  if (any) load(r_first);
  __syncthreads();
  const R alpha2 = (R)a.alpha, alpha1 = (R)(0.5 * a.alpha);
  for (int k = 1; k <= a.n_terms; ++k) {
    const Pack<R, V>* src = (k & 1) ? a.p0 : a.p1;
    Pack<R, V>* dst = (k & 1) ? a.p1 : a.p0;
    const R al = k == 1 ? alpha1 : alpha2;
    double nrm[V], cre[V];
#pragma unroll
    for (int v = 0; v < V; ++v) nrm[v] = cre[v] = 0.0;
    if (any) {
      for (int64_t r = r_first; r < n; r += stride) {
        const int64_t e = r * tpr + lane;
        Pack<R, V> x[kPersistDeg];
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u)
          if (c[u] >= 0) x[u] = ldcg_pack(src + (int64_t)c[u] * tpr + lane);
        const Pack<R, V> own = ldcg_pack(src + e);
        Pack<R, V> pm2;
        if (k >= 2) {
          pm2 = ldcg_pack(dst + e);
        } else {
#pragma unroll
          for (int q = 0; q < 2 * V; ++q) pm2.v[q] = (R)0;
        }
        R sre[V], sim[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          sre[v] = d.x * own.v[2 * v] - d.y * own.v[2 * v + 1];
          sim[v] = d.x * own.v[2 * v + 1] + d.y * own.v[2 * v];
        }
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u)
          if (c[u] >= 0) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
              sre[v] = fma(h[u].x, x[u].v[2 * v], fma(-h[u].y, x[u].v[2 * v + 1], sre[v]));
              sim[v] = fma(h[u].x, x[u].v[2 * v + 1], fma(h[u].y, x[u].v[2 * v], sim[v]));
            }
          }
        for (int j = j0 + kPersistDeg; j < j1; ++j) {
          const C hj = ldg_c(a.hop + j);
          const Pack<R, V> xj = ldcg_pack(src + (int64_t)__ldg(a.indices + j) * tpr + lane);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            sre[v] = fma(hj.x, xj.v[2 * v], fma(-hj.y, xj.v[2 * v + 1], sre[v]));
            sim[v] = fma(hj.x, xj.v[2 * v + 1], fma(hj.y, xj.v[2 * v], sim[v]));
          }
        }
        load(r + stride < n ? r + stride : r_first);
        Pack<R, V> pk;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          pk.v[2 * v] = fma(al, sre[v], -pm2.v[2 * v]);
          pk.v[2 * v + 1] = fma(al, sim[v], -pm2.v[2 * v + 1]);
          const double xr = (double)pk.v[2 * v], xi = (double)pk.v[2 * v + 1];
          nrm[v] += xr * xr + xi * xi;
          cre[v] += xr * (double)own.v[2 * v] + xi * (double)own.v[2 * v + 1];
        }
        stwb_pack(dst + e, pk);
      }
    }
    // arrive, reduce this block's products, then wait for the others
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && k < a.n_terms) atomicAdd(a.bar, 1u);
    if (in) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        psm[slot * width + (lane * V + v) * 2] = nrm[v];
        psm[slot * width + (lane * V + v) * 2 + 1] = cre[v];
      }
    }
    __syncthreads();
    tree_reduce_slots(psm, rpp, width, slot, lane, tpr);
    for (int q = threadIdx.x; q < width; q += blockDim.x)
      a.partials[((int64_t)(k - 1) * ld2 + q) * gridDim.x + blockIdx.x] = psm[q];
    if (k == a.n_terms) break;
    if (threadIdx.x == 0) {
      const unsigned int want = (unsigned int)k * gridDim.x;
      unsigned long long t0 = 0;
      for (unsigned int spin = 0;; ++spin) {
        unsigned int seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
        if (seen >= want) break;
        if ((spin & 255u) == 255u) {
          unsigned long long now;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          if (now - t0 > kPersistWaitNs) {
            atomicOr(a.status, 1u);
            stop = 1;
            break;
          }
        }
      }
      __threadfence();
    }
    __syncthreads();
    if (stop) break;
  }
}

// ---- packed realisations ------------------------------------------------------

// <x|x> and Re <x|y> per (segment, column):
// partials[((seg*ns + col)*2 + q)*n_chunks + chunk]; launch shape of seg_corr_kernel
template <typename R>
__global__ void __launch_bounds__(256) seg_dots_kernel(const int64_t* seg_off, int ns,
                                                       int64_t rows_per_chunk,
                                                       const typename Cx<R>::t* x,
                                                       const typename Cx<R>::t* y,
                                                       double* partials) {
  __shared__ double smem[256 * 2];
  const int seg = blockIdx.y;
  const int slot = threadIdx.x / ns;
  const int col = threadIdx.x - slot * ns;
  const int rpp = blockDim.x / ns;
  const int64_t s0 = seg_off[seg], s1 = seg_off[seg + 1];
  const int64_t c0 = s0 + (int64_t)blockIdx.x * rows_per_chunk;
  const int64_t c1 = min(c0 + rows_per_chunk, s1);
  double v[2] = {0.0, 0.0};
  if (slot < rpp) {
#pragma unroll 4
    for (int64_t r = c0 + slot; r < c1; r += rpp) {
      const typename Cx<R>::t p = ldg_c(x + r * ns + col);
      const typename Cx<R>::t q = ldg_c(y + r * ns + col);
      const double pr = (double)p.x, pi = (double)p.y;
      v[0] += pr * pr + pi * pi;
      v[1] += pr * (double)q.x + pi * (double)q.y;
    }
  }
  seg_block_reduce(smem, v, 2, slot, col, rpp, ns);
  if (slot == 0) {
    for (int q = 0; q < 2; ++q)
      partials[(((int64_t)seg * ns + col) * 2 + q) * gridDim.x + blockIdx.x] = smem[col * 2 + q];
  }
}

// ---- quasi-eigenstates as energy filters ---------------------------------------

// Phase 1 of tbpm_dccond (tbpm.f90:600-638) accumulates
//   QE_i = wf0 + sum_t W(t) [e^{i E_i t dt} P(H)^t + e^{-i E_i t dt} conj(P)(H)^t] wf0,
// W(t) = (1 + cos(pi t / T)) / 2: a real function f_i of H.  With its Chebyshev
// coefficients, QE_i = sum_k c_ki T_k(H/a) wf0 needs one block of Chebyshev
// vectors (3.0 products with H per time step) instead of the forward and the
// backward propagation of 19 products each.

// The window and phase factors c_ti = W(t) e^{i E_i t dt} are taken as the same
// doubles that time stepping multiplies with (far from the spectrum QE_i is a
// small difference of them), and the powers of P come from extended-precision
// phases, so the filters carry no more rounding than the sums over t did.

// s + e += v without loss (two-sum)
__device__ __forceinline__ void filter_add(double* s, double* e, double v) {
  const double t = *s + v;
  const double z = t - *s;
  *e += (*s - (t - z)) + (v - z);
  *s = t;
}

// f[j*n_en + i] = 1 + 2 Re sum_t c[(t-1)*n_en + i] P(x_j)^t.  Block: 32 nodes x 8
// energies; per 32 time steps the powers of the nodes are formed once and
// shared by the energies.
static __global__ void __launch_bounds__(256) filter_values_kernel(const PolyNode* nodes, int M,
                                                                   const double2* c, int n_en,
                                                                   int T, double* f) {
  __shared__ double pre[32][33], pim[32][33];
  __shared__ double2 cc[32][8];
  const int jj = threadIdx.x & 31, ii = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + jj;
  const int i = blockIdx.y * 8 + ii;
  PolyNode p = {0.0, 0.0, 0.0};
  if (j < M) p = nodes[j];
  double s = 0.0, e = 0.0;
  for (int t0 = 1; t0 <= T; t0 += 32) {
    __syncthreads();
    for (int q = ii; q < 32; q += 8) {
      const double t = (double)(t0 + q);
      double re, im;
      node_power(p, t, &re, &im);
      const double g = 1.0 + t * p.lnabs;  // |P|^t, lnabs of the order of rounding
      pre[q][jj] = re * g;
      pim[q][jj] = im * g;
    }
    {
      const int q = threadIdx.x >> 3, k = threadIdx.x & 7;
      const int ik = blockIdx.y * 8 + k;
      cc[q][k] = t0 + q <= T && ik < n_en ? c[(int64_t)(t0 + q - 1) * n_en + ik]
                                          : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < 32; ++q)
      filter_add(&s, &e, cc[q][ii].x * pre[q][jj] - cc[q][ii].y * pim[q][jj]);
  }
  if (j < M && i < n_en) f[(int64_t)j * n_en + i] = 1.0 + 2.0 * (s + e);
}

// c[k*n_en + i] = (2 - delta_k0)/M sum_j f[j*n_en + i] cos(k theta_j).  Block: one
// k and up to 256 energies; the threads left over split the nodes.
static __global__ void __launch_bounds__(256) filter_coef_kernel(const double* f, int M, int n_en,
                                                                 double* c) {
  __shared__ double cs[256];
  __shared__ double red[2][256];
  const int k = blockIdx.x;
  const int i0 = blockIdx.y * 256;
  const int ni = min(256, n_en - i0);
  const int parts = 256 / ni;
  const int part = threadIdx.x / ni;
  const int i = threadIdx.x - part * ni;
  double s = 0.0, e = 0.0;
  for (int j0 = 0; j0 < M; j0 += 256) {
    __syncthreads();
    if (j0 + threadIdx.x < M) cs[threadIdx.x] = node_cos(k, j0 + threadIdx.x, M);
    __syncthreads();
    if (part < parts) {
      const int nj = min(256, M - j0);
      for (int j = part; j < nj; j += parts)
        filter_add(&s, &e, cs[j] * f[(int64_t)(j0 + j) * n_en + i0 + i]);
    }
  }
  red[0][threadIdx.x] = s;
  red[1][threadIdx.x] = e;
  __syncthreads();
  if (threadIdx.x < ni) {
    double t = 0.0, r = 0.0;
    for (int q = 0; q < parts; ++q) {
      filter_add(&t, &r, red[0][q * ni + threadIdx.x]);
      r += red[1][q * ni + threadIdx.x];
    }
    c[(int64_t)k * n_en + i0 + threadIdx.x] = (k ? 2.0 : 1.0) / M * (t + r);
  }
}

constexpr int kFilterWindow = 32;  // Chebyshev vectors folded into QE per pass

template <typename R>
struct FilterPtrs {
  const typename Cx<R>::t* p[kFilterWindow];
};

// Shared memory of qe_filter_mma_kernel: the window's values of a tile,
// [tau][pair], rows padded by 4 pairs (64 bytes), so that the four tau of a
// fragment load lie in different banks.
constexpr int kFilterPad = 4;
__host__ __device__ constexpr size_t qe_filter_smem(int nb) {
  return (size_t)kFilterWindow * (qe_mma_rows(nb) * nb + kFilterPad) * sizeof(double2);
}

// QE[r][i][b] (+)= sum_{tau < T} c[tau][i] p_tau[r][b], c real: per tile of
// (row, state) pairs a real product A (energies x 32) . B (32 x (pair, re/im)),
// with the fragments and the split over warps of qe_accum_mma_kernel (whose
// +/- windows need 2 x 16 coefficients for 16 steps).  A window of 32 vectors
// per pass over QE: at 16 the pass over QE (32 bytes a complex128 element
// against 32 FMAs) was the longer side.  A warp's QE elements of the next
// column tile are loaded before the products of the current one.
template <typename R>
__global__ void __launch_bounds__(kQeMmaWarps * 32, 2) qe_filter_mma_kernel(
    typename Cx<R>::t* qe, int64_t n_rows, int n_en, int nb,
    const __grid_constant__ FilterPtrs<R> win, int T, const double* coef, int init) {
  using C = typename Cx<R>::t;
  extern __shared__ double2 qsm[];
  const int RT = qe_mma_rows(nb);
  const int P = RT * nb;  // pairs of a tile; P % 4 == 0
  const int PS = P + kFilterPad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n_mt = (n_en + 7) / 8;
  const int mt_b = blockIdx.y * kQeMmaWarps * kQeMmaMT;
  const int n_mt_b = min(kQeMmaWarps * kQeMmaMT, n_mt - mt_b);
  const int n_mg = (n_mt_b + kQeMmaMT - 1) / kQeMmaMT;
  const int mg = warp % n_mg;
  const int nt_first = warp / n_mg;
  const int nt_step = (kQeMmaWarps - mg + n_mg - 1) / n_mg;
  const int mt0 = mt_b + mg * kQeMmaMT;
  double afr[kQeMmaMT][kFilterWindow / 4];
#pragma unroll
  for (int m = 0; m < kQeMmaMT; ++m) {
    const int i = (mt0 + m) * 8 + g;
#pragma unroll
    for (int st = 0; st < kFilterWindow / 4; ++st) {
      const int tau = 4 * st + t;
      afr[m][st] = i < n_en && tau < T ? coef[(int64_t)tau * n_en + i] : 0.0;
    }
  }
  for (int64_t r0 = (int64_t)blockIdx.x * RT; r0 < n_rows; r0 += (int64_t)gridDim.x * RT) {
    const int nr = (int)min((int64_t)RT, n_rows - r0);
    const int np = nr * nb;  // pairs in range
    auto load_c = [&](int nt, C* v) {
      const int pc = 4 * nt + t;
      const int rr = pc / nb, bb = pc - rr * nb;
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        const int i = (mt0 + m) * 8 + g;
        v[m].x = v[m].y = (R)0;
        if (!init && nt < P / 4 && pc < np && i < n_en)
          v[m] = qe[((r0 + rr) * n_en + i) * nb + bb];
      }
    };
    C cv[kQeMmaMT];
    load_c(nt_first, cv);
    __syncthreads();  // the previous tile's values are consumed
    for (int q = threadIdx.x; q < kFilterWindow * P; q += blockDim.x) {
      const int tau = q / P;
      const int pr = q - tau * P;
      double2 v = make_double2(0.0, 0.0);
      if (tau < T && pr < np) {
        const C x = ldg_c(win.p[tau] + r0 * nb + pr);
        v = make_double2((double)x.x, (double)x.y);
      }
      qsm[tau * PS + pr] = v;
    }
    __syncthreads();
    for (int nt = nt_first; nt < P / 4; nt += nt_step) {
      // B fragment: B[k = 4*s + t][n = g]; column g is pair 4*nt + g/2, part g&1
      const double* b = reinterpret_cast<const double*>(qsm + 4 * nt) + g;
      double bfr[kFilterWindow / 4];
#pragma unroll
      for (int st = 0; st < kFilterWindow / 4; ++st) bfr[st] = b[(4 * st + t) * 2 * PS];
      double c0[kQeMmaMT], c1[kQeMmaMT];
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        c0[m] = (double)cv[m].x;
        c1[m] = (double)cv[m].y;
      }
      load_c(nt + nt_step, cv);
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        if (mt0 + m < n_mt) {
#pragma unroll
          for (int st = 0; st < kFilterWindow / 4; ++st)
            dmma_8x8x4(c0[m], c1[m], afr[m][st], bfr[st]);
        }
      }
      const int pc = 4 * nt + t;
      const int rr = pc / nb, bb = pc - rr * nb;
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        const int i = (mt0 + m) * 8 + g;
        if (pc < np && i < n_en) {
          C o;
          o.x = (R)c0[m];
          o.y = (R)c1[m];
          qe[((r0 + rr) * n_en + i) * nb + bb] = o;
        }
      }
    }
  }
}

// ---- several time steps from one expansion ----------------------------------------

constexpr int kCombineWindow = 16;  // Chebyshev vectors per pass
constexpr int kCombineSteps = 16;   // most time steps per expansion
constexpr int kCombineBatch = 8;    // vectors loaded together

template <typename R>
struct CombineArgs {
  const typename Cx<R>::t* p[kCombineWindow];
  typename Cx<R>::t* out[kCombineSteps];
  double w[kCombineSteps][kCombineWindow];  // zero where an output has no such term
  int64_t total;                            // values of a block
  int np;                                   // vectors of this pass
  int j0, m;                                // outputs j0 <= j < m take part
  unsigned int init;                        // bit j: out_j starts here (is not read)
};

// out_j[e] (+)= sum_tau w[j][tau] p_tau[e] for up to 16 outputs: the states
// after 1..m time steps all come from the same Chebyshev vectors, so m steps of
// phase tau take n(m tau) products with H instead of m n(tau) (AC: 57 instead of
// 240 for 16 steps).  One complex value per thread; the weights are
// compile-time offsets into the parameter bank.  Sums in FP64.  Bound by memory: 16
// values read for 32 FMAs each, 9 TB/s of reads at the FP64 peak.
// p_0 may be out_{m-1}: a thread reads every p of its value before it writes.
template <typename R, int M>
__global__ void __launch_bounds__(256, 2) combine_kernel(const __grid_constant__ CombineArgs<R> a) {
  using C = typename Cx<R>::t;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.total) return;
  double re[M], im[M];
#pragma unroll
  for (int j = 0; j < M; ++j) {
    re[j] = im[j] = 0.0;
    if (j >= a.j0 && j < a.m && !((a.init >> j) & 1u)) {
      const C o = a.out[j][e];
      re[j] = (double)o.x;
      im[j] = (double)o.y;
    }
  }
#pragma unroll
  for (int q0 = 0; q0 < kCombineWindow; q0 += kCombineBatch) {
    if (q0 < a.np) {
      C p[kCombineBatch];
#pragma unroll
      for (int q = 0; q < kCombineBatch; ++q) {
        p[q].x = p[q].y = (R)0;
        if (q0 + q < a.np) p[q] = a.p[q0 + q][e];
      }
#pragma unroll
      for (int q = 0; q < kCombineBatch; ++q) {
        const double x = (double)p[q].x, y = (double)p[q].y;
#pragma unroll
        for (int j = 0; j < M; ++j) {
          re[j] = fma(a.w[j][q0 + q], x, re[j]);
          im[j] = fma(a.w[j][q0 + q], y, im[j]);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < M; ++j)
    if (j >= a.j0 && j < a.m) {
      C o;
      o.x = (R)re[j];
      o.y = (R)im[j];
      a.out[j][e] = o;
    }
}

}  // namespace tbpm
