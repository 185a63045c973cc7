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
// 1600 x 1500 graphene, 16 FP64 states, 64 steps: 1061 -> 99 ms; 1024 x 1000, 16
// FP32 states, 128 steps: 494 -> 43 ms; 100 x 100, one state, 256 steps: 14.2 ->
// 1.04 ms; 20 packed samples, 4 states, 128 steps: 178 -> 27 ms.  The error against
// exact propagation stays where it was (1e-15 to 1e-14).
//
//  ham_spectrum_kernel    Gershgorin bounds of H and of its anti-Hermitian part.
//  moment_density_kernel  moments -> weights rho_j of Gauss-Chebyshev nodes.
//  moment_curve_kernel    C(t) = sum_j P(x_j)^t rho_j, and the norms.
//  cheb_persist_kernel    all terms of a small problem in one launch.
//  cheb_cluster_kernel    the same for a tiny one, in the shared memory of one
//                         cluster.
//  seg_closed_kernel      whether packed samples are uncoupled.
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
// double, ordered like it), info[1]: the same of the anti-Hermitian part (H - H^+)/2,
// off-diagonal deviations of up to `rounding` (relative) left out: those have no
// common sign and average out, info[2]: nonzero when an entry is not the conjugate of
// its transpose
// to `tol` (relative) or a row is longer than kSpectrumMaxRow.  One thread per row; a
// row's transposed entries lie in its neighbours' rows, which are near in
// memory.  Runs once per Hamiltonian.
template <typename R>
__global__ void __launch_bounds__(256) ham_spectrum_kernel(const int32_t* indptr,
                                                           const int32_t* indices,
                                                           const typename Cx<R>::t* hop,
                                                           const typename Cx<R>::t* diag,
                                                           int64_t n, double tol,
                                                           double rounding,
                                                           unsigned long long* info) {
  double bound = 0.0, skew = 0.0;
  bool bad = false;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int j0 = indptr[r], j1 = indptr[r + 1];
    double s = 0.0, sk = 0.0;
    if (diag) {
      const typename Cx<R>::t d = diag[r];
      s = fabs((double)d.x);
      sk = fabs((double)d.y);
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
      const double dev = hypot(fr - br, fi + bi);
      if (dev > rounding * (fabs(fr) + fabs(fi))) sk += 0.5 * dev;
    }
    if (!(s <= 1e300)) bad = true;
    bound = fmax(bound, s);
    skew = fmax(skew, sk);
  }
  for (int w = 16; w > 0; w >>= 1) {
    bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, w));
    skew = fmax(skew, __shfl_xor_sync(0xffffffffu, skew, w));
  }
  const bool any = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(info, (unsigned long long)__double_as_longlong(bound));
    atomicMax(info + 1, (unsigned long long)__double_as_longlong(skew));
    if (any) atomicOr(info + 2, 1ull);
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
// steps, and the largest |mu_m|: for unitary P the norms are mu_0 whatever the terms
// computed, but no moment of a state with spectrum in [-1, 1] exceeds mu_0.
// out[(row*n_cols + col)*2 + {re, im}].
static __global__ void __launch_bounds__(128) moment_curve_kernel(const PolyNode* nodes,
                                                                  const double* mu,
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
#pragma unroll
      for (int c = 0; c < kMomentCols; ++c)
        if (c < nc) ai[c] = fmax(ai[c], fabs(mu[(int64_t)(c0 + c) * M + j]));
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
      const double o = __shfl_xor_sync(0xffffffffu, ai[c], s);
      ai[c] = norm ? fmax(ai[c], o) : ai[c] + o;
    }
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5][2 * c] = ar[c];
      red[threadIdx.x >> 5][2 * c + 1] = ai[c];
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * nc) {
    const double a = red[0][threadIdx.x], b = red[1][threadIdx.x], c = red[2][threadIdx.x],
                 d = red[3][threadIdx.x];
    out[((int64_t)row * n_cols + c0) * 2 + threadIdx.x] =
        norm && (threadIdx.x & 1) ? fmax(fmax(a, b), fmax(c, d)) : (a + b) + (c + d);
  }
}

// ---- all terms of a small problem in one launch -----------------------------

constexpr int kPersistRing = 34;  // most vectors kept

template <typename R, int V>
struct PersistArgs {
  const int32_t* indptr;
  const int32_t* indices;
  const typename Cx<R>::t* hop;
  const typename Cx<R>::t* diag;
  int64_t n_rows;
  int tpr;
  const Pack<R, V>* p0;          // p_0
  Pack<R, V>* ring[kPersistRing];  // p_k, k >= 1, is ring[k % slots]
  int slots;
  double alpha;       // 2 / a
  int turn;           // 1: the vectors times (-i)^k
  int k0, k1;         // terms k0 <= k <= k1 of this launch
  // ACC kernels: the weighted sum of the vectors is folded into acc every third
  // term (k = 2, 5, 8, ...; k0 is 1), weights w[set*n_w + k]
  Pack<R, V>* acc;
  const double* w;
  int n_w;
  unsigned long long set_mask;  // columns that use set 1
  int k_dots;         // products are formed for k <= k_dots
  double* partials;   // [((k-k0)*ld*2 + col*2 + q) * gridDim.x + block]
  unsigned int* bar;      // grid barrier, zero on entry
  unsigned int* status;  // bit 0: a bounded wait ran out
  unsigned int absent;   // arrivals expected beside the grid's (the self-test's: never come)
  unsigned long long wait_ns;  // longest wait
};

// most threads of a block: 128 registers a thread for 32-byte packs, 85 for
// 16-byte ones, 64 for 8-byte ones
template <typename R, int V>
constexpr int kPersistThreads = sizeof(R) * V == 16 ? 512 : (sizeof(R) * V == 8 ? 768 : 1024);
// the same of the cluster kernel, whose items take more registers
template <typename R, int V>
constexpr int kClusterThreads = sizeof(R) * V == 16 ? 512 : (sizeof(R) * V == 8 ? 640 : 768);
constexpr int kPersistDeg = 3;  // row entries whose gathers are issued together
constexpr int kPersistBatch = 4;  // terms whose products are reduced together

// The terms p_k = (2/a) H p_{k-1} - p_{k-2}, k0 <= k <= k1, of a problem whose
// vectors stay in L2 for the most part (persist_shape: up to 160 MB of matrix and
// vectors, where L2 has 126), under one cooperative launch: a grid barrier per
// term instead of a launch per term.  What bounds it is latency, not bytes: a
// barrier round trip and a gather per item of a thread (a row's pack of V columns).
// So nothing else waits: an item's columns (up to kPersistDeg) are in registers when
// its turn comes, the first one's when the barrier opens, and its matrix values, the
// next item's columns and the row bounds of the one after it are loaded beside its
// gathers (values and columns one item ahead, but after the gathers: 19.8 us a term for
// 320,000 orbitals x 5 FP64 states, 17.3 us so; 32,768 x 1: 3.3 and 2.9).  p_k, which other SMs wrote in this launch, is read by
// ordinary loads: the acquire and the fence after the barrier make the writes
// visible, and neighbouring rows of a tile then hit L1.  A term's two products per
// column stay in shared memory per thread and are reduced every kPersistBatch terms, one
// warp per product: the reduction's barriers were as long as the grid's.
//
// ACC: expansions (Fermi operators, psi_t's jumps) instead of moments; the sums
// are formed in FP64 as in the launched terms, so states are bit-identical.
template <typename R, int V, bool ACC>
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
  // columns and row bounds of the current item, row bounds of the next one
  int j0 = 0, j1 = 0, n0 = 0, n1 = 0;
  int c[kPersistDeg];
  auto next_row = [&](int64_t r) { return r + stride < n ? r + stride : r_first; };
  const bool any = in && r_first < n;
  if (any) {
    j0 = __ldg(a.indptr + r_first);
    j1 = __ldg(a.indptr + r_first + 1);
    n0 = __ldg(a.indptr + next_row(r_first));
    n1 = __ldg(a.indptr + next_row(r_first) + 1);
#pragma unroll
    for (int u = 0; u < kPersistDeg; ++u)
      c[u] = j0 + u < j1 ? __ldg(a.indices + j0 + u) : -1;
  }
  __syncthreads();
  const R alpha2 = (R)a.alpha, alpha1 = (R)(0.5 * a.alpha);
  const R sgn = a.turn ? (R)1 : (R)-1;  // of p_{k-2}
  for (int k = a.k0; k <= a.k1; ++k) {
    const Pack<R, V>* src = k == 1 ? a.p0 : a.ring[(k - 1) % a.slots];
    const Pack<R, V>* prv = k == 2 ? a.p0 : a.ring[(k + a.slots - 2) % a.slots];
    Pack<R, V>* dst = a.ring[k % a.slots];
    const bool dots = !ACC && k <= a.k_dots;
    const bool flush = ACC && k % 3 == 2;
    double fw[2][3];
    if (flush) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        fw[0][q] = __ldg(a.w + k - 2 + q);
        fw[1][q] = __ldg(a.w + a.n_w + k - 2 + q);
      }
    }
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
          if (c[u] >= 0) x[u] = ld_pack(src + (int64_t)c[u] * tpr + lane);
        const Pack<R, V> own = ld_pack(src + e);
        Pack<R, V> pm2;
        if (k >= 2) {
          pm2 = ld_pack(prv + e);
        } else {
#pragma unroll
          for (int q = 0; q < 2 * V; ++q) pm2.v[q] = (R)0;
        }
        // beside the gathers: this item's values, the next one's columns and the
        // bounds of the one after it
        C h[kPersistDeg];
        C d;
        d.x = d.y = (R)0;
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u)
          if (c[u] >= 0) h[u] = ldg_c(a.hop + j0 + u);
        if (a.diag) d = ldg_c(a.diag + r);
        int c_next[kPersistDeg];
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u)
          c_next[u] = n0 + u < n1 ? __ldg(a.indices + n0 + u) : -1;
        const int64_t r2 = next_row(next_row(r));
        const int m0 = __ldg(a.indptr + r2), m1 = __ldg(a.indptr + r2 + 1);
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
        for (int jb = j0 + kPersistDeg; jb < j1; jb += kPersistDeg) {  // longer rows
#pragma unroll
          for (int u = 0; u < kPersistDeg; ++u)
            if (jb + u < j1) {
              h[u] = ldg_c(a.hop + jb + u);
              x[u] = ld_pack(src + (int64_t)__ldg(a.indices + jb + u) * tpr + lane);
            }
#pragma unroll
          for (int u = 0; u < kPersistDeg; ++u)
            if (jb + u < j1) {
#pragma unroll
              for (int v = 0; v < V; ++v) {
                sre[v] = fma(h[u].x, x[u].v[2 * v], fma(-h[u].y, x[u].v[2 * v + 1], sre[v]));
                sim[v] = fma(h[u].x, x[u].v[2 * v + 1], fma(h[u].y, x[u].v[2 * v], sim[v]));
              }
            }
        }
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u) c[u] = c_next[u];
        j0 = n0;
        j1 = n1;
        n0 = m0;
        n1 = m1;
        Pack<R, V> pk;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const R br = a.turn ? sim[v] : sre[v], bi = a.turn ? -sre[v] : sim[v];
          pk.v[2 * v] = fma(al, br, sgn * pm2.v[2 * v]);
          pk.v[2 * v + 1] = fma(al, bi, sgn * pm2.v[2 * v + 1]);
          if (!ACC) {
            const double xr = (double)pk.v[2 * v], xi = (double)pk.v[2 * v + 1];
            nrm[v] += xr * xr + xi * xi;
            cre[v] += xr * (double)own.v[2 * v] + xi * (double)own.v[2 * v + 1];
          }
        }
        if (flush) {
          Pack<R, V> acc;
          if (k > 2) acc = ld_pack(a.acc + e);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int set = (int)(a.set_mask >> (lane * V + v)) & 1;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int i = 2 * v + q;
              double sum = k > 2 ? (double)acc.v[i] : 0.0;
              sum += (set ? fw[1][0] : fw[0][0]) * (double)pm2.v[i];
              sum += (set ? fw[1][1] : fw[0][1]) * (double)own.v[i];
              sum += (set ? fw[1][2] : fw[0][2]) * (double)pk.v[i];
              acc.v[i] = (R)sum;
            }
          }
          stwb_pack(a.acc + e, acc);
        }
        stwb_pack(dst + e, pk);
      }
    }
    // the products of this term: psm[slot of the batch][column value][thread row]
    const int bs = (k - a.k0) % kPersistBatch;
    if (dots && in) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        psm[(bs * width + (lane * V + v) * 2) * rpp + slot] = nrm[v];
        psm[(bs * width + (lane * V + v) * 2 + 1) * rpp + slot] = cre[v];
      }
    }
    // arrive, then reduce a full batch of products while the others arrive
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && k < a.k1) atomicAdd(a.bar, 1u);
    const int k_end = min(a.k1, a.k_dots);  // last term with products
    if (dots && (bs == kPersistBatch - 1 || k == k_end)) {
      const int warp = threadIdx.x >> 5, wl = threadIdx.x & 31;
      const int full = blockDim.x >> 5;  // a partial last warp takes no part
      const int64_t k_first = k - bs - a.k0;
      for (int q = warp < full ? warp : (bs + 1) * width; q < (bs + 1) * width; q += full) {
        double t = 0.0;
        for (int i = wl; i < rpp; i += 32) t += psm[q * rpp + i];
        for (int sft = 16; sft > 0; sft >>= 1) t += __shfl_xor_sync(0xffffffffu, t, sft);
        if (wl == 0) a.partials[(k_first * ld2 + q) * gridDim.x + blockIdx.x] = t;
      }
    }
    if (k == a.k1) break;
    if (threadIdx.x == 0) {
      const unsigned int want = (unsigned int)(k - a.k0 + 1) * gridDim.x + a.absent;
      unsigned long long t0 = 0;
      for (unsigned int spin = 0;; ++spin) {
        unsigned int seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
        if (seen >= want) break;
        if ((spin & 255u) == 255u) {
          unsigned long long now;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          if (now - t0 > a.wait_ns) {
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

// ---- tiny problems in the shared memory of one cluster -------------------------

template <typename R, int V>
struct ClusterArgs {
  const int32_t* indptr;
  const int32_t* indices;
  const typename Cx<R>::t* hop;
  const typename Cx<R>::t* diag;
  int n_rows;
  int tpr;
  Pack<R, V>* even;    // p_{k0-1} and p_{k0-2} (absent at k0 = 1) by their parity;
  Pack<R, V>* odd;     // with `keep`, p_{k1} and p_{k1-1} on return
  double alpha;        // 2 / a
  int k0, k1;          // terms k0 <= k <= k1 of this launch
  int keep;
  int rows;            // rows per block: block q owns rows [q*rows, (q+1)*rows)
  unsigned int magic;  // ceil(2^32 / rows): c / rows = umulhi(c, magic) for c*rows < 2^32
  double* partials;    // [((k-k0)*ld*2 + col*2 + q) * gridDim.x + block]
};

constexpr int kClusterBlocks = 16;
constexpr int kClusterItems = 2;  // most items of a thread (their matrix rows stay in registers)

__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Arrival and wait of every thread of the cluster, releasing its writes.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// 16 bytes (8 for one complex64) of a block of the cluster
__device__ __forceinline__ void cluster_ld(uint32_t a, double* v) {
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a)
               : "memory");
}
__device__ __forceinline__ void cluster_ld(uint32_t a, float* v) {
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(a)
               : "memory");
}
__device__ __forceinline__ void cluster_ld4(uint32_t a, float* v) {
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(a)
               : "memory");
}
template <typename R, int V>
__device__ __forceinline__ Pack<R, V> cluster_ld_pack(uint32_t a) {
  Pack<R, V> p;
  if constexpr (sizeof(R) == 4 && V >= 2) {
#pragma unroll
    for (int q = 0; q < V / 2; ++q) cluster_ld4(a + 16 * q, p.v + 4 * q);
  } else {
#pragma unroll
    for (int q = 0; q < V; ++q) cluster_ld(a + 2 * sizeof(R) * q, p.v + 2 * q);
  }
  return p;
}

// The moments' terms of a problem whose two vectors fit the shared memory of one
// cluster of 16 blocks.  A term of cheb_persist_kernel is a grid barrier through L2
// and a gather from L2; here it is the hardware barrier of the cluster and a
// gather from distributed shared memory, on 16 SMs instead of 148, so it is
// the better one while a thread has few items: their matrix rows then stay in
// registers.
template <typename R, int V>
__global__ void __launch_bounds__((kClusterThreads<R, V>), 1)
    cheb_cluster_kernel(const __grid_constant__ ClusterArgs<R, V> a) {
  using C = typename Cx<R>::t;
  extern __shared__ __align__(128) char csm[];
  const int tpr = a.tpr, rows = a.rows;
  const int slot = threadIdx.x / tpr;
  const int lane = threadIdx.x - slot * tpr;
  const int rpp = blockDim.x / tpr;
  const int r_base = blockIdx.x * rows;
  const int n_own = max(0, min(rows, a.n_rows - r_base));
  const int vec = rows * tpr;  // packs of a vector per block
  Pack<R, V>* buf = reinterpret_cast<Pack<R, V>*>(csm);  // p_even | p_odd
  double* psm = reinterpret_cast<double*>(csm + 2 * (size_t)vec * sizeof(Pack<R, V>));
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(csm);
  const uint32_t odd = (uint32_t)(vec * sizeof(Pack<R, V>));
  const int width = tpr * V * 2;
  const bool any = slot < rpp && slot < n_own;
  for (int q = threadIdx.x; q < n_own * tpr; q += blockDim.x) {
    const int64_t e = (int64_t)r_base * tpr + q;
    buf[q] = a.even[e];
    if (a.k0 > 1) buf[vec + q] = a.odd[e];
  }
  // matrix entries of the thread's items; ca: address of a neighbour in p_even
  constexpr int NI = kClusterItems;
  int j0[NI], j1[NI];
  uint32_t ca[NI][kPersistDeg];
  C h[NI][kPersistDeg], d[NI];
  auto neighbour = [&](int c) {
    const uint32_t q = __umulhi((uint32_t)c, a.magic);
    const uint32_t l = (uint32_t)c - q * (uint32_t)rows;
    return cluster_map(base + (l * (uint32_t)tpr + (uint32_t)lane) * (uint32_t)sizeof(Pack<R, V>),
                       q);
  };
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int r = slot + i * rpp;
    j0[i] = j1[i] = 0;
    d[i].x = d[i].y = (R)0;
    if (any && r < n_own) {
      j0[i] = __ldg(a.indptr + r_base + r);
      j1[i] = __ldg(a.indptr + r_base + r + 1);
      if (a.diag) d[i] = ldg_c(a.diag + r_base + r);
    }
#pragma unroll
    for (int u = 0; u < kPersistDeg; ++u)
      if (j0[i] + u < j1[i]) {
        ca[i][u] = neighbour(__ldg(a.indices + j0[i] + u));
        h[i][u] = ldg_c(a.hop + j0[i] + u);
      }
  }
  cluster_sync();
  const R alpha2 = (R)a.alpha, alpha1 = (R)(0.5 * a.alpha);
  for (int k = a.k0; k <= a.k1; ++k) {
    const uint32_t so = (k & 1) ? 0u : odd;  // p_{k-1}
    const Pack<R, V>* src = buf + ((k & 1) ? 0 : vec);
    Pack<R, V>* dst = buf + ((k & 1) ? vec : 0);
    const R al = k == 1 ? alpha1 : alpha2;
    double nrm[V], cre[V];
#pragma unroll
    for (int v = 0; v < V; ++v) nrm[v] = cre[v] = 0.0;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int r = slot + i * rpp;
      if (any && r < n_own) {
        const int e = r * tpr + lane;
        Pack<R, V> x[kPersistDeg];
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u)
          if (j0[i] + u < j1[i]) x[u] = cluster_ld_pack<R, V>(ca[i][u] + so);
        const Pack<R, V> own = src[e];
        Pack<R, V> pm2;
        if (k >= 2) {
          pm2 = dst[e];
        } else {
#pragma unroll
          for (int q = 0; q < 2 * V; ++q) pm2.v[q] = (R)0;
        }
        R sre[V], sim[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          sre[v] = d[i].x * own.v[2 * v] - d[i].y * own.v[2 * v + 1];
          sim[v] = d[i].x * own.v[2 * v + 1] + d[i].y * own.v[2 * v];
        }
#pragma unroll
        for (int u = 0; u < kPersistDeg; ++u)
          if (j0[i] + u < j1[i]) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
              sre[v] = fma(h[i][u].x, x[u].v[2 * v], fma(-h[i][u].y, x[u].v[2 * v + 1], sre[v]));
              sim[v] = fma(h[i][u].x, x[u].v[2 * v + 1], fma(h[i][u].y, x[u].v[2 * v], sim[v]));
            }
          }
        for (int j = j0[i] + kPersistDeg; j < j1[i]; ++j) {
          const C hj = ldg_c(a.hop + j);
          const Pack<R, V> xj = cluster_ld_pack<R, V>(neighbour(__ldg(a.indices + j)) + so);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            sre[v] = fma(hj.x, xj.v[2 * v], fma(-hj.y, xj.v[2 * v + 1], sre[v]));
            sim[v] = fma(hj.x, xj.v[2 * v + 1], fma(hj.y, xj.v[2 * v], sim[v]));
          }
        }
        Pack<R, V> pk;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          pk.v[2 * v] = fma(al, sre[v], -pm2.v[2 * v]);
          pk.v[2 * v + 1] = fma(al, sim[v], -pm2.v[2 * v + 1]);
          const double xr = (double)pk.v[2 * v], xi = (double)pk.v[2 * v + 1];
          nrm[v] += xr * xr + xi * xi;
          cre[v] += xr * (double)own.v[2 * v] + xi * (double)own.v[2 * v + 1];
        }
        dst[e] = pk;
      }
    }
    // products per thread, reduced in batches as in cheb_persist_kernel
    const int bs = (k - a.k0) % kPersistBatch;
    if (slot < rpp) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        psm[(bs * width + (lane * V + v) * 2) * rpp + slot] = nrm[v];
        psm[(bs * width + (lane * V + v) * 2 + 1) * rpp + slot] = cre[v];
      }
    }
    cluster_sync();
    if (bs == kPersistBatch - 1 || k == a.k1) {
      const int warp = threadIdx.x >> 5, wl = threadIdx.x & 31;
      const int full = blockDim.x >> 5;  // a partial last warp takes no part
      const int64_t k_first = k - a.k0 - bs;
      for (int q = warp < full ? warp : (bs + 1) * width; q < (bs + 1) * width; q += full) {
        double t = 0.0;
        for (int i = wl; i < rpp; i += 32) t += psm[q * rpp + i];
        for (int sft = 16; sft > 0; sft >>= 1) t += __shfl_xor_sync(0xffffffffu, t, sft);
        if (wl == 0) a.partials[(k_first * width + q) * gridDim.x + blockIdx.x] = t;
      }
      __syncthreads();  // the batch's slots are free again
    }
  }
  if (a.keep)
    for (int q = threadIdx.x; q < n_own * tpr; q += blockDim.x) {
      const int64_t e = (int64_t)r_base * tpr + q;
      a.even[e] = buf[q];
      a.odd[e] = buf[vec + q];
    }
}

// ---- packed realisations ------------------------------------------------------

// *coupled becomes nonzero when an entry leads from one realisation to another
// (1.4M rows: 14 us beside 16 ms of terms).
// Block (row chunk, realisation), threads over rows.
static __global__ void __launch_bounds__(256) seg_closed_kernel(const int64_t* seg_off,
                                                                const int32_t* indptr,
                                                                const int32_t* indices,
                                                                unsigned int* coupled) {
  const int64_t s0 = seg_off[blockIdx.y], s1 = seg_off[blockIdx.y + 1];
  bool out = false;
  for (int64_t r = s0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < s1;
       r += (int64_t)gridDim.x * blockDim.x)
    for (int j = indptr[r]; j < indptr[r + 1]; ++j) out |= indices[j] < s0 || indices[j] >= s1;
  if (__syncthreads_or(out) && threadIdx.x == 0) atomicOr(coupled, 1u);
}

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

// out[(seg*ns2 + v)] = sum of the entries [first[seg], first[seg+1]) x per_tile of one
// term, entries of ns2 values; block (seg, term), fixed order.  Terms follow
// each other at `stride` doubles in `partials`, n_seg*ns2 doubles in `out`.
static __global__ void __launch_bounds__(256) seg_tile_reduce_kernel(const double* partials,
                                                                     int64_t stride,
                                                                     const int* first, int per_tile,
                                                                     int ns2, double* out) {
  __shared__ double red[256];
  const int seg = blockIdx.x;
  const int groups = 256 / ns2;
  const int grp = threadIdx.x / ns2;
  const int v = threadIdx.x - grp * ns2;
  const double* p = partials + blockIdx.y * stride;
  const int64_t e0 = (int64_t)first[seg] * per_tile, e1 = (int64_t)first[seg + 1] * per_tile;
  double s = 0.0;
  if (grp < groups)
    for (int64_t e = e0 + grp; e < e1; e += groups) s += p[e * ns2 + v];
  red[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < ns2) {
    double t = 0.0;
    for (int g = 0; g < groups; ++g) t += red[g * ns2 + threadIdx.x];
    out[((int64_t)blockIdx.y * gridDim.x + seg) * ns2 + threadIdx.x] = t;
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

// (row, state) pairs per staged tile of qe_filter_mma_kernel: 32 KB a buffer
template <typename R>
constexpr int kFilterPairs = sizeof(R) == 8 ? 64 : 128;
// Rows per tile: about that many pairs, rows * nb a multiple of 4.
template <typename R>
__host__ __device__ constexpr int qe_filter_rows(int nb) {
  const int q = nb % 4 == 0 ? 1 : (nb % 2 == 0 ? 2 : 4);  // rows that make whole 8-column tiles
  const int r = (kFilterPairs<R> + nb - 1) / nb;
  return (r + q - 1) / q * q;
}
// Shared memory: two buffers of the window's values of a tile, [tau][pair], the
// pairs padded by 64 bytes, so that the four tau of a fragment load lie in
// different banks.
template <typename R>
constexpr int kFilterPad = sizeof(R) == 8 ? 4 : 8;
template <typename R>
__host__ __device__ constexpr size_t qe_filter_smem(int nb) {
  return 2 * (size_t)kFilterWindow * (qe_filter_rows<R>(nb) * nb + kFilterPad<R>) * 2 * sizeof(R);
}

// QE[r][i][b] (+)= sum_{tau < T} c[tau][i] p_tau[r][b], c real: per tile of
// (row, state) pairs a real product A (energies x 32) . B (32 x (pair, re/im)),
// with the fragments and the split over warps of qe_accum_mma_kernel (whose
// +/- windows need 2 x 16 coefficients for 16 steps).  A window of 32 vectors
// per pass over QE: at 16 the pass over QE (32 bytes a complex128 element
// against 32 FMAs) was the longer side.  The next tile's values are on their
// way into the other buffer (cp.async) during the products, and a warp's QE
// elements of the next column tile are loaded before the products of the
// current one: one barrier per tile.  (Staged by plain loads in tiles of 32
// pairs: 57 energies x 4 FP32 states of 307,200 rows took 843 us per pass, 1.3
// TB/s; 7 energies x 2 FP64 states of 192,640 rows 189 us.)
template <typename R>
__global__ void __launch_bounds__(kQeMmaWarps * 32, 2) qe_filter_mma_kernel(
    typename Cx<R>::t* qe, int64_t n_rows, int n_en, int nb,
    const __grid_constant__ FilterPtrs<R> win, int T, const double* coef, int init) {
  using C = typename Cx<R>::t;
  extern __shared__ double2 qsm[];
  const int RT = qe_filter_rows<R>(nb);
  const int P = RT * nb;  // pairs of a tile; P % 4 == 0
  const int PS = P + kFilterPad<R>;
  C* buf[2] = {reinterpret_cast<C*>(qsm), reinterpret_cast<C*>(qsm) + kFilterWindow * PS};
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
  // vectors past the window (tau >= T) are zeroed once; their coefficients are
  // zero too, but what lies in shared memory need not be finite
  for (int q = threadIdx.x; q < 2 * kFilterWindow * PS; q += blockDim.x) {
    C z;
    z.x = z.y = (R)0;
    buf[0][q] = z;
  }
  __syncthreads();
  auto issue = [&](int64_t r0, C* dst) {
    if (r0 < n_rows) {
      const int np = (int)min((int64_t)RT, n_rows - r0) * nb;
      // a warp per vector: consecutive lanes copy consecutive pairs
      for (int tau = warp; tau < T; tau += kQeMmaWarps) {
        const C* src = win.p[tau] + r0 * nb;
        for (int q = lane; q < np; q += 32) qe_cp_async(dst + tau * PS + q, src + q);
      }
    }
    qe_cp_commit();
  };
  const int64_t r_first = (int64_t)blockIdx.x * RT, r_step = (int64_t)gridDim.x * RT;
  issue(r_first, buf[0]);
  int cur = 0;
  for (int64_t r0 = r_first; r0 < n_rows; r0 += r_step, cur ^= 1) {
    const int nr = (int)min((int64_t)RT, n_rows - r0);
    const int np = nr * nb;  // pairs in range
    C* base = qe + r0 * n_en * nb;
    // offset of the lane's element of energy tile 0 in the rows of this tile
    auto at = [&](int pc) {
      const int rr = pc / nb;
      return (rr * n_en + mt0 * 8 + g) * nb + (pc - rr * nb);
    };
    auto load_c = [&](int nt, C* v) {
      const int pc = 4 * nt + t;
      const int o = at(pc);
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        v[m].x = v[m].y = (R)0;
        if (!init && pc < np && (mt0 + m) * 8 + g < n_en) v[m] = base[o + 8 * m * nb];
      }
    };
    // (FP64 elements are loaded at their use: a second set spilled)
    constexpr bool ahead = sizeof(R) == 4;
    C cv[kQeMmaMT];
    if (ahead) load_c(nt_first, cv);
    qe_cp_wait_all();
    __syncthreads();  // this tile has landed; the other buffer is consumed
    issue(r0 + r_step, buf[cur ^ 1]);
    const R* tile = reinterpret_cast<const R*>(buf[cur]);
    for (int nt = nt_first; 4 * nt < np; nt += nt_step) {
      // B fragment: B[k = 4*s + t][n = g]; column g is pair 4*nt + g/2, part g&1
      const R* b = tile + 8 * nt + g;
      double bfr[kFilterWindow / 4];
#pragma unroll
      for (int st = 0; st < kFilterWindow / 4; ++st) bfr[st] = (double)b[(4 * st + t) * 2 * PS];
      double c0[kQeMmaMT], c1[kQeMmaMT];
      if (!ahead) load_c(nt, cv);
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        c0[m] = (double)cv[m].x;
        c1[m] = (double)cv[m].y;
      }
      if (ahead) load_c(nt + nt_step, cv);
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        if (mt0 + m < n_mt) {
#pragma unroll
          for (int st = 0; st < kFilterWindow / 4; ++st)
            dmma_8x8x4(c0[m], c1[m], afr[m][st], bfr[st]);
        }
      }
      const int pc = 4 * nt + t;
      const int o = at(pc);
#pragma unroll
      for (int m = 0; m < kQeMmaMT; ++m) {
        if (pc < np && (mt0 + m) * 8 + g < n_en) {
          C v;
          v.x = (R)c0[m];
          v.y = (R)c1[m];
          base[o + 8 * m * nb] = v;
        }
      }
    }
  }
  qe_cp_wait_all();
}

// ---- several time steps from one expansion ----------------------------------------

constexpr int kCombineWindow = 32;  // Chebyshev vectors per pass
constexpr int kCombineSteps = 16;   // most time steps per expansion

template <typename R>
struct CombineArgs {
  const typename Cx<R>::t* p[kCombineWindow];
  typename Cx<R>::t* out[kCombineSteps];
  double w[kCombineSteps][kCombineWindow];  // zero where an output has no such term
  int64_t total;                            // values of a block
  int np;                                   // vectors of this pass
  int j0, m;                                // outputs j0 <= j < m take part
  int init;                                 // 1: the outputs start here (are not read)
};

// out_j[e] (+)= sum_tau w[j][tau] p_tau[e] for up to 16 outputs: the states
// after 1..m time steps all come from the same Chebyshev vectors, so m steps of
// phase tau take n(m tau) products with H instead of m n(tau) (AC: 57 instead of
// 240 for 16 steps).  Sums in FP64; both kernels are bound by memory when their
// loads are in flight early enough:
//  combine_kernel (FP64): one value per thread, 16 accumulators, the weights
//    compile-time offsets into the parameter bank.  Blocks of 196 MB, 16 steps: 3.1 ms
//    an expansion in windows of 32 vectors, 4.2 ms in windows of 16 (the outputs are
//    read and written more often), 6.3 TB/s; the product on mma.sync took 25% more.
//  combine_mma_kernel (FP32): blocks of 20 MB, 8 steps of 42 vectors: 0.61 ms an
//    expansion; 0.83 ms with 8-byte loads, pointers from the parameter bank in the
//    loop and windows of 16.  combine_kernel took 1.4 times that, with a conversion
//    for every 32 FMAs.
// p_0 may be an output: every p of a value is read before the value is written.
template <typename R, int M>
__global__ void __launch_bounds__(256, 2) combine_kernel(const __grid_constant__ CombineArgs<R> a) {
  using C = typename Cx<R>::t;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.total) return;
  double re[M], im[M];
#pragma unroll
  for (int j = 0; j < M; ++j) {
    re[j] = im[j] = 0.0;
    if (!a.init && j >= a.j0 && j < a.m) {
      const C o = a.out[j][e];
      re[j] = (double)o.x;
      im[j] = (double)o.y;
    }
  }
#pragma unroll
  for (int q0 = 0; q0 < kCombineWindow; q0 += 8) {
    if (q0 < a.np) {
      C p[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        p[q].x = p[q].y = (R)0;
        if (q0 + q < a.np) p[q] = a.p[q0 + q][e];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
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

// W (8 x window) . P (window x values) on mma.sync m8n8k4 f64.  A warp takes 16
// values at a time: lane (g, t) loads p_tau of values 2g and 2g + 1 for tau = 4s + t;
// the even and the odd values, real and imaginary parts, are the 8 columns of four
// products, so that a lane's accumulators are values 4t .. 4t + 3 of output g: 32
// bytes in a row.  W and the pointers (read by lane, so not from the parameter bank
// in the loop) stay in registers.  WIDE: whole groups of four values at 16-byte
// boundaries; else each value is checked and moved by itself.
template <bool WIDE>
__global__ void __launch_bounds__(256, 2)
    combine_mma_kernel(const __grid_constant__ CombineArgs<float> a) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  constexpr int NS = kCombineWindow / 4;
  double w[NS];
  const float2* p[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) p[s] = 4 * s + t < a.np ? a.p[4 * s + t] : nullptr;
#pragma unroll
  for (int s = 0; s < NS; ++s) w[s] = a.w[g][4 * s + t];
  const bool in = g >= a.j0 && g < a.m;
  float2* const out = in ? a.out[g] : nullptr;
  const int64_t step = 16 * (int64_t)gridDim.x * (blockDim.x >> 5);
  // values e, e + 1
  auto ld2 = [&](const float2* q, int64_t e) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if constexpr (WIDE) {
      if (e < a.total) v = *reinterpret_cast<const float4*>(q + e);
    } else {
      if (e < a.total) {
        const float2 u = q[e];
        v.x = u.x;
        v.y = u.y;
      }
      if (e + 1 < a.total) {
        const float2 u = q[e + 1];
        v.z = u.x;
        v.w = u.y;
      }
    }
    return v;
  };
  for (int64_t e0 = 16 * ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
       e0 < a.total; e0 += step) {
    float4 x[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s)
      x[s] = p[s] ? ld2(p[s], e0 + 2 * g) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int64_t e = e0 + 4 * t;
    double re[2][2], im[2][2];  // [odd value][column 2t, 2t + 1]
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (!a.init && in) o = ld2(out, e + 2 * q);
      re[0][q] = (double)o.x;
      im[0][q] = (double)o.y;
      re[1][q] = (double)o.z;
      im[1][q] = (double)o.w;
    }
#pragma unroll
    for (int s = 0; s < NS; ++s)
      if (4 * s < a.np) {
        dmma_8x8x4(re[0][0], re[0][1], w[s], (double)x[s].x);
        dmma_8x8x4(im[0][0], im[0][1], w[s], (double)x[s].y);
        dmma_8x8x4(re[1][0], re[1][1], w[s], (double)x[s].z);
        dmma_8x8x4(im[1][0], im[1][1], w[s], (double)x[s].w);
      }
    __syncwarp();  // an output may be p_0: the warp has read these values
    if (in) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 o = make_float4((float)re[0][q], (float)im[0][q], (float)re[1][q],
                                     (float)im[1][q]);
        const int64_t f = e + 2 * q;
        if constexpr (WIDE) {
          if (f < a.total) *reinterpret_cast<float4*>(out + f) = o;
        } else {
          if (f < a.total) out[f] = make_float2(o.x, o.y);
          if (f + 1 < a.total) out[f + 1] = make_float2(o.z, o.w);
        }
      }
    }
  }
}

}  // namespace tbpm
