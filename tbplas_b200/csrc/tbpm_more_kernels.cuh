// Kernels of the TBPM drivers beyond DOS / AC / DC / psi(t):
//  dynamical polarisation  (tbpm.f90:355-493, funcs.f90:125-149)
//  quasi-eigenstates       (tbpm.f90:721-830; the QE accumulation is shared with DC)
//  Kubo-Bastin mu_mn       (tbpm.f90:836-960)
//  Haydock recursion       (propagation.f90:85-155)
#pragma once

#include "tbpm_common.cuh"
#include "tbpm_kernels.cuh"

namespace tbpm {

// up to kMaxCols q-points per launch
struct QBlock {
  double q[kMaxCols][3];
};

// q.r in the reference's order (q1*x + q2*y) + q3*z, without FMA contraction
__device__ __forceinline__ double q_dot_r(const double* q, double x, double y, double z) {
  return __dadd_rn(__dadd_rn(__dmul_rn(q[0], x), __dmul_rn(q[1], y)), __dmul_rn(q[2], z));
}

// Block of nq*nb + nb columns: psi1 of q-point k and state b at column k*nb + b
// gets exp(-i q_k.r) wf0_b (tbpm.f90:456), psi2 of state b (column nq*nb + b)
// gets wf0_b.
template <typename R>
__global__ void dens_init_kernel(const typename Cx<R>::t* W, const double* sx, const double* sy,
                                 const double* sz, QBlock qb, int nq, int nb, int64_t n_rows,
                                 typename Cx<R>::t* A) {
  const int ld = (nq + 1) * nb;
  const int64_t total = n_rows * ld;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = g / ld;
    const int col = (int)(g - r * ld);
    const int k = col / nb;
    const int b = col - k * nb;
    const typename Cx<R>::t w = W[r * nb + b];
    typename Cx<R>::t o = w;
    if (k < nq) {
      double sn, cs;
      sincos(q_dot_r(qb.q[k], sx[r], sy[r], sz[r]), &sn, &cs);
      // (cs - i sn) * w
      const double wr = (double)w.x, wi = (double)w.y;
      o.x = (R)(cs * wr + sn * wi);
      o.y = (R)(cs * wi - sn * wr);
    }
    A[g] = o;
  }
}

// Partials of <psi2_b | exp(i q_k.r) psi1_{k,b}> (re, im) and <psi2_b|psi2_b>
// for every (k, b): partials[((k*nb + b)*3 + v) * gridDim.x + block].
// One thread per (k, b) column of a row slot; rows grid-stride.
template <typename R>
__global__ void __launch_bounds__(256) dens_corr_kernel(const typename Cx<R>::t* A,
                                                        const double* sx, const double* sy,
                                                        const double* sz, QBlock qb, int nq,
                                                        int nb, int64_t n_rows,
                                                        double* partials) {
  extern __shared__ double smem[];
  const int tpr = nq * nb;
  const int slot = threadIdx.x / tpr;
  const int lane = threadIdx.x - slot * tpr;
  const int rpp = blockDim.x / tpr;
  const int k = lane / nb;
  const int b = lane - k * nb;
  const int ld = (nq + 1) * nb;
  double cr = 0.0, ci = 0.0, nn = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * rpp + slot; r < n_rows;
       r += (int64_t)gridDim.x * rpp) {
    const typename Cx<R>::t p1 = A[r * ld + lane];
    const typename Cx<R>::t p2 = A[r * ld + nq * nb + b];
    double sn, cs;
    sincos(q_dot_r(qb.q[k], sx[r], sy[r], sz[r]), &sn, &cs);
    const double ar = (double)p1.x, ai = (double)p1.y;
    const double wr = cs * ar - sn * ai, wi = cs * ai + sn * ar;  // exp(i q.r) psi1
    const double qr = (double)p2.x, qi = (double)p2.y;
    cr += qr * wr + qi * wi;
    ci += qr * wi - qi * wr;
    nn += qr * qr + qi * qi;
  }
  const int width = tpr * 3;
  smem[slot * width + lane * 3 + 0] = cr;
  smem[slot * width + lane * 3 + 1] = ci;
  smem[slot * width + lane * 3 + 2] = nn;
  __syncthreads();
  tree_reduce_slots(smem, rpp, width, slot, lane, tpr);
  if (slot == 0) {
#pragma unroll
    for (int v = 0; v < 3; ++v)
      partials[(int64_t)(lane * 3 + v) * gridDim.x + blockIdx.x] = smem[lane * 3 + v];
  }
}

// Block partials of sum_r |QE[r][ib]|^2, one thread per (energy, state) ib;
// partials[ib * gridDim.x + block].
template <typename R>
__global__ void __launch_bounds__(256) qe_sqnorm_kernel(const typename Cx<R>::t* qe,
                                                        int64_t n_rows, int64_t rows_per_tile,
                                                        int n_ib, double* partials) {
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_tile;
  const int64_t r1 = min(r0 + rows_per_tile, n_rows);
  for (int ib = threadIdx.x; ib < n_ib; ib += blockDim.x) {
    double s = 0.0;
    for (int64_t r = r0; r < r1; ++r) {
      const typename Cx<R>::t q = qe[r * n_ib + ib];
      s += (double)q.x * (double)q.x + (double)q.y * (double)q.y;
    }
    partials[(int64_t)ib * gridDim.x + blockIdx.x] = s;
  }
}

// acc[r][i] += scale * sum_b |QE[r][i][b]|^2 / nrm2[i*nb + b]   (tbpm.f90:803-813)
template <typename R>
__global__ void qe_density_kernel(const typename Cx<R>::t* qe, int64_t n_rows, int n_en, int nb,
                                  const double* nrm2, double scale, double* acc) {
  const int64_t total = n_rows * n_en;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = g / n_en;
    const int i = (int)(g - r * n_en);
    double s = 0.0;
    for (int b = 0; b < nb; ++b) {
      const typename Cx<R>::t q = qe[(r * n_en + i) * nb + b];
      s += ((double)q.x * (double)q.x + (double)q.y * (double)q.y) / nrm2[i * nb + b];
    }
    acc[g] += scale * s;
  }
}

// ---- single-vector kernels (Kubo-Bastin, Haydock) ---------------------------

// y = alpha * (H x) + beta * z, H = D + O (z may alias y; beta == 0 ignores z)
template <typename R>
__global__ void cheb_vec_kernel(const int32_t* indptr, const int32_t* indices,
                                const typename Cx<R>::t* hop, const typename Cx<R>::t* diag,
                                int64_t n_rows, double alpha, double beta,
                                const typename Cx<R>::t* x, const typename Cx<R>::t* z,
                                typename Cx<R>::t* y) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows;
       r += (int64_t)gridDim.x * blockDim.x) {
    double vr = 0.0, vi = 0.0;
    if (diag) {
      const typename Cx<R>::t d = diag[r], w = x[r];
      vr = (double)d.x * (double)w.x - (double)d.y * (double)w.y;
      vi = (double)d.x * (double)w.y + (double)d.y * (double)w.x;
    }
    const int j0 = __ldg(indptr + r), j1 = __ldg(indptr + r + 1);
    for (int j = j0; j < j1; ++j) {
      const typename Cx<R>::t h = ldg_c(hop + j);
      const typename Cx<R>::t w = ldg_c(x + __ldg(indices + j));
      vr += (double)h.x * (double)w.x - (double)h.y * (double)w.y;
      vi += (double)h.x * (double)w.y + (double)h.y * (double)w.x;
    }
    double orr = alpha * vr, oi = alpha * vi;
    if (beta != 0.0) {
      const typename Cx<R>::t zz = z[r];
      orr += beta * (double)zz.x;
      oi += beta * (double)zz.y;
    }
    typename Cx<R>::t o;
    o.x = (R)orr;
    o.y = (R)oi;
    y[r] = o;
  }
}

// y = J_d x with J_d = i * rescale * hop * d on the off-diagonal entries
// (funcs.f90:12-33 + csr.F90:71-101)
template <typename R>
__global__ void current_vec_kernel(const int32_t* indptr, const int32_t* indices,
                                   const typename Cx<R>::t* hop, const R* d, double rescale,
                                   int64_t n_rows, const typename Cx<R>::t* x,
                                   typename Cx<R>::t* y) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows;
       r += (int64_t)gridDim.x * blockDim.x) {
    double vr = 0.0, vi = 0.0;
    const int j0 = __ldg(indptr + r), j1 = __ldg(indptr + r + 1);
    for (int j = j0; j < j1; ++j) {
      const typename Cx<R>::t h = ldg_c(hop + j);
      const double dd = (double)__ldg(d + j);
      const double jr = -rescale * (double)h.y * dd, ji = rescale * (double)h.x * dd;
      const typename Cx<R>::t w = ldg_c(x + __ldg(indices + j));
      vr += jr * (double)w.x - ji * (double)w.y;
      vi += jr * (double)w.y + ji * (double)w.x;
    }
    typename Cx<R>::t o;
    o.x = (R)vr;
    o.y = (R)vi;
    y[r] = o;
  }
}

// One ket step of the Kubo-Bastin moments: y = alpha*(H x) + beta*z (y null: not
// formed) and q = J_d x, from one pass over the matrix and one gather of x.
template <typename R>
__global__ void __launch_bounds__(256) cheb_current_kernel(
    const int32_t* indptr, const int32_t* indices, const typename Cx<R>::t* hop,
    const typename Cx<R>::t* diag, const R* d, double rescale, int64_t n_rows, double alpha,
    double beta, const typename Cx<R>::t* x, const typename Cx<R>::t* z, typename Cx<R>::t* y,
    typename Cx<R>::t* q) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows;
       r += (int64_t)gridDim.x * blockDim.x) {
    double vr = 0.0, vi = 0.0, cr = 0.0, ci = 0.0;
    typename Cx<R>::t zz;
    zz.x = zz.y = (R)0;
    if (y && beta != 0.0) zz = z[r];
    if (y && diag) {
      const typename Cx<R>::t g = diag[r], w = x[r];
      vr = (double)g.x * (double)w.x - (double)g.y * (double)w.y;
      vi = (double)g.x * (double)w.y + (double)g.y * (double)w.x;
    }
    const int j0 = __ldg(indptr + r), j1 = __ldg(indptr + r + 1);
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      const typename Cx<R>::t h = ldg_c(hop + j);
      const double dd = (double)__ldg(d + j);
      const typename Cx<R>::t w = ldg_c(x + __ldg(indices + j));
      vr += (double)h.x * (double)w.x - (double)h.y * (double)w.y;
      vi += (double)h.x * (double)w.y + (double)h.y * (double)w.x;
      const double jr = -rescale * (double)h.y * dd, ji = rescale * (double)h.x * dd;
      cr += jr * (double)w.x - ji * (double)w.y;
      ci += jr * (double)w.y + ji * (double)w.x;
    }
    typename Cx<R>::t o;
    o.x = (R)cr;
    o.y = (R)ci;
    q[r] = o;
    if (y) {
      o.x = (R)(alpha * vr + beta * (double)zz.x);
      o.y = (R)(alpha * vi + beta * (double)zz.y);
      y[r] = o;
    }
  }
}

// ---- Haydock recursion ------------------------------------------------------

template <typename R>
struct HaydockArgs {
  const int32_t* indptr;
  const int32_t* indices;
  const typename Cx<R>::t* hop;
  const typename Cx<R>::t* diag;
  int64_t n_rows;
  double rescale;
  typename Cx<R>::t* w0;  // start vector (overwritten)
  typename Cx<R>::t* w1;
  typename Cx<R>::t* y;
  int n_depth;
  double* a;         // [2 * n_depth]
  double* b;         // [n_depth]
  double* partials;  // [3 * gridDim.x]: <v|y> (re, im), <w|w>
  int cap;               // own rows of w, w_prev and y a thread keeps in shared memory
  unsigned int* bar;     // grid barrier, zero on entry
  unsigned int* status;  // bit 0: a bounded wait ran out
  unsigned int absent;   // arrivals expected beside the grid's (the self-test's: never come)
  unsigned long long wait_ns;  // longest wait
};

constexpr int kHaydockDeg = 3;  // row entries whose gathers are issued together
constexpr size_t kHaydockSmem = 192 * 1024;  // for the threads' own rows

// Arrival of the block on the grid barrier and bounded wait for `want` arrivals;
// false when the wait ran out.  Every thread of the block calls it.
__device__ __forceinline__ bool haydock_barrier(unsigned int* bar, unsigned int want,
                                                unsigned int* status, int* stop,
                                                unsigned long long wait_ns) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(bar, 1u);
    unsigned long long t0 = 0;
    for (unsigned int spin = 0;; ++spin) {
      unsigned int seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if (seen >= want) break;
      if ((spin & 255u) == 255u) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (t0 == 0) t0 = now;
        if (now - t0 > wait_ns) {
          atomicOr(status, 1u);
          *stop = 1;
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *stop == 0;
}

// Sums of a block's N per-thread values, fixed order: value i to out[i * stride].
template <int N>
__device__ __forceinline__ void haydock_block_sums(double (&v)[N], double (*red)[32], double* out,
                                                   int stride) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    for (int s = 16; s > 0; s >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], s);
    if (lane == 0) red[i][warp] = v[i];
  }
  __syncthreads();
  if (warp < N) {  // one warp per value (a block has four warps or more)
    double t = lane < (blockDim.x >> 5) ? red[warp][lane] : 0.0;
    for (int s = 16; s > 0; s >>= 1) t += __shfl_xor_sync(0xffffffffu, t, s);
    if (lane == 0) out[warp * stride] = t;
  }
}

// Sums over the grid's partials of N values, read past L1 (other blocks wrote them in
// this launch), in the same order in every block; to every thread.
template <int N>
__device__ __forceinline__ void haydock_grid_sums(const double* p, int n, double* bcast,
                                                  double (&sum)[N]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < N) {
    double t = 0.0;
    for (int i = lane; i < n; i += 32) t += __ldcg(p + warp * n + i);
    for (int s = 16; s > 0; s >>= 1) t += __shfl_xor_sync(0xffffffffu, t, s);
    if (lane == 0) bcast[warp] = t;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) sum[i] = bcast[i];
}

// Ordinary loads of vectors that other SMs wrote before the last grid barrier
// (volatile: not moved across it, and not through the read-only path); rows that
// neighbours share hit L1.
__device__ __forceinline__ double2 ld_c(const double2* p) {
  const Pack<double, 1> v = ld_pack(reinterpret_cast<const Pack<double, 1>*>(p));
  return make_double2(v.v[0], v.v[1]);
}
__device__ __forceinline__ float2 ld_c(const float2* p) {
  const Pack<float, 1> v = ld_pack(reinterpret_cast<const Pack<float, 1>*>(p));
  return make_float2(v.v[0], v.v[1]);
}

// The whole recursion (propagation.f90:85-155) in one cooperative launch.  With
// w the unnormalised vector and v = w / b_{d-1}:
//   y = rescale H v, a_d = <v|y>;  w' = y - a_d v - b_{d-1} v_prev, b_d = |w'|.
// Two grid barriers per depth (one per inner product) replace five launches, and
// the division by b_d is folded into the next depth instead of taking a pass.
// The matrix and w stay in L2 for some hundred thousand orbitals; what a depth
// then costs is latency: the barriers and the chain from a row's entries to the
// gathered values.  So a row's entries are loaded one item ahead (the first row's
// before the barrier), its gathers are issued together, and a thread's own rows of
// w, w_prev and y (as many as fit the shared memory: `cap` per thread) never leave
// the SM: the second half of a depth then reads nothing from L2.  524,288
// orbitals, per depth: 12.6 us, 16.5 us with the entries in the loop and all
// vectors in L2, 35 us as five launches.
template <typename R, int T_MAX>
__global__ void __launch_bounds__(T_MAX, 1)
    haydock_kernel(const __grid_constant__ HaydockArgs<R> k) {
  using C = typename Cx<R>::t;
  extern __shared__ __align__(16) char hsm[];
  __shared__ double red[2][32];
  __shared__ double bcast[3];
  __shared__ int stop;
  if (threadIdx.x == 0) stop = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int T = blockDim.x, cap = k.cap;
  // own rows: item i of the thread at [i * T]
  C* sw = reinterpret_cast<C*>(hsm) + threadIdx.x;
  C* sp = sw + (size_t)cap * T;
  C* const sy = sp + (size_t)cap * T;
  unsigned int want = k.absent;
  double s = 1.0, s_prev = 0.0, b_prev = 0.0;  // v = s w, v_prev = s_prev w_prev
  C* w = k.w0;
  C* w_prev = k.w1;
  {
    int i = 0;
    for (int64_t r = r0; r < k.n_rows && i < cap; r += stride, ++i) sw[i * T] = ld_c(w + r);
  }
  // columns and row bounds of the current item, row bounds of the next one
  int j0 = 0, j1 = 0, n0 = 0, n1 = 0;
  int c[kHaydockDeg];
  auto next_row = [&](int64_t r) { return r + stride < k.n_rows ? r + stride : r0; };
  if (r0 < k.n_rows) {
    j0 = __ldg(k.indptr + r0);
    j1 = __ldg(k.indptr + r0 + 1);
    n0 = __ldg(k.indptr + next_row(r0));
    n1 = __ldg(k.indptr + next_row(r0) + 1);
#pragma unroll
    for (int u = 0; u < kHaydockDeg; ++u)
      c[u] = j0 + u < j1 ? __ldg(k.indices + j0 + u) : -1;
  }
  __syncthreads();
  for (int d = 0; d < k.n_depth; ++d) {
    double cs[2] = {0.0, 0.0};
    int i = 0;
    for (int64_t r = r0; r < k.n_rows; r += stride, ++i) {
      C x[kHaydockDeg];
#pragma unroll
      for (int u = 0; u < kHaydockDeg; ++u)
        if (c[u] >= 0) x[u] = ld_c(w + c[u]);
      const C own = i < cap ? sw[i * T] : ld_c(w + r);
      // beside the gathers: this item's values, the next one's columns and the
      // bounds of the one after it
      C h[kHaydockDeg];
#pragma unroll
      for (int u = 0; u < kHaydockDeg; ++u)
        if (c[u] >= 0) h[u] = ldg_c(k.hop + j0 + u);
      C g;
      g.x = g.y = (R)0;
      if (k.diag) g = ldg_c(k.diag + r);
      int c_next[kHaydockDeg];
#pragma unroll
      for (int u = 0; u < kHaydockDeg; ++u)
        c_next[u] = n0 + u < n1 ? __ldg(k.indices + n0 + u) : -1;
      const int64_t r2 = next_row(next_row(r));
      const int m0 = __ldg(k.indptr + r2), m1 = __ldg(k.indptr + r2 + 1);
      double vr = 0.0, vi = 0.0;
      if (k.diag) {
        vr = (double)g.x * (double)own.x - (double)g.y * (double)own.y;
        vi = (double)g.x * (double)own.y + (double)g.y * (double)own.x;
      }
#pragma unroll
      for (int u = 0; u < kHaydockDeg; ++u)
        if (c[u] >= 0) {
          vr += (double)h[u].x * (double)x[u].x - (double)h[u].y * (double)x[u].y;
          vi += (double)h[u].x * (double)x[u].y + (double)h[u].y * (double)x[u].x;
        }
      for (int jb = j0 + kHaydockDeg; jb < j1; jb += kHaydockDeg) {  // longer rows
#pragma unroll
        for (int u = 0; u < kHaydockDeg; ++u)
          if (jb + u < j1) {
            h[u] = ldg_c(k.hop + jb + u);
            x[u] = ld_c(w + __ldg(k.indices + jb + u));
          }
#pragma unroll
        for (int u = 0; u < kHaydockDeg; ++u)
          if (jb + u < j1) {
            vr += (double)h[u].x * (double)x[u].x - (double)h[u].y * (double)x[u].y;
            vi += (double)h[u].x * (double)x[u].y + (double)h[u].y * (double)x[u].x;
          }
      }
#pragma unroll
      for (int u = 0; u < kHaydockDeg; ++u) c[u] = c_next[u];
      j0 = n0;
      j1 = n1;
      n0 = m0;
      n1 = m1;
      C o;
      o.x = (R)(vr * s * k.rescale);
      o.y = (R)(vi * s * k.rescale);
      if (i < cap)
        sy[i * T] = o;
      else
        k.y[r] = o;
      const double xr = s * (double)own.x, xi = s * (double)own.y;
      cs[0] += xr * (double)o.x + xi * (double)o.y;
      cs[1] += xr * (double)o.y - xi * (double)o.x;
    }
    haydock_block_sums(cs, red, k.partials + blockIdx.x, (int)gridDim.x);
    want += gridDim.x;
    if (!haydock_barrier(k.bar, want, k.status, &stop, k.wait_ns)) return;
    double a[2];
    haydock_grid_sums(k.partials, (int)gridDim.x, bcast, a);
    const double ar = a[0], ai = a[1];
    double nn[1] = {0.0};
    i = 0;
    for (int64_t r = r0; r < k.n_rows; r += stride, ++i) {
      const bool in = i < cap;
      const C x = in ? sw[i * T] : ld_c(w + r), z = in ? sy[i * T] : ld_c(k.y + r);
      const double xr = s * (double)x.x, xi = s * (double)x.y;
      double vr = (double)z.x - (ar * xr - ai * xi);
      double vi = (double)z.y - (ar * xi + ai * xr);
      if (d > 0) {
        const C p = in ? sp[i * T] : ld_c(w_prev + r);
        vr -= b_prev * (s_prev * (double)p.x);
        vi -= b_prev * (s_prev * (double)p.y);
      }
      C o;
      o.x = (R)vr;
      o.y = (R)vi;
      w_prev[r] = o;
      if (in) sp[i * T] = o;
      nn[0] += (double)o.x * (double)o.x + (double)o.y * (double)o.y;
    }
    haydock_block_sums(nn, red, k.partials + 2 * gridDim.x + blockIdx.x, (int)gridDim.x);
    want += gridDim.x;
    if (!haydock_barrier(k.bar, want, k.status, &stop, k.wait_ns)) return;
    double bb[1];
    haydock_grid_sums(k.partials + 2 * gridDim.x, (int)gridDim.x, bcast + 2, bb);
    const double b = sqrt(bb[0]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      k.a[2 * d] = ar;
      k.a[2 * d + 1] = ai;
      k.b[d] = b;
    }
    C* t = w;
    w = w_prev;
    w_prev = t;
    t = sw;
    sw = sp;
    sp = t;
    s_prev = s;
    s = 1.0 / b;
    b_prev = b;
  }
}

// G00(E + i delta) of the continued fraction (funcs.f90:152-172), one thread per energy.
static __global__ void haydock_green_kernel(const double* a, const double* b, int n_depth,
                                            const double* energies, int n_e, double delta,
                                            double2* g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_e) return;
  const double e = energies[i];
  double gr = 0.0, gi = 0.0;
  for (int d = n_depth - 1; d >= 0; --d) {
    const double b2 = b[d] * b[d];
    const double zr = e - a[2 * d] - b2 * gr;
    const double zi = delta - a[2 * d + 1] - b2 * gi;
    const double q = 1.0 / (zr * zr + zi * zi);
    gr = zr * q;
    gi = -zi * q;
  }
  g[i] = make_double2(gr, gi);
}

}  // namespace tbpm

namespace tbpm {

// analysis.f90:6-69 (cond_from_trace) with kpm.f90:31-56 (get_gamma_mn):
// out[k-1] = sum_{m,n} Re(Gamma_mn(x_k) mu_mn), x_k = k * pi / ne_integral,
// one block per energy; cos(m x), sin(m x) are tabulated in shared memory and
// the threads walk the rows m of mu (column-major), so the reads coalesce.
//   Gamma_mn = (cos x - i n sin x) cos(m x) e^{i n x} + (cos x + i m sin x) cos(n x) e^{-i m x}
__global__ void __launch_bounds__(256) gamma_trace_kernel(const double2* mu, int nk,
                                                          int ne_integral, double* out) {
  extern __shared__ double tab[];  // [0, nk): cos(m x), [nk, 2nk): sin(m x)
  __shared__ double red[256];
  const int k = blockIdx.x + 1;
  const double x = k * (3.14159265358979323846 / ne_integral);
  for (int m = threadIdx.x; m < nk; m += blockDim.x) {
    double s, c;
    sincos(m * x, &s, &c);
    tab[m] = c;
    tab[nk + m] = s;
  }
  __syncthreads();
  double sx, cx;
  sincos(x, &sx, &cx);
  double acc = 0.0;
  for (int n = 0; n < nk; ++n) {
    const double cn = tab[n], sn = tab[nk + n];
    const double a1 = cx * cn + n * sx * sn;  // Re of (cx - i n sx)(Cn + i Sn)
    const double b1 = cx * sn - n * sx * cn;  // Im of the same
    const double2* col = mu + (int64_t)n * nk;
    for (int m = threadIdx.x; m < nk; m += blockDim.x) {
      const double cm = tab[m], sm = tab[nk + m];
      const double re = cm * a1 + cn * (cx * cm + m * sx * sm);
      const double im = cm * b1 + cn * (m * sx * cm - cx * sm);
      const double2 v = col[m];
      acc += re * v.x - im * v.y;
    }
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

}  // namespace tbpm
