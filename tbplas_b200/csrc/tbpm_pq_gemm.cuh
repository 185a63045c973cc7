// The Kubo-Bastin moment contraction of tbpm_kbdc (tbpm.f90:898-957) as one
// complex GEMM with split K:
//
//   cs[i][j] = sum_n conj(P[n, i]) * Q[n, j]      i < m (bra vectors of a chunk),
//                                                 j < nk (ket vectors), n < N
//
// P and Q are column-major N x m and N x nk (column i of P starts at P + i*N):
// both operands are contiguous along the reduction index, as in a "TN" GEMM.
// The reference forms these m*nk inner products one at a time (n_kernel^2
// serial dot products); here a grid of 64 x 64 output tiles and S slices of
// the N rows each accumulate their share in registers.
//
// FP64 runs on pq_dmma_kernel (mma.sync f64, below); pq_gemm_kernel is the FP32
// kernel: 256 threads, output tile 64 (i) x 64 (j), 16 rows of n per
// step staged in shared memory (row length padded to 65 complex values, so the
// transposing stores and the broadcast reads are free of bank conflicts).
// Thread (tx, ty) owns outputs i = ty + 16a, j = tx + 16b (a, b < 4): per step
// it reads 4 + 4 staged values and does 16 complex FMAs.  The next step's
// loads are issued into registers before the current step is computed.  The
// block writes its slice's partial tile to ws[slice][j][i] (FP64).
//
// pq_reduce_kernel sums the slices in a fixed order and adds
// g_i g_j * scale * cs[i][j] to mu[i0 + i + nk*j] (FP64), so results are
// deterministic.  FP32 operands accumulate in FP32 within a slice and in FP64
// across slices.
#pragma once

#include "tbpm_common.cuh"
#include "tbpm_dc_kernels.cuh"

namespace tbpm {

constexpr int kPqTile = 64;
constexpr int kPqK = 16;
constexpr int kPqPad = kPqTile + 1;

template <typename R>
__global__ void __launch_bounds__(256) pq_gemm_kernel(const typename Cx<R>::t* __restrict__ P,
                                                      const typename Cx<R>::t* __restrict__ Q,
                                                      int64_t N, int m, int nk, int64_t rows_per_slice,
                                                      double2* __restrict__ ws) {
  using C = typename Cx<R>::t;
  __shared__ C sP[kPqK][kPqPad];
  __shared__ C sQ[kPqK][kPqPad];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int j0 = blockIdx.x * kPqTile, i0 = blockIdx.y * kPqTile;
  const int slice = blockIdx.z;
  const int64_t n_lo = (int64_t)slice * rows_per_slice;
  const int64_t n_hi = n_lo + rows_per_slice < N ? n_lo + rows_per_slice : N;
  // loader mapping: row k = tid & 15 of the step, columns (tid >> 4) + 16q
  const int lk = tid & 15, lc = tid >> 4;
  R acc_re[4][4], acc_im[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc_re[a][b] = acc_im[a][b] = (R)0;
  C pr[4], qr[4];
  auto load = [&](int64_t n0) {
    const int64_t n = n0 + lk;
    const bool in = n < n_hi;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + lc + 16 * q, j = j0 + lc + 16 * q;
      C zero;
      zero.x = zero.y = (R)0;
      pr[q] = (in && i < m) ? P[(int64_t)i * N + n] : zero;
      qr[q] = (in && j < nk) ? Q[(int64_t)j * N + n] : zero;
    }
  };
  if (n_lo < n_hi) load(n_lo);
  for (int64_t n0 = n_lo; n0 < n_hi; n0 += kPqK) {
    __syncthreads();  // the previous step's reads are done
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      sP[lk][lc + 16 * q] = pr[q];
      sQ[lk][lc + 16 * q] = qr[q];
    }
    __syncthreads();
    if (n0 + kPqK < n_hi) load(n0 + kPqK);  // in flight during the step
#pragma unroll
    for (int k = 0; k < kPqK; ++k) {
      C p[4], q[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) p[a] = sP[k][ty + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) q[b] = sQ[k][tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          // conj(p) * q
          acc_re[a][b] = fma(p[a].x, q[b].x, fma(p[a].y, q[b].y, acc_re[a][b]));
          acc_im[a][b] = fma(p[a].x, q[b].y, fma(-p[a].y, q[b].x, acc_im[a][b]));
        }
    }
  }
  double2* out = ws + (int64_t)slice * m * nk;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      if (i < m && j < nk)
        out[(int64_t)j * m + i] = make_double2((double)acc_re[a][b], (double)acc_im[a][b]);
    }
}

// The FP64 contraction as a real product on mma.sync m8n8k4 f64.  A column of P
// or Q is read as 2N doubles (re, im, re, im, ...):
//   Re cs[i][j] = sum_k P[k] Q[k],   Im cs[i][j] = sum_k P[k] Q'[k],
// with Q'[2n] = Q[2n+1], Q'[2n+1] = -Q[2n]: the same A fragments serve both, and
// the second B fragment is the neighbouring double with a sign.  64 x 64 tiles of
// 4 warps (32 x 32 complex outputs each, 128 accumulator registers), 16 rows
// of n (32 doubles) per stage, three stages filled by cp.async; a column's
// stage takes 36 doubles, so a half warp's fragment loads touch every bank once.
// Bound by the FP64 pipe (4 FMAs per complex product; ncu: tensor pipe 89% busy):
// 128 x 768 moments of 72,000 rows take 1.75 ms, 16 TFMA/s, in the 24 slices of pq_split.
constexpr int kPqStages = 3;
constexpr int kPqLd = 2 * kPqK + 4;  // doubles per column of a stage
constexpr size_t kPqSmem = (size_t)kPqStages * 2 * kPqTile * kPqLd * sizeof(double);

__device__ __forceinline__ void pq_cp_async(double* dst, const double2* src, bool in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = in ? 16 : 0;  // 0: the 16 bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes)
               : "memory");
}

static __global__ void __launch_bounds__(128, 2)
    pq_dmma_kernel(const double2* __restrict__ P, const double2* __restrict__ Q, int64_t N, int m,
                   int nk, int64_t rows_per_slice, double2* __restrict__ ws) {
  extern __shared__ __align__(16) double pqs[];
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wi = (warp & 1) * 32, wj = (warp >> 1) * 32;
  const int j0 = blockIdx.x * kPqTile, i0 = blockIdx.y * kPqTile;
  const int64_t n_lo = (int64_t)blockIdx.z * rows_per_slice;
  const int64_t n_hi = n_lo + rows_per_slice < N ? n_lo + rows_per_slice : N;
  const int n_steps = n_hi > n_lo ? (int)((n_hi - n_lo + kPqK - 1) / kPqK) : 0;
  const int lr = tid & 15, lc = tid >> 4;  // row of the step, first column
  auto issue = [&](int s) {
    if (s < n_steps) {
      double* sp = pqs + (size_t)(s % kPqStages) * 2 * kPqTile * kPqLd;
      double* sq = sp + kPqTile * kPqLd;
      const int64_t n = n_lo + (int64_t)s * kPqK + lr;
#pragma unroll
      for (int q = 0; q < kPqTile / 8; ++q) {
        const int c = lc + 8 * q;
        const bool pin = n < n_hi && i0 + c < m, qin = n < n_hi && j0 + c < nk;
        pq_cp_async(sp + c * kPqLd + 2 * lr, pin ? P + (int64_t)(i0 + c) * N + n : P, pin);
        pq_cp_async(sq + c * kPqLd + 2 * lr, qin ? Q + (int64_t)(j0 + c) * N + n : Q, qin);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double re[4][4][2], im[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) re[a][b][0] = re[a][b][1] = im[a][b][0] = im[a][b][1] = 0.0;
#pragma unroll
  for (int s = 0; s < kPqStages - 1; ++s) issue(s);
  for (int s = 0; s < n_steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPqStages - 2) : "memory");
    __syncthreads();  // stage s has landed; stage s-1 is consumed
    issue(s + kPqStages - 1);
    const double* sp = pqs + (size_t)(s % kPqStages) * 2 * kPqTile * kPqLd;
    const double* sq = sp + kPqTile * kPqLd;
#pragma unroll
    for (int k = 0; k < 2 * kPqK; k += 4) {
      double fa[4], fb[4], fc[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) fa[a] = sp[(wi + 8 * a + g) * kPqLd + k + t];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const double* col = sq + (wj + 8 * b + g) * kPqLd + k;
        fb[b] = col[t];
        const double o = col[t ^ 1];
        fc[b] = (t & 1) ? -o : o;
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          dmma_8x8x4(re[a][b][0], re[a][b][1], fa[a], fb[b]);
          dmma_8x8x4(im[a][b][0], im[a][b][1], fa[a], fc[b]);
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  double2* out = ws + (int64_t)blockIdx.z * m * nk;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + wi + 8 * a + g, j = j0 + wj + 8 * b + 2 * t + q;
        if (i < m && j < nk) out[(int64_t)j * m + i] = make_double2(re[a][b][q], im[a][b][q]);
      }
}

// mu[(i0 + i) + nk*j] += g[i0+i] g[j] * scale * sum_s ws[s][j][i]
__global__ void pq_reduce_kernel(const double2* __restrict__ ws, int slices, int m, int nk,
                                 int i0, const double* __restrict__ g, double scale,
                                 double2* __restrict__ mu) {
  const int64_t total = (int64_t)m * nk;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    double re = 0.0, im = 0.0;
    for (int s = 0; s < slices; ++s) {
      const double2 v = ws[(int64_t)s * total + e];
      re += v.x;
      im += v.y;
    }
    const int ii = (int)(e % m);
    const int j = (int)(e / m);
    const int i = i0 + ii;
    const double w = g[i] * g[j];
    double2& o = mu[(int64_t)i + (int64_t)nk * j];
    o.x += w * re * scale;
    o.y += w * im * scale;
  }
}

}  // namespace tbpm
