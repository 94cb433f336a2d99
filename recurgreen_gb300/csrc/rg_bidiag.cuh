// Eigenvalues of t^H t for a matrix in global memory, by one thread-block
// cluster (the blocked sweeps of more than 64 modes): Householder
// bidiagonalisation with its columns dealt to the CTAs, then bisection
// (rg_device.cuh).
//
// Step k works on A(k:m, k:n) and makes two passes over it.  With z, u the
// right reflection of the step before (A <- A - z u^H still to be done):
//   1. every CTA forms column k of A - z u^H and its reflector v, tau for
//      itself; then for its own columns j > k: A_j <- A_j - z conj(u_j),
//      w_j = v^H A_j, and publishes row k of the reflected matrix,
//      y_j = A_kj - tau w_j;
//   2. every CTA forms the reflector u, tau' of conj(y); then for its own
//      columns A_j <- A_j - tau w_j v and its part of z = conj(tau') A u.
// So an entry is read and written twice a step, 16 FP64 multiply-adds in all,
// 16/3 n^3 for the matrix: the FP64 pipe bounds it (51 M clocks for 256 x
// 256), where nine sweeps of one-sided Jacobi at 4 n^3 complex rotations took
// 0.9 G.  By this stage alone: 152 guides of 256 modes and 40 slices 1,435 ->
// 287 ms, one guide of 60 slices on 8 CTAs 316 -> 150.
#pragma once

#include <cooperative_groups.h>

#include "rg_device.cuh"

namespace rg {

// A: m x n (m >= n), column-major with leading dimension m, overwritten.
// pub: global scratch of the cluster, n + 8 m double2 (n + m with C = 0).  sh: shared memory of
// each CTA, 80 m + 16 NT bytes.  The largest neig squared singular values,
// descending, go to out.  Called by every thread (NT per CTA) of the whole
// cluster, with its size C (1, 2, 4 or 8) and the CTA's rank, or of one CTA
// for matrices that never have a cluster, with C = 0; A was written before a
// barrier of theirs, and the call ends with none.  The result does not depend
// on C.
template <int NT>
__device__ __forceinline__ void cluster_tt_eigenvalues(int C, const int rank, double2* A, int m, int n, int neig,
                                                       double2* pub, double2* sh, double* out) {
  constexpr int NW = NT / 32;
  const int K = C ? 8 : 1;  // classes of columns
  if (!C) C = 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* v = sh;       // [m]
  double2* u = v + m;    // [n]
  double2* tw = u + n;   // [n] tau w_j of this CTA's columns
  double2* z = tw + n;   // [m]
  double* d = reinterpret_cast<double*>(z + m);  // [n]
  double* e = d + n;                             // [n]
  double2* s_z = z + 2 * m;                      // [NT] (d, e take at most m double2)
  __shared__ double s_part[NW];
  __shared__ double2 s_tau, s_scale;
  double2* ypub = pub;
  double2* zpub = pub + n;
  auto sync = [&]() {
    if (C > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  };
  // v (or u) holds a vector x of L elements: its reflector, in place.
  auto reflect = [&](double2* x, int L, double* beta) {
    double xn2 = 0.0;
    for (int i = 1 + tid; i < L; i += NT) xn2 = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, xn2));
#pragma unroll
    for (int off = 16; off; off >>= 1) xn2 += __shfl_xor_sync(0xffffffffu, xn2, off);
    if (lane == 0) s_part[warp] = xn2;
    __syncthreads();
    if (warp == 0) {
      double s = 0.0;
      for (int k = 0; k < NW; ++k) s += s_part[k];
      const Reflector r = reflector(x[0], s);
      if (lane == 0) {
        s_tau = r.tau;
        s_scale = r.scale;
        *beta = r.beta;
      }
    }
    __syncthreads();
    const double2 sc = s_scale;
    for (int i = tid; i < L; i += NT) x[i] = i == 0 ? make_double2(1.0, 0.0) : cmul(x[i], sc);
    __syncthreads();
  };
  __shared__ int s_top;
  if (tid == 0) s_top = 0;
  __syncthreads();
  int top = 0;
#pragma unroll 4
  for (int64_t q = tid; q < (int64_t)m * n; q += NT) top = max(top, biased_exp(__ldcg(A + q)));
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&s_top, top);
  __syncthreads();
  double unscale;
  const double scale = range_scale(s_top, &unscale);
  if (scale != 1.0) {
    sync();  // every CTA has read A
    for (int64_t q = rank * NT + tid; q < (int64_t)m * n; q += C * NT) A[q] = cscale(scale, __ldcg(A + q));
    sync();
  }
  for (int i = tid; i < m; i += NT) z[i] = make_double2(0.0, 0.0);
  for (int j = tid; j < n; j += NT) u[j] = make_double2(0.0, 0.0);
  double2 tr = make_double2(0.0, 0.0);  // conj(tau') of the step before
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    if (k > 0) {
      for (int i = k + tid; i < m; i += NT) {
        double2 s = make_double2(0.0, 0.0);
        for (int c = 0; c < K; ++c) {
          const double2 q = __ldcg(zpub + (int64_t)c * m + i);
          s.x += q.x;
          s.y += q.y;
        }
        z[i] = cmul(tr, s);
      }
      __syncthreads();
    }
    const double2 uk = make_double2(u[k].x, -u[k].y);
    for (int i = k + tid; i < m; i += NT) v[i - k] = csub(__ldcg(A + (int64_t)k * m + i), cmul(z[i], uk));
    __syncthreads();
    reflect(v, m - k, d + k);
    const double2 tau = s_tau;
    // this CTA's columns: the smallest j > k with j = rank (mod C), and on
    const int j0 = k + 1 + ((rank - (k + 1)) % C + C) % C;
    for (int j = j0 + C * warp; j < n; j += C * NW) {
      double2* col = A + (int64_t)j * m;
      const double2 uj = make_double2(u[j].x, -u[j].y);
      double re = 0.0, im = 0.0;
      double2 first = make_double2(0.0, 0.0);
#pragma unroll 2
      for (int i = k + lane; i < m; i += 32) {
        const double2 a = csub(__ldcg(col + i), cmul(z[i], uj));
        const double2 q = v[i - k];
        re = fma(q.x, a.x, fma(q.y, a.y, re));
        im = fma(q.x, a.y, fma(-q.y, a.x, im));
        if (i == k) first = a;
        else col[i] = a;
      }
      // lanes 0..15 sum re, lanes 16..31 im
      const double other = __shfl_xor_sync(0xffffffffu, lane < 16 ? im : re, 16);
      double h = (lane < 16 ? re : im) + other;
#pragma unroll
      for (int off = 8; off; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
      const double hi = __shfl_sync(0xffffffffu, h, 16);
      if (lane == 0) {
        const double2 t = cmul(tau, make_double2(h, hi));
        tw[j] = t;
        ypub[j] = csub(first, t);
      }
    }
    if (k + 1 >= n) break;
    sync();
    for (int j = k + 1 + tid; j < n; j += NT) {
      const double2 y = __ldcg(ypub + j);
      u[j] = make_double2(y.x, -y.y);
    }
    __syncthreads();
    reflect(u + k + 1, n - k - 1, e + k);
    tr = make_double2(s_tau.x, -s_tau.y);
    // Rows to threads; below NT/2 rows several groups of threads share the
    // columns.  The columns of class c (j = c mod K) are summed apart, so that
    // z, the sum over the classes, does not depend on which CTA has which.
    const int L = m - k - 1, L32 = (L + 31) & ~31;
    const int G = L32 >= NT ? 1 : NT / L32;
    const int grp = L32 >= NT ? 0 : tid / L32;
    for (int c = rank; c < K; c += C) {
      const int jc = k + 1 + ((c - (k + 1)) % K + K) % K;
      double2* zc = zpub + (int64_t)c * m;
      for (int i0 = L32 >= NT ? tid : tid % L32; i0 < (L32 >= NT ? L : L32); i0 += L32 >= NT ? NT : L32) {
        const bool on = i0 < L && grp < G;
        const int i = k + 1 + (i0 < L ? i0 : 0);
        const double2 vi = v[i - k];
        double zr = 0.0, zi = 0.0;
        if (on) {
#pragma unroll 4
          for (int j = jc + K * grp; j < n; j += K * G) {
            double2* p = A + (int64_t)j * m + i;
            const double2 a = cfms(__ldcg(p), tw[j], vi), uj = u[j];
            *p = a;
            zr = fma(a.x, uj.x, fma(-a.y, uj.y, zr));
            zi = fma(a.x, uj.y, fma(a.y, uj.x, zi));
          }
        }
        if (G == 1) {
          if (on) zc[i] = make_double2(zr, zi);
        } else {
          s_z[tid] = make_double2(zr, zi);
        }
      }
      if (G > 1) {
        __syncthreads();
        if (tid < L) {
          double2 s = s_z[tid];
          for (int q = 1; q < G; ++q) {
            s.x += s_z[q * L32 + tid].x;
            s.y += s_z[q * L32 + tid].y;
          }
          zc[k + 1 + tid] = s;
        }
        __syncthreads();
      }
    }
    sync();
  }
  bidiag_values<NT>(d, e, n, neig, out, unscale, rank, C);
}

}  // namespace rg
