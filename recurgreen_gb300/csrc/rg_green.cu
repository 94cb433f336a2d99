// Full Green-function column: the kernels behind the transmission-eigenstate
// profiles (compute_tprofile, compute_tprofile_group, compute_itx_profile,
// src/waveguide.f90:764-997), the deposition matrix (compute_deposition,
// src/waveguide.f90:710-745) and the wavefunction (compute_wavefunction,
// src/waveguide.f90:636-698).
//
// The reference solves the block tridiagonal system for every slice with
// solve_block_tridiag (src/base_utils.f90:296-335): a forward loop S_n =
// inv(A_n - B S_{n-1} B), Z_n = S_n (I_n - B Z_{n-1}) and a backward loop
// X_n = Z_n - S_n B X_{n+1}, each block M x M.  Here the forward loop is a
// sweep kernel, symmetric or pivoted (its state after slice n is (Gss, Gs1) =
// (S_n, Z_n), kept for every slice), and the backward loop runs only on the
// few source vectors W the caller needs: X_n W for the eigenvectors of t^H t
// inside a window of T, or one column for the deposition and the
// wavefunction.  That cuts the backward work from 8 M^3 to 16 M^2 k per slice
// for k vectors, and the profiles |X_n W|^2 come out of the same loop.
#include <algorithm>

#include "rg_device.cuh"
#include "rg_ozaki.cuh"

namespace rg {
namespace {

constexpr int kNT = 256;
constexpr int kKC = 8;  // source vectors per CTA of the back-substitution (one warp each in the reduction)

// One-sided Jacobi on the nv columns (length L) of A, with the right
// rotations accumulated in V (nv x nv): at convergence A_0 V = A has
// orthogonal columns, so A_0^H A_0 = V diag(|a_v|^2) V^H.  Both matrices are
// column-major in per-item global memory owned by this CTA (written and read
// by its threads only, ordered by __syncthreads).  A pair is rotated while its
// columns' product exceeds tol of their norms.  Returns false after 60 sweeps.
__device__ bool jacobi_with_vectors(double2* A, int lda, int L, int nv, double2* V, int* rot) {
  constexpr int NW = kNT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int NP = (nv + 1) & ~1;
  const double tol = 2.220446049250313e-16 * L;
  int sweep = 0;
  for (; sweep < 60; ++sweep) {
    if (threadIdx.x == 0) *rot = 0;
    __syncthreads();
    for (int rr = 0; rr < NP - 1; ++rr) {
      for (int pk = warp; pk < NP / 2; pk += NW) {
        const int pos1 = pk, pos2 = NP - 1 - pk;
        const int vp = pos1 == 0 ? 0 : ((pos1 - 1 + rr) % (NP - 1)) + 1;
        const int vq = ((pos2 - 1 + rr) % (NP - 1)) + 1;
        if (vp >= nv || vq >= nv) continue;
        double2* xp = A + (int64_t)vp * lda;
        double2* xq = A + (int64_t)vq * lda;
        double al = 0.0, be = 0.0, gr = 0.0, gi = 0.0;
        for (int i = lane; i < L; i += 32) {
          const double2 u = xp[i], w = xq[i];
          al = fma(u.x, u.x, fma(u.y, u.y, al));
          be = fma(w.x, w.x, fma(w.y, w.y, be));
          gr = fma(u.x, w.x, fma(u.y, w.y, gr));
          gi = fma(u.x, w.y, fma(-u.y, w.x, gi));
        }
#pragma unroll
        for (int off = 16; off; off >>= 1) {
          al += __shfl_xor_sync(0xffffffffu, al, off);
          be += __shfl_xor_sync(0xffffffffu, be, off);
          gr += __shfl_xor_sync(0xffffffffu, gr, off);
          gi += __shfl_xor_sync(0xffffffffu, gi, off);
        }
        const double ga = sqrt(gr * gr + gi * gi);
        if (ga > tol * sqrt(al * be) && ga > 1e-300) {
          if (lane == 0) *rot = 1;
          const double zeta = (be - al) / (2.0 * ga);
          const double t = fabs(zeta) > 1e100 ? 0.5 / zeta
                                              : copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
          const double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
          const double2 ph = make_double2(gr / ga, -gi / ga);
          for (int i = lane; i < L; i += 32) {
            const double2 u = xp[i];
            const double2 w = cmul(ph, xq[i]);
            xp[i] = make_double2(c * u.x - s * w.x, c * u.y - s * w.y);
            xq[i] = make_double2(s * u.x + c * w.x, s * u.y + c * w.y);
          }
          double2* yp = V + (int64_t)vp * nv;
          double2* yq = V + (int64_t)vq * nv;
          for (int i = lane; i < nv; i += 32) {
            const double2 u = yp[i];
            const double2 w = cmul(ph, yq[i]);
            yp[i] = make_double2(c * u.x - s * w.x, c * u.y - s * w.y);
            yq[i] = make_double2(s * u.x + c * w.x, s * u.y + c * w.y);
          }
        }
      }
      __syncthreads();
    }
    if (!*rot) break;
    __syncthreads();
  }
  return sweep < 60;
}

// Singular values and right singular vectors of the m x n matrix A (m >= n,
// column-major, leading dimension m, overwritten) by one CTA: Householder
// bidiagonalisation U^H A Q = B, V = Q, then the implicit-shift QR iteration of
// Golub and Kahan on B, whose right rotations V takes (its sweeps start from
// (|d| - sigma)(sign d + sigma/d), the form that LAPACK documents for xBDSQR).
// d[n], e[n]: the singular values end up in d, up to sign, in no order.  V: n x n
// column-major.  sc: 7 n + 4 doubles and 2 m double2 of shared memory.  Warp 0
// runs the rotations of a sweep, a serial chain, while the other warps apply
// those of the sweep before.
// As accurate as the reference's zgesvd: absolutely, to the norm of A.
// Returns false when the iteration does not end or A is not finite (then d is NaN).
__device__ bool svd_with_vectors(double2* A, const int m, const int n, double2* V, double* sc) {
  constexpr int NW = kNT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* d = sc;
  double* e = d + n;
  double* rot = e + n;                                   // [2][n][2] c, s of a sweep
  int* col = reinterpret_cast<int*>(rot + 4 * n);        // [2][n] columns i and j of a rotation, i + j 2^16
  double2* v = reinterpret_cast<double2*>(sc + ((7 * n + 1) & ~1));  // [m] reflection vector
  double2* tq = v + m;                                   // [n] factors of the right reflections
  __shared__ double2 s_tau;
  __shared__ int s_count[2], s_more, s_bad;
  // warp 0: the reflector of the L elements at x (stride st), conjugated for a row
  auto reflect = [&](const double2* x, int st, int L, double sg, double* beta) {
    double xn2 = 0.0;
    for (int i = 1 + lane; i < L; i += 32) {
      const double2 u = x[(int64_t)i * st];
      xn2 = fma(u.x, u.x, fma(u.y, u.y, xn2));
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) xn2 += __shfl_xor_sync(0xffffffffu, xn2, off);
    const Reflector r = reflector(make_double2(x[0].x, sg * x[0].y), xn2);
    for (int i = 1 + lane; i < L; i += 32) {
      const double2 u = x[(int64_t)i * st];
      v[i] = cmul(make_double2(u.x, sg * u.y), r.scale);
    }
    if (lane == 0) {
      v[0] = make_double2(1.0, 0.0);
      s_tau = r.tau;
      *beta = r.beta;
    }
  };
  // x <- x - f (v^H x) v, or with conjugated v for a row, by one warp
  auto apply = [&](double2* x, int st, int L, double2 f, double sg, const double2* v) {
    double re = 0.0, im = 0.0;
    for (int i = lane; i < L; i += 32) {
      const double2 q = v[i], u = x[(int64_t)i * st];
      re = fma(q.x, u.x, fma(sg * q.y, u.y, re));
      im = fma(q.x, u.y, fma(-sg * q.y, u.x, im));
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, off);
      im += __shfl_xor_sync(0xffffffffu, im, off);
    }
    const double2 w = cmul(f, make_double2(re, im));
    for (int i = lane; i < L; i += 32) {
      const double2 q = v[i], u = x[(int64_t)i * st];
      x[(int64_t)i * st] =
          make_double2(fma(-w.x, q.x, fma(sg * w.y, q.y, u.x)), fma(-w.x, sg * q.y, fma(-w.y, q.x, u.y)));
    }
  };
  __shared__ int s_top;
  if (tid == 0) s_top = 0;
  __syncthreads();
  int top = 0;
  for (int64_t q = tid; q < (int64_t)m * n; q += kNT) top = max(top, biased_exp(A[q]));
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&s_top, top);
  __syncthreads();
  double unscale;
  const double scale = range_scale(s_top, &unscale);
  if (scale != 1.0) {
    for (int64_t q = tid; q < (int64_t)m * n; q += kNT) A[q] = cscale(scale, A[q]);
    __syncthreads();
  }
  for (int k = 0; k < n; ++k) {
    double2* akk = A + (int64_t)k * m + k;
    if (warp == 0) reflect(akk, 1, m - k, 1.0, d + k);
    __syncthreads();
    for (int j = 1 + warp; j < n - k; j += NW) apply(akk + (int64_t)j * m, 1, m - k, s_tau, 1.0, v);
    __syncthreads();
    if (k + 1 >= n) break;
    if (warp == 0) reflect(akk + m, m, n - k - 1, -1.0, e + k);
    __syncthreads();
    const double2 tc = make_double2(s_tau.x, -s_tau.y);
    for (int i = 1 + warp; i < m - k; i += NW) apply(akk + m + i, m, n - k - 1, tc, -1.0, v);
    if (warp == 0) {  // column k is done with: it keeps the right reflection vector
      for (int i = lane; i < n - k - 1; i += 32) A[(int64_t)k * m + i] = v[i];
      if (lane == 0) tq[k] = tc;
    }
    __syncthreads();
  }
  // V = H_0 H_1 ..., H_k = I - tq_k v_k v_k^H on rows k + 1 and on
  for (int64_t q = tid; q < (int64_t)n * n; q += kNT) V[q] = make_double2(q % (n + 1) == 0 ? 1.0 : 0.0, 0.0);
  __syncthreads();
  for (int j = 1 + warp; j < n; j += NW)  // (column j starts as e_j: reflections k < j alone change it)
    for (int k = j - 1; k >= 0; --k) {
      apply(V + (int64_t)j * n + k + 1, 1, n - k - 1, tq[k], 1.0, A + (int64_t)k * m);
      __syncwarp();
    }
  double norm = 0.0;
  bool finite = true;
  for (int i = lane; i < n; i += 32) {
    const double a = fabs(d[i]), b = i + 1 < n ? fabs(e[i]) : 0.0;
    norm = fmax(norm, fmax(a, b));
    finite = finite && a + b < INFINITY;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) norm = fmax(norm, __shfl_xor_sync(0xffffffffu, norm, off));
  finite = __all_sync(0xffffffffu, finite);
  if (tid == 0) {
    s_bad = 0;
    s_count[0] = s_count[1] = 0;
  }
  __syncthreads();
  if (!finite) {
    for (int i = tid; i < n; i += kNT) d[i] = NAN;
    __syncthreads();
    return false;
  }
  const double eps = 0x1p-53, tiny = 0x1p-56 * norm;
  // (c, s) with [c s; -s c] (f, g) = (r, 0)
  auto givens = [](double f, double g, double& c, double& s, double& r) {
    const double h = fma(f, f, g * g);
    if (h < 1e-290) {
      const double a = fmax(fabs(f), fabs(g));
      if (a == 0.0) {
        c = 1.0, s = 0.0, r = 0.0;
        return;
      }
      const double x = f / a, y = g / a, q = sqrt(fma(x, x, y * y));
      c = x / q, s = y / q, r = a * q;
      return;
    }
    const double q = rsqrt(h);
    c = f * q, s = g * q, r = h * q;
  };
  int hi = n - 1, sweeps = 0;  // warp 0: B below row hi is diagonal
  for (int it = 0;; ++it) {
    const int b = it & 1;
    if (warp == 0) {
      if (lane == 0) {
        double* rb = rot + 2 * n * b;
        int* cb = col + n * b;
        int cnt = 0;
        auto put = [&](int i, int j, double c, double s) {
          rb[2 * cnt] = c;
          rb[2 * cnt + 1] = s;
          cb[cnt++] = i | j << 16;
        };
        while (hi > 0 && fabs(e[hi - 1]) <= fmax(tiny, eps * (fabs(d[hi - 1]) + fabs(d[hi])))) --hi;
        bool more = hi > 0;
        if (more && ++sweeps > 40 * n) {
          s_bad = 1;
          more = false;
        }
        if (more) {
          int lo = hi - 1;  // the unreduced block lo .. hi
          while (lo > 0 && fabs(e[lo - 1]) > fmax(tiny, eps * (fabs(d[lo - 1]) + fabs(d[lo])))) --lo;
          int z = -1;  // a zero on the diagonal
          for (int i = lo; i <= hi; ++i)
            if (fabs(d[i]) <= tiny) z = i;
          if (z == hi) {  // the last column is rotated to zero
            double f = e[hi - 1];
            e[hi - 1] = 0.0;
            for (int k = hi - 1; k >= lo; --k) {
              double c, s, r;
              givens(d[k], f, c, s, r);
              d[k] = r;
              put(k, hi, c, s);
              if (k > lo) {
                f = -s * e[k - 1];
                e[k - 1] *= c;
              }
            }
          } else if (z >= 0) {  // row z is rotated to zero, from the left
            double f = e[z];
            e[z] = 0.0;
            for (int k = z + 1; k <= hi; ++k) {
              double c, s, r;
              givens(d[k], f, c, s, r);
              d[k] = r;
              if (k < hi) {
                f = -s * e[k];
                e[k] *= c;
              }
            }
          } else {
            // shift: the eigenvalue of the last 2 x 2 of B^T B next to its corner
            const double dm = d[hi - 1], dn = d[hi], fm = hi - 1 > lo ? e[hi - 2] : 0.0, fn = e[hi - 1];
            const double tm = fma(dm, dm, fm * fm), tn = fma(dn, dn, fn * fn), to = dm * fn;
            const double dl = 0.5 * (tm - tn), root = sqrt(fma(dl, dl, to * to));
            const double den = dl + copysign(root, dl);
            const double mu = den == 0.0 ? tn : tn - to * to / den;
            // (d^2 - mu) / d and e: the first column of B^T B - mu, over d
            const double sg = sqrt(fmax(mu, 0.0));
            double y = (fabs(d[lo]) - sg) * (copysign(1.0, d[lo]) + sg / d[lo]), g = e[lo];
            double dk = d[lo], ek = e[lo];
            for (int k = lo; k < hi; ++k) {
              double c, s, r;
              givens(y, g, c, s, r);
              if (k > lo) e[k - 1] = r;
              put(k, k + 1, c, s);
              // columns k, k + 1
              const double d1 = d[k + 1];
              y = fma(c, dk, s * ek);
              ek = fma(c, ek, -s * dk);
              g = s * d1;
              const double dn1 = c * d1;
              // rows k, k + 1
              givens(y, g, c, s, r);
              d[k] = r;
              y = fma(c, ek, s * dn1);
              dk = fma(c, dn1, -s * ek);
              if (k + 1 < hi) {
                const double e1 = e[k + 1];
                g = s * e1;
                ek = c * e1;
              }
            }
            e[hi - 1] = y;
            d[hi] = dk;
          }
        }
        s_count[b] = cnt;
        s_more = more ? 1 : 0;
      }
      __syncwarp();
    } else {
      // the rotations of the sweep before, on the columns of V
      const int cnt = s_count[1 - b];
      const double* rb = rot + 2 * n * (1 - b);
      const int* cb = col + n * (1 - b);
      double* Vd = reinterpret_cast<double*>(V);
      for (int q = tid - 32; q < 2 * n; q += kNT - 32) {
        int last = -1;
        double keep = 0.0;  // entry of column `last`
        for (int k = 0; k < cnt; ++k) {
          const int i = cb[k] & 0xffff, j = cb[k] >> 16;
          const double c = rb[2 * k], s = rb[2 * k + 1];
          if (last >= 0 && last != i && last != j) Vd[(int64_t)last * 2 * n + q] = keep;
          const double x = last == i ? keep : Vd[(int64_t)i * 2 * n + q];
          const double y = last == j ? keep : Vd[(int64_t)j * 2 * n + q];
          Vd[(int64_t)i * 2 * n + q] = fma(c, x, s * y);
          keep = fma(c, y, -s * x);
          last = j;
        }
        if (last >= 0) Vd[(int64_t)last * 2 * n + q] = keep;
      }
    }
    __syncthreads();
    const bool more = s_more != 0;
    if (!more && s_count[0] == 0 && s_count[1] == 0) break;
    __syncthreads();
    // (s_count[b] is zero after the last sweep, so the loop ends one pass later)
  }
  for (int i = tid; i < n; i += kNT) d[i] *= unscale;
  __syncthreads();
  return s_bad == 0;
}

__host__ __device__ inline size_t eigvec_head_bytes(int nc) {
  return (sizeof(double) * nc + sizeof(int) * 2 * nc + 15) & ~(size_t)15;
}
// svd_with_vectors' scratch, and whether its matrices fit shared memory beside it
__host__ __device__ inline size_t eigvec_qr_bytes(int m, int nc) {
  return (sizeof(double) * (size_t)((7 * nc + 1) & ~1) + sizeof(double2) * (size_t)(m + nc) + 15) & ~(size_t)15;
}
__host__ __device__ inline bool eigvec_in_smem(int m, int nc) {
  return eigvec_head_bytes(nc) + eigvec_qr_bytes(m, nc) + sizeof(double2) * ((size_t)m * nc + (size_t)nc * nc) <=
         200 * 1024;
}

// One CTA per item: the block of t, its singular values and right vectors (QR
// iteration or Jacobi, see launch_eigvec), eigenvalues in descending order with
// their eigenvectors, then the window selection.
template <bool QR>
__global__ void __launch_bounds__(kNT) eigvec_kernel(EigvecArgs a) {
  extern __shared__ double sh[];
  double* tv = sh;                        // [nc] |a_v|^2 by column
  int* order = (int*)(tv + a.nc);         // [nc] column of rank k
  int* selcol = order + a.nc;             // [nc] column of selected vector k
  __shared__ int s_rot, s_k;
  const int r = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = kNT / 32;
  const int nr = a.nr, nc = a.nc;
  const int mr = QR && nr < nc ? nc : nr;  // rows of A, with zeros up to the columns
  double* qs = reinterpret_cast<double*>(reinterpret_cast<char*>(sh) + eigvec_head_bytes(nc));
  double2* A = a.work + (int64_t)r * a.work_stride;
  if (QR && eigvec_in_smem(mr, nc))
    A = reinterpret_cast<double2*>(reinterpret_cast<char*>(qs) + eigvec_qr_bytes(mr, nc));
  double2* V = A + (int64_t)mr * nc;
  const double2* src = a.a + (int64_t)r * a.astride;
  for (int64_t e = tid; e < (int64_t)mr * nc; e += kNT) {
    const int i = (int)(e % mr), j = (int)(e / mr);
    A[e] = i < nr ? src[(int64_t)(a.col0 + j) * a.lda + a.row0 + i] : make_double2(0.0, 0.0);
  }
  bool ok;
  if (QR) {
    ok = svd_with_vectors(A, mr, nc, V, qs);
    for (int v = tid; v < nc; v += kNT) tv[v] = qs[v] * qs[v];
  } else {
    for (int64_t e = tid; e < (int64_t)nc * nc; e += kNT)
      V[e] = make_double2((e % nc) == (e / nc) ? 1.0 : 0.0, 0.0);
    __syncthreads();
    ok = jacobi_with_vectors(A, nr, nr, nc, V, &s_rot);
  }
  for (int v = warp; v < nc && !QR; v += NW) {
    const double2* x = A + (int64_t)v * nr;
    double s = 0.0;
    for (int i = lane; i < nr; i += 32) s = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, s));
#pragma unroll
    for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) tv[v] = s;
  }
  __syncthreads();
  for (int v = tid; v < nc; v += kNT) {
    const int k = descending_rank(tv, nc, v);
    order[k] = v;
    a.tvals[(int64_t)r * nc + k] = tv[v];
    ok = ok && tv[v] < INFINITY;
  }
  ok = __syncthreads_and(ok) != 0;  // no decomposition of a matrix that is not finite
  if (a.u) {
    double2* u = a.u + (int64_t)r * nc * nc;
    for (int64_t e = tid; e < (int64_t)nc * nc; e += kNT) {
      const int i = (int)(e % nc), k = (int)(e / nc);
      u[e] = V[(int64_t)order[k] * nc + i];
    }
  }
  if (a.wsel) {
    // Selection in rank order (the reference's loop over iv of tvals).
    if (tid == 0) {
      int k = 0;
      for (int w = 0; w < a.nprof; ++w) a.nt[(int64_t)r * a.nprof + w] = 0;
      double sum = 0.0;
      for (int q = 0; q < nc; ++q) {
        const double t = tv[order[q]];
        sum += t;
        uint32_t bits = 0;
        for (int w = 0; w < a.nprof; ++w) {
          const bool in = a.centered ? (fabs(t - a.wa[w]) <= a.wb[w]) : (a.wa[w] <= t && t <= a.wb[w]);
          if (in) {
            bits |= 1u << w;
            a.nt[(int64_t)r * a.nprof + w] += 1;
          }
        }
        if (bits) {
          a.member[(int64_t)r * nc + k] = bits;
          selcol[k] = order[q];
          ++k;
        }
      }
      s_k = k;
      a.ksel[r] = k;
      if (a.tavg) a.tavg[r] = sum / nc;
    }
    __syncthreads();
    const int k = s_k;
    double2* ws = a.wsel + (int64_t)r * nc * a.M;
    for (int64_t e = tid; e < (int64_t)k * a.M; e += kNT) {
      const int s = (int)(e / a.M), m = (int)(e % a.M);
      const int j = m - a.col0;
      ws[e] = (j >= 0 && j < nc) ? cmul(a.sqmu[m], V[(int64_t)selcol[s] * nc + j]) : make_double2(0.0, 0.0);
    }
  }
  if (tid == 0) a.status[r] = ok ? RG_OK : RG_ERR_NOCONV;
}

// Back-substitution.  Block (chunk, item): the nv <= kKC source vectors
// s0 .. s0+nv-1 of item blockIdx.y.  The M*nv outputs are dealt to the
// threads, e = tid + kNT*j -> row m = e / nv, vector v = e % nv, so the FP64
// work is 16 M^2 nv per slice whatever nv is (an FP64 warp instruction costs
// the same with idle lanes; whole idle warps cost nothing).  Ysh holds
// B Y_{n+1} and Wsh the source vectors, [M][kKC]; Psh the |Y|^2 terms of
// the profile, summed per vector in a fixed order.
template <int JMAX>
__global__ void __launch_bounds__(kNT) back_kernel(BackArgs a) {
  extern __shared__ double2 shb[];
  const int M = a.M;
  double2* Ysh = shb;
  double2* Wsh = shb + M * kKC;
  double* Psh = (double*)(Wsh + M * kKC);
  const int r = blockIdx.y;
  const int kr = a.kcount ? a.kcount[r] : a.kmax;
  const int s0 = blockIdx.x * kKC;
  if (s0 >= kr) return;  // uniform over the block
  const int nv = min(kKC, kr - s0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nout = M * nv;  // <= kNT * JMAX (checked by the launcher)
  for (int e = tid; e < M * kKC; e += kNT) {
    const int m = e / kKC, vv = e % kKC;
    Wsh[e] = vv < nv ? a.src[(int64_t)r * a.src_stride + (int64_t)(s0 + vv) * M + m] : make_double2(0.0, 0.0);
    Ysh[e] = make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int64_t mm = (int64_t)M * M;
  const int nslices = a.only_lo ? 1 : a.nx - a.i_lo;
  int mj[JMAX], vj[JMAX];  // row and vector of output j (the divisions once, outside the slice loop)
#pragma unroll
  for (int j = 0; j < JMAX; ++j) {
    const int e = tid + kNT * j;
    mj[j] = e < nout ? e / nv : 0;
    vj[j] = e < nout ? e % nv : 0;
  }
  for (int n = a.nx - 1; n >= a.i_lo; --n) {
    const double2* S = a.dump + ((int64_t)r * a.nx + n) * 2 * mm;
    const double2* Z = S + mm;
    const bool first = (n == a.nx - 1);
    double2 acc[JMAX];
#pragma unroll
    for (int j = 0; j < JMAX; ++j) acc[j] = make_double2(0.0, 0.0);
    if (tid < nout) {
      for (int c = 0; c < M; ++c) {
#pragma unroll
        for (int j = 0; j < JMAX; ++j) {
          if (tid + kNT * j < nout) {
            const int m = mj[j], v = vj[j];
            const double2 wc = Wsh[c * kKC + v];
            const double2 z = __ldg(Z + (int64_t)m * M + c);
            acc[j] = make_double2(fma(z.x, wc.x, fma(-z.y, wc.y, acc[j].x)), fma(z.x, wc.y, fma(z.y, wc.x, acc[j].y)));
            if (!first) {
              const double2 yc = Ysh[c * kKC + v];
              const double2 sv = __ldg(S + (int64_t)m * M + c);
              acc[j] = make_double2(fma(-sv.x, yc.x, fma(sv.y, yc.y, acc[j].x)),
                                    fma(-sv.x, yc.y, fma(-sv.y, yc.x, acc[j].y)));
            }
          }
        }
      }
    }
    __syncthreads();  // every thread has read Ysh
#pragma unroll
    for (int j = 0; j < JMAX; ++j) {
      if (tid + kNT * j < nout) {
        const int m = mj[j], v = vj[j];
        const double2 y = acc[j];
        Ysh[m * kKC + v] = cmul(a.bmat[m], y);
        Psh[m * kKC + v] = fma(y.x, y.x, y.y * y.y);
        if (a.out_mode == kBackColumns && (!a.only_lo || n == a.i_lo)) {
          const int64_t sl = a.only_lo ? 0 : n - a.i_lo;
          double2 o = y;
          if (a.left) {
            const double2 q = cmul(a.left[m], y);
            o = make_double2(-2.0 * q.y, 2.0 * q.x);
          }
          a.cols[(((int64_t)r * nslices + sl) * a.kmax + s0 + v) * M + m] = o;
        }
      }
    }
    __syncthreads();  // Ysh and Psh complete
    if (a.out_mode == kBackProfile) {
      for (int v = warp; v < nv; v += kNT / 32) {  // warp v sums vector v over the rows
        double p = 0.0;
        for (int m = lane; m < M; m += 32) p += Psh[m * kKC + v];
#pragma unroll
        for (int off = 16; off; off >>= 1) p += __shfl_xor_sync(0xffffffffu, p, off);
        if (lane == 0) a.prof[((int64_t)r * a.kmax + s0 + v) * a.nx + n] = p;
      }
    }
  }
}

// The same for up to 64 modes on the FP16 tensor cores: eight vectors are the n8
// side of mma.m16n8k16.  Per slice the 16 warps turn S and Z into six 9-bit
// digits a part (rg_ozaki.cuh; a warp per tile), then each has one row tile, one
// part and one of the two products; the vectors' digits, W in one word pair and B
// Y_{n+1} in the other, follow those of S and Z in every plane.  The FP64 form
// takes 32 M^2 multiply-adds a slice and vector at 1.7 lanes per clock: 25 ms of
// 152 items, 300 slices and some eight vectors at 64 modes, 6.4 here
// (profiles 90 -> 71 ms).
constexpr int kBackNT = 512;
template <int T>
struct BackTile {
  static constexpr int MP = 16 * T, TILES = 2 * T * T + T;  // tiles of a plane: S, Z, vectors
  static constexpr int kPlane = TILES * 512;                // bytes
  static constexpr size_t bytes() {
    return 12 * (size_t)kPlane + sizeof(double2) * MP * kKC + sizeof(double) * 2 * kKC +
           sizeof(int) * (2 * T * MP + 3 * kKC);
  }
};
template <int T>
__global__ void __launch_bounds__(kBackNT, 1) back_tile_kernel(BackArgs a) {
  using Cf = BackTile<T>;
  constexpr int MP = Cf::MP, TILES = Cf::TILES, kPlane = Cf::kPlane, NW = kBackNT / 32, QT = (2 * T * T + NW - 1) / NW;
  static_assert(kKC == 8 && 4 * T <= NW && 2 * kKC == NW, "warps' tasks");
  extern __shared__ uint4 shp[];
  char* P = reinterpret_cast<char*>(shp);
  double2* R = reinterpret_cast<double2*>(P + 12 * kPlane);   // [MP][kKC] vectors
  double* psum = reinterpret_cast<double*>(R + MP * kKC);     // [2 kKC] |Y|^2 by vector and half of the rows
  int* ex = reinterpret_cast<int*>(psum + 2 * kKC);           // [2][T][MP] row exponents of S, Z by tile column
  int* exw = ex + 2 * T * MP;                                 // [kKC] exponents of W,
  int* exy = exw + kKC;                                       // [2 kKC] of B Y by half of the rows
  const int M = a.M, r = blockIdx.y, kr = a.kcount ? a.kcount[r] : a.kmax, s0 = blockIdx.x * kKC;
  if (s0 >= kr) return;  // uniform over the block
  const int nv = min(kKC, kr - s0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, odd = (lane >> 3) & 1;
  const int vv = warp >> 1, vm = (warp & 1) * 32 + lane;  // element steps: vector and row of a thread
  // Digits of the vectors in R with exponents e(v), to word pair `slot`: warps
  // (k tile, part); the vectors are the rows of the operand's transpose.
  auto put_vectors = [&](int slot, auto e) {
    if (warp >= 2 * T) return;
    const int tk = warp >> 1, part = warp & 1;
    const double* Rd = reinterpret_cast<const double*>(R);
    const int ev = e(g);
    long long bias = 0;
#pragma unroll
    for (int p = 0; p < 6; ++p) bias += 256LL << (oz::kDigitBits * p);
    unsigned long long y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int m = tk * 16 + 2 * t4 + (k & 1) + 8 * (k >> 1);
      y[k] = (unsigned long long)(oz::sfixed53(Rd[2 * (m * kKC + g) + part], ev) + bias);
    }
#pragma unroll
    for (int p = 0; p < 6; ++p) {
      const uint32_t mask = p ? 511u : 1023u;
      uint32_t w[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
        w[k] = oz::field_pair((uint32_t)(y[2 * k] >> (oz::kDigitBits * (5 - p))) & mask,
                              (uint32_t)(y[2 * k + 1] >> (oz::kDigitBits * (5 - p))) & mask);
      *reinterpret_cast<uint2*>(P + (6 * part + p) * kPlane + (2 * T * T + tk) * 512 + lane * 16 + 8 * (odd ^ slot)) =
          make_uint2(w[0], w[1]);
    }
  };
  double2 w0 = make_double2(0.0, 0.0);
  if (vm < M && vv < nv) w0 = a.src[(int64_t)r * a.src_stride + (int64_t)(s0 + vv) * M + vm];
  const double2 bm = vm < M ? a.bmat[vm] : w0;
  if (vm < MP) R[vm * kKC + vv] = w0;
  int ew = __reduce_max_sync(0xffffffffu, oz::fexp2(w0));
  if (lane == 0) exy[warp] = ew;
  __syncthreads();
  if (tid < kKC) exw[tid] = max(exy[2 * tid], exy[2 * tid + 1]);
  put_vectors(0, [&](int v) { return max(exy[2 * v], exy[2 * v + 1]); });
  __syncthreads();
  const int64_t mm = (int64_t)M * M;
  const int nslices = a.only_lo ? 1 : a.nx - a.i_lo;
  for (int n = a.nx - 1; n >= a.i_lo; --n) {
    const double2* S = a.dump + ((int64_t)r * a.nx + n) * 2 * mm;  // Z follows
    const bool first = n == a.nx - 1;
    double2 x[QT][8];
#pragma unroll
    for (int q = 0; q < QT; ++q) {
      const int task = warp + NW * q, mat = task / (T * T), tile = task % (T * T);
      if (task < 2 * T * T) {
        const int ti = tile / T, tj = tile % T;
        int e0 = oz::kNoExp, e1 = oz::kNoExp;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int i = ti * 16 + g + 8 * ((k >> 1) & 1), j = tj * 16 + 2 * t4 + (k & 1) + 8 * (k >> 2);
          x[q][k] = i < M && j < M ? __ldg(S + mat * mm + (int64_t)i * M + j) : make_double2(0.0, 0.0);
          if ((k >> 1) & 1) e1 = max(e1, oz::fexp2(x[q][k]));
          else e0 = max(e0, oz::fexp2(x[q][k]));
        }
        oz::put_row_exps(ex + (mat * T + tj) * MP, ti, lane, e0, e1);
      }
    }
    __syncthreads();  // the exponents, and B Y's digits
#pragma unroll
    for (int q = 0; q < QT; ++q) {
      const int task = warp + NW * q, mat = task / (T * T), tile = task % (T * T);
      if (task < 2 * T * T) {
        const int row = (tile / T) * 16 + g;
        const int e0 = oz::row_exp<T>(ex + mat * T * MP, MP, row), e1 = oz::row_exp<T>(ex + mat * T * MP, MP, row + 8);
        long long f[16];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          f[k] = oz::sfixed53(x[q][k].x, (k >> 1) & 1 ? e1 : e0);
          f[8 + k] = oz::sfixed53(x[q][k].y, (k >> 1) & 1 ? e1 : e0);
        }
        oz::put_planes<53, 8>(f, 6, reinterpret_cast<uint4*>(P) + (mat * T * T + tile) * 32 + lane, TILES * 32, 6, 0);
      }
    }
    __syncthreads();
    // warps 0 .. 2 T - 1: S (B Y), the next 2 T: Z W; the difference meets in R
    const int mat = warp / (2 * T), rt = (warp >> 1) % T, part = warp & 1;
    double val[4];
    if (warp < 4 * T && !(first && mat == 0)) {
      const char* pa = P + (mat * T * T + rt * T) * 512 + lane * 16;
      long long hi[4], lo[4];
      oz::half_product<T, 6, 6, oz::kLmax, 2>(pa + 8 * odd, pa + 8 * (1 - odd), 6 * kPlane,
                                              P + 2 * T * T * 512 + lane * 16 + 8 * (odd ^ (1 - mat)), 6 * kPlane,
                                              kPlane, hi, lo, nullptr, part);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const int v = 2 * t4 + (w & 1);
        const int e = oz::row_exp<T>(ex + mat * T * MP, MP, rt * 16 + g + 8 * (w >> 1));
        val[w] = oz::fold_to_double(hi[w], lo[w], e + (mat ? exw[v] : max(exy[2 * v], exy[2 * v + 1])));
      }
    } else {
#pragma unroll
      for (int w = 0; w < 4; ++w) val[w] = 0.0;
    }
    double* Rd = reinterpret_cast<double*>(R) + 2 * ((rt * 16 + g) * kKC + 2 * t4) + part;
    if (mat == 0) {
#pragma unroll
      for (int w = 0; w < 4; ++w) Rd[2 * (8 * (w >> 1) * kKC + (w & 1))] = val[w];
    }
    __syncthreads();
    if (mat == 1) {
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        double* d = Rd + 2 * (8 * (w >> 1) * kKC + (w & 1));
        *d = val[w] - *d;
      }
    }
    __syncthreads();
    double2 by = make_double2(0.0, 0.0);
    double p = 0.0;
    if (vm < M && vv < nv) {
      const double2 y = R[vm * kKC + vv];
      by = cmul(bm, y);
      p = fma(y.x, y.x, y.y * y.y);
      if (a.out_mode == kBackColumns && (!a.only_lo || n == a.i_lo)) {
        const int64_t sl = a.only_lo ? 0 : n - a.i_lo;
        double2 o = y;
        if (a.left) {
          const double2 q = cmul(a.left[vm], y);
          o = make_double2(-2.0 * q.y, 2.0 * q.x);
        }
        a.cols[(((int64_t)r * nslices + sl) * a.kmax + s0 + vv) * M + vm] = o;
      }
    }
    if (vm < MP) R[vm * kKC + vv] = by;
    ew = __reduce_max_sync(0xffffffffu, oz::fexp2(by));
    if (a.out_mode == kBackProfile) {
#pragma unroll
      for (int off = 16; off; off >>= 1) p += __shfl_xor_sync(0xffffffffu, p, off);
    }
    if (lane == 0) {
      exy[warp] = ew;
      psum[warp] = p;
    }
    __syncthreads();
    if (a.out_mode == kBackProfile && tid < nv)
      a.prof[((int64_t)r * a.kmax + s0 + tid) * a.nx + n] = psum[2 * tid] + psum[2 * tid + 1];
    put_vectors(1, [&](int v) { return max(exy[2 * v], exy[2 * v + 1]); });
  }
}

template <int T>
int launch_back_tile(const BackArgs& a, cudaStream_t s) {
  RG_CUDA(allow_smem((const void*)back_tile_kernel<T>, BackTile<T>::bytes()));
  back_tile_kernel<T><<<dim3((a.kmax + kKC - 1) / kKC, a.nreal), kBackNT, BackTile<T>::bytes(), s>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

__global__ void windows_kernel(WindowArgs a) {
  const int64_t total = (int64_t)a.nreal * a.nprof * a.nx;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int n = (int)(e % a.nx);
    const int w = (int)((e / a.nx) % a.nprof);
    const int r = (int)(e / ((int64_t)a.nx * a.nprof));
    const int k = a.ksel[r];
    double s = 0.0;
    for (int q = 0; q < k; ++q)
      if ((a.member[(int64_t)r * a.kmax + q] >> w) & 1u) s += a.prof[((int64_t)r * a.kmax + q) * a.nx + n];
    if (a.kind == RG_PROFILE_ITX) {
      s = (s * 2.0) / ((3.141592653589793 * a.wol) * fabs(a.wb[w] - a.wa[w]));
    } else {
      const int nt = a.nt[(int64_t)r * a.nprof + w];
      if (nt != 0) s = s * (4.0 / nt);
    }
    a.out[e] = s;
  }
}

__global__ void wavefun_kernel(WavefunArgs a) {
  const int64_t rows = (int64_t)a.nx * a.ny;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < rows; e += (int64_t)gridDim.x * blockDim.x) {
    const int n = (int)(e / a.ny), j = (int)(e % a.ny);
    const double2* y = a.y + (int64_t)n * a.M;
    const double2* md = a.modal + (int64_t)j * a.M;
    double re = 0.0, im = 0.0;
    for (int m = 0; m < a.M; ++m) {
      const double2 c = md[m], g = y[m];
      re = fma(c.x, g.x, fma(-c.y, g.y, re));
      im = fma(c.x, g.y, fma(c.y, g.x, im));
    }
    const int id = n - a.nxfree;
    a.out[e] = a.xmesh[n];
    a.out[rows + e] = a.ymesh[j];
    a.out[2 * rows + e] = re;
    a.out[3 * rows + e] = im;
    a.out[4 * rows + e] = (id >= 0 && id < a.nxdiso) ? a.upot[(int64_t)id * a.ny + j] : 0.0;
  }
}

template <int JMAX>
int launch_back_t(const BackArgs& a, cudaStream_t s) {
  const size_t smem = (2 * sizeof(double2) + sizeof(double)) * (size_t)a.M * kKC;
  RG_CUDA(allow_smem((const void*)back_kernel<JMAX>, smem));
  const dim3 grid((a.kmax + kKC - 1) / kKC, a.nreal);
  back_kernel<JMAX><<<grid, kNT, smem, s>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

}  // namespace

int64_t eigvec_work_stride(int nr, int nc) {
  return (((int64_t)(nr > nc ? nr : nc) * nc + (int64_t)nc * nc) + 15) & ~(int64_t)15;
}

// Vectors for a selection by windows of T come from the QR iteration, whose
// values are accurate to the norm of t.  So is t itself: profiles of localised
// guides in windows down to T = 1e-18 are as far from an extended-precision
// reference as with one-sided Jacobi (1e-12 .. 1e-9 there, 1e-14 above 1e-5).  An
// eigenvector call by itself, whose matrix may be better than that, keeps Jacobi
// and its relative accuracy.  152 matrices of 64 x
// 64: 41 ms by Jacobi, 6.4 by QR (profiles of 152 guides of 64 modes and 300
// slices 125 -> 90 ms).
int launch_eigvec(const EigvecArgs& a, cudaStream_t s) {
  if (a.nreal <= 0) return RG_OK;
  if (a.nc < 1 || a.nr < 1 || a.nprof > 32) return fail(RG_ERR_INVALID_ARG, "eigvec: invalid sizes");
  const bool qr = a.wsel != nullptr && a.nc < 65536;
  const int m = a.nr > a.nc ? a.nr : a.nc;
  size_t smem = eigvec_head_bytes(a.nc);
  if (qr) {
    smem += eigvec_qr_bytes(m, a.nc);
    if (eigvec_in_smem(m, a.nc)) smem += sizeof(double2) * ((size_t)m * a.nc + (size_t)a.nc * a.nc);
  }
  const auto kernel = qr ? eigvec_kernel<true> : eigvec_kernel<false>;
  RG_CUDA(allow_smem((const void*)kernel, smem));
  kernel<<<a.nreal, kNT, smem, s>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

int launch_back(const BackArgs& a, cudaStream_t s) {
  if (a.nreal <= 0 || a.kmax <= 0) return RG_OK;
  if (a.i_lo < 0 || a.i_lo >= a.nx) return fail(RG_ERR_INVALID_ARG, "back-substitution: slice out of range");
  if (a.M <= 16) return launch_back_tile<1>(a, s);
  if (a.M <= 32) return launch_back_tile<2>(a, s);
  if (a.M <= 48) return launch_back_tile<3>(a, s);
  if (a.M <= 64) return launch_back_tile<4>(a, s);
  const int J = (a.M * kKC + kNT - 1) / kNT;
  if ((2 * sizeof(double2) + sizeof(double)) * (size_t)a.M * kKC > 200 * 1024)
    return fail(RG_ERR_INVALID_ARG, "back-substitution: too many modes");
  if (J <= 4) return launch_back_t<4>(a, s);
  if (J <= 8) return launch_back_t<8>(a, s);
  if (J <= 16) return launch_back_t<16>(a, s);
  return launch_back_t<32>(a, s);
}

int launch_windows(const WindowArgs& a, cudaStream_t s) {
  const int64_t total = (int64_t)a.nreal * a.nprof * a.nx;
  if (total <= 0) return RG_OK;
  const int grid = (int)std::min<int64_t>((total + 255) / 256, 4096);
  windows_kernel<<<grid, 256, 0, s>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

int launch_wavefun(const WavefunArgs& a, cudaStream_t s) {
  const int64_t rows = (int64_t)a.nx * a.ny;
  if (rows <= 0) return RG_OK;
  const int grid = (int)std::min<int64_t>((rows + 255) / 256, 4096);
  wavefun_kernel<<<grid, 256, 0, s>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

}  // namespace rg
