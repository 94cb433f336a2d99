// Device helpers shared by the sweep kernels: complex FP64 arithmetic, the
// gfortran-style xoshiro256** generator and the integer pivot key.
#pragma once

#include "rg_internal.h"

namespace rg {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// w - f * r with four FMAs.
__device__ __forceinline__ double2 cfms(double2 w, double2 f, double2 r) {
  return make_double2(fma(-f.x, r.x, fma(f.y, r.y, w.x)), fma(-f.x, r.y, fma(-f.y, r.x, w.y)));
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cscale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
__device__ __forceinline__ uint64_t rotl64(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }

struct Xoshiro {
  uint64_t s0, s1, s2, s3;
  __device__ __forceinline__ void step() {
    const uint64_t t = s1 << 17;
    s2 ^= s0;
    s3 ^= s1;
    s1 ^= s2;
    s0 ^= s3;
    s2 ^= t;
    s3 = rotl64(s3, 45);
  }
  __device__ __forceinline__ uint64_t next() {
    const uint64_t r = rotl64(s1 * 5, 7) * 9;
    step();
    return r;
  }
};

// Seed array of random_seed(put=) from the ANSI-C LCG (randi_ansic,
// src/random_normal.f90:20-31), scrambled into the 256-bit state the way
// gfortran's runtime does it (last put element first, XOR keys).
__device__ __forceinline__ Xoshiro seeded_state(int32_t seed) {
  uint32_t s = (uint32_t)seed, put[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s = 1103515245u * s + 12345u;
    put[i] = s;
  }
  const uint64_t k0 = 0xbd0c5b6e50c2df49ULL, k1 = 0xd46061cd46e1df38ULL;
  const uint64_t k2 = 0xbb4f4d4ed6103544ULL, k3 = 0x114a583d0756ad39ULL;
  Xoshiro x;
  x.s0 = ((uint64_t)put[7] | ((uint64_t)put[6] << 32)) ^ k0;
  x.s1 = ((uint64_t)put[5] | ((uint64_t)put[4] << 32)) ^ k1;
  x.s2 = ((uint64_t)put[3] | ((uint64_t)put[2] << 32)) ^ k2;
  x.s3 = ((uint64_t)put[1] | ((uint64_t)put[0] << 32)) ^ k3;
  return x;
}

__device__ __forceinline__ unsigned long long pivot_key(double2 x) {
  const unsigned long long a = (unsigned long long)__double_as_longlong(x.x) & 0x7fffffffffffffffULL;
  const unsigned long long b = (unsigned long long)__double_as_longlong(x.y) & 0x7fffffffffffffffULL;
  const unsigned long long m = a > b ? a : b;
  return m > 0x7ff0000000000000ULL ? 0ULL : m;  // NaN never wins
}

// Advances st by the jump polynomial poly (4 words, bit i = coefficient of
// x^i): the state after d steps is poly(T) applied to st when
// poly = x^d mod the characteristic polynomial of the xoshiro256 map T.
__device__ __forceinline__ Xoshiro jump_state(Xoshiro st, const uint64_t* poly) {
  Xoshiro acc{0, 0, 0, 0};
  for (int w = 0; w < 4; ++w) {
    const uint64_t pw = poly[w];
    for (int b = 0; b < 64; ++b) {
      if ((pw >> b) & 1ULL) {
        acc.s0 ^= st.s0;
        acc.s1 ^= st.s1;
        acc.s2 ^= st.s2;
        acc.s3 ^= st.s3;
      }
      st.step();
    }
  }
  return acc;
}

// One scaled normal from two draws: random_number's real(8) conversion (top
// 53 bits) and Box-Muller as src/random_normal.f90:63-65, times stdu
// (src/waveguide.f90:371).
__device__ __forceinline__ double scaled_normal(double stdu, Xoshiro& st) {
  const double twopi = 2.0 * 3.141592653589793;
  const double u1 = (double)(st.next() >> 11) * 0x1.0p-53;
  const double u2 = (double)(st.next() >> 11) * 0x1.0p-53;
  return stdu * (sqrt(-2.0 * log(u1)) * cos(twopi * u2));
}

// ---------------------------------------------------------------------------
// Singular values: Householder bidiagonalisation, then bisection.
// ---------------------------------------------------------------------------

// 1/x to one ulp where x and 1/x are normal (NaN elsewhere): the hardware's
// approximation and two Newton steps (a division instruction sequence is twice as
// long).  For bidiag_count, whose divisors lie in between.
__device__ __forceinline__ double fast_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// The reductions below square entries, so a matrix is brought to order 1 when
// its largest entry lies outside 2^-300 .. 2^300 (t of a strongly absorbing guide
// comes down to 1e-300).  Powers of two: the singular values scale exactly.
// Biased exponent of the larger part of x:
__device__ __forceinline__ int biased_exp(double2 x) {
  const int a = (__double2hiint(x.x) >> 20) & 0x7ff, b = (__double2hiint(x.y) >> 20) & 0x7ff;
  return a > b ? a : b;
}
// The factor for a matrix whose entries have exponents up to e, and the one that
// undoes it; 1 where no scaling is needed.
__device__ __forceinline__ double range_scale(int e, double* undo) {
  const bool on = e > 0 && (e < 1023 - 300 || e > 1023 + 300) && e < 2046;
  *undo = on ? __longlong_as_double((long long)e << 52) : 1.0;
  return on ? __longlong_as_double((long long)(2046 - e) << 52) : 1.0;
}

// Reflection of a complex vector x (first element a, squared norm xn2 of the
// others): (I - tau v v^H) x = beta e_1 with v = (1, x[1:] * scale), beta real.
struct Reflector {
  double beta;
  double2 tau, scale;
};
__device__ __forceinline__ Reflector reflector(double2 a, double xn2) {
  Reflector r;
  const double n2 = fma(a.x, a.x, fma(a.y, a.y, xn2));
  // (below 1e-145 of a matrix of order 1: zero, whose square would underflow)
  if ((xn2 == 0.0 && a.y == 0.0) || n2 < 1e-290) {
    r.beta = n2 < 1e-290 ? 0.0 : a.x;
    r.tau = r.scale = make_double2(0.0, 0.0);
    return r;
  }
  r.beta = -copysign(sqrt(n2), a.x);
  const double rb = 1.0 / r.beta;
  r.tau = make_double2((r.beta - a.x) * rb, a.y * rb);
  const double dx = a.x - r.beta;  // no cancellation: beta has the sign opposite to a.x
  const double den = 1.0 / fma(dx, dx, a.y * a.y);
  r.scale = make_double2(dx * den, -a.y * den);
  return r;
}

// Eigenvalues below mu of B^T B, for the upper bidiagonal B with squared
// diagonal dd[n] and superdiagonal ee[n - 1]: the negative pivots of its
// factorisation shifted by mu, in the differential form that never forms B^T B.
__device__ __forceinline__ int bidiag_count(const double* dd, const double* ee, int n, double mu, double tiny) {
  double s = -mu;
  int c = 0;
  for (int i = 0; i < n; ++i) {
    double q = dd[i] + s;
    if (fabs(q) < tiny) q = -tiny;
    c += q < 0.0 ? 1 : 0;
    s = fma(ee[i], s * fast_rcp(q), -mu);
  }
  return c;
}

// The largest neig squared singular values of the bidiagonal d[n], e[n - 1]
// (shared memory; squared in place), descending, to out.  Bisection on sigma,
// down to 2^-52 of the value itself; a warp's lanes share out its values, S lanes cutting an interval
// into S + 1 parts; `unscale` multiplies the singular values.  Called by NT threads of one CTA, or by CTA
// `rank` of `parts` (then S = 1: the bits of a value do not depend on the sharing).
template <int NT>
__device__ void bidiag_values(double* d, double* e, int n, int neig, double* out, double unscale, int rank = 0,
                              int parts = 0) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  double bound = 0.0, top = 0.0;  // every thread: ||B|| <= bound, largest square
  bool finite = true;
  for (int i = lane; i < n; i += 32) {
    const double di = fabs(d[i]), e0 = i > 0 ? fabs(e[i - 1]) : 0.0, e1 = i + 1 < n ? fabs(e[i]) : 0.0;
    bound = fmax(bound, di + fmax(e0, e1));
    top = fmax(top, fmax(di * di, e1 * e1));
    finite = finite && di + e1 < INFINITY;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, off));
    top = fmax(top, __shfl_xor_sync(0xffffffffu, top, off));
  }
  finite = __all_sync(0xffffffffu, finite);
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += NT) {
    d[i] *= d[i];
    e[i] = i + 1 < n ? e[i] * e[i] : 0.0;
  }
  __syncthreads();
  const int share = parts ? (neig + parts - 1) / parts : neig, j0 = rank * share, cnt = min(share, neig - j0);
  if (!finite) {
    for (int k = threadIdx.x; k < cnt; k += NT) out[j0 + k] = NAN;
    return;
  }
  // warps in use: at least one per scheduler, then a warp per 32 values
  const int wn = min(NW, max(4, (cnt + 31) / 32));
  if (warp >= wn) return;
  const int per = (cnt + wn - 1) / wn;           // values of a warp
  const double tiny = fmax(1e-120 * top, 1e-300);  // (its reciprocal times two squares is finite)
  for (int v0 = 0; v0 < per; v0 += 32) {
    const int here = min(32, per - v0), S = parts ? 1 : 32 / here;
    const int grp = lane / S, s = lane % S;
    const int k = warp * per + v0 + grp;          // position among this sharer's values
    const bool on = grp < here && k < cnt;
    const int want = n - 1 - (j0 + k);            // the value has this many below it
    const unsigned mask = S == 32 ? ~0u : (1u << S) - 1u;
    // the first of a group's S cuts, falling or rising, that `hit`s
    auto first = [&](bool hit) {
      const unsigned b = (__ballot_sync(0xffffffffu, hit) >> (grp * S)) & mask;
      return b ? __ffs(b) - 1 : S;
    };
    // Its octave first, bound 2^-p1 .. bound 2^-p0: the bidiagonal gives a small
    // value to as many digits as a large one, and so does t where modes hardly
    // mix (a clean absorbing guide).  (54 halvings of 0 .. bound took 1 % less of
    // 256 modes and lost the small ones.)
    int p0 = 0, p1 = 192;  // (zero below)
    while (__any_sync(0xffffffffu, on && p1 - p0 > 1)) {
      const bool go = on && p1 - p0 > 1;
      const int p = p0 + (p1 - p0) * (s + 1) / (S + 1);
      const double x = bound * __longlong_as_double((long long)(1023 - p) << 52);
      const int f = first(go && bidiag_count(d, e, n, x * x, tiny) <= want), lo0 = p0, w = p1 - p0;
      if (go && f < S) p1 = lo0 + w * (f + 1) / (S + 1);
      if (go && f > 0) p0 = lo0 + w * f / (S + 1);
    }
    double hi = bound * __longlong_as_double((long long)(1023 - p0) << 52), lo = p1 == 192 ? 0.0 : 0.5 * hi;
    const double rs = 1.0 / (S + 1);
    // 52 halvings, or as many cuts into S + 1 parts as shrink the interval alike
    const int steps = (int)ceilf(52.0f / log2f((float)(S + 1)));
    for (int it = 0; it < steps; ++it) {
      const double x = fma(hi - lo, (s + 1) * rs, lo);
      const int f = first(on ? bidiag_count(d, e, n, x * x, tiny) > want : true);  // the first cut above the value
      const double w = hi - lo, base = lo;
      if (f < S) hi = fma(w, (f + 1) * rs, base);
      if (f > 0) lo = fma(w, f * rs, base);
    }
    if (on && s == 0) {
      const double x = 0.5 * (lo + hi) * unscale;
      out[j0 + k] = x * x;
    }
  }
}

// Eigenvalues of t^H t for the nrow x ncol matrix t held in shared memory at
// W[i * LDW + j]: the largest neigv, descending, to out.  Every thread of the
// NT-thread block calls this; sc is shared scratch of 2 n + 2 max(nrow, ncol)
// + 4 doubles, n the smaller dimension.
//
// Householder reflections from both sides make t real bidiagonal (4/3 n^3
// complex multiply-adds) and bisection gives the values, as accurate as the
// reference's zgesvd (absolutely, to the norm of t, where modes mix).  One-sided Jacobi took
// nine sweeps of 4 n^3 on the same FP64 pipe: 57 M clocks for 64 x 64.
template <int NT>
__device__ void tt_eigenvalues(double2* W, int LDW, int nrow, int ncol, int neigv, double* sc, double* out) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool tall = nrow >= ncol;
  const int m = tall ? nrow : ncol, n = tall ? ncol : nrow;
  const int rs = tall ? LDW : 1, cs = tall ? 1 : LDW;  // A(i, j) = W[i rs + j cs], t or its transpose
  double* d = sc;
  double* e = d + n;
  double2* v = reinterpret_cast<double2*>(e + n);  // [max(m, n)] reflection vector
  double2* tau = v + m;                            // [1]
  // warp 0: the reflector of L elements at x (stride st), conjugated for a row
  auto reflect = [&](const double2* x, int st, int L, double sg, double* beta) {
    double xn2 = 0.0;
    for (int i = 1 + lane; i < L; i += 32) {
      const double2 u = x[i * st];
      xn2 = fma(u.x, u.x, fma(u.y, u.y, xn2));
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) xn2 += __shfl_xor_sync(0xffffffffu, xn2, off);
    const Reflector r = reflector(make_double2(x[0].x, sg * x[0].y), xn2);
    for (int i = 1 + lane; i < L; i += 32) v[i] = cmul(make_double2(x[i * st].x, sg * x[i * st].y), r.scale);
    if (lane == 0) {
      v[0] = make_double2(1.0, 0.0);
      *tau = r.tau;
      *beta = r.beta;
    }
  };
  // x <- x - f (v^H x) v for the L elements at x, by one warp (f tau of a
  // column; for a row both are conjugated, which conjugates v)
  auto apply = [&](double2* x, int st, int L, double2 f, double sg) {
    double re = 0.0, im = 0.0;
    for (int i = lane; i < L; i += 32) {
      const double2 q = v[i], u = x[i * st];
      re = fma(q.x, u.x, fma(sg * q.y, u.y, re));
      im = fma(q.x, u.y, fma(-sg * q.y, u.x, im));
    }
    // lanes 0..15 sum re, lanes 16..31 im
    const double other = __shfl_xor_sync(0xffffffffu, lane < 16 ? im : re, 16);
    double h = (lane < 16 ? re : im) + other;
#pragma unroll
    for (int off = 8; off; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
    const double2 w = cmul(f, make_double2(__shfl_sync(0xffffffffu, h, 0), __shfl_sync(0xffffffffu, h, 16)));
    for (int i = lane; i < L; i += 32) {
      const double2 q = v[i], u = x[i * st];
      x[i * st] = make_double2(fma(-w.x, q.x, fma(sg * w.y, q.y, u.x)), fma(-w.x, sg * q.y, fma(-w.y, q.x, u.y)));
    }
  };
  __shared__ int s_top;
  if (threadIdx.x == 0) s_top = 0;
  __syncthreads();
  int top = 0;
  for (int q = threadIdx.x; q < nrow * ncol; q += NT) top = max(top, biased_exp(W[(q / ncol) * LDW + q % ncol]));
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&s_top, top);
  __syncthreads();
  double unscale;
  const double scale = range_scale(s_top, &unscale);
  if (scale != 1.0) {
    for (int q = threadIdx.x; q < nrow * ncol; q += NT) {
      double2* x = W + (q / ncol) * LDW + q % ncol;
      *x = cscale(scale, *x);
    }
    __syncthreads();
  }
  for (int k = 0; k < n; ++k) {
    if (warp == 0) reflect(W + k * rs + k * cs, rs, m - k, 1.0, d + k);
    __syncthreads();
    for (int j = k + 1 + warp; j < n; j += NW) apply(W + k * rs + j * cs, rs, m - k, *tau, 1.0);
    __syncthreads();
    if (k + 1 >= n) break;
    if (warp == 0) reflect(W + k * rs + (k + 1) * cs, cs, n - k - 1, -1.0, e + k);
    __syncthreads();
    const double2 tc = make_double2(tau->x, -tau->y);
    for (int i = k + 1 + warp; i < m; i += NW) apply(W + i * rs + (k + 1) * cs, cs, n - k - 1, tc, -1.0);
    __syncthreads();
  }
  bidiag_values<NT>(d, e, n, min(neigv, n), out, unscale);
}

}  // namespace rg
